"""The one-kernel OC update of 2D designs against the bisection written out in
numpy: grids of one tile, at and past tile edges, several tiles a CTA, the
first grid past the most a CTA takes, radii of every unrolled column height and
past them (the graph form), with and without the threshold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cone_2d(x, r):
    k = int(r) + 1

    def stencil(v):
        out = np.zeros_like(v)
        for j in range(-k, k + 1):
            for i in range(-k, k + 1):
                d = np.hypot(i, j)
                if d > r or abs(j) >= v.shape[0] or abs(i) >= v.shape[1]:
                    continue
                to = tuple(slice(max(0, -t), n - max(0, t)) for t, n in zip((j, i), v.shape))
                fr = tuple(slice(max(0, t), n - max(0, -t)) for t, n in zip((j, i), v.shape))
                out[to] += (r - d) * v[fr]
        return out

    return stencil(x) / stencil(np.ones_like(x))


def bisection(x, df, dg, g, lo, hi, move, volume):
    """OCSolver.hpp:33-60: the last evaluated candidate"""
    l0, l1, n, gaps = 0.0, 1e4, 0, []
    while (l1 - l0) / (l1 + l0) > 1e-5 and n < 100:
        lam = 0.5 * (l1 + l0)
        y = np.sqrt(np.maximum(0.0, -df / (dg * lam))) * x
        y = np.clip(y, np.maximum(lo, (1 - move) * x), np.minimum(hi, (1 + move) * x))
        v = volume(y) - g
        gaps.append(abs(v) / g)
        l0, l1 = (lam, l1) if v > 0.0 else (l0, lam)
        n += 1
    return y, n, min(gaps)


@pytest.mark.parametrize("beta", [0.0, 2.0])
@pytest.mark.parametrize("nx,ny,r", [(32, 32, 1.0), (33, 31, 1.5), (5, 3, 2.4), (64, 65, 4.2),
                                     (40, 1, 3.0), (120, 40, 1.5), (500, 420, 2.4), (640, 320, 4.9),
                                     (1200, 700, 1.2), (60, 44, 5.2), (45, 30, 9.5)])
def test_oc_update_matches_bisection(ctx, nx, ny, r, beta):
    import icarat_b200 as icb
    p = icb.Problem(ctx, 2, nx, ny)
    p.finalize()
    rng = np.random.default_rng(nx + ny)
    n = nx * ny
    x = rng.uniform(0.05, 1.0, n)
    df = -rng.uniform(0.0, 2.0, n) ** 3
    df[:3] = 0.0
    dg = rng.uniform(0.8, 1.2, n)
    lo, hi = np.full(n, 1e-4), np.ones(n)

    def volume(y):
        v = cone_2d(y.reshape(ny, nx), r)
        if beta > 0.0:
            t = np.tanh(0.5 * beta)
            v = 0.5 * (t + np.tanh(beta * (v - 0.5))) / t
        return v.sum()

    g = 0.97 * volume(x)
    y, steps, gap = bisection(x, df, dg, g, lo, hi, 0.2, volume)
    # every step's volume is further from g than the sums' rounding (n terms of
    # a few eps each), so both bisections take the same turns
    assert gap > 1e-9
    cone = icb.Cone(p, r)
    for _ in range(2):
        out, k = icb.oc_update(p, cone, x, df, g, dg, lo, hi, 0.2, beta=beta)
        assert k == steps
        # the same lambda; a division, a square root and a product each
        np.testing.assert_allclose(out, y, rtol=8 * np.finfo(float).eps)
    cone.close()
    p.close()
