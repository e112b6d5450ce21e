"""The cone filter's tiled form against a direct sum, at the edges of its tiles:
grids of one tile, one element past a tile and smaller than one, both 3D
splits (eight and four outputs a thread), every unrolled half height and a
radius past them (the general kernel), and unequal element edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def direct(x, h, r):
    """filtered and adjoint of x (z, y, x) with weights r - |offset h|"""
    R = [0 if np.isinf(hh) else int(r / hh) + 1 for hh in h]
    offs = [(k, j, i) for k in range(-R[0], R[0] + 1) for j in range(-R[1], R[1] + 1)
            for i in range(-R[2], R[2] + 1)]

    def stencil(v):
        out = np.zeros_like(v)
        for o in offs:
            d = np.sqrt(sum((t * hh) ** 2 for t, hh in zip(o, h) if t))
            if d > r or any(abs(t) >= n for t, n in zip(o, v.shape)):
                continue
            to = tuple(slice(max(0, -t), n - max(0, t)) for t, n in zip(o, v.shape))
            fr = tuple(slice(max(0, t), n - max(0, -t)) for t, n in zip(o, v.shape))
            out[to] += (r - d) * v[fr]
        return out

    w = stencil(np.ones_like(x))
    return stencil(x) / w, stencil(x / w)


@pytest.mark.parametrize("dims,radius,edge", [
    ((32, 32), 1.0, 1.0), ((33, 33), 1.5, 1.0), ((5, 3), 2.4, 1.0), ((64, 65), 4.0, 1.0),
    ((40, 24), 5.2, 1.0), ((37, 31), 2.0, 0.5),
    ((32, 8, 8), 1.5, 1.0), ((33, 9, 9), 3.0, 1.0), ((7, 5, 3), 2.2, 1.0), ((31, 7, 4), 4.2, 1.0),
    ((200, 60, 61), 2.5, 1.0), ((24, 12, 12), 5.2, 1.0), ((40, 17, 13), 2.0, 0.6)])
def test_cone_tiles_match_direct_sum(ctx, dims, radius, edge):
    import icarat_b200 as icb
    d = len(dims)
    # the x edge differs from the others
    lens = [dims[0] * edge] + [float(n) for n in dims[1:]]
    p = icb.Problem(ctx, d, *dims, lx=lens[0], ly=lens[1], lz=lens[2] if d == 3 else None)
    fixed = np.zeros(p.neq, np.uint8)
    fixed[:2 * d] = 1
    p.dirichlet_mask(fixed)
    p.finalize()
    x = np.random.default_rng(3).uniform(0.01, 1.0, p.nel)
    shape = (1,) * (3 - d) + tuple(reversed(dims))
    f, a = direct(x.reshape(shape), [1.0, 1.0, edge], radius) if d == 3 else \
        direct(x.reshape(shape), [np.inf, 1.0, edge], radius)
    c = icb.Cone(p, radius)
    # sums of at most ~600 positive terms, each with two roundings: 600 * 2 eps
    # bounds the relative error of either side
    tol = 2 * 1200 * np.finfo(float).eps
    np.testing.assert_allclose(c.apply(x), f.reshape(-1), rtol=tol)
    np.testing.assert_allclose(c.apply(x, sens=True), a.reshape(-1), rtol=tol)
    c.close()
    p.close()
