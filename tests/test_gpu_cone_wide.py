"""The 3D cone filter on elements a millionth as wide as they are tall: a stencil
whose tile would exceed 2^31 bytes takes the gather kernel, as any too large one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_stencil_wider_than_any_tile(ctx):
    import icarat_b200 as icb
    n, h, r = (2, 2, 2), (1e-6, 2.0, 0.26), 1.06
    p = icb.Problem(ctx, 3, *n, lx=n[0] * h[0], ly=n[1] * h[1], lz=n[2] * h[2])
    p.finalize()
    x = np.random.default_rng(1).uniform(0.1, 1.0, p.nel)
    at = np.array([[i * h[0], j * h[1], k * h[2]]
                   for k in range(n[2]) for j in range(n[1]) for i in range(n[0])])
    w = np.maximum(0.0, r - np.linalg.norm(at[:, None] - at[None], axis=2))
    cone = icb.Cone(p, r)
    # at most eight terms a sum
    np.testing.assert_allclose(cone.apply(x), w @ x / w.sum(1), rtol=64 * np.finfo(float).eps)
    np.testing.assert_allclose(cone.apply(x, sens=True), w @ (x / w.sum(1)),
                               rtol=64 * np.finfo(float).eps)
    cone.close()
    p.close()
