"""The one-kernel Jacobi-PCG of the 3D Helmholtz filter: against the oracle on
boxes cut short, thin and single-element grids, and by its own identities on
larger ones up to and past the largest that fits."""
import numpy as np
import pytest

import pyoracle as po

pytestmark = pytest.mark.gpu


def build(ctx, dims):
    import icarat_b200 as icb
    g = icb.Problem(ctx, 3, *dims)
    g.finalize()
    return g


# both solve to a residual of 1e-10; the Jacobi-scaled operator's condition
# number is at most 8 + 48 (R / (2 sqrt 3))^2 < 300 for R <= 8: errors below 1e-7
@pytest.mark.parametrize("dims,R", [((1, 1, 1), 1.5), ((2, 2, 2), 8.0), ((7, 7, 3), 2.2),
                                    ((33, 16, 17), 2.2), ((40, 20, 20), 1.5), ((1, 40, 9), 3.0),
                                    ((97, 2, 1), 3.0), ((5, 3, 61), 3.0)])
def test_helm_tiles_match_oracle(ctx, dims, R):
    import icarat_b200 as icb
    o, g = po.Problem(3, *dims), build(ctx, dims)
    x = np.random.default_rng(4).uniform(0.01, 1.0, o.nel)
    h = icb.Helmholtz(g, R)
    for sens in (False, True):
        a, b = o.helmholtz(R, x, sens=sens), h.apply(x, sens=sens)
        assert np.abs(a - b).max() <= 1e-7 * np.abs(a).max()
        assert np.array_equal(b, h.apply(x, sens=sens))  # a repeat is bitwise the same


# a constant stays one (the gradient term vanishes); the map and its adjoint
# differ by the load's and the mean's 1 / ne only, so <y, F x> = <F' y, x> up to
# the solves' 1e-10
@pytest.mark.parametrize("dims", [(80, 40, 40), (100, 50, 50), (128, 64, 64), (131, 64, 64),
                                  (160, 80, 80)])
def test_helm_tiles_identities(ctx, dims):
    import icarat_b200 as icb
    g = build(ctx, dims)
    h = icb.Helmholtz(g, 2.2)
    assert np.abs(h.apply(np.full(g.nel, 0.7)) - 0.7).max() <= 1e-7
    r = np.random.default_rng(5)
    x, y = r.uniform(0.01, 1.0, g.nel), r.uniform(0.01, 1.0, g.nel)
    a, b = float(y @ h.apply(x)), float(h.apply(y, sens=True) @ x)
    assert abs(a - b) <= 1e-7 * abs(a)
