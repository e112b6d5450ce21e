"""The multigrid's coarse levels as one launch: grids at the sizes where the
tail begins a level later, thin and odd grids, every smoothing degree it takes
and the first it does not, FP64 and FP32 V-cycles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(ctx, dims, seed=5):
    import icarat_b200 as icb
    d = len(dims)
    p = icb.Problem(ctx, d, *dims)
    fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (d,), np.uint8)
    fixed[..., 0, :] = 1
    fixed[(0,) * (d - 1) + (dims[0] // 2, d - 1)] = 1  # a point support at an odd or even node
    p.dirichlet_mask(fixed.reshape(-1))
    p.nodal_load(p.nnode - 1, [0.3, -1.0, 0.5][:d])
    p.finalize()
    p.set_density(np.random.default_rng(seed).uniform(0.3, 1.0, p.nel))
    return p


# 127 x 127: 16384 nodes, the largest 2D first level; 128 x 127 starts a level lower;
# 15 x 15 x 15: 4096 nodes, 16 x 15 x 15 starts lower
@pytest.mark.parametrize("dims", [(127, 127), (128, 127), (255, 64), (61, 1), (9, 33), (24, 13),
                                  (15, 15, 15), (16, 15, 15), (20, 10, 10), (7, 6, 5)])
def test_tail_solves_match_jacobi(ctx, dims):
    import icarat_b200 as icb
    p = build(ctx, dims)
    p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-13, maxit=200000)
    u = p.displacement()
    for precision in (icb.FP64, icb.MIXED):
        info = p.solve(precision=precision, precond=icb.GMG, tol=1e-12)
        # a V-cycle with a wrong level would not contract: unknowns by the
        # thousand, tens of iterations
        assert info["iters"] <= 60, (precision, info)
        # |u - u*| <= cond(K) * relres * |u|: two solves of relres 1e-12 and
        # 1e-13 on systems of condition number below 1e5
        assert np.abs(p.displacement() - u).max() <= 1e-7 * np.abs(u).max(), precision
    p.close()


@pytest.mark.parametrize("dims", [(50, 31), (12, 9, 7)])
@pytest.mark.parametrize("nu", [1, 2, 3, 4, 8, 9])
def test_tail_smoothing_degrees(ctx, dims, nu):
    import icarat_b200 as icb
    p = build(ctx, dims)
    p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-13, maxit=200000)
    u = p.displacement()
    info = p.solve(precision=icb.FP64, precond=icb.GMG, tol=1e-12, mg_smooth=nu)
    assert info["iters"] <= 80, info
    assert np.abs(p.displacement() - u).max() <= 1e-7 * np.abs(u).max()
    p.close()


@pytest.mark.parametrize("dims", [(15, 15, 15), (21, 11, 12), (33, 9, 1)])
def test_tail_matches_the_levels_on_the_dense_operator(ctx, dims):
    """with the corner-mode operator off the levels run as launches of their
    own on the dense element product: the same V-cycle up to rounding"""
    import icarat_b200 as icb
    p = build(ctx, dims)
    a = p.solve(precision=icb.FP64, precond=icb.GMG, tol=1e-10)
    u = p.displacement()
    icb.set_option("hex8_modal", 0)
    try:
        b = p.solve(precision=icb.FP64, precond=icb.GMG, tol=1e-10)
        v = p.displacement()
    finally:
        icb.set_option("hex8_modal", 1)
    assert abs(a["iters"] - b["iters"]) <= 1
    # both stop at relres 1e-10
    assert np.abs(u - v).max() <= 1e-5 * np.abs(v).max()
    p.close()
