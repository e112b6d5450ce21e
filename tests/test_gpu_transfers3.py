"""The 3D multigrid transfers that take several nodes a thread: every parity of
the fine grid's axes (a last fine row between two coarse ones or on one), coarse
plane counts that are and are not multiples of the restriction's, and a grid
wider than one block, all large enough that the fine levels run as launches of
their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 14, 12), (17, 14, 12), (16, 15, 12), (16, 14, 13),
                                  (17, 15, 13), (15, 9, 30), (22, 10, 31), (270, 6, 5), (131, 7, 8)])
def test_transfers_give_a_contracting_cycle(ctx, dims):
    import icarat_b200 as icb
    p = icb.Problem(ctx, 3, *dims)
    fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (3,), np.uint8)
    fixed[:, :, 0, :] = 1  # two clamped faces: a well-conditioned system
    fixed[0, :, :, :] = 1
    fixed[-1, dims[1] // 2, dims[0] // 2, 1] = 1  # a point support
    p.dirichlet_mask(fixed.reshape(-1))
    p.nodal_load(p.nnode - 1, [0.3, -1.0, 0.5])
    p.finalize()
    p.set_density(np.random.default_rng(6).uniform(0.5, 1.0, p.nel))
    p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-13, maxit=100000)
    u = p.displacement()
    its = []
    for precision in (icb.FP64, icb.MIXED):
        info = p.solve(precision=precision, precond=icb.GMG, tol=1e-11)
        its.append(info["iters"])
        # |u - u*| <= cond(K) relres |u|, condition number below 1e5
        assert np.abs(p.displacement() - u).max() <= 1e-6 * np.abs(u).max()
    # the dense element product runs the same transfers on the same levels; a
    # transfer pair that is not adjoint, or a row it misses, costs iterations in
    # the flexible CG whatever the operator: a two-step Chebyshev cycle on moduli
    # within a factor of eight contracts by more than two an iteration
    assert max(its) <= 35, its
    p.close()
