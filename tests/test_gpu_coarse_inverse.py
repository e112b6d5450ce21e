"""The multigrid's coarsest level: its assembled matrix and its inverse, at the
sizes where the register form changes shape (32, 64, 96, 128 unknowns), at its
largest (160) and past it.  A grid that is its own coarsest level makes the
V-cycle the exact inverse, so one preconditioned step solves the system."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,coarse", [
    ((1, 1), 0), ((3, 3), 0), ((7, 1), 0), ((5, 5), 0), ((8, 4), 0), ((11, 3), 0), ((7, 7), 0),
    ((9, 7), 0), ((11, 5), 0), ((15, 4), 0), ((39, 1), 0), ((16, 9), 400),
    ((1, 1, 1), 0), ((2, 2, 1), 0), ((4, 2, 2), 0), ((5, 2, 2), 200), ((4, 4, 3), 400)])
def test_coarsest_level_is_the_inverse(ctx, dims, coarse):
    import icarat_b200 as icb
    d = len(dims)
    p = icb.Problem(ctx, d, *dims)
    fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (d,), np.uint8)
    fixed[..., 0, :] = 1  # the face x = 0
    p.dirichlet_mask(fixed.reshape(-1))
    last = p.nnode - 1
    p.nodal_load(last, [0.3, -1.0, 0.5][:d])
    n = p.finalize()
    p.set_density(np.random.default_rng(len(dims)).uniform(0.3, 1.0, p.nel))
    K = np.stack([p.matvec(e) for e in np.eye(n)], 1)
    u = np.linalg.solve(K, p.load())
    info = p.solve(precision=icb.FP64, precond=icb.GMG, tol=1e-10, mg_coarse_dofs=coarse)
    assert info["iters"] <= 1, info
    # both sides solve with a relative error of about cond(K) eps
    tol = 100 * np.linalg.cond(K) * np.finfo(float).eps
    assert np.abs(p.displacement() - u).max() <= tol * np.abs(u).max()
    p.close()
