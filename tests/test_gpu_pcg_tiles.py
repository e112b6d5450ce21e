"""The one-kernel Jacobi-PCG of small grids against the three-kernel form
(icb_solve_noalloc runs the same iteration launch by launch): grids of one box
and of many, boxes cut short by the grid's edge, thin grids, the largest boxes,
and the first grids past them, which fall back to the three kernels."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(ctx, dims, clamp=True):
    import icarat_b200 as icb
    d = len(dims)
    p = icb.Problem(ctx, d, *dims)
    fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (d,), np.uint8)
    fixed[..., 0, :] = 1
    fixed[(0,) * (d - 1) + (dims[0], d - 1)] = 1
    p.dirichlet_mask(fixed.reshape(-1))
    p.nodal_load(p.nnode - 1, [0.3, -1.0, 0.5][:d])
    p.finalize()
    p.set_density(np.random.default_rng(11).uniform(0.2, 1.0, p.nel))
    return p


def three_kernels(p, tol, maxit):
    """(iterations, compliance f.u, solution on the unknowns) of the launch by launch form"""
    import torch
    import icarat_b200 as icb
    L = icb.lib()
    free = p.dof_map() < p.numeq  # node-major, interleaved
    d = p.dim
    ld = p.soa_length() // d
    f = np.zeros(p.neq)
    f[free] = p.load()
    b = torch.zeros((d, ld), dtype=torch.float64)
    b[:, :p.nnode] = torch.from_numpy(f.reshape(-1, d).T.copy())
    b = b.cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    info = icb.SolveInfo()
    icb.check(L.icb_solve_noalloc(p.h, b.data_ptr(), x.data_ptr(), tol, maxit, C.byref(info)))
    p.ctx.synchronize()
    u = x.cpu().numpy()[:, :p.nnode].T.reshape(-1)[free]
    return info.iters, float(f[free] @ u), u


@pytest.mark.parametrize("dims", [(1, 1), (15, 15), (16, 16), (120, 40), (97, 3), (2, 61), (250, 151),
                                  (380, 380), (540, 540), (640, 600),
                                  (1, 1, 1), (7, 7, 3), (8, 8, 4), (60, 20, 20), (33, 2, 2),
                                  (5, 40, 3), (41, 41, 41), (48, 46, 45), (54, 54, 50)])
def test_one_kernel_pcg_matches_three(ctx, dims):
    import icarat_b200 as icb
    p = build(ctx, dims)
    tol = 1e-10
    it, c, u = three_kernels(p, tol, 100000)
    info = p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=tol, maxit=100000)
    # the sums are associated differently: the last iterations' residuals, and
    # with them the converging iteration, may differ by a few
    assert abs(info["iters"] - it) <= max(2, it // 50), (info, it)
    # the recurrence's residual drifts from the true one by rounding, in either form
    true3 = np.linalg.norm(p.load() - p.matvec(u)) / np.linalg.norm(p.load())
    assert info["true_relres"] <= 2 * max(tol, true3)
    assert abs(p.compliance() - c) <= 1e-7 * abs(c)
    # both have relres 1e-10 on systems of condition number below 1e6
    assert np.abs(p.displacement() - u).max() <= 1e-4 * np.abs(u).max()
    # a second solve repeats the first bitwise
    v = p.displacement()
    p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=tol, maxit=100000)
    assert np.array_equal(p.displacement(), v)
    p.close()


def test_one_kernel_pcg_statuses(ctx):
    """the iteration limit, a singular system and a non-finite one end the
    kernel with their status"""
    import icarat_b200 as icb
    p = build(ctx, (40, 20))
    r = p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-12, maxit=7, raise_on_error=False)
    assert r["status"] == -4 and r["iters"] == 7 and r["matvecs"] == 7
    p.set_density(np.full(p.nel, np.nan))
    r = p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-12, raise_on_error=False)
    assert r["status"] in (-3, -6)
    p.set_density(np.full(p.nel, 0.7))  # the context stays usable
    assert p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-10)["status"] == 0
    p.close()
