"""Batched launches many waves long, whose CTAs take several blocks of one design
at a time: vector sums, bisection steps, operator rows.  And the 2D multigrid
transfers on grids whose fine levels run as launches of their own: every parity
of both axes, widths around a block's, an axis too short to be halved."""
import numpy as np
import pytest

import cases
import icarat_b200 as icb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,count", [(icb.MIXED, 14), (icb.FP64, 9)])
def test_long_batched_launches_equal_each_problem_alone(precision, count):
    rng = np.random.default_rng(29)
    insts = [cases.random_instance2d(rng, nelx_range=(300, 640)) for _ in range(count)]
    insts += [cases.random_instance2d(rng, nelx_range=(12, 40)) for _ in range(2)]
    ctxs = [icb.Context(0) for _ in insts]
    probs = [cases.build_instance(c, i) for c, i in zip(ctxs, insts)]
    opts = [icb.loop_opts(2, i["r"], move=0.2, precision=precision) for i in insts]
    rho0 = [np.full(p.nel, i["vf"]) for p, i in zip(probs, insts)]
    h, x, st = icb.run_batch(probs, [0] * len(probs), opts, rho0, nworkers=1)
    assert (st == 0).all()
    for k, (p, i) in enumerate(zip(probs, insts)):
        ha, xa = icb.run_loop(p, "oc", rho0[k], 2, i["r"], move=0.2, precision=precision)
        assert np.array_equal(ha, h[k]), k
        assert np.array_equal(xa, x[k]), k
    for p in probs:
        p.close()
    for c in ctxs:
        c.close()


@pytest.mark.parametrize("dims", [(300, 200), (301, 200), (300, 201), (301, 203), (255, 160),
                                  (256, 161), (127, 254), (700, 5), (5, 700), (900, 90)])
def test_2d_transfers_give_a_contracting_cycle(ctx, dims):
    p = icb.Problem(ctx, 2, *dims)
    fixed = np.zeros((dims[1] + 1, dims[0] + 1, 2), np.uint8)
    fixed[:, 0, :] = 1
    fixed[0, :, :] = 1
    fixed[-1, dims[0] // 2, 1] = 1  # a point support
    p.dirichlet_mask(fixed.reshape(-1))
    p.nodal_load(p.nnode - 1, [0.3, -1.0])
    p.finalize()
    p.set_density(np.random.default_rng(6).uniform(0.5, 1.0, p.nel))
    p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-13, maxit=100000)
    u = p.displacement()
    for precision in (icb.FP64, icb.MIXED):
        info = p.solve(precision=precision, precond=icb.GMG, tol=1e-11)
        # |u - u*| <= cond(K) relres |u|; two clamped sides of a body at most 160
        # elements from either keep the condition number below 1e6
        assert np.abs(p.displacement() - u).max() <= 1e-5 * np.abs(u).max()
        if min(dims) > 5:
            # a transfer pair that is not adjoint, or a row it misses, costs
            # iterations; a two-step Chebyshev cycle contracts by more than two
            assert info["iters"] <= 35, (precision, info["iters"])
    p.close()
