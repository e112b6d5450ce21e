"""The one-kernel Jacobi-PCG on a singular system: an unsupported body under a load
that is not in equilibrium has no solution, so the solve ends with a status of its own
and the context stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(40, 20), (12, 8, 6)])
def test_singular_system_ends_with_a_status(ctx, dims):
    import icarat_b200 as icb
    d = len(dims)
    p = icb.Problem(ctx, d, *dims)
    p.nodal_load(p.nnode - 1, [0.3, -1.0, 0.5][:d])
    p.finalize()
    p.set_density(np.full(p.nel, 0.7))
    r = p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-12, maxit=5000, raise_on_error=False)
    # the recurrence leaves the range of K: a breakdown (p.Kp <= 0), the iteration
    # limit, or values past the largest double
    assert r["status"] in (-3, -4, -6) and r["rc"] == r["status"]
    p.close()
    q = icb.Problem(ctx, d, *dims)
    q.dirichlet_box([1] * 6, [0.0] * 6, [0.0, 0.0, -1e9, 1e9, -1e9, 1e9])
    q.nodal_load(q.nnode - 1, [0.3, -1.0, 0.5][:d])
    q.finalize()
    q.set_density(np.full(q.nel, 0.7))
    assert q.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-10)["status"] == 0
    q.close()
