"""The waits between the CTAs of a cooperative kernel: with a limit of no polls every
wait gives up at once, the call says so, and the context stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ICB_ERR_TIMEOUT = -5


@pytest.fixture
def no_polls():
    import icarat_b200 as icb
    default = icb.get_option("exchange_spin_limit")
    assert default == 1 << 22
    icb.set_option("exchange_spin_limit", 0)
    yield lambda: icb.set_option("exchange_spin_limit", default)
    icb.set_option("exchange_spin_limit", default)


@pytest.mark.parametrize("dims", [(1, 1), (120, 40), (7, 7, 3), (40, 20, 20)])
def test_solve_reports_the_timeout(ctx, no_polls, dims):
    import icarat_b200 as icb
    d = len(dims)
    p = icb.Problem(ctx, d, *dims)
    fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (d,), np.uint8)
    fixed[..., 0, :] = 1
    p.dirichlet_mask(fixed.reshape(-1))
    p.nodal_load(p.nnode - 1, [0.3, -1.0, 0.5][:d])
    p.finalize()
    p.set_density(np.random.default_rng(3).uniform(0.2, 1.0, p.nel))
    r = p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-10, raise_on_error=False)
    assert r["rc"] == ICB_ERR_TIMEOUT and r["status"] == ICB_ERR_TIMEOUT
    no_polls()
    r = p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-10)
    assert r["status"] == 0 and r["true_relres"] <= 1e-9
    p.close()


def test_filter_reports_the_timeout(ctx, no_polls):
    import icarat_b200 as icb
    p = icb.Problem(ctx, 3, 40, 20, 20)
    p.finalize()
    h = icb.Helmholtz(p, 2.2)
    x = np.full(p.nel, 0.7)
    with pytest.raises(icb.IcbError) as e:
        h.apply(x)
    assert e.value.code == ICB_ERR_TIMEOUT
    no_polls()
    assert np.abs(h.apply(x) - 0.7).max() <= 1e-7
    h.close()
    p.close()


@pytest.mark.parametrize("dims", [(20, 10), (500, 420)])
def test_oc_update_reports_the_timeout(ctx, no_polls, dims):
    import icarat_b200 as icb
    p = icb.Problem(ctx, 2, *dims)
    p.finalize()
    cone = icb.Cone(p, 1.5)
    n = p.nel
    x, df, dg = np.full(n, 0.5), -np.linspace(0.1, 2.0, n), np.ones(n)
    lo, hi = np.full(n, 1e-4), np.ones(n)
    with pytest.raises(icb.IcbError) as e:
        icb.oc_update(p, cone, x, df, 0.5 * n, dg, lo, hi, 0.2)
    assert e.value.code == ICB_ERR_TIMEOUT
    no_polls()
    out, steps = icb.oc_update(p, cone, x, df, 0.5 * n, dg, lo, hi, 0.2)
    assert 0 < steps <= 100 and abs(out.mean() - 0.5) <= 1e-2
    cone.close()
    p.close()
