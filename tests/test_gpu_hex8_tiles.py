"""The corner-mode Hex8 operator at the edges of its tiles (31 x 7 nodes; FP64
product and residual 31 x 11) and of its z chunks against the dense element
product: the operator, the smoothing step and the fused forms inside a solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (30, 6, 5), (31, 7, 4), (29, 10, 3), (30, 11, 9),
                                  (62, 21, 2), (61, 22, 7), (12, 23, 17), (5, 44, 3), (93, 13, 40)])
def test_corner_mode_tiles_match_dense_product(ctx, dims):
    import torch
    import icarat_b200 as icb
    p = icb.Problem(ctx, 3, *dims)
    fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (3,), np.uint8)
    fixed[..., 0, :] = 1
    fixed[-1, -1, -1, 1] = 1
    p.dirichlet_mask(fixed.reshape(-1))
    p.nodal_load(p.nnode - 2, [0.3, -1.0, 0.5])
    p.finalize()
    p.set_density(np.random.default_rng(2).uniform(0.05, 1.0, p.nel))
    n = p.soa_length()
    ld = n // 3
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    free = torch.zeros((3, ld), dtype=torch.bool, device="cuda")
    free[:, :p.nnode] = torch.from_numpy(np.ascontiguousarray(fixed.reshape(-1, 3).T) == 0).cuda()
    for precision, dt, eps in ((icb.FP64, torch.float64, 2.3e-16), (icb.MIXED, torch.float32, 1.2e-7)):
        u, b = (torch.randn((3, ld), dtype=dt, device="cuda", generator=g) * free for _ in range(2))
        dinv = torch.rand((3, ld), dtype=dt, device="cuda", generator=g) * free
        out = []
        for modal in (1, 0):
            icb.set_option("hex8_modal", modal)
            try:
                y = torch.full((3, ld), 7.0, dtype=dt, device="cuda")
                w = b.clone()
                torch.cuda.synchronize()
                p.operator_apply_device(u.data_ptr(), y.data_ptr(), precision)
                p.smoother_apply_device(u.data_ptr(), w.data_ptr(), b.data_ptr(), dinv.data_ptr(),
                                        0.3, 0.4, precision=precision)
                ctx.synchronize()
            finally:
                icb.set_option("hex8_modal", 1)
            out.append((y, w))
        for a, c in zip(out[0], out[1]):
            # 24 products and as many sums of eight elements, entries of K0 below 1
            # and |u| below 6
            assert float((a - c)[:, :p.nnode].abs().max()) <= 24 * 8 * 6 * eps
        assert bool((out[0][0][:, p.nnode:] == 7.0).all())  # the padding is not written
    p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-12, maxit=100000)
    v = p.displacement()
    info = p.solve(precision=icb.FP64, precond=icb.GMG, tol=1e-12)
    assert info["true_relres"] <= 1e-9
    assert np.abs(p.displacement() - v).max() <= 1e-6 * np.abs(v).max()
    p.close()
