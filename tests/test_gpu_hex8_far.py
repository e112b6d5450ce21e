"""The corner-mode Hex8 operator's form for grids of more than 2^32 bytes a component
(offsets counted from each z chunk's first plane), forced onto small ones: the bits of
the usual form, for one chunk and several, FP64 and FP32, and in a solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (30, 6, 5), (31, 7, 4), (12, 23, 17), (62, 21, 2),
                                  (33, 65, 50), (100, 50, 50)])
def test_far_form_has_the_usual_bits(ctx, dims):
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
    ld = p.soa_length() // 3
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    free = torch.zeros((3, ld), dtype=torch.bool, device="cuda")
    free[:, :p.nnode] = torch.from_numpy(np.ascontiguousarray(fixed.reshape(-1, 3).T) == 0).cuda()
    out = {0: [], 1: []}
    for precision, dt in ((icb.FP64, torch.float64), (icb.MIXED, torch.float32)):
        u, b = (torch.randn((3, ld), dtype=dt, device="cuda", generator=g) * free for _ in range(2))
        dinv = torch.rand((3, ld), dtype=dt, device="cuda", generator=g) * free
        for far in (0, 1):
            icb.set_option("hex8_far", far)
            try:
                y = torch.full((3, ld), 7.0, dtype=dt, device="cuda")
                w = b.clone()
                torch.cuda.synchronize()
                p.operator_apply_device(u.data_ptr(), y.data_ptr(), precision)
                p.smoother_apply_device(u.data_ptr(), w.data_ptr(), b.data_ptr(), dinv.data_ptr(),
                                        0.3, 0.4, precision=precision)
                ctx.synchronize()
            finally:
                icb.set_option("hex8_far", 0)
            out[far] += [y, w]
    for a, c in zip(out[0], out[1]):
        assert torch.equal(a, c)
    # a solve: its residuals and the fused dot (whose tiles may differ)
    res = []
    for far in (0, 1):
        icb.set_option("hex8_far", far)
        try:
            info = p.solve(precision=icb.FP64, precond=icb.GMG, tol=1e-10)
        finally:
            icb.set_option("hex8_far", 0)
        res.append((info["iters"], p.displacement()))
    assert abs(res[0][0] - res[1][0]) <= 1
    # both have relres 1e-10 on systems of condition number below 1e5
    assert np.abs(res[0][1] - res[1][1]).max() <= 1e-5 * np.abs(res[0][1]).max()
    p.close()
