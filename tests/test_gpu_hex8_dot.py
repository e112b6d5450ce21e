"""The fused p.Kp of the corner-mode Hex8 operator, directly: after one iteration of
the Jacobi-PCG x = (r.z / p.Kp) p with r = b, so b.x = x.Kx, the right side taken with
the dense element product and summed exactly.  Grids ending inside, at and just past
tiles of 7 and of 11 node rows, with one and with several z chunks."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# up to (12, 23, 17), and 30x87x60 and 61x54x80, in tiles of 8 element rows on 148 SMs,
# the others in tiles of 12
@pytest.mark.parametrize("dims", [(1, 1, 1), (30, 6, 5), (31, 7, 4), (29, 10, 3), (30, 11, 9),
                                  (62, 21, 2), (12, 23, 17), (30, 87, 60), (61, 54, 80),
                                  (100, 50, 50), (92, 65, 33), (93, 66, 34), (31, 88, 61)])
def test_fused_dot_matches_dense_product(ctx, dims):
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
    L = icb.lib()
    n = p.soa_length()
    assert n <= L.icb_noalloc_max_soa()
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    b = torch.zeros((3, n // 3), dtype=torch.float64, device="cuda")
    free = torch.from_numpy(np.ascontiguousarray(fixed.reshape(-1, 3).T) == 0).cuda()
    b[:, :p.nnode] = torch.randn((3, p.nnode), dtype=torch.float64, device="cuda", generator=g) * free
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    torch.cuda.synchronize()
    info = icb.SolveInfo()
    rc = L.icb_solve_noalloc(p.h, b.data_ptr(), x.data_ptr(), 1e-30, 1, C.byref(info))
    assert rc == -4 and info.iters == 1  # the iteration limit
    icb.set_option("hex8_modal", 0)
    try:
        p.operator_apply_device(x.data_ptr(), y.data_ptr(), icb.FP64)
        ctx.synchronize()
    finally:
        icb.set_option("hex8_modal", 1)
    xs, ys, bs = (v.cpu().numpy()[:, :p.nnode].reshape(-1) for v in (x, y, b))
    bx, xkx = math.fsum(bs * xs), math.fsum(xs * ys)
    # either operator's entries have 24 products and eight elements' sums, a sum of
    # terms passes fewer than 100 additions on its way through thread, warp and blocks
    tol = (2 * 24 * 8 + 100) * np.finfo(float).eps * math.fsum(np.abs(xs * ys)) / xkx
    assert tol < 1e-11
    assert abs(bx / xkx - 1.0) <= tol
    p.close()
