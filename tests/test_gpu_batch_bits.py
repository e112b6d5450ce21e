"""A batch's designs are bitwise those of their own runs also where the bisection
hangs on the last bit of a volume: every element starts at its upper bound, so
every lambda up to the first element's own leaves the volume at the target, and
whether it lies above is rounding.  Grids of one tile and of many, several tiles a
CTA, the first ones past the one-kernel update, and a radius past its stencils."""
import numpy as np
import pytest

import icarat_b200 as icb

pytestmark = pytest.mark.gpu

GRIDS = [(20, 9, 1.2), (33, 31, 1.5), (64, 65, 2.4), (96, 40, 3.3), (120, 40, 1.5), (131, 77, 4.2),
         (200, 61, 2.1), (250, 130, 1.8), (300, 150, 3.0), (333, 222, 2.4), (420, 210, 1.5),
         (500, 260, 2.7), (640, 320, 2.4), (700, 400, 4.6), (60, 44, 5.2), (830, 800, 1.5)]


@pytest.mark.parametrize("precision", [icb.MIXED, icb.FP64])
def test_designs_on_a_volume_plateau(precision):
    def build(nx, ny):
        c = icb.Context(0)
        p = icb.Problem(c, 2, nx, ny)
        fixed = np.zeros((ny + 1, nx + 1, 2), np.uint8)
        fixed[:, 0, :] = 1
        p.dirichlet_mask(fixed.reshape(-1))
        p.nodal_load((ny // 2) * (nx + 1) + nx, [0.1, -1.0])
        p.finalize()
        return c, p

    pairs = [build(nx, ny) for nx, ny, _ in GRIDS]
    probs = [p for _, p in pairs]
    opts = [icb.loop_opts(3, r, move=0.2, use_threshold=k % 2 == 1, precision=precision)
            for k, (_, _, r) in enumerate(GRIDS)]
    rho0 = [np.ones(p.nel) for p in probs]
    h, x, st = icb.run_batch(probs, [icb.JOB_OC] * len(probs), opts, rho0, nworkers=1)
    assert (st == 0).all()
    for k, (p, (_, _, r)) in enumerate(zip(probs, GRIDS)):
        ha, xa = icb.run_loop(p, "oc", rho0[k], 3, r, move=0.2, use_threshold=k % 2 == 1,
                              precision=precision)
        assert np.array_equal(ha, h[k]) and np.array_equal(xa, x[k]), GRIDS[k]
    for c, p in pairs:
        p.close()
        c.close()
