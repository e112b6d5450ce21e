"""The V-cycle's forms that claim one another's bits: the coarse levels as one launch
against their own launches, on grids whose first tail level is the largest it takes
and one past it (in 2D 48 rows of up to 32 nodes in FP64 and 64 in FP32, 480 nodes in
3D), thin and odd ones, and a problem that is all tail; and the 3D restriction with one, two, four and
five coarse planes a thread, on every parity of the axes and on a grid past the size
where it takes four by itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(ctx, dims):
    import icarat_b200 as icb
    d = len(dims)
    p = icb.Problem(ctx, d, *dims)
    fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (d,), np.uint8)
    fixed[..., 0, :] = 1
    fixed[(0,) * (d - 1) + (dims[0] // 2, d - 1)] = 1  # a point support at an odd or even node
    p.dirichlet_mask(fixed.reshape(-1))
    p.nodal_load(p.nnode - 1, [0.3, -1.0, 0.5][:d])
    p.finalize()
    p.set_density(np.random.default_rng(3).uniform(0.2, 1.0, p.nel))
    return p


def solves(p, option, values, smooth=(0,)):
    """(iterations, displacement) per precision and degree, for every value of an option"""
    import icarat_b200 as icb
    default = icb.get_option(option)
    out = []
    for v in values:
        icb.set_option(option, v)
        try:
            out.append([])
            for precision in (icb.FP64, icb.MIXED):
                for nu in smooth:
                    i = p.solve(precision=precision, precond=icb.GMG, tol=1e-10, mg_smooth=nu)
                    out[-1].append((i["iters"], p.displacement()))
        finally:
            icb.set_option(option, default)
    return out


@pytest.mark.parametrize("dims", [(63, 23), (63, 24), (31, 47), (31, 48), (64, 15), (64, 16),
                                  (63, 31), (63, 32), (31, 63), (31, 64), (126, 62), (57, 57), (68, 78),
                                  (120, 40), (61, 1), (9, 33), (24, 13), (333, 222),
                                  (7, 9, 5), (7, 9, 6), (7, 7, 7), (15, 15, 15), (16, 15, 15), (20, 10, 10),
                                  (33, 9, 1), (7, 6, 5), (40, 21, 18)])
def test_tail_has_the_bits_of_its_levels_launches(ctx, dims):
    p = build(ctx, dims)
    a, b = solves(p, "mg_tail", (1, 0), smooth=(0, 1, 3))
    for (ia, ua), (ib, ub) in zip(a, b):
        assert ia == ib
        assert np.array_equal(ua, ub)
    p.close()


@pytest.mark.parametrize("dims", [(16, 14, 12), (17, 14, 12), (16, 15, 12), (16, 14, 13), (17, 15, 13),
                                  (15, 9, 30), (22, 10, 31), (270, 6, 5), (33, 31, 37),
                                  (257, 65, 63), (256, 66, 67), (256, 73, 62)])
def test_restriction_has_the_same_bits_for_any_planes(ctx, dims):
    p = build(ctx, dims)
    first, *rest = solves(p, "mg_restrict_planes", (1, 2, 4, 5, 0))
    for r in rest:
        for (ia, ua), (ib, ub) in zip(first, r):
            assert ia == ib
            assert np.array_equal(ua, ub)
    p.close()
