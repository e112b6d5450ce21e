"""Several one-kernel solves at a time: the more of them are in flight the fewer CTAs
each takes, several boxes of its cut a CTA.  The iterates are bitwise those of the
solve alone: 2D and 3D Jacobi-PCG and the 3D Helmholtz filter, cuts of one box, of
few and of as many as there are SMs, boxes too large to share a CTA."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = 6


def together(jobs):
    """every job of a list in a thread of its own; their results"""
    out, go = [None] * len(jobs), threading.Barrier(len(jobs))

    def run(k):
        go.wait()
        try:
            out[k] = jobs[k]()
        except Exception as e:  # noqa: BLE001 -- reported by the caller
            out[k] = e

    ts = [threading.Thread(target=run, args=(k,)) for k in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for r in out:
        if isinstance(r, Exception):
            raise r
    return out


@pytest.mark.parametrize("dims", [(15, 15), (120, 40), (97, 3), (250, 151), (540, 540), (7, 7, 3),
                                  (40, 15, 15), (60, 20, 20), (33, 2, 2), (41, 41, 41), (48, 46, 45)])
def test_concurrent_solves_equal_the_solve_alone(dims):
    import icarat_b200 as icb
    d = len(dims)
    ctxs = [icb.Context(0) for _ in range(THREADS)]
    probs = []
    for k, c in enumerate(ctxs):
        p = icb.Problem(c, d, *dims)
        fixed = np.zeros(tuple(n + 1 for n in reversed(dims)) + (d,), np.uint8)
        fixed[..., 0, :] = 1
        p.dirichlet_mask(fixed.reshape(-1))
        p.nodal_load(p.nnode - 1, [0.3, -1.0, 0.5][:d])
        p.finalize()
        p.set_density(np.random.default_rng(k).uniform(0.2, 1.0, p.nel))
        probs.append(p)

    def solve(p):
        info = p.solve(precision=icb.FP64, precond=icb.JACOBI, tol=1e-9, maxit=20000)
        return info["iters"], p.displacement()

    alone = [solve(p) for p in probs]
    for _ in range(3):
        for (it, u), (i0, u0) in zip(together([lambda p=p: solve(p) for p in probs]), alone):
            assert it == i0
            assert np.array_equal(u, u0)
    for p in probs:
        p.close()
    for c in ctxs:
        c.close()


@pytest.mark.parametrize("dims", [(7, 7, 3), (20, 10, 10), (40, 20, 20), (80, 40, 40), (128, 64, 64)])
def test_concurrent_filters_equal_the_filter_alone(dims):
    import icarat_b200 as icb
    ctxs = [icb.Context(0) for _ in range(THREADS)]
    probs, filters, xs = [], [], []
    for k, c in enumerate(ctxs):
        p = icb.Problem(c, 3, *dims)
        p.finalize()
        probs.append(p)
        filters.append(icb.Helmholtz(p, 2.2))
        xs.append(np.random.default_rng(k).uniform(0.01, 1.0, p.nel))

    def calls(k):
        return [filters[k].apply(xs[k], sens=bool(q % 2)) for q in range(10)]

    alone = [calls(k) for k in range(THREADS)]
    for got, ref in zip(together([lambda k=k: calls(k) for k in range(THREADS)]), alone):
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
    for f, p, c in zip(filters, probs, ctxs):
        f.close()
        p.close()
        c.close()
