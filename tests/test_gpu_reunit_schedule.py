"""The scheduled reunitarization where its threads take several links each (a
remainder of links among them), and its cost on a small lattice."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one, two, three (4 V not a multiple) and eight links per thread
@pytest.mark.parametrize("N,prec,lay,dims", [(2, "f32", 0, (18, 18, 18, 18)), (2, "f32", 0, (20, 20, 20, 20)),
                                             (3, "f32", 1, (22, 22, 22, 22)), (2, "f64", 0, (28, 28, 28, 28))])
def test_due_sweeps_reunitarize_every_link(ctx, N, prec, lay, dims):
    from sun_b200 import Batch, Reunitarize, Sweep, gauge
    small = (4, 4, 4, 6)
    a, b, c, d, e = (gauge(ctx, N=N, dims=x, beta=2.5, atype=lay, prec=prec, seed=6, reunit_every=r)
                     for x, r in ((dims, 0), (dims, 1), (dims, 1), (small, 0), (small, 1)))
    for g in (a, b, c, d, e):
        g.Init(hot=True)
    Sweep(b, 0, 1, 1)
    batch = Batch(ctx)  # the small lattice shares the large one's launch
    batch.add(c)
    batch.add(e)
    batch.sweep(0, 1, 1)
    for g in (a, d):
        Sweep(g, 0, 1, 1)
        Reunitarize(g).Run()
    assert np.array_equal(a.get_image(), b.get_image()) and np.array_equal(a.get_image(), c.get_image())
    assert np.array_equal(d.get_image(), e.get_image())
    batch.close()
    for g in (a, b, c, d, e):
        g.Release()


def test_due_launch_of_a_small_lattice_uses_the_gpu(ctx):
    """A due sweep costs no more than an undue one and twice a reunitarization
    call (SU(6) 8^4 FP32: 92 + 2 x 33 us; 115 us measured, 247 us with eight links
    per thread)."""
    import torch
    from sun_b200 import Reunitarize, Sweep, gauge

    def best(f, n=20):
        f(1)
        t = []
        for _ in range(10):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            f(n)
            torch.cuda.synchronize()
            t.append((time.perf_counter() - t0) / n)
        return min(t)

    never, due = (gauge(ctx, N=6, dims=(8, 8, 8, 8), beta=25.0, prec="f32", seed=2, reunit_every=r) for r in (0, 1))
    never.Init(hot=True)
    due.Init(hot=True)
    once = Reunitarize(never)
    t_call = best(lambda n: [once.Run() for _ in range(n)])
    assert best(lambda n: Sweep(due, 0, 1, n)) < best(lambda n: Sweep(never, 0, 1, n)) + 2 * t_call
    never.Release()
    due.Release()
