"""Branches that only certain sizes, schedules and masks reach: measured sweeps
of lattices whose plaquette takes one thread per site, batches with both
plaquette forms in one launch, reunitarization against a sweep limit and inside a
caller's capture, and HYP and stout smearing of mixed directions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gauge(ctx, dims, prec="f32", lay=1, **kw):
    from sun_b200 import gauge
    g = gauge(ctx, N=3, dims=dims, beta=6.0, atype=lay, prec=prec, seed=13, **kw)
    g.Init(hot=True)
    return g


def _same_as_single_calls(g, h, n, plaq, poly):
    """h, swept and measured call by call, gives g's values, links and counters."""
    from sun_b200 import OnePolyakovLoop, PlaquetteCUB, Sweep
    for i in range(n):
        Sweep(h, 1, 2, 1)
        p = PlaquetteCUB(h).Run()
        assert plaq[i, 0] == p.real and plaq[i, 1] == p.imag and poly[i] == OnePolyakovLoop(h).Run(), i
    assert np.array_equal(g.get_image(), h.get_image()) and g.rng_state() == h.rng_state()


# 32,928 and 36,864 sites: one thread per site from 32,768
@pytest.mark.parametrize("dims,prec,lay", [((14, 14, 14, 12), "f32", 1), ((14, 14, 14, 12), "f64", 0),
                                           ((16, 12, 12, 16), "f32", 2)])
def test_measured_sweeps_of_large_lattices(ctx, dims, prec, lay):
    from sun_b200 import SweepMeasure
    g, h = (_gauge(ctx, dims, prec, lay, reunit_every=2) for _ in range(2))
    _same_as_single_calls(g, h, 5, *SweepMeasure(g, 1, 2, 5))


def test_measured_sweeps_stop_at_the_sweep_limit(ctx):
    """The limit is a due sweep: the sweeps a lattice sits out leave it as it is."""
    from sun_b200 import SweepMeasure
    g, h = (_gauge(ctx, (4, 4, 6, 4), reunit_every=2) for _ in range(2))
    g.set_sweep_limit(4)
    h.set_sweep_limit(4)
    plaq, poly = SweepMeasure(g, 1, 2, 7)
    assert np.array_equal(plaq[3], plaq[6]) and not np.array_equal(plaq[2], plaq[3])
    _same_as_single_calls(g, h, 7, plaq, poly)


@pytest.mark.parametrize("prec,lay", [("f32", 1), ("f64", 0)])
def test_batch_plaquettes_on_both_sides_of_the_limit(ctx, prec, lay):
    from sun_b200 import Batch, OnePolyakovLoop, PlaquetteCUB
    gs = [_gauge(ctx, d, prec, lay) for d in ((4, 4, 4, 6), (14, 14, 14, 12), (12, 12, 14, 16))]
    b = Batch(ctx)
    for g in gs:
        b.add(g)
    for (s, t), l, g in zip(b.plaquette(), b.polyakov(), gs):
        p, q = PlaquetteCUB(g).Run(), OnePolyakovLoop(g).Run()
        assert (s, t) == (p.real, p.imag) and complex(*l) == q
    b.close()


def test_reunitarization_inside_a_callers_capture(ctx):
    """A captured sun_sweep of a lattice that has run a heatbath before."""
    import torch
    from sun_b200 import HeatBath, Sweep
    from sun_b200._native import check, lib
    g, h = (_gauge(ctx, (4, 4, 4, 6), reunit_every=2) for _ in range(2))
    for x in (g, h):
        HeatBath(x).Run(1)
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        check(lib().sun_sweep(g.h, 1, 2, 1, stream.cuda_stream), ctx.h)
    for _ in range(4):
        graph.replay()
    torch.cuda.synchronize()
    Sweep(h, 1, 2, 4)
    torch.cuda.synchronize()
    assert np.array_equal(g.get_image(), h.get_image()) and g.rng_state() == h.rng_state()


@pytest.mark.parametrize("prec,lay,eo", [("f64", 0, True), ("f32", 1, False)])
@pytest.mark.parametrize("mask", [5, 7, 8, 10, 15])
@pytest.mark.parametrize("kind", ["hyp", "stout"])
def test_smearing_of_mixed_directions(ctx, kind, mask, prec, lay, eo):
    """One step against the oracle (the tolerances of the space and time masks),
    and two and three steps against as many calls."""
    import ctypes as C
    from oracle import oracle as O
    from sun_b200._native import check, lib
    alpha = (C.c_double * 3)(0.75, 0.6, 0.3)

    def smear(g, steps):
        if kind == "hyp":
            check(lib().sun_smear_hyp(g.h, alpha, steps, 8, 1e-10, mask, None), ctx.h)
        else:
            check(lib().sun_smear_stout(g.h, 0.1, steps, mask, None), ctx.h)

    dims = (4, 4, 4, 6)
    src = _gauge(ctx, dims, prec, lay, evenodd=eo)
    U = O.hot(3, list(dims), 31)
    O.sweeps(U, list(dims), 5.8, 1, 1, 2, seed=31)
    src.Set(U)
    many, one = (_gauge(ctx, dims, prec, lay, evenodd=eo) for _ in range(2))
    one.Copy(src)
    for steps in (1, 2, 3):
        smear(one, 1)
        many.Copy(src)
        smear(many, steps)
        assert np.array_equal(many.get_image(), one.get_image()), steps
        if steps == 1:
            ref = src.Get()
            if kind == "hyp":
                O.hyp(ref, list(dims), (0.75, 0.6, 0.3), 1, 8, 1e-10, mask)
            else:
                O.stout(ref, list(dims), 0.1, 1, mask)
            tol = 1e-12 if prec == "f64" else (2e-4 if kind == "hyp" else 5e-5)
            assert np.abs(one.Get() - ref).max() < tol
