"""The plaquette's two decompositions on either side of their volume limit and
the Polyakov loop's two lane counts, against the FP64 oracle on the stored
links (FP64 sums: 1e-12), in both orders; scheduled reunitarization with fewer
threads than links; smearing scratch shared by calls of different sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# N, dims, prec, layout, even/odd: volumes just below and above 2^15 sites, and
# spatial volumes below and above 8192, T not a multiple of the lanes
VOLUMES = [(3, (14, 14, 12, 12), "f32", 1, True), (3, (14, 14, 14, 12), "f32", 1, True),
           (3, (22, 20, 20, 4), "f32", 0, False), (3, (22, 20, 20, 6), "f64", 0, True),
           (3, (18, 22, 26, 10), "f64", 1, False), (3, (14, 12, 14, 14), "f32", 2, True),
           (2, (24, 22, 18, 6), "f32", 0, True), (2, (16, 16, 12, 12), "f64", 0, False),
           (4, (16, 16, 12, 14), "f32", 0, True), (6, (4, 4, 4, 10), "f64", 0, True)]


@pytest.mark.parametrize("N,dims,prec,lay,eo", VOLUMES)
def test_plaquette_and_polyakov_match_oracle_at_kernel_limits(ctx, N, dims, prec, lay, eo):
    from oracle import oracle as O
    from sun_b200 import OnePolyakovLoop, PlaquetteCUB, gauge
    g = gauge(ctx, N=N, dims=dims, beta=6.0, atype=lay, evenodd=eo, prec=prec, seed=4)
    g.Init(hot=True)
    U, X = g.Get(), list(dims)
    p, l = PlaquetteCUB(g).Run(), OnePolyakovLoop(g).Run()
    po, lo = O.plaquette(U, X), O.polyakov(U, X)
    assert abs(p.real - po[0]) < 1e-12 and abs(p.imag - po[1]) < 1e-12
    assert abs(l - (lo[0] + 1j * lo[1])) < 1e-12


@pytest.mark.parametrize("N,prec,lay,dims", [(3, "f32", 1, (4, 4, 4, 6)), (3, "f64", 0, (6, 6, 4, 10)), (2, "f32", 0, (4, 4, 4, 4))])
def test_scheduled_reunitarization_is_the_full_one(ctx, N, prec, lay, dims):
    """A due sweep, alone or measured, leaves the links of the sweep followed by
    a full reunitarization."""
    from sun_b200 import Reunitarize, Sweep, SweepMeasure, gauge
    gs = [gauge(ctx, N=N, dims=dims, beta=2.3 * N / 2, atype=lay, prec=prec, seed=8, reunit_every=e) for e in (0, 2, 2)]
    for g in gs:
        g.Init(hot=True)
    Sweep(gs[0], 1, 2, 2)
    Reunitarize(gs[0]).Run()
    Sweep(gs[1], 1, 2, 2)
    SweepMeasure(gs[2], 1, 2, 2)
    ref = gs[0].get_image()
    assert np.array_equal(ref, gs[1].get_image()) and np.array_equal(ref, gs[2].get_image())
    assert gs[0].rng_state() == gs[1].rng_state() == gs[2].rng_state()


@pytest.mark.parametrize("mask", [7, 8, 5, 15])
@pytest.mark.parametrize("steps", [1, 2, 3])
def test_smearing_steps_and_scratch(ctx, mask, steps):
    """n steps in one call are n calls of one step, whichever directions are
    smeared, with the scratch of a larger call in between."""
    from sun_b200 import gauge
    from sun_b200._native import check, lib
    a, b, big = (gauge(ctx, N=3, dims=d, atype=1, prec="f32", seed=5) for d in ((4, 6, 4, 8), (4, 6, 4, 8), (8, 8, 8, 8)))
    a.Init(hot=True)
    big.Init(hot=True)
    b.Copy(a)
    assert np.array_equal(a.get_image(), b.get_image())
    check(lib().sun_smear_ape(a.h, 0.2, steps, 4, 0.0, mask, None), ctx.h)
    for _ in range(steps):
        check(lib().sun_smear_ape(b.h, 0.2, 1, 4, 0.0, mask, None), ctx.h)
        check(lib().sun_smear_ape(big.h, 0.2, 1, 4, 0.0, 7, None), ctx.h)
    assert np.array_equal(a.get_image(), b.get_image())
