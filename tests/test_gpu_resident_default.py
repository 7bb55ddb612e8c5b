"""Resident sweeps of sun_sweep_measure: what they cost beside the replayed
graph, and which lattices take them by default."""
import os
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA = {3: 6.0, 4: 10.5}


def _context(**env):
    """A context made with these variables and no other SUN_B200_RESIDENT* ones."""
    from sun_b200 import Context
    names = set(env) | {"SUN_B200_RESIDENT", "SUN_B200_RESIDENT_MAX_HALFV"}
    old = {k: os.environ.pop(k, None) for k in names}
    os.environ.update(env)
    try:
        return Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


def _lattice(ctx, N, dims, prec, lay):
    from sun_b200 import gauge
    g = gauge(ctx, N=N, dims=dims, beta=BETA[N], atype=lay, prec=prec, seed=21, reunit_every=2)
    g.Init(hot=True)
    return g


@pytest.mark.parametrize("N,prec,lay", [(3, "f64", 0), (3, "f32", 1), (4, "f64", 0)])
def test_resident_sweeps_cost_little_more_than_the_graph(N, prec, lay):
    """8^4: 1.02 to 1.17 times the graph's time measured; 2.4 to 2.7 times when the
    warps stay split behind their waits."""
    from sun_b200 import SweepMeasure
    t = {}
    for how in "01":
        with _context(SUN_B200_RESIDENT=how) as c:
            g = _lattice(c, N, (8, 8, 8, 8), prec, lay)
            SweepMeasure(g, 1, 4, 20)
            t[how] = 1e9
            for _ in range(8):
                t0 = time.perf_counter()
                SweepMeasure(g, 1, 4, 20)
                t[how] = min(t[how], time.perf_counter() - t0)
            g.Release()
    assert t["1"] < 1.6 * t["0"]


def _runs_resident(c, g):
    """A CTA told to skip its first barrier makes a resident call fail."""
    from sun_b200 import SunError, SweepMeasure
    from sun_b200._native import lib
    assert lib().sun_debug_resident_barrier(c.h, 2_000_000, 0) == 0
    try:
        SweepMeasure(g, 1, 1, 1)
        return False
    except SunError as e:
        assert "ran out" in str(e)
        return True
    finally:
        assert lib().sun_debug_resident_barrier(c.h, 0, -1) == 0


# prec, layout, dims, environment, resident: both ends of the default's range
# (6,145 and 9,216 to 16,383 half-sites), classes outside it, and the limit set
DEFAULTS = [("f32", 1, (8, 8, 12, 16), {}, False), ("f32", 1, (10, 10, 8, 16), {}, True),
            ("f32", 0, (8, 16, 16, 8), {}, False), ("f32", 0, (16, 16, 18, 4), {}, True),
            ("f32", 0, (14, 14, 14, 10), {}, True), ("f32", 1, (16, 16, 16, 8), {}, False),
            ("f64", 0, (12, 12, 12, 12), {}, False), ("f32", 2, (12, 12, 12, 12), {}, False),
            ("f32", 1, (12, 12, 12, 12), {"SUN_B200_RESIDENT_MAX_HALFV": "10367"}, False),
            ("f32", 1, (12, 12, 12, 12), {"SUN_B200_RESIDENT_MAX_HALFV": "10368"}, True),
            ("f32", 1, (12, 12, 12, 12), {"SUN_B200_RESIDENT": "auto"}, True)]


@pytest.mark.parametrize("prec,lay,dims,env,resident", DEFAULTS)
def test_default_takes_the_faster_path_with_the_same_bits(prec, lay, dims, env, resident):
    from sun_b200 import SweepMeasure
    with _context(**env) as c, _context(SUN_B200_RESIDENT="0") as graph:
        g = _lattice(c, 3, dims, prec, lay)
        assert _runs_resident(c, g) == resident
        g.Release()
        g, h = _lattice(c, 3, dims, prec, lay), _lattice(graph, 3, dims, prec, lay)
        for n in (3, 2):
            for x, y in zip(SweepMeasure(g, 1, 4, n), SweepMeasure(h, 1, 4, n)):
                assert np.array_equal(x, y)
        assert np.array_equal(g.get_image(), h.get_image()) and g.rng_state() == h.rng_state()
        g.Release()
        h.Release()


@pytest.mark.parametrize("N,prec,dims", [(3, "f32", (12, 12, 12, 12)), (4, "f64", (8, 8, 12, 12)), (3, "f64", (10, 10, 10, 16))])
def test_forced_row_split_resident_sweeps_keep_the_bits(N, prec, dims):
    """More row-split CTAs than SMs: the resident launch takes one thread per
    half-site."""
    from sun_b200 import SweepMeasure
    with _context(SUN_B200_RESIDENT="1", SUN_B200_UPDATE_KERNEL="rows") as c, _context(SUN_B200_RESIDENT="0") as graph:
        g, h = _lattice(c, N, dims, prec, 0), _lattice(graph, N, dims, prec, 0)
        for x, y in zip(SweepMeasure(g, 1, 2, 3), SweepMeasure(h, 1, 2, 3)):
            assert np.array_equal(x, y)
        assert np.array_equal(g.get_image(), h.get_image())
        g.Release()
        h.Release()
