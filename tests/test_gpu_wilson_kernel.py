"""k_wilson at the edges of its decomposition, against the FP64 oracle: every
CTA size (it depends on N, R and T), volumes that fill no whole tile, CTAs of
several items, odd and even T (values leave the warp two t's at a time), and
extents without loops.  The sums are FP64 products of the stored links, so
1e-12 as for the other measurements."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # N, dims, prec, layout, even/odd, R, T
    (2, (4, 4, 4, 6), "f32", 0, True, 3, 5),
    (3, (6, 4, 10, 8), "f32", 1, True, 3, 3),
    (3, (4, 6, 4, 10), "f64", 0, False, 1, 8),
    (3, (10, 10, 10, 4), "f64", 0, True, 8, 1),
    (3, (10, 10, 10, 10), "f64", 1, False, 8, 8),
    (3, (6, 6, 4, 4), "f32", 2, True, 2, 2),
    (3, (20, 20, 20, 20), "f32", 1, True, 2, 4),
    (4, (4, 4, 6, 6), "f32", 0, True, 3, 5),
    (4, (4, 4, 4, 10), "f64", 0, False, 2, 8),
    (6, (4, 4, 4, 10), "f32", 0, True, 2, 8),
    (3, (4, 4, 4, 4), "f64", 0, True, 0, 3),
    (3, (4, 4, 4, 4), "f64", 0, True, 3, 0),
    (3, (4, 4, 4, 4), "f64", 0, True, 0, 0),
]


@pytest.mark.parametrize("N,dims,prec,lay,eo,R,T", CASES)
def test_wilson_loops_match_oracle_at_tile_edges(ctx, N, dims, prec, lay, eo, R, T):
    from oracle import oracle as O
    from sun_b200 import WilsonLoop, gauge
    g = gauge(ctx, N=N, dims=dims, beta=6.0, atype=lay, evenodd=eo, prec=prec, seed=3)
    g.Init(hot=True)
    ref = O.wilson_loops(g.Get(), list(dims), R, T)
    got = WilsonLoop(g, R, T)
    assert np.abs(got - (ref[..., 0] + 1j * ref[..., 1])).max() < 1e-12
