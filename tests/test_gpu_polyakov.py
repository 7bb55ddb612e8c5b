"""The Polyakov loop of SU(6), whose lanes load each link where it is used:
time extents shorter than the lanes, one link per lane and remainders, with 8 and
with 2 lanes per spatial site, against the FP64 oracle on the stored links (FP64
products: 1e-12)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,prec,eo", [((4, 4, 4, 2), "f32", True), ((4, 4, 6, 8), "f64", False),
                                          ((4, 4, 4, 22), "f32", False), ((22, 20, 20, 2), "f64", True),
                                          ((20, 22, 20, 6), "f32", True), ((20, 20, 22, 10), "f64", False)])
def test_su6_polyakov_matches_oracle(ctx, dims, prec, eo):
    from oracle import oracle as O
    from sun_b200 import OnePolyakovLoop, gauge
    g = gauge(ctx, N=6, dims=dims, beta=25.0, evenodd=eo, prec=prec, seed=4)
    g.Init(hot=True)
    l = O.polyakov(g.Get(), list(dims))
    assert abs(OnePolyakovLoop(g).Run() - (l[0] + 1j * l[1])) < 1e-12
    g.Release()
