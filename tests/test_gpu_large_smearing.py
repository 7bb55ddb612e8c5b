"""Smearing a lattice whose image is above the documented limit of a pitched
copy (the four directions of one element take 2^31 bytes or more: 2^25 sites in
FP64, 2^26 in FP32).  The large lattice is a small one repeated along T, and
spatial staples do not leave a time slice, so every slice must come out with
the small lattice's bits."""
import pytest

pytestmark = pytest.mark.gpu


class _Image:
    def __init__(self, g, real):
        self.lattice = g
        self.__cuda_array_interface__ = dict(shape=(g.Bytes() // real,), typestr=f"<f{real}", data=(g.GetPtr(), False),
                                             version=3, strides=None)


def _view(g):
    """The device image as [element, direction, T, re/im of a time slice]."""
    import torch
    x, y, z, t = g.dims
    elems = 4  # SU(2) full links
    return torch.as_tensor(_Image(g, 4 if g.prec == "f32" else 8), device="cuda").view(elems, 4, t, 2 * x * y * z)


@pytest.mark.parametrize("prec,space", [("f64", (64, 64, 64)), ("f32", (64, 64, 128))])
def test_odd_step_counts_above_the_pitch_limit(ctx, prec, space):
    import torch
    from sun_b200 import gauge
    from sun_b200._native import check, lib
    small, big = (gauge(ctx, N=2, dims=space + (t,), beta=2.5, evenodd=False, prec=prec, seed=3) for t in (2, 128))
    try:
        assert 4 * big.volume * (16 if prec == "f64" else 8) >= 2 ** 31
        for mask, steps in ((7, 1), (5, 3)):  # one run of directions, two runs
            small.Init(hot=True)
            s, b = _view(small), _view(big)
            b.view(4, 4, 64, 2, -1).copy_(s[:, :, None])
            torch.cuda.synchronize()
            for g in (small, big):
                check(lib().sun_smear_ape(g.h, 0.2, steps, 3, 1e-10, mask, None), ctx.h)
            for e in range(4):
                assert torch.equal(b[e].view(4, 64, 2, -1), s[e][:, None].expand(4, 64, 2, -1)), (mask, e)
    finally:
        small.Release()
        big.Release()
