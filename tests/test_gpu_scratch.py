"""Scratch images kept between calls: given back on request, and to an
allocation that would otherwise fail, also while their context is busy in
another thread."""
import threading
import time

import pytest

pytestmark = pytest.mark.gpu

HYP_BYTES = 2 * 16 * 9 * 16 * 16 ** 4  # both levels of SU(3) FP64 16^4: 302 MB
SLACK = 32 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _keep_scratch(c):
    """A context's lattice after one HYP step, whose scratch it keeps."""
    from sun_b200 import ApplyHYPinSpace, gauge
    g = gauge(c, N=3, dims=(16, 16, 16, 16), prec="f64", seed=1)
    g.Init(hot=True)
    free = _free()
    ApplyHYPinSpace(g, 1, 2, 1e-3)
    assert free - _free() >= HYP_BYTES - SLACK
    return g, free


def _fill(left):
    """All of the device's free memory but `left` bytes."""
    import torch
    torch.cuda.empty_cache()
    return torch.empty(_free() - left, dtype=torch.uint8, device="cuda")


def test_release_scratch_gives_the_memory_back():
    from sun_b200 import Context
    with Context(0) as c:
        g, free = _keep_scratch(c)
        c.release_scratch()
        assert abs(_free() - free) <= SLACK
        g.Release()


@pytest.mark.parametrize("busy", [False, True])
def test_kept_scratch_makes_room_for_a_lattice(busy):
    """24^4 FP64 (191 MB) with 96 MB free beside the kept scratch."""
    import torch
    from sun_b200 import Context, SunError, SweepMeasure, gauge
    with Context(0) as a, Context(0) as b:
        g, _ = _keep_scratch(a)
        h = gauge(a, N=3, dims=(8, 8, 8, 8), prec="f64", seed=2)
        h.Init(hot=True)
        n = 12000
        SweepMeasure(h, 1, 4, n)  # its buffers, before the memory is filled
        fill = _fill(96 << 20)
        t = threading.Thread(target=SweepMeasure, args=(h, 1, 4, n))
        try:
            if busy:
                t.start()
                time.sleep(0.3)
            big = gauge(b, N=3, dims=(24, 24, 24, 24), prec="f64")
            assert not busy or t.is_alive()
            with pytest.raises(SunError) as e:  # 3 GB: more than any context keeps
                gauge(b, N=3, dims=(48, 48, 48, 48), prec="f64")
            assert e.value.status == 3
        finally:
            if busy:
                t.join()
            del fill
            torch.cuda.empty_cache()
        for x in (g, h, big):
            x.Release()
