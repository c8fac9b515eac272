"""GPU test of ray queues whose length is on the device, walked by a context that chose no kernel: the shares
follow from the length that a queue has, so frames whose queues begin on either side of the lines between share
sizes equal the per-thread walk's bit for bit, and short queues of a large frame do not leave the chip idle."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _view(nb, w, h, spp, depth):
    return nb.view_pinhole((0, 60, -180), (0, 0, 0), width=w, height=h, spp=spp, max_depth=depth, seed=3)


# 148 SMs: equal shares up to 132,608 paths, shares of 32 rays up to 1,363,968, of 64 up to 2,727,936
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (33, 1, 1), (259, 16, 1), (259, 512, 1), (148, 128, 7), (1300, 103, 1),
                                     (1184, 1152, 1), (1185, 1152, 1), (1369, 997, 2), (1433, 1003, 3)])
def test_frames_equal_the_per_thread_walk(nb, small_city, w, h, spp):
    v = _view(nb, w, h, spp, 3)
    out = []
    for kernel in (0, 1):
        c = nb.Context(0)
        try:
            c.upload(small_city[1])
            c.set_kernel(kernel)
            out.append(c.render(v)[0])
            assert c.status() == 0
        finally:
            c.close()
    assert np.array_equal(out[0].view(np.int32), out[1].view(np.int32))


def test_short_queues_of_a_large_frame(nb, small_city):
    """Six bounces of 921,600 paths, whose queues shrink to a few thousand rays: the untuned context takes at
    most 1.3 times as long as the same kernel fed from a cursor (1.8 with shares of the capacity)."""
    v = _view(nb, 1280, 720, 1, 6)
    best = []
    for kernel in (0, 4):
        c = nb.Context(0)
        try:
            c.upload(small_city[1])
            c.set_kernel(kernel)
            times = []
            for _ in range(9):
                t0 = time.perf_counter()
                c.render(v, graph=True)
                c.sync()
                times.append(time.perf_counter() - t0)
            best.append(min(times))
        finally:
            c.close()
    assert best[0] <= 1.3 * best[1], best
