"""GPU test that a trace call reads and writes its own rays alone: batches that end inside a warp's share, in
buffers that go on beyond them (by more than the largest share), leave every result behind the batch as it was, and
write each one in it, with every kernel, for closest and any hits."""
import numpy as np
import pytest

from tests import raysets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1, 2, 3, 4, 5, 6])
def test_results_of_the_batch_alone(nb, small_city, kernel):
    import torch

    sb = small_city[1]
    base = raysets.aimed_rays(sb, 4096, 5)
    # ends of shares of 8, 12, 32, 64 and 96 rays (148 SMs) and of the cursor's 32, and one more, one less
    sizes = [1, 7, 9, 18, 31, 33, 100, 2001, 40_007, 132_607, 132_609, 1_363_975, 2_727_941]
    n = max(sizes) + 256
    rays = torch.from_numpy(np.tile(base, -(-n // base.shape[0]))[:n].view(np.float32).reshape(-1, 8)).cuda()
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        ctx.set_kernel(kernel)
        for m in sizes:
            hits = torch.full((n, 5), -77, dtype=torch.int32, device="cuda")
            occ = torch.full((n,), 77, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            ctx.reset_object_hits()
            ctx.trace_closest_dev(rays.data_ptr(), m, hits.data_ptr(), count_hits=True)
            ctx.trace_any_dev(rays.data_ptr(), m, occ.data_ptr())
            ctx.sync()
            wrote = (hits != -77).any(1)
            assert wrote[:m].all() and not wrote[m:].any(), m
            assert (occ[:m] != 77).all() and (occ[m:] == 77).all(), m
            assert int(ctx.object_hits().sum()) == int((hits[:m, 1] >= 0).sum()), m
    finally:
        ctx.close()
