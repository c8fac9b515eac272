"""GPU test of the library's own choice of a traversal: it can be taken up again on a context whose only node layout
is a paged wide one."""
import numpy as np
import pytest

from tests import raysets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 4, 8])
def test_automatic_again_while_paging(nb, small_city, width):
    sb = small_city[1]
    rays = raysets.aimed_rays(sb, 3000, 1)
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        want = ctx.trace_closest(rays)
        ctx.paging_enable(1 << 40, width=width, max_onloads=sb.object_count)
        for _ in range(8):
            ctx.paging_update()
            ctx.paging_wait()
        ctx.set_traversal(width=width, persistent=2, short_stack=16, regroup=24)
        tuned = ctx.trace_closest(rays)
        ctx.set_kernel(nb.KERNEL_AUTO)
        auto = ctx.trace_closest(rays)
        assert np.array_equal(auto, tuned) and np.array_equal(auto["prim"], want["prim"])
        if width != 2:
            with pytest.raises(nb.NomadError, match="paged"):
                ctx.set_kernel(nb.KERNEL_BVH2)
        assert ctx.status() == 0
    finally:
        ctx.close()
