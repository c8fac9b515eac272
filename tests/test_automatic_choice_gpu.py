"""GPU test of the library's own choice of a traversal: it can be taken up again on a context whose only node layout
is a paged wide one, and it goes with a configuration that is read from one context and set on another."""
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


def test_unchosen_configuration_goes_with_the_dict(nb, small_city):
    sb = small_city[1]
    a, b = nb.Context(0), nb.Context(0)
    try:
        for c in (a, b):
            c.upload(sb)
        b.set_kernel(nb.KERNEL_BVH8)
        b.set_traversal(**a.traversal())
        assert b.traversal() == a.traversal()
        # changed in a field, it is an ordinary configuration
        for change in (dict(width=4, persistent=2, short_stack=16), dict(persistent=1), dict(min_blocks=10), dict(block=64)):
            b.set_traversal(**dict(a.traversal(), **change))
            assert b.traversal() == dict(a.traversal(), regroup=1, **change)
        # and so is the per-thread binary walk by its own numbers
        b.set_traversal(**dict(a.traversal(), regroup=1))
        assert b.traversal()["regroup"] == 1 and a.traversal()["regroup"] != 1
        b.set_kernel(nb.KERNEL_AUTO)
        assert b.traversal() == a.traversal()
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("leaves", ["several records", "one record"])
def test_sweep_times_no_build_twice(nb, small_city, leaves):
    """The cooperative walk has one build, so the sweep lists min_blocks for it only where the scene's leaves hold
    one record, which the lane-by-lane walk serves."""
    sb = small_city[1]
    if leaves == "one record":
        geom = np.zeros((64, 15), np.float32)
        geom[:, :9] = np.random.default_rng(1).uniform(-5, 5, (64, 9))
        sb = nb.SceneBVH(nb.HostScene(np.ones(64, np.int32), geom, np.full((64, 20), 0.5, np.float32), np.arange(64),
                                      np.ones(64, np.uint32)))
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        res = ctx.autotune_sweep(raysets.aimed_rays(sb, 6000, 1), repeats=1)
        bounded = sorted(name for name, cfg, ms, bad in res["entries"] if cfg["persistent"] == 1 and cfg["min_blocks"])
        assert len(bounded) == (9 if leaves == "one record" else 0)
        assert all(bad == 0 for _, _, ms, bad in res["entries"] if ms >= 0)
    finally:
        ctx.close()
