"""GPU test of the shading kernel's block appends: frames of one partial block up to several rounds of every
block, ragged, equal bit for bit to the same paths rendered in tiles of a few blocks, with the same counts of
rays, escapes and hits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (31, 1, 1), (255, 3, 1), (257, 1, 2), (517, 401, 1), (389, 311, 5)])
def test_frame_equals_tiles(nb, small_city, w, h, spp):
    scene, sb = small_city
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        view = nb.view_pinhole((0, 60, -180), (0, 0, 0), width=w, height=h, spp=spp, max_depth=4, seed=11)
        ctx.reset_render_stats()
        whole = ctx.render(view)[0]
        stats = ctx.render_stats().copy()
        ctx.reset_render_stats()
        rows = max(1, (4000 + w * spp - 1) // (w * spp))
        for y in range(0, h, rows):
            n = min(rows, h - y)
            tile = ctx.render_tiles(view, [(0, y, w, n)])[0]
            assert np.array_equal(tile.view(np.int32), whole[y:y + n].view(np.int32))
        assert np.array_equal(ctx.render_stats(), stats)
        assert int(stats[0]) >= w * h * spp
    finally:
        ctx.close()


@pytest.mark.parametrize("mode", ["plain", "restir", "reference"])
@pytest.mark.parametrize("w,h,spp", [(301, 299, 1), (8, 4, 2400), (211, 213, 2), (179, 167, 3), (150, 101, 6), (2, 7001, 6)])
def test_ray_order_does_not_show(nb, small_city, w, h, spp, mode):
    """The camera rays of a large batch are queued in pixel blocks, those of a small one in rows: the first of
    two views is the same bit for bit alone (below 132,608 paths, rows) and with the second (blocks)."""
    scene, sb = small_city
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        flags = nb.VIEW_RESTIR if mode != "plain" else 0
        if mode != "plain":
            kw = dict(candidates=8, temporal=True)
            if mode == "restir":
                kw.update(spatial=3, radius_px=20.0, m_cap=20.0)
            ctx.set_restir(reference_mode=mode == "reference", **kw)
        a = nb.view_pinhole((0, 60, -180), (0, 0, 0), width=w, height=h, spp=spp, max_depth=2, seed=5, flags=flags)
        b = nb.view_pinhole((40, 60, -150), (0, 0, 0), width=333, height=401, spp=1, max_depth=2, seed=6, flags=flags)
        assert w * h * spp < 132_608 < w * h * spp + 333 * 401
        alone = ctx.render(a)[0]
        ctx.upload(sb)  # no history
        both = ctx.render(np.concatenate([a, b]))[0]
        assert np.array_equal(alone.view(np.int32), both.view(np.int32))
        assert ctx.status() == 0
    finally:
        ctx.close()
