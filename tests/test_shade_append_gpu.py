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
