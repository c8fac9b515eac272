"""GPU test of persistent walks fed from a cursor over queues whose length is on the device: the kernels around a
trace clear its cursor, so a frame of more paths than are dealt out in shares (132,608), of several bounces and
estimators, replayed and launched directly, equals the per-thread walk's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(nb, sb, kernel, mode):
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        ctx.set_kernel(kernel)
        flags = 0
        if mode != "plain":
            flags = nb.VIEW_RESTIR
            kw = {} if mode == "reference" else dict(spatial=3, radius_px=20.0, m_cap=20.0)
            ctx.set_restir(candidates=8, temporal=True, reference_mode=mode == "reference", **kw)
        out = []
        for f, graph in enumerate((True, True, False)):
            v = nb.view_pinhole((f, 60, -180), (0, 0, 0), width=487, height=311, spp=1, max_depth=4, seed=9, frame=f,
                                flags=flags)
            out.append(ctx.render(v, graph=graph)[0].view(np.int32))
        assert ctx.status() == 0
        return out
    finally:
        ctx.close()


@pytest.fixture(scope="module")
def triangles(nb):
    """4,096 objects of one triangle, whose leaves the lane-by-lane walk tests."""
    rng = np.random.default_rng(2)
    n = 4096
    geom = np.zeros((n, 15), np.float32)
    c = rng.uniform([-90, 0, -90], [90, 60, 90], (n, 3))
    for k in range(3):
        geom[:, 3 * k:3 * k + 3] = c + rng.normal(size=(n, 3)) * 4
    mat = np.tile(nb.synth_city(seed=5, grid=2, size_m=50.0, target_tris=500, median_tris=50, max_tris=200).prim_material[0],
                  (n, 1)).astype(np.float32)
    mat[::64, 8:12] = 1.0
    return nb.SceneBVH(nb.HostScene(np.ones(n, np.int32), geom, mat, np.arange(n), np.ones(n, np.uint32)))


@pytest.mark.parametrize("mode", ["plain", "restir", "reference"])
@pytest.mark.parametrize("scene", ["city", "one-record leaves"])
def test_frames_fed_from_the_cursor(nb, small_city, triangles, scene, mode):
    sb = small_city[1] if scene == "city" else triangles
    want = _frames(nb, sb, 1, mode)
    for kernel in (2, 4, 6):
        for f, (a, b) in enumerate(zip(_frames(nb, sb, kernel, mode), want)):
            assert np.array_equal(a, b), (kernel, f)
