"""Device compaction at the edges of its tiles: primitive and node counts around a warp, a block and
the 4,096-item scan tile, one object and many, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(nb, prims, objects):
    rng = np.random.default_rng(prims * 31 + objects)
    geom = np.zeros((prims, 15), np.float32)
    c = rng.uniform(-10, 10, (prims, 3))
    for k in range(3):
        geom[:, 3 * k:3 * k + 3] = c + rng.normal(size=(prims, 3)) * 0.3
    cuts = np.linspace(0, prims, objects + 1).astype(np.uint32)
    mat = rng.uniform(0, 1, (prims, 20)).astype(np.float32)
    mat[:, 16:19] = -1.0
    return nb.SceneBVH(nb.HostScene(np.ones(prims, np.int32), geom, mat, cuts[:-1], np.diff(cuts)))


@pytest.mark.parametrize("prims,objects", [(1, 1), (31, 1), (33, 3), (255, 2), (257, 40), (4095, 1), (4096, 7),
                                           (4097, 300), (12289, 5)])
def test_tile_edges(nb, orc, prims, objects):
    sb = _scene(nb, prims, objects)
    comp = nb.native.Compactor(sb)
    rng = np.random.default_rng(prims)
    for active in (np.ones(prims, np.uint8), np.zeros(prims, np.uint8), (rng.random(prims) < 0.5).astype(np.uint8),
                   (rng.random(prims) < 0.03).astype(np.uint8)):
        comp.run(active)
        got, want = comp.result(), orc.compact(sb, active)
        assert got["prim_count"] == want["prim_count"] and got["bvh_node_count"] == want["bvh_node_count"]
        for k in ("bvh_nodes", "prims", "materials", "prim_indices", "remap", "prim_to_resident", "instances"):
            assert got[k].tobytes() == np.ascontiguousarray(want[k]).tobytes(), k
