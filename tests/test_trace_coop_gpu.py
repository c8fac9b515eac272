"""The persistent kernels' cooperative leaf tests at the sizes where they can go wrong: leaves below,
at and above the eight records of one pass, batches around a warp, and rays with non-finite or zero
components. Closest and any hits equal the oracle's and the per-thread kernel's bit for bit."""
import types

import numpy as np
import pytest

from tests import raysets

pytestmark = pytest.mark.gpu


def _bits(h):
    return np.ascontiguousarray(h).view(np.int32).reshape(-1, 5)


def _one_leaf_objects(nb, per_object, seed):
    """Two objects of `per_object` random triangles, each object one leaf."""
    rng = np.random.default_rng(seed)
    n = 2 * per_object
    geom = np.zeros((n, 15), np.float32)
    c = rng.uniform(-1, 1, (n, 3))
    c[per_object:, 0] += 1.0
    for k in range(3):
        geom[:, 3 * k:3 * k + 3] = c + rng.normal(size=(n, 3)) * 0.4
    scene = nb.HostScene(np.ones(n, np.int32), geom, np.full((n, 20), 0.5, np.float32), [0, per_object],
                         [per_object, per_object])
    sb = nb.SceneBVH(scene)
    v = sb.prims.reshape(-1, 28)[:, [0, 1, 2, 4, 5, 6, 8, 9, 10]].reshape(2, per_object * 3, 3)
    nodes = np.zeros((2, 8), np.float32)
    nodes[:, 0:3], nodes[:, 4:7] = v.min(1), v.max(1)
    nodes[:, 3] = np.array([0, per_object], np.int32).view(np.float32)
    nodes[:, 7] = np.array([per_object, per_object], np.int32).view(np.float32)
    inst = sb.instances.copy()
    inst["blas_root_index"] = [0, 1]
    return types.SimpleNamespace(
        bvh_nodes=nodes.reshape(-1), bvh_node_count=2, tlas_nodes=sb.tlas_nodes, tlas_node_count=sb.tlas_node_count,
        prims=sb.prims, materials=sb.materials, prim_indices=np.arange(n, dtype=np.int32), prim_count=n, instances=inst,
        object_count=2, object_bounds=sb.object_bounds, prim_object=sb.prim_object)


@pytest.fixture(scope="module")
def ctx(nb):
    c = nb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kernel", [2, 4, 6])
@pytest.mark.parametrize("records", [1, 7, 8, 9, 16, 17, 40])
def test_leaf_sizes(nb, orc, ctx, records, kernel):
    sb = _one_leaf_objects(nb, records, records)
    ctx.upload(sb)
    ctx.set_kernel(kernel)
    ctx.set_primitive_active(records // 2, False)
    ctx.flush()
    active = np.ones(sb.prim_count, np.uint8)
    active[records // 2] = 0
    root = sb.instances["blas_root_index"].copy()
    if records == 1:
        root[0] = -1
    ref = orc.OracleScene(sb, active=active, blas_root=root)
    rays = np.concatenate([raysets.aimed_rays(sb, 4000, 1), raysets.random_rays(sb, 1000, 2),
                           raysets.edge_case_rays(sb, 3)])
    assert np.array_equal(_bits(ctx.trace_closest(rays)), _bits(ref.closest(rays)))
    assert np.array_equal(ctx.trace_any(rays), ref.any(rays))
    assert ctx.status() == 0


@pytest.mark.parametrize("kernel", [2, 4, 6])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 4097])
def test_batch_sizes(nb, orc, ctx, small_city, n, kernel):
    sb = small_city[1]
    ctx.upload(sb)
    ctx.set_kernel(kernel)
    rays = raysets.aimed_rays(sb, n, 5)
    ref = orc.OracleScene(sb)
    ctx.reset_object_hits()
    got = ctx.trace_closest(rays, count_hits=True)
    want = ref.closest(rays)
    assert np.array_equal(_bits(got), _bits(want))
    assert np.array_equal(ctx.object_hits(), np.bincount(want["inst"][want["prim"] >= 0], minlength=sb.object_count))
    assert np.array_equal(ctx.trace_any(rays), ref.any(rays))


@pytest.mark.parametrize("kernel", [2, 4, 6])
def test_odd_rays(nb, ctx, small_city, kernel):
    """Zero, infinite and NaN components, and bounds that are negative, NaN or the largest float."""
    sb = small_city[1]
    ctx.upload(sb)
    rays = raysets.aimed_rays(sb, 2048, 7)
    rng = np.random.default_rng(8)
    odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-30, 3e38], np.float32)
    for name in ("ox", "oy", "oz", "dx", "dy", "dz"):
        at = rng.random(rays.shape[0]) < 0.04
        rays[name][at] = odd[rng.integers(0, odd.size, at.sum())]
    at = rng.random(rays.shape[0]) < 0.2
    rays["tmax"][at] = np.array([-1.0, 0.0, np.nan, 3.4e38, 1e-4, 50.0], np.float32)[rng.integers(0, 6, at.sum())]
    ctx.set_kernel(1)
    want, occ = ctx.trace_closest(rays), ctx.trace_any(rays)
    ctx.set_kernel(kernel)
    assert np.array_equal(_bits(ctx.trace_closest(rays)), _bits(want))
    assert np.array_equal(ctx.trace_any(rays), occ)


@pytest.mark.parametrize("n", [1, 1000, 150_001, 700_003])
def test_unchosen_kernel(nb, small_city, n):
    """A context that never chose a kernel returns the per-thread binary walk's hits, also when two
    of its calls overlap on two streams, and still reports that walk's configuration."""
    import torch

    sb = small_city[1]
    base = raysets.aimed_rays(sb, min(n, 50_000), 5)
    rays = torch.from_numpy(np.tile(base, -(-n // base.shape[0]))[:n].view(np.float32).reshape(-1, 8)).cuda()
    c = nb.Context(0)
    try:
        c.upload(sb)
        assert c.traversal()["width"] == 2 and c.traversal()["persistent"] == 0
        streams = [torch.cuda.Stream() for _ in range(2)]
        outs = [torch.zeros((n, 5), dtype=torch.int32, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        for s, o in zip(streams, outs):
            c.set_stream(s.cuda_stream)
            c.trace_closest_dev(rays.data_ptr(), n, o.data_ptr())
        torch.cuda.synchronize()
        c.set_stream(0)
        c.set_kernel(1)
        c.trace_closest_dev(rays.data_ptr(), n, outs[2].data_ptr())
        c.sync()
        assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[2])
    finally:
        c.close()
