"""Device compaction of more nodes (4.19M) and primitives (67.1M) than the tiles that add up the sums before them
themselves, where one block scans the sums first."""
import ctypes as C
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _complete_trees(nb, objects, levels):
    """`objects` complete trees of 2**levels one-primitive leaves in pre-order, with random boxes and records."""
    leaves = 1 << levels
    per = 2 * leaves - 1
    first, count = np.zeros(per, np.int64), np.zeros(per, np.int64)
    stack, node = [(0, leaves)], 0
    while stack:  # pre-order: left child next, right child behind the left subtree
        lo, n = stack.pop()
        if n == 1:
            first[node], count[node] = lo, 1
        else:
            first[node], count[node] = node + 1, -(node + n)
            stack += [(lo + n // 2, n // 2), (lo, n // 2)]
        node += 1
    n, nodes = objects * leaves, objects * per
    rng = np.random.default_rng(1)
    bvh = rng.random((nodes, 8), dtype=np.float32)
    o = np.repeat(np.arange(objects), per)
    leaf = np.tile(count > 0, objects)
    base = np.where(leaf, o * leaves, o * per)
    bvh[:, 3] = (np.tile(first, objects) + base).astype(np.int32).view(np.float32)
    bvh[:, 7] = np.where(leaf, 1, np.tile(count, objects) - base).astype(np.int32).view(np.float32)
    inst = np.zeros(objects, nb.native.INSTANCE_DTYPE)
    inst["primitive_base"] = inst["primitive_index_base"] = np.arange(objects) * leaves
    inst["primitive_count"] = leaves
    inst["blas_root_index"] = np.arange(objects) * per
    return types.SimpleNamespace(
        prim_count=n, bvh_node_count=nodes, object_count=objects, bvh_nodes=bvh.reshape(-1),
        prims=rng.random(n * 28, dtype=np.float32), materials=rng.random(n * 20, dtype=np.float32),
        prim_indices=np.arange(n, dtype=np.int32), instances=inst, prim_object=np.repeat(np.arange(objects), leaves))


@pytest.mark.parametrize("objects", [2048, 2051])  # 4,192,256 nodes (sums of 4,194,304: none to scan) and 4,198,397
def test_many_nodes(nb, orc, objects):
    sb = _complete_trees(nb, objects, 10)
    comp = nb.native.Compactor(sb)
    rng = np.random.default_rng(2)
    active = (rng.random(objects) < 0.5)[sb.prim_object].astype(np.uint8)
    active &= (rng.random(sb.prim_count) < 0.6).astype(np.uint8)
    comp.run(active)
    got, want = comp.result(), orc.compact(sb, active)
    assert got["prim_count"] == want["prim_count"] and got["bvh_node_count"] == want["bvh_node_count"]
    for k in ("bvh_nodes", "prims", "materials", "prim_indices", "remap", "prim_to_resident", "instances"):
        assert got[k].tobytes() == np.ascontiguousarray(want[k]).tobytes(), k


def test_many_primitives(nb):
    """67.2M primitives in one leaf, 1 in 1,000 of them active. Arrays that a compaction reads and writes at active
    primitives only are allocated whole and left as they are."""
    import torch

    lib, native = nb.load(), nb.native
    n = (16384 + 20) * 4096 + 7
    g = torch.Generator(device="cuda").manual_seed(3)
    active = (torch.rand(n, device="cuda", generator=g) < 1e-3).to(torch.uint8)
    idx = torch.arange(n, dtype=torch.int32, device="cuda").flip(0).contiguous()
    prims = torch.empty(n * 28, dtype=torch.float32, device="cuda")
    mats = torch.empty(n * 20, dtype=torch.float32, device="cuda")
    on = active.nonzero()[:, 0]
    prims.view(n, 28)[on] = torch.rand((on.numel(), 28), device="cuda", generator=g)
    mats.view(n, 20)[on] = torch.rand((on.numel(), 20), device="cuda", generator=g)
    inst = torch.tensor([0, 0, n, 0], dtype=torch.int32, device="cuda")
    nodes = torch.tensor([0, 0, 0, 0, 0, 0, 0, n], dtype=torch.int32, device="cuda")
    out = dict(bvh=torch.full((8,), 9, dtype=torch.int32, device="cuda"), prims=torch.zeros((on.numel(), 28), device="cuda"),
               mats=torch.zeros((on.numel(), 20), device="cuda"), idx=torch.zeros(n, dtype=torch.int32, device="cuda"),
               remap=torch.zeros(n, dtype=torch.int32, device="cuda"), p2r=torch.full((n,), -7, dtype=torch.int32, device="cuda"),
               inst=torch.zeros(4, dtype=torch.int32, device="cuda"), counts=torch.zeros(3, dtype=torch.int32, device="cuda"))
    size = int(lib.nomad_compact_workspace_bytes(n, 1, 1))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    inp = native.ScenebvhDevice(n, 1, 1, 0, nodes.data_ptr(), prims.data_ptr(), mats.data_ptr(), idx.data_ptr(),
                                inst.data_ptr())
    cout = native.CompactOut(*[out[k].data_ptr() for k in ("bvh", "prims", "mats", "idx", "remap", "p2r", "inst", "counts")])
    torch.cuda.synchronize()
    assert lib.nomad_scenebvh_compact_gpu(C.byref(inp), active.data_ptr(), ws.data_ptr(), size, C.byref(cout), None) == 0
    torch.cuda.synchronize()
    assert out["counts"].tolist() == [on.numel(), 1, 0]
    assert out["bvh"].tolist() == [0, 0, 0, 0, 0, 0, 0, on.numel()] and out["inst"].tolist() == [0, 0, on.numel(), 0]
    want = on.flip(0)  # leaf order is the reverse of the global one
    m = on.numel()
    assert torch.equal(out["remap"][:m].long(), want)
    assert torch.equal(out["idx"][:m].long(), torch.arange(m, device="cuda"))
    assert torch.equal(out["prims"], prims.view(n, 28)[want]) and torch.equal(out["mats"], mats.view(n, 20)[want])
    assert torch.equal(out["p2r"][want].long(), torch.arange(m, device="cuda"))
    assert int((out["p2r"] == -1).sum()) == n - m
