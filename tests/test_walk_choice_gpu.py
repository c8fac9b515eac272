"""GPU test of the choice between cooperative leaf tests and the lane-by-lane walk: scenes and batches on both
sides of its lines (one-record leaves, few primitives, one ray for each of 28 warps per SM = 4,144 rays) trace the
oracle's hits bit for bit with every persistent configuration, from the host and from a frame's device queues, and
an untuned context is not slower on one-record leaves than the per-thread walk."""
import time

import numpy as np
import pytest

from tests import raysets

pytestmark = pytest.mark.gpu


def _scene(nb, kind, prims, objects, seed=1):
    rng = np.random.default_rng(seed)
    geom = np.zeros((prims, 15), np.float32)
    c = rng.uniform(-20, 20, (prims, 3))
    c = c[np.argsort(c[:, 0])]
    size = 20.0 / prims ** (1 / 3)
    if kind == 0:
        geom[:, 0:3], geom[:, 3] = c, rng.uniform(0.2, 1.0, prims) * size
    elif kind == 1:
        for k in range(3):
            geom[:, 3 * k:3 * k + 3] = c + rng.normal(size=(prims, 3)) * size
    else:
        u = rng.normal(size=(prims, 3))
        w = np.cross(u, rng.normal(size=(prims, 3)))
        geom[:, 0:3] = c
        geom[:, 3:6] = u / np.linalg.norm(u, axis=1, keepdims=True) * size
        geom[:, 6:9] = w / np.linalg.norm(w, axis=1, keepdims=True) * size
    cuts = np.linspace(0, prims, objects + 1).astype(np.int64)
    return nb.SceneBVH(nb.HostScene(np.full(prims, kind, np.int32), geom, np.full((prims, 20), 0.5, np.float32),
                                    cuts[:-1], np.diff(cuts)))


def _bits(h):
    return np.ascontiguousarray(h).view(np.int32).reshape(-1, 5)


@pytest.mark.parametrize("kind,prims,objects", [(1, 1, 1), (1, 7, 2), (1, 15, 1), (1, 16, 1), (1, 300, 300), (1, 300, 150),
                                                (0, 300, 4), (2, 300, 4), (0, 40, 40)])
def test_every_side_of_the_lines(nb, orc, kind, prims, objects):
    sb = _scene(nb, kind, prims, objects)
    ref = orc.OracleScene(sb)
    rays = np.concatenate([raysets.aimed_rays(sb, 3000, 1), raysets.random_rays(sb, 1000, 2)] +
                          ([raysets.edge_case_rays(sb, 3)] if kind == 1 else []) + [raysets.aimed_rays(sb, 4200, 4)])
    want, occ = ref.closest(rays), ref.any(rays)
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        for cfg in [None] + [(w, mb) for w in (2, 4, 8) for mb in (0, 10, 12, 16)]:
            if cfg:
                ctx.set_traversal(width=cfg[0], persistent=1, min_blocks=cfg[1])
            for n in (1, 4144, 4145, rays.shape[0]):
                ctx.reset_object_hits()
                assert np.array_equal(_bits(ctx.trace_closest(rays[:n], count_hits=True)), _bits(want[:n])), (cfg, n)
                hit = want["inst"][:n][want["prim"][:n] >= 0]
                assert np.array_equal(ctx.object_hits(), np.bincount(hit, minlength=objects)), (cfg, n)
                assert np.array_equal(ctx.trace_any(rays[:n]), occ[:n]), (cfg, n)
        assert ctx.status() == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("kind,prims,objects", [(1, 300, 300), (1, 12, 1), (0, 300, 4)])
@pytest.mark.parametrize("w,h,spp", [(61, 67, 1), (383, 401, 1)])
def test_frames(nb, kind, prims, objects, w, h, spp):
    sb = _scene(nb, kind, prims, objects)
    v = nb.view_pinhole((0, 10, -60), (0, 0, 0), width=w, height=h, spp=spp, max_depth=4, seed=3)
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        out = []
        for kernel in (1, 0, 2, 4, 6):
            ctx.set_kernel(kernel)
            out.append([ctx.render(v, graph=g)[0].view(np.int32) for g in (True, True, False)])
        for o in out[1:]:
            assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))
        assert ctx.status() == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("width", [2, 4, 8])
def test_paged_one_record_leaves(nb, width):
    """An untuned context whose only layout is a paged one, batches and frames on both sides of the lines."""
    sb = _scene(nb, 1, 300, 300)
    rays = np.concatenate([raysets.aimed_rays(sb, 4144, 1), raysets.random_rays(sb, 2000, 2)])
    v = nb.view_pinhole((0, 10, -60), (0, 0, 0), width=383, height=401, spp=1, max_depth=3, seed=3)
    out = []
    for paged in (False, True):
        ctx = nb.Context(0)
        try:
            ctx.upload(sb)
            if paged:
                ctx.paging_enable(1 << 40, width=width, max_onloads=sb.object_count)
                for _ in range(4):
                    ctx.paging_update()
                    ctx.paging_wait()
                assert ctx.paging_stats()["resident"] == sb.object_count
            out.append([_bits(ctx.trace_closest(rays[:n])) for n in (1, 4144, 4145, 6144)] +
                       [ctx.trace_any(rays), ctx.render(v)[0].view(np.int32), ctx.render(v[:1])[0].view(np.int32)])
            assert ctx.status() == 0
        finally:
            ctx.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def _times(nb, sb, kernels, paged=0):
    """Milliseconds of a million coherent closest hits with each kernel, the best of twelve."""
    import torch

    n = 1 << 20
    i = torch.arange(n, device="cuda")
    d = torch.stack([(i % 1024) / 1024.0 - 0.5, (i // 1024) / 1024.0 - 0.6, torch.full((n,), 1.0, device="cuda")], 1)
    rays = torch.zeros((n, 8), device="cuda")
    rays[:, 1], rays[:, 2] = 8.0, -70.0
    rays[:, 3], rays[:, 4:7], rays[:, 7] = 1e-4, d / d.norm(dim=1, keepdim=True), float("inf")
    hits = torch.empty((n, 5), dtype=torch.int32, device="cuda")
    ctx = nb.Context(0)
    try:
        ctx.upload(sb)
        if paged:
            ctx.paging_enable(1 << 40, width=paged, max_onloads=sb.object_count)
            for _ in range(4):
                ctx.paging_update()
                ctx.paging_wait()
        best = []
        for kernel in kernels:
            ctx.set_kernel(kernel)
            times = []
            for _ in range(12):
                ctx.sync()
                t0 = time.perf_counter()
                for _ in range(5):
                    ctx.trace_closest_dev(rays.data_ptr(), n, hits.data_ptr())
                ctx.sync()
                times.append((time.perf_counter() - t0) * 200.0)
            best.append(min(times))
    finally:
        ctx.close()
    return best


def test_untuned_on_one_record_leaves(nb):
    """A million rays into 8,192 objects of one triangle: the untuned context takes at most 1.1 times as long as
    the per-thread binary walk (1.2 to 1.45 with cooperative leaf tests)."""
    auto, walk = _times(nb, _scene(nb, 1, 8192, 8192), (0, 1))
    assert auto <= 1.1 * walk, (auto, walk)


def test_paged_untuned_on_one_record_leaves(nb):
    """The same with a paged 4-wide layout, against its per-thread walk."""
    auto, walk = _times(nb, _scene(nb, 1, 8192, 8192), (0, 3), paged=4)
    assert auto <= 1.1 * walk, (auto, walk)


def test_spheres(nb):
    """A million rays into 500 spheres: the 4-wide cooperative walk takes at most 1.35 times as long as the
    per-thread binary walk (1.19 when a record runs its own test alone, 1.56 with the triangle test before it)."""
    coop, walk = _times(nb, _scene(nb, 0, 500, 1), (4, 1))
    assert coop <= 1.35 * walk, (coop, walk)
