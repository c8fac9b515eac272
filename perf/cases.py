"""Measured workloads of the framework, each reached through its public entry points.

``listed()`` names the fixed cases and ``draw(rng)`` gives more of the same ranges; ``prepare``
builds what a program holds before the call (scene, context, rays, views, model), ``run`` makes one
pass and returns its whole outputs, ``work`` states the bytes a pass cannot do without and ``exact``
gives the float64 values of outputs that have a closed form.

Scenes come from the framework's own seeded generators at the sizes of its bench, residency
workload and tests (icospheres; cities of 120k, 600k and 2.5M triangles). A scene stands for an
asset file, so one process builds each once and every context uploads it anew; rays, cameras,
random streams, masks, models and samples come from the seed.
"""
import functools
import math

import numpy as np
import torch

import nomad_b200 as nb
from nomad_b200.native import Compactor

# The traversal that a tuned program selects for cities (the bench's sweep and the residency
# workload use it); cases with "tuned": False keep the context's default, as a program does that
# never tunes.
TUNED = dict(width=4, persistent=1, short_stack=0, regroup=1, staged_nodes=0, block=128, postpone_leaves=0,
             min_blocks=10)


def listed():
    return [
        # A picking or probe query of a viewer: a thousand rays into a small scene, untuned. The
        # call's latency is the cost.
        {"name": "probe rays", "kind": "closest", "scene": "ico", "tris": 64, "width": 37, "height": 27, "spp": 1,
         "bounce": False, "count": False, "tuned": False},
        # The headline step: the closest hits of a 1080p x 4 frame of the 2.5M-triangle city, the
        # coherent primary rays and then one incoherent diffuse bounce of each hit, with the
        # per-object hit counts that the residency policies read.
        {"name": "closest city 1080p", "kind": "closest", "scene": "city", "tris": 2_500_000, "width": 1920,
         "height": 1080, "spp": 4, "bounce": True, "count": True, "tuned": True},
        # A caller whose rays and hits live in pinned host memory (the C ABI's plain form).
        {"name": "closest host buffers", "kind": "host", "scene": "city", "tris": 600_000, "width": 1280,
         "height": 720, "spp": 1, "tuned": True},
        # Shadow queries: any-hit from the visible points to points on the emissive quads.
        {"name": "any-hit shadows", "kind": "any", "scene": "city", "tris": 600_000, "width": 1279, "height": 717,
         "spp": 2, "tuned": True},
        # The production frame: path traced 1080p x 4 spp, three bounces, next-event estimation.
        {"name": "frame 1080p", "kind": "frame", "scene": "city", "tris": 2_500_000, "width": 1920, "height": 1080,
         "spp": 4, "depth": 3, "views": 1, "tuned": True},
        # An interactive preview at an odd size, one sample, read back to the host, untuned.
        {"name": "frame preview", "kind": "frame", "scene": "city", "tris": 120_000, "width": 321, "height": 181,
         "spp": 1, "depth": 2, "views": 1, "tuned": False},
        # Many uneven views of one scene in one batch (data-set rendering).
        {"name": "frame views", "kind": "frame", "scene": "city", "tris": 600_000, "width": 641, "height": 479,
         "spp": 3, "depth": 2, "views": 7, "tuned": True},
        # Direct light of 4,096 emissive triangles by ReSTIR, one 1080p frame of a moving camera.
        {"name": "restir 1080p", "kind": "restir", "scene": "lights", "tris": 600_000, "width": 1920, "height": 1080,
         "candidates": 32, "reference": False, "tuned": True},
        # The same light transport with the reference renderer's own estimator, whose candidates
        # each cast a visibility ray.
        {"name": "restir reference mode", "kind": "restir", "scene": "lights", "tris": 600_000, "width": 961,
         "height": 541, "candidates": 32, "reference": True, "tuned": True},
        # The residency loop: render a frame with hit counting, take a learned residency step under
        # a 40 % byte budget, read the resident set.
        {"name": "residency loop", "kind": "residency", "scene": "objects", "tris": 600_000, "width": 640,
         "height": 360, "spp": 2, "depth": 2, "policy": "learned", "budget": 0.4, "tuned": True},
        # Residency compaction of the whole city under a 40 % object mask.
        {"name": "compaction", "kind": "compact", "scene": "city", "tris": 2_500_000, "keep": 0.4},
        # Training the residency scorer on recorded samples.
        {"name": "scorer training", "kind": "train", "samples": 262_144, "steps": 300, "batch": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "closest", "host", "any", "frame", "frame", "restir", "residency", "compact",
                       "train"])
    if kind == "train":
        return {"kind": kind, "samples": _log(rng, 20_000, 262_144), "steps": _log(rng, 50, 300),
                "batch": 64 * _log(rng, 4, 64)}
    tris = rng.choice([120_000, 600_000])
    if kind == "compact":
        return {"kind": kind, "scene": "city", "tris": tris, "keep": round(rng.uniform(0.05, 0.95), 3)}
    px = _log(rng, 2_000, 2_000_000)
    w = max(8, int(math.sqrt(px * rng.uniform(1.0, 2.0))))
    h = max(8, px // w)
    c = {"kind": kind, "scene": "city", "tris": tris, "width": w, "height": h, "tuned": rng.random() < 0.75}
    if kind == "closest" and rng.random() < 0.2:
        c.update(scene="ico", tris=64)
    if kind in ("closest", "host", "any"):
        c["spp"] = rng.choice([1, 1, 2, 4]) if px < 1_000_000 else 1
    if kind == "closest":
        c.update(bounce=rng.random() < 0.5, count=rng.random() < 0.5)
    if kind == "frame":
        c.update(spp=rng.choice([1, 2, 3, 4]), depth=rng.choice([1, 2, 3, 6]), views=1 if px > 300_000 else
                 rng.choice([1, 1, 2, 5]))
    if kind == "restir":
        ref = rng.random() < 0.4
        if ref:
            c.update(width=max(8, w // 2), height=max(8, h // 2))
        c.update(scene="lights", tris=600_000, candidates=rng.choice([4, 16, 31, 32]), reference=ref)
    if kind == "residency":
        c.update(scene="objects", width=max(8, w // 2), height=max(8, h // 2), spp=rng.choice([1, 2]),
                 depth=rng.choice([1, 2, 3]), policy=rng.choice(["learned", "rayhit"]),
                 budget=round(rng.uniform(0.15, 0.9), 3))
    return c


# ---------------------------------------------------------------------------------------------
# Scenes and rays


@functools.lru_cache(maxsize=None)
def _scene(scene, tris):
    if scene == "ico":
        return nb.SceneBVH(nb.synth_icospheres(seed=1, instances=tris))
    if scene == "lights":
        return nb.SceneBVH(nb.synth_city(seed=2, target_tris=tris, emissive_tris=4096, emissive_sigma=1.5))
    if scene == "objects":  # 2,048 objects, the residency workload's layout
        return nb.SceneBVH(nb.synth_city(seed=17, grid=64, grid_z=32, size_m=2000.0, target_tris=tris))
    return nb.SceneBVH(nb.synth_city(seed=2, target_tris=tris))


def _context(case):
    sb = _scene(case["scene"], case["tris"])
    ctx = nb.Context(0)
    ctx.upload(sb)
    if case["tuned"]:
        ctx.set_traversal(**TUNED)
    return ctx, sb


def _camera(case, rng):
    """Position and target of the bench's cameras, moved a little by the seed."""
    j = rng.uniform(-1.0, 1.0, 3)
    if case["scene"] == "ico":
        return (2.0 * j[0], 40.0 + 2.0 * j[1], 170.0 + 2.0 * j[2]), (0.0, 0.0, 0.0)
    if case["scene"] == "objects":
        return (100.0 * j[0], 60.0 + 5.0 * j[1], 50.0 * j[2]), (100.0 * j[0], 35.0, 60.0 + 50.0 * j[2])
    return (15.0 * j[0], 220.0 + 4.0 * j[1], -620.0 + 10.0 * j[2]), (0.0, 0.0, 60.0)


def _unit(v):
    return v / v.square().sum(1, keepdim=True).sqrt()


def _pack(o, d, tmax):
    n = d.shape[0]
    rays = torch.empty((n, 8), dtype=torch.float32, device=d.device)
    rays[:, 0:3] = o
    rays[:, 3] = 1e-4
    rays[:, 4:7] = d
    rays[:, 7] = tmax
    return rays


def _primary(case, seed):
    """Jittered pinhole rays, pixel-major and then sample, on the GPU."""
    rng = np.random.default_rng(seed)
    pos, look = _camera(case, rng)
    w, h, spp = case["width"], case["height"], case["spp"]
    cam = nb.Camera(pos, look, width=w, height=h)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    i = torch.arange(w * h * spp, device="cuda") // spp
    n = i.numel()
    ux = (((i % w).float() + torch.rand(n, device="cuda", generator=g)) / w)[:, None]
    uy = (((i // w).float() + torch.rand(n, device="cuda", generator=g)) / h)[:, None]
    def dev(a):
        return torch.from_numpy(np.asarray(a, np.float32)).cuda()[None, :]
    d = dev(cam.first_pixel) + ux * dev(cam.viewport_u) + uy * dev(cam.viewport_v) - dev(cam.position)
    return _pack(dev(cam.position), _unit(d), math.inf)


def _surface(rays, hits, sb):
    """Hit points and the normals facing the incoming rays, of 6 in 10 rays: the hits in their order,
    thinned or repeated evenly to that count."""
    keep = (hits[:, 1] >= 0).nonzero()[:, 0]
    n = max(1, int(0.6 * rays.shape[0]))
    keep = keep[torch.arange(n, device="cuda") * keep.numel() // n]
    r, h = rays[keep], hits[keep]
    t = h[:, 2].contiguous().view(torch.float32)[:, None]
    p = r[:, 0:3] + t * r[:, 4:7]
    nrm = torch.from_numpy(np.ascontiguousarray(sb.prims.reshape(-1, 28)[:, 24:27])).cuda()[h[:, 1].long()]
    nrm = _unit(nrm)
    return p, torch.where((nrm * r[:, 4:7]).sum(1, keepdim=True) > 0, -nrm, nrm)


def _bounce(rays, hits, sb, seed):
    """One cosine-weighted ray from each surface point."""
    p, n = _surface(rays, hits, sb)
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    u = torch.rand((2, p.shape[0]), device="cuda", generator=g)
    up = torch.where(n[:, 2:3].abs() < 0.999, torch.tensor([[0.0, 0.0, 1.0]], device="cuda"),
                     torch.tensor([[0.0, 1.0, 0.0]], device="cuda"))
    t = _unit(torch.linalg.cross(up, n))
    b = _unit(torch.linalg.cross(n, t))
    rr, th = u[0].sqrt()[:, None], (2 * math.pi * u[1])[:, None]
    d = t * (rr * th.cos()) + b * (rr * th.sin()) + n * (1 - u[0]).clamp_min(0).sqrt()[:, None]
    return _pack(p + 1e-4 * n, _unit(d), math.inf)


def _shadow(rays, hits, sb, seed):
    """One ray from each surface point to a point of a uniformly drawn emissive quad, ending before it."""
    p, n = _surface(rays, hits, sb)
    m = sb.materials.reshape(-1, 20)
    light = sb.prims.reshape(-1, 28)[(m[:, 11] > 0) & (m[:, 8:11].sum(1) > 0)]
    light = torch.from_numpy(np.ascontiguousarray(light)).cuda()
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 2)
    k = torch.randint(0, light.shape[0], (p.shape[0],), device="cuda", generator=g)
    u = torch.rand((2, p.shape[0], 1), device="cuda", generator=g) * 2 - 1
    q = light[k]
    o = p + 5e-4 * n
    to = q[:, 0:3] + u[0] * q[:, 4:7] + u[1] * q[:, 8:11] - o
    dist = to.square().sum(1).sqrt().clamp_min(2e-3)
    return _pack(o, to / dist[:, None], dist - 1e-3)


def _hits(n):
    return torch.zeros((n, 5), dtype=torch.int32, device="cuda")


def _trace(ctx, rays):
    hits = _hits(rays.shape[0])
    torch.cuda.synchronize()  # the context runs on a stream of its own
    ctx.trace_closest_dev(rays.data_ptr(), rays.shape[0], hits.data_ptr())
    ctx.sync()
    return hits


def _views(case, seed):
    """The frame's views: the bench camera, or uneven views around it."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case.get("views", 1)):
        pos, look = _camera(case, rng)
        w, h = case["width"], case["height"]
        if i:
            w, h = max(8, w * (11 - i) // 12), max(8, h * (5 + i) // 12)
        out.append(nb.view_pinhole(pos, look, width=w, height=h, spp=case.get("spp", 1), max_depth=case.get("depth", 1),
                                   seed=int(seed) * 64 + i))
    return np.concatenate(out)


# ---------------------------------------------------------------------------------------------
# What a program holds, one pass, and what a pass has to move


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, t = _samples(case, seed)
        ctx = nb.Context(0)
        ctx.mlp_init(int(seed) & 0x7FFFFFFF)
        return {"case": case, "ctx": ctx, "x": x, "t": t, "blob": ctx.mlp_get(), "seed": int(seed)}
    if kind == "compact":
        sb = _scene(case["scene"], case["tris"])
        comp = Compactor(sb)
        for o in (comp.o_bvh, comp.o_prims, comp.o_mats, comp.o_idx, comp.o_remap, comp.o_p2r, comp.o_inst):
            o.zero_()  # the arrays past the compacted lengths are the caller's
        keep = np.random.default_rng(seed).random(sb.object_count) < case["keep"]
        return {"case": case, "comp": comp, "mask": torch.from_numpy(keep[sb.prim_object].astype(np.uint8)).cuda()}
    ctx, sb = _context(case)
    s = {"case": case, "ctx": ctx}
    if kind in ("closest", "any", "host"):
        rays = _primary(case, seed)
        if kind == "any":
            rays = _shadow(rays, _trace(ctx, rays), sb, seed)
            s["occ"] = torch.zeros(rays.shape[0], dtype=torch.uint8, device="cuda")
            s["rays"] = rays
        elif kind == "host":
            s["rays"] = rays.cpu().pin_memory()
            s["hits"] = torch.zeros((rays.shape[0], 5), dtype=torch.int32).pin_memory()
        else:
            s["batches"] = [(rays, _hits(rays.shape[0]))]
            if case["bounce"]:
                b = _bounce(rays, _trace(ctx, rays), sb, seed)
                s["batches"].append((b, _hits(b.shape[0])))
        torch.cuda.synchronize()
        return s
    s["views"] = _views(case, seed)
    s["pixels"] = [int(v["width"]) * int(v["height"]) for v in s["views"]]
    s["image"] = torch.zeros(sum(s["pixels"]) * 3, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    if kind == "restir":
        s["views"]["flags"] |= nb.VIEW_RESTIR
        ctx.set_restir(candidates=case["candidates"], temporal=True, spatial=3, radius_px=30.0, m_cap=20.0,
                       reference_mode=case["reference"])
        _render(s)  # the frame before: the reservoirs that this one reuses
        ctx.sync()
    if kind == "residency":
        if case["policy"] == "learned":
            ctx.mlp_init(int(seed) & 0x7FFFFFFF)
        ctx.residency_step(nb.ResidencyParams.make(nb.POLICY_ALWAYS), s["views"])
        ctx.reset_object_hits()
        policy = nb.POLICY_LEARNED if case["policy"] == "learned" else nb.POLICY_RAYHIT_BUDGET
        s["params"] = nb.ResidencyParams.make(policy, budget_bytes=int(case["budget"] * int(ctx.object_bytes().sum())),
                                              camera_motion=0.3)
    return s


def _render(s, count=False):
    s["views"]["frame"] += 1
    s["ctx"].render_dev(s["views"], s["image"].data_ptr(), count_hits=count)
    return s["image"]


def _split(hits):
    """Hits as their ids and their distances and barycentrics."""
    return {"ids": hits[:, 0:2], "tuv": hits[:, 2:5].view(torch.float32)}


def run(s):
    case = s["case"]
    kind, ctx = case["kind"], s.get("ctx")
    if kind == "closest":
        for rays, hits in s["batches"]:
            ctx.trace_closest_dev(rays.data_ptr(), rays.shape[0], hits.data_ptr(), count_hits=case["count"])
        return [_split(h) for _, h in s["batches"]]
    if kind == "host":
        st = ctx.lib.nomad_trace_closest(ctx.h, s["rays"].data_ptr(), s["rays"].shape[0], s["hits"].data_ptr(), 0)
        if st != 0:
            raise nb.NomadError(st)
        return _split(s["hits"])
    if kind == "any":
        ctx.trace_any_dev(s["rays"].data_ptr(), s["rays"].shape[0], s["occ"].data_ptr())
        return s["occ"]
    if kind == "frame":
        if not case["tuned"]:  # the preview reads its images back
            s["views"]["frame"] += 1
            return ctx.render(s["views"])
        return _render(s)
    if kind == "restir":
        return _render(s)
    if kind == "residency":
        image = _render(s, count=True)
        ctx.residency_step(s["params"], s["views"], toggles=False)
        return {"image": image, "resident": ctx.residency_flags()}
    if kind == "compact":
        c = s["comp"]
        c.run(s["mask"])
        i32 = torch.int32
        return {"nodes": c.o_bvh.view(i32), "prims": c.o_prims.view(i32), "materials": c.o_mats.view(i32),
                "indices": c.o_idx, "remap": c.o_remap, "to_resident": c.o_p2r, "instances": c.o_inst,
                "counts": c.o_counts}
    ctx.mlp_set(s["blob"])
    loss = ctx.mlp_train(s["x"], s["t"], steps=case["steps"], batch=case["batch"], lr=2e-3, seed=s["seed"] & 0xFFFF)
    return {"loss": loss, "weights": ctx.mlp_get()}


def _samples(case, seed):
    """Recorded scorer samples: non-negative features of varying scale, log hit counts."""
    rng = np.random.default_rng(seed)
    x = np.abs(rng.standard_normal((case["samples"], nb.N_FEATURES), np.float32))
    x *= rng.uniform(0.2, 4.0, nb.N_FEATURES).astype(np.float32)
    w = rng.standard_normal(nb.N_FEATURES).astype(np.float32)
    t = np.log1p(np.maximum(x @ w, 0.0)).astype(np.float32)
    return np.ascontiguousarray(x), t


def work(case):
    """Bytes each pass has to read and write once (rays, hits, geometry, images, samples), and the
    multiply-adds where the path is a contraction."""
    kind = case["kind"]
    if kind == "train":
        macs = case["steps"] * case["batch"] * (nb.N_FEATURES * 128 + 128 * 128 + 128) * 3
        return {"bytes": case["samples"] * (nb.N_FEATURES + 1) * 4 + 2 * nb.MLP_PARAMS * 4, "flops": 2 * macs}
    sb = _scene(case["scene"], case["tris"])
    n, nodes = sb.prim_count, sb.bvh_node_count
    if kind == "compact":
        moved = 2 * 192 * n * case["keep"] + 2 * 32 * nodes * case["keep"] + n * 9 + n * 4 + 8 * n * case["keep"]
        return {"bytes": moved, "flops": 0}
    geometry = 48 * n + 32 * nodes
    paths = case["width"] * case["height"] * case.get("spp", 1)
    if kind in ("closest", "host", "any"):
        rays = paths * (0.6 if kind == "any" else 1.6 if case.get("bounce") else 1.0)
        return {"bytes": rays * (32 + (1 if kind == "any" else 20)) + geometry, "flops": 0}
    pixels = case["width"] * case["height"] * case.get("views", 1)
    rays = paths * case.get("views", 1) * case.get("depth", 1) * 2  # a segment and a shadow ray per bounce
    if kind == "restir" and case["reference"]:
        rays += paths * case["candidates"]
    return {"bytes": pixels * 12 + rays * 52 + geometry, "flops": 0}


def exact(case, seed):
    """Closest hits in float64 against every triangle, where that is affordable."""
    if case["kind"] not in ("closest", "host") or case.get("bounce"):
        return None
    sb = _scene(case["scene"], case["tris"])
    n_rays = case["width"] * case["height"] * case["spp"]
    if n_rays * sb.prim_count > 4e9 or case["scene"] != "ico":
        return None
    rays = _primary(case, seed).double()
    g = torch.from_numpy(sb.prims.reshape(-1, 28)).cuda().double()
    assert bool((g[:, 3] == 1).all())
    v0, e1, e2 = g[:, 0:3], g[:, 4:7] - g[:, 0:3], g[:, 8:11] - g[:, 0:3]
    # distance, then the barycentrics, by the scalar triple products of Moller and Trumbore
    out = torch.zeros((n_rays, 3), dtype=torch.float64, device="cuda")
    step = max(1, int(2e8) // max(1, sb.prim_count))
    for a in range(0, n_rays, step):
        o, d = rays[a:a + step, None, 0:3], rays[a:a + step, None, 4:7]
        pv = torch.linalg.cross(d, e2[None].expand(d.shape[0], -1, -1))
        det = (pv * e1).sum(2)
        s = o - v0[None]
        u = (s * pv).sum(2) / det
        q = torch.linalg.cross(s, e1[None].expand(s.shape))
        v = (q * d).sum(2) / det
        t = (q * e2).sum(2) / det
        ok = (det.abs() > 1e-5) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-4)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        tb, k = t.min(1)
        hit = torch.isfinite(tb)
        at = torch.arange(k.numel(), device="cuda")
        out[a:a + step, 0] = tb
        out[a:a + step, 1] = torch.where(hit, u[at, k], torch.zeros_like(tb))
        out[a:a + step, 2] = torch.where(hit, v[at, k], torch.zeros_like(tb))
    tuv = {"ids": None, "tuv": out.cpu()}
    return tuv if case["kind"] == "host" else [tuv]
