"""The workloads whose speed is watched: ray queries, tree builds, path-traced frames,
inverse-rendering steps and scene batches, through the package's public calls.

listed() names them, draw(rng) gives more of the same ranges; prepare(case, seed) makes a
case's inputs and what a program keeps between calls (contexts, trees, scenes, output
buffers), run(state) is one pass and returns its outputs, work(case) the bytes and
operations such a pass cannot do without, exact(case, seed) the outputs in 64 bits where a
brute-force answer is affordable.
"""
import ctypes
import math

import numpy as np
import torch

import visionaray_gb300 as vg
from visionaray_gb300 import inverse, scenes
from visionaray_gb300 import runtime as rt
from visionaray_gb300.types import (BATCH_ORDER_BLOCKS, CAMERA, GLASS, MATERIAL, MATTE, MIRROR, PLASTIC, PT_PARAMS,
                                    PT_NO_RUSSIAN_ROULETTE, PT_SHADOW_RANGE_FIX)

DEVICE = 0
FLT_MAX = float(np.finfo(np.float32).max)


def listed():
    return [
        # Picking and line-of-sight queries of an interactive program: a thousand rays into
        # a small mesh, where the call itself is what costs.
        {"name": "trace_pick", "kind": "trace", "scene": "soup", "size": 4099, "rays": "primary", "width": 33,
         "height": 31, "query": "closest", "sort": False},
        # Camera rays of a whole image into a soup of 65,536 triangles, in pixel order.
        {"name": "trace_primary", "kind": "trace", "scene": "soup", "size": 65536, "rays": "primary", "width": 1024,
         "height": 1024, "query": "closest", "sort": False},
        # Secondary rays from the surface of an 8.4 M triangle heightfield, in random
        # order, the library sorting them: the incoherent closest-hit workload.
        {"name": "trace_incoherent", "kind": "trace", "scene": "heightfield", "size": 2048, "rays": "surface",
         "width": 2048, "height": 2048, "query": "closest", "sort": True},
        # Ambient-occlusion rays (eight short ones per surface point) over 2.1 M triangles.
        {"name": "trace_ao", "kind": "trace", "scene": "heightfield", "size": 1024, "rays": "ao", "width": 1024,
         "height": 1024, "query": "any", "sort": True},
        # A tree over a few thousand triangles, built anew: one of many small objects.
        {"name": "build_small", "kind": "build", "scene": "soup", "size": 5003, "mode": "build"},
        # The tree of the 8.4 M triangle heightfield, built anew and handed out in the
        # reference's node layout.
        {"name": "build_large", "kind": "build", "scene": "heightfield", "size": 2048, "mode": "build"},
        # The high-quality builder on about a million triangles, then camera rays through
        # its tree.
        {"name": "build_quality", "kind": "quality", "scene": "heightfield", "size": 701, "width": 513, "height": 511},
        # One progressive frame of an interactive viewer: small image, one sample, few
        # bounces; launches and latency.
        {"name": "frame_preview", "kind": "frame", "scene": "box", "blobs": 10, "subdiv": 8, "width": 160,
         "height": 120, "spp": 1, "depth": 4, "builder": "lbvh"},
        # The box of 2.5 M triangles at full HD, eight samples per pixel, eight bounces.
        {"name": "frame_hd", "kind": "frame", "scene": "box", "blobs": 256, "subdiv": 22, "width": 1920,
         "height": 1080, "spp": 8, "depth": 8, "builder": "ploc"},
        # Instances of one blob in mirror, glass, plastic and matte, lit by area, point and
        # spot lights, at an odd image size.
        {"name": "frame_instanced", "kind": "frame", "scene": "instanced", "blobs": 64, "subdiv": 16, "width": 641,
         "height": 479, "spp": 4, "depth": 6, "builder": "lbvh"},
        # One step of inverse rendering: a frame with per-triangle albedos, the image loss
        # and the backward pass.
        {"name": "inverse_step", "kind": "inverse", "blobs": 204, "width": 512, "height": 512, "spp": 16, "depth": 6},
        # Many scenes at once: 64 trees of 1 k to 1 M triangles rebuilt, one frame of each.
        {"name": "batch_scenes", "kind": "batch", "scenes": 64, "largest": 1000000, "spp": 1, "depth": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "build", "build", "quality", "frame", "frame", "inverse", "batch"])
    scene = rng.choice(["soup", "heightfield"])
    if kind == "trace":
        side = _log(rng, 16, 1800)
        rays = rng.choice(["primary", "surface", "ao"])
        if rays == "ao":
            side = min(side, 1000)
        return {"kind": kind, "scene": scene, "size": _log(rng, 1000, 1000000) if scene == "soup" else _log(rng, 24, 1800),
                "rays": rays, "width": side, "height": max(1, side - rng.randrange(0, 9)),
                "query": "any" if rays == "ao" else rng.choice(["closest", "closest", "any"]),
                "sort": rng.choice([True, False])}
    if kind == "build":
        return {"kind": kind, "scene": scene, "size": _log(rng, 1000, 6000000) if scene == "soup" else _log(rng, 24, 1900),
                "mode": rng.choice(["build", "rebuild"])}
    if kind == "quality":
        return {"kind": kind, "scene": scene, "size": _log(rng, 1000, 900000) if scene == "soup" else _log(rng, 24, 700),
                "width": rng.randrange(300, 600), "height": rng.randrange(200, 500)}
    if kind == "frame":
        scene = rng.choice(["box", "box", "instanced"])
        width = _log(rng, 64, 1280)
        return {"kind": kind, "scene": scene, "blobs": _log(rng, 4, 128), "subdiv": _log(rng, 3, 20), "width": width,
                "height": max(8, width * 9 // 16 + rng.randrange(0, 5)), "spp": rng.choice([1, 2, 3, 4, 8]),
                "depth": rng.randrange(2, 9), "builder": rng.choice(["lbvh", "ploc"])}
    if kind == "inverse":
        side = _log(rng, 64, 500)
        return {"kind": kind, "blobs": _log(rng, 16, 204), "width": side, "height": max(8, side - rng.randrange(0, 20)),
                "spp": rng.choice([1, 3, 4, 8, 16]), "depth": rng.randrange(3, 7)}
    return {"kind": kind, "scenes": _log(rng, 4, 60), "largest": _log(rng, 20000, 900000), "spp": rng.choice([1, 1, 2]),
            "depth": rng.randrange(2, 4)}


def _mesh(case, seed):
    n = case["size"]
    if case["scene"] == "heightfield":
        return scenes.heightfield(n, seed=seed)
    return scenes.soup(n, seed=seed, offset=0.5 / n ** (1.0 / 3.0))


def _num_tris(case):
    return 2 * case["size"] ** 2 if case["scene"] == "heightfield" else case["size"]


def _rays(case, tris, seed):
    w, h = case["width"], case["height"]
    if case["rays"] == "primary":
        k = 0.1 * ((seed * 7919) % 101) / 101.0
        return scenes.pinhole_rays(w, h, eye=(0.45 + k, 0.5 + 0.5 * k, -1.5 - k))
    closest, ao = scenes.surface_rays(tris, w * h, seed=seed + 7, ao_per_origin=8, ao_tmax=0.05,
                                      closest=case["rays"] == "surface", ao=case["rays"] == "ao")
    return closest if case["rays"] == "surface" else ao


def _context(sort=False):
    ctx = vg.Context(DEVICE)
    if sort:
        ctx.set_trace_flags(vg.Context.TRACE_SORT_RAYS)
    return ctx


def _prepare_trace(case, seed):
    tris = _mesh(case, seed)
    ctx = _context(case["sort"])
    bvh = vg.lbvh_builder(ctx).build(rt.as_device_bytes(tris, DEVICE))
    rays = rt.device_rays(_rays(case, tris, seed), DEVICE)
    hits = torch.empty((rays.shape[0], 4), dtype=torch.float32, device=rays.device)
    return {"kind": "trace", "ctx": ctx, "bvh": bvh, "rays": rays, "hits": hits, "any": case["query"] == "any"}


def _hits(hits):
    return {"prim_id": hits.view(torch.int32)[:, 0], "t": hits[:, 1], "uv": hits[:, 2:]}


def _prepare_build(case, seed):
    ctx = _context()
    tris = rt.as_device_bytes(_mesh(case, seed), DEVICE)
    n = _num_tris(case)
    state = {"kind": "build", "ctx": ctx, "tris": tris, "mode": case["mode"],
             "nodes": torch.empty((2 * n - 1) * 32, dtype=torch.uint8, device=tris.device),
             "indices": torch.empty(n, dtype=torch.int32, device=tris.device)}
    if case["mode"] == "rebuild":
        # a program that rebuilds one tree every frame: here over the geometry of another
        state["bvh"] = vg.lbvh_builder(ctx).build(rt.as_device_bytes(_mesh(case, seed + 1000), DEVICE))
    return state


def _run_build(s):
    ctx = s["ctx"]
    if s["mode"] == "rebuild":
        bvh = s["bvh"].rebuild(s["tris"])
    else:
        bvh = vg.lbvh_builder(ctx).build(s["tris"])
    # the C ABI's export into the caller's device buffers, in the reference's node layout
    ctx.check(ctx.lib.gbrt_bvh_export_bvh2(ctx.h, bvh.h, ctypes.c_void_p(s["nodes"].data_ptr()),
                                           ctypes.c_void_p(s["indices"].data_ptr())))
    return {"nodes": s["nodes"], "indices": s["indices"]}


def _prepare_quality(case, seed):
    ctx = _context()
    tris = rt.as_device_bytes(_mesh(case, seed), DEVICE)
    rays = rt.device_rays(_rays(dict(case, rays="primary"), None, seed), DEVICE)
    hits = torch.empty((rays.shape[0], 4), dtype=torch.float32, device=rays.device)
    return {"kind": "quality", "ctx": ctx, "tris": tris, "rays": rays, "hits": hits}


def _prepare_frame(case, seed):
    ctx = _context()
    builder = vg.ploc_builder(ctx) if case["builder"] == "ploc" else vg.lbvh_builder(ctx)
    keep = []
    if case["scene"] == "box":
        tris, mats, lights = scenes.box_scene(n_blobs=case["blobs"], subdiv=case["subdiv"], seed=seed)
        bvh = builder.build(rt.as_device_bytes(tris, DEVICE))
        scene = vg.PTScene(bvh, mats, lights)
        keep.append(bvh)
    else:
        d = scenes.instanced_box_scene(n_blobs=case["blobs"], subdiv=case["subdiv"], seed=seed, albedo_seed=seed + 9)
        mats = d["materials"]
        per = len(d["blob"])
        for b in range(case["blobs"]):
            m = mats[14 + b * per:14 + (b + 1) * per]
            if b % 4 == 1:
                m["kind"], m["ior"], m["absorption"] = MIRROR, (0.27, 0.42, 1.35), (3.4, 2.3, 1.8)
            elif b % 4 == 2:
                m["kind"], m["color"], m["color2"], m["scale2"], m["ior"] = GLASS, 1.0, 1.0, 1.0, 1.5
            elif b % 4 == 3:
                m["kind"], m["color2"], m["scale2"], m["exponent"] = PLASTIC, 0.4, 1.0, 32.0
        room = builder.build(rt.as_device_bytes(d["room"], DEVICE))
        blob = builder.build(rt.as_device_bytes(d["blob"], DEVICE))
        identity = np.array([1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0], np.float32)
        tlas = vg.TLAS([(room, identity)] + [(blob, x) for x in d["transforms"]], ctx)
        scene = vg.PTScene.over_instances(tlas, mats, scenes.mixed_lights(d["lights"]), d["inst_geom"])
        keep += [room, blob, tlas]
    params = scenes.pt_params(case["width"], case["height"], case["spp"], num_bounces=case["depth"], frame_id=seed)
    shape = (case["height"], case["width"], 4)
    accum = torch.zeros(shape, dtype=torch.float32, device=f"cuda:{DEVICE}")
    color = torch.zeros(shape, dtype=torch.float32, device=f"cuda:{DEVICE}")
    return {"kind": "frame", "ctx": ctx, "scene": scene, "params": params, "camera": scenes.box_camera(),
            "accum": accum, "color": color, "keep": keep}


def _prepare_inverse(case, seed):
    ctx = _context()
    scene, tris, mats, lights, hidden, emission = inverse.setup(n_blobs=case["blobs"], seed=seed, hidden_seed=seed + 5,
                                                                ctx=ctx, builder="ploc")
    w, h, flags = case["width"], case["height"], PT_SHADOW_RANGE_FIX | PT_NO_RUSSIAN_ROULETTE
    camera = scenes.box_camera()
    target = rt.pathtrace_forward(scene, camera, scenes.pt_params(w, h, 16, num_bounces=case["depth"],
                                                                  frame_id=inverse.TARGET_FRAME, flags=flags),
                                  hidden, emission)
    # an albedo state in mid-optimisation
    rng = np.random.default_rng(seed + 11)
    albedo = torch.from_numpy(rng.uniform(0.3, 0.7, size=tuple(hidden.shape)).astype(np.float32)).to(hidden.device)
    return {"kind": "inverse", "ctx": ctx, "scene": scene, "camera": camera, "target": target, "albedo": albedo,
            "emission": emission, "image": torch.empty_like(target),
            "forward": scenes.pt_params(w, h, case["spp"], num_bounces=case["depth"], frame_id=seed, flags=flags),
            "backward": scenes.pt_params(w, h, case["spp"], num_bounces=case["depth"],
                                         frame_id=seed + inverse.GRAD_FRAME_OFFSET, flags=flags)}


def _run_inverse(s):
    image = rt.pathtrace_forward(s["scene"], s["camera"], s["forward"], s["albedo"], s["emission"], image=s["image"])
    loss, adjoint = inverse.l2_adjoint(image, s["target"])
    grad_albedo, grad_emission = rt.pathtrace_backward(s["scene"], s["camera"], s["backward"], s["albedo"],
                                                       s["emission"], adjoint)
    return {"image": image, "loss": loss, "grad_albedo": grad_albedo, "grad_emission": grad_emission}


def _batch_scenes(case, seed):
    """The scenes of a batch: triangle counts log-uniform in [1000, largest] and image
    sides of 64 to 512 that depend on the case alone, soups and cameras on the seed."""
    num = case["scenes"]
    counts = [int(round(math.exp(math.log(1000.0) + scenes.u01(17, 1, s) * math.log(case["largest"] / 1000.0))))
              for s in range(num)]
    sides = [scenes.BATCH_SIDES[min(int(scenes.u01(17, 2, s) * 4), 3)] for s in range(num)]
    tris = np.concatenate([scenes.soup(n, seed=seed * 1000003 + s, offset=0.5 / n ** (1.0 / 3.0))
                           for s, n in enumerate(counts)])
    cams, params = np.zeros(num, CAMERA), np.zeros(num, PT_PARAMS)
    for s in range(num):
        z, phi = 2.0 * scenes.u01(seed, 3, s) - 1.0, 2.0 * math.pi * scenes.u01(seed, 4, s)
        r = math.sqrt(max(0.0, 1.0 - z * z))
        eye = (0.5 + 1.6 * r * math.cos(phi), 0.5 + 1.6 * r * math.sin(phi), 0.5 + 1.6 * z)
        cams[s] = scenes.box_camera(eye, (0.5, 0.5, 0.5), (0.0, 0.0, 1.0) if abs(r * math.sin(phi)) > 0.9
                                    else (0.0, 1.0, 0.0), 50.0)
        params[s] = scenes.pt_params(sides[s], sides[s], case["spp"], num_bounces=case["depth"], frame_id=seed,
                                     ambient=(1.0, 1.0, 1.0))
    mats = np.zeros(1, MATERIAL)
    mats["kind"], mats["color"], mats["scale"] = MATTE, 0.7, 1.0
    return tris, np.concatenate([[0], np.cumsum(counts)]), cams, params, mats


def _prepare_batch(case, seed):
    ctx = _context()
    tris, offsets, cams, params, mats = _batch_scenes(case, seed)
    batch = vg.Batch(offsets, ctx)
    batch.set_frames(cams, params, mats)
    batch.launch = (128, 32, 64, BATCH_ORDER_BLOCKS)
    return {"kind": "batch", "ctx": ctx, "batch": batch, "tris": rt.as_device_bytes(tris, DEVICE),
            "images": batch.new_images()}


_PREPARE = {"trace": _prepare_trace, "build": _prepare_build, "quality": _prepare_quality, "frame": _prepare_frame,
            "inverse": _prepare_inverse, "batch": _prepare_batch}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    kind = state["kind"]
    if kind == "trace":
        query = vg.any_hit if state["any"] else vg.closest_hit
        return _hits(query(state["rays"], state["bvh"], state["hits"]))
    if kind == "build":
        return _run_build(state)
    if kind == "quality":
        bvh = vg.ploc_builder(state["ctx"]).build(state["tris"])
        return _hits(vg.closest_hit(state["rays"], bvh, state["hits"]))
    if kind == "frame":
        vg.pathtrace_frame(state["scene"], state["camera"], state["params"], state["accum"], state["color"])
        return {"accum": state["accum"], "color": state["color"]}
    if kind == "inverse":
        return _run_inverse(state)
    state["batch"].build(state["tris"])
    return {"images": state["batch"].pathtrace(state["images"])}


def _segment_flops(n):
    # a closest-hit query: a box pair per level of a balanced tree, one triangle test
    return 48.0 * math.log2(max(n, 2)) + 50.0


def work(case):
    kind = case["kind"]
    if kind in ("trace", "build", "quality"):
        n = _num_tris(case)
    if kind == "trace":
        rays = case["width"] * case["height"] * (8 if case["rays"] == "ao" else 1)
        # a ray in and a hit out, and the part of the tree that the rays can reach
        tree = min(112.0 * n, rays * (64.0 * math.log2(max(n, 2)) + 48.0))
        return {"bytes": 48.0 * rays + tree, "flops": rays * _segment_flops(n)}
    if kind == "build":
        # triangles in, 2n - 1 exported nodes and n indices out
        return {"bytes": 44.0 * n + 64.0 * n + 4.0 * n, "flops": 60.0 * n}
    if kind == "quality":
        rays = case["width"] * case["height"]
        # triangles in, node pairs and leaf triangles out, then the rays; each cluster
        # level compares 32 neighbours, the levels sum to about 3 n clusters
        return {"bytes": 44.0 * n + 112.0 * n + 48.0 * rays, "flops": 3.0 * n * 32 * 14 + rays * _segment_flops(n)}
    if kind == "frame":
        per = 20 * case["subdiv"] ** 2
        n = 14 + per * (case["blobs"] if case["scene"] == "box" else 1)
        pixels = case["width"] * case["height"]
        segments = pixels * case["spp"] * min(case["depth"], 3)
        return {"bytes": 32.0 * pixels + 112.0 * n, "flops": segments * (2 * _segment_flops(n) + 300.0)}
    if kind == "inverse":
        n = 14 + 20 * case["blobs"]
        pixels = case["width"] * case["height"]
        segments = pixels * case["spp"] * case["depth"]
        # forward and replayed segments, each with a shadow ray
        return {"bytes": 48.0 * pixels + 112.0 * n + 24.0 * n, "flops": 2.0 * segments * (2 * _segment_flops(n) + 300.0)}
    mean = (case["largest"] - 1000.0) / math.log(case["largest"] / 1000.0)   # of log-uniform counts
    n = case["scenes"] * mean
    pixels = case["scenes"] * 87040.0                                        # mean of 64^2, 128^2, 256^2, 512^2
    segments = pixels * case["spp"] * case["depth"] * 0.6
    return {"bytes": (44.0 + 112.0) * n + 16.0 * pixels, "flops": 60.0 * n + segments * (_segment_flops(mean) + 200.0)}


def exact(case, seed):
    """The closest hits in 64 bits by testing every triangle, for small queries."""
    if case["kind"] != "trace" or case["query"] != "closest":
        return None
    rays_n = case["width"] * case["height"]
    if rays_n * _num_tris(case) > 2_000_000_000:
        return None
    dev = f"cuda:{DEVICE}"
    tris = _mesh(case, int(seed))
    rays = _rays(case, tris, int(seed))
    v1, e1, e2 = (torch.from_numpy(np.ascontiguousarray(tris[k])).to(dev).double() for k in ("v1", "e1", "e2"))
    ori, d = (torch.from_numpy(np.ascontiguousarray(rays[k])).to(dev).double() for k in ("ori", "dir"))
    tmin, tmax = (torch.from_numpy(np.ascontiguousarray(rays[k])).to(dev).double() for k in ("tmin", "tmax"))
    out = {k: torch.zeros(rays_n, dtype=torch.float64, device=dev) for k in ("t", "u", "v")}
    step = max(1, 20_000_000 // len(tris))
    for b in range(0, rays_n, step):
        o, r = ori[b:b + step, None, :], d[b:b + step, None, :]
        s1 = torch.linalg.cross(r.expand(-1, len(tris), -1), e2[None].expand(r.shape[0], -1, -1))
        inv = 1.0 / (s1 * e1[None]).sum(-1)
        q = o - v1[None]
        u = (q * s1).sum(-1) * inv
        s2 = torch.linalg.cross(q, e1[None].expand(q.shape[0], -1, -1))
        v = (r * s2).sum(-1) * inv
        t = (e2[None] * s2).sum(-1) * inv
        hit = (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t >= tmin[b:b + step, None]) & (t <= tmax[b:b + step, None])
        best, at = torch.where(hit, t, math.inf).min(dim=1)
        found = torch.isfinite(best)
        out["t"][b:b + step] = torch.where(found, best, FLT_MAX)
        out["u"][b:b + step] = torch.where(found, u.gather(1, at[:, None])[:, 0], 0.0)
        out["v"][b:b + step] = torch.where(found, v.gather(1, at[:, None])[:, 0], 0.0)
    return {"prim_id": None, "t": out["t"], "uv": torch.stack([out["u"], out["v"]], dim=1)}
