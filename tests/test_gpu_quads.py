"""Queries through the quad nodes return what the node pairs return, byte for byte: the
tree is traced as built (quads) and uploaded again from its export (pairs only, the same
children in the same order).  The rays include axis-parallel ones, ones that start on
planes and pass through shared edges and vertices, negative and empty ranges, directions
of any length, and zero, infinite and NaN components; the trees flat, tiny, far from the
origin, full of coincident triangles, and with triangles whose boxes the quads refuse."""
import numpy as np
import pytest

import visionaray_gb300 as vg
from visionaray_gb300 import scenes

pytestmark = pytest.mark.gpu


def grid_scene(k, scale=1.0, shift=0.0):
    """k x k axis-aligned squares (two triangles each) in the plane z = shift."""
    x, y = np.meshgrid(np.arange(k), np.arange(k), indexing="ij")
    x, y = x.ravel(), y.ravel()
    tris = np.zeros(2 * k * k, vg.TRIANGLE)
    for half, (dx, e1, e2) in enumerate((((0, 0), (1, 0, 0), (0, 1, 0)), ((1, 1), (-1, 0, 0), (0, -1, 0)))):
        t = tris[half::2]
        t["v1"] = np.stack([x + dx[0], y + dx[1], np.zeros(len(x))], 1) / k * scale + np.float32(shift)
        t["e1"], t["e2"] = np.array(e1) / k * scale, np.array(e2) / k * scale
    tris["prim_id"] = np.arange(len(tris))
    return tris


def scene(kind):
    if kind == "soup":
        return scenes.soup(5000, seed=3, offset=0.1)
    if kind == "heightfield":
        return scenes.heightfield(48, seed=2)
    if kind == "box":
        return scenes.box_scene(n_blobs=4, subdiv=4, seed=2)[0]
    if kind == "flat":
        return grid_scene(20)
    if kind == "coincident":
        t = np.concatenate([scenes.soup(300, seed=8, offset=0.2)] * 5)
        t["prim_id"] = np.arange(len(t))
        return t
    if kind == "tiny":
        return grid_scene(16, 1e-6, 1e-6)
    if kind == "mixed_scales":
        t = np.concatenate([grid_scene(8, 1e-7), scenes.soup(500, seed=5, offset=0.3)])
        t["prim_id"] = np.arange(len(t))
        return t
    if kind == "far":
        t = scenes.soup(2000, seed=6, offset=0.2)
        t["v1"] += np.float32(1000.0)
        return t
    if kind == "nan":
        t = scenes.soup(700, seed=7, offset=0.2)
        t["v1"][::50] = np.nan
        return t
    if kind == "huge":
        t = scenes.soup(700, seed=9, offset=0.2)
        t["v1"][5] = 3e38
        return t
    return scenes.soup(int(kind), seed=11, offset=0.5)


def ray_set(tris, seed):
    rng = np.random.default_rng(seed)
    fin = np.isfinite(tris["v1"]).all(1) & (np.abs(tris["v1"]) < 1e30).all(1)
    v = tris["v1"][fin]
    lo, hi = v.min(0) - 1e-3, v.max(0) + 1e-3
    ext = float((hi - lo).max()) or 1.0
    n = 6000
    r = np.zeros(n, vg.RAY)
    pick = lambda m: tris[fin][rng.integers(0, fin.sum(), m)]   # noqa: E731
    r["ori"] = rng.uniform(lo - 0.3 * ext, hi + 0.3 * ext, size=(n, 3))
    t = pick(n)
    w = rng.dirichlet((1, 1, 1), n).astype(np.float32)
    w[::3] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, len(w[::3]))]       # through vertices
    w[1::3, 0] = 0.0                                                            # through edges
    target = t["v1"] + t["e1"] * w[:, 1:2] + t["e2"] * w[:, 2:3]
    r["dir"] = target - r["ori"]
    r["dir"] /= np.linalg.norm(r["dir"], axis=1, keepdims=True)
    r["tmax"] = np.finfo(np.float32).max
    r["ori"][1000:2000] = target[1000:2000]                                     # from the surface
    r["dir"][1000:2000] = rng.normal(size=(1000, 3))
    axis = rng.integers(0, 3, 1000)
    r["dir"][2000:3000] = np.eye(3)[axis] * rng.choice([-1, 1], (1000, 1))       # along an axis
    r["ori"][2000:2500] = target[2000:2500] - r["dir"][2000:2500] * ext
    r["dir"][3000:3200, 0] = 0.0
    r["dir"][3200:3400, 1:] *= np.float32(1e-9)
    r["dir"][3400:3800] *= 10.0 ** rng.uniform(-6, 6, (400, 1))
    r["tmin"][3800:4200], r["tmax"][3800:4200] = -ext, 0.5 * ext
    r["tmin"][4200:4400], r["tmax"][4200:4400] = 0.1 * ext, 0.3 * ext
    r["tmin"][4400:4420], r["tmax"][4400:4420] = 1.0, 0.5                        # empty
    special = [(0, 0, 0), (np.nan, 1, 0), (np.inf, 1, 0), (1e-30, 1e-30, 1e-30), (1e30, 1e30, 0), (1e-42, 1, 0),
               (1e-20, 1, 1e-20), (3e38, -3e38, 1)]
    for k, d in enumerate(special):
        r["dir"][4420 + 20 * k:4440 + 20 * k] = d
    r["ori"][4600:4610] = np.nan
    r["ori"][4610:4620] = 1e25
    r["ori"][4620:4640] *= np.float32(1e6)
    return r


@pytest.mark.parametrize("sort", [0, 1])
@pytest.mark.parametrize("builder", ["lbvh", "ploc"])
@pytest.mark.parametrize("kind", ["2", "3", "5", "64", "soup", "heightfield", "box", "flat", "coincident", "tiny",
                                  "mixed_scales", "far", "nan", "huge"])
def test_quads_equal_pairs(kind, builder, sort):
    if sort and kind not in ("soup", "heightfield"):
        pytest.skip("the ray order does not depend on the tree's kind")
    ctx = vg.Context(0)
    ctx.set_trace_flags(sort)
    tris = scene(kind)
    make = vg.ploc_builder if builder == "ploc" else vg.lbvh_builder
    if kind == "huge" and builder == "ploc":
        # PLOC refuses boxes whose union area overflows
        with pytest.raises(vg.GbrtError):
            make(ctx).build(vg.as_device_bytes(tris))
        return
    bvh = make(ctx).build(vg.as_device_bytes(tris))
    nodes, idx = bvh.export_bvh2()
    pairs = vg.IndexBVH.upload(nodes, idx, tris, ctx)
    rays = ray_set(tris, 1)
    if sort:
        rays = np.tile(rays, 12)   # enough rays to be sorted
    for m in (1, 31, 33, len(rays)):
        d = vg.device_rays(rays[:m])
        for query in (vg.closest_hit, vg.any_hit):
            got, want = vg.hits_to_numpy(query(d, bvh)), vg.hits_to_numpy(query(d, pairs))
            bad = np.flatnonzero(got.view(np.uint32).reshape(m, 4) != want.view(np.uint32).reshape(m, 4))
            assert got.tobytes() == want.tobytes(), (query.__name__, m, bad[:4] // 4, rays[bad[:2] // 4])
    moved = tris.copy()
    moved["v1"] += np.float32(0.01)
    bvh.refit(vg.as_device_bytes(moved))
    nodes, idx = bvh.export_bvh2()
    pairs = vg.IndexBVH.upload(nodes, idx, moved, ctx)
    d = vg.device_rays(rays)
    assert vg.hits_to_numpy(vg.closest_hit(d, bvh)).tobytes() == vg.hits_to_numpy(vg.closest_hit(d, pairs)).tobytes()
    ctx.synchronize()
