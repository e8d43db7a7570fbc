"""Queries through the quad nodes return what the node pairs return, byte for byte, where
their arithmetic is at its limits (the tree traced as built, and uploaded again from its
export, which traverses the pairs only): rays with zero direction components among
triangles far thinner than their distance, from near and far, along directions of any
length; rays in the plane of a surface that is turned against the axes, whose hits are
rounding errors."""
import numpy as np
import pytest

import visionaray_gb300 as vg
from visionaray_gb300 import scenes

pytestmark = pytest.mark.gpu

FLT_MAX = np.finfo(np.float32).max


def assert_quads_equal_pairs(tris, rays, builder="lbvh", ctx=None):
    ctx = ctx or vg.Context(0)
    make = vg.ploc_builder if builder == "ploc" else vg.lbvh_builder
    bvh = make(ctx).build(vg.as_device_bytes(tris))
    nodes, idx = bvh.export_bvh2()
    pairs = vg.IndexBVH.upload(nodes, idx, tris, ctx)
    d = vg.device_rays(rays)
    for query in (vg.closest_hit, vg.any_hit):
        got, want = vg.hits_to_numpy(query(d, bvh)), vg.hits_to_numpy(query(d, pairs))
        bad = np.flatnonzero((got.view(np.uint32).reshape(-1, 4) != want.view(np.uint32).reshape(-1, 4)).any(1))
        assert len(bad) == 0, (query.__name__, len(bad), rays[bad[:2]], got[bad[:2]], want[bad[:2]])
    ctx.synchronize()
    return want


def thin_strips(scale, thin, seed=0, n=200):
    """Triangles across the y axis: x extents of scale * thin around x = 0, z extents of
    about scale, at random heights."""
    rng = np.random.default_rng(seed)
    t = np.zeros(n, vg.TRIANGLE)
    w = scale * thin * rng.uniform(0.2, 1.0, n)
    t["v1"][:, 0] = w * rng.uniform(-1.0, 0.0, n)
    t["v1"][:, 1] = rng.uniform(-1.0, 1.0, n) * scale
    t["v1"][:, 2] = rng.uniform(-1.0, 0.5, n) * scale
    t["e1"][:, 0] = w
    t["e2"][:, 2] = rng.uniform(0.1, 0.5, n) * scale
    t["prim_id"] = np.arange(n)
    return t


def rays_across(t, n, length, distance, seed):
    """Rays along y (every other one a little along z too) through points of the triangles."""
    rng = np.random.default_rng(seed)
    s = t[rng.integers(0, len(t), n)]
    w = rng.dirichlet((1, 1, 1), n)
    p = s["v1"].astype(float) + s["e1"] * w[:, 1:2] + s["e2"] * w[:, 2:3]
    d = np.zeros((n, 3))
    d[:, 1] = rng.choice([-1.0, 1.0], n)
    d[::2, 2] = rng.uniform(-0.3, 0.3, len(d[::2]))
    r = np.zeros(n, vg.RAY)
    r["ori"], r["dir"], r["tmax"] = p - d * distance, d * length, FLT_MAX
    return r


@pytest.mark.parametrize("builder", ["lbvh", "ploc"])
@pytest.mark.parametrize("scale", [2.0 ** -30, 1.0, 2.0 ** 30])
def test_thin_triangles_along_zero_components(scale, builder):
    hits = 0
    for k, thin in enumerate((2.0 ** -12, 2.0 ** -30, 2.0 ** -50, 2.0 ** -70, 2.0 ** -90)):
        t = thin_strips(scale, thin, k)
        r = np.concatenate([rays_across(t, 1500, length, distance * scale, 10 * k + j)
                            for j, (length, distance) in enumerate(((1.0, 3.0), (1.0, 1e3), (1e-9, 3.0), (1e9, 3.0),
                                                                    (1.0, 1e6), (2.0 ** -13, 1e4)))])
        want = assert_quads_equal_pairs(t, r, builder)
        hits += int((want["prim_id"] != 0xFFFFFFFF).sum())
    assert hits > 10000


def test_a_ray_of_tiny_direction_into_a_narrow_box():
    t = np.zeros(4, vg.TRIANGLE)
    t["v1"][:, 1] = (1.0, 1.5, 2.0, 2.5)
    t["e1"], t["e2"] = (2.0 ** -25, 0, 0), (0, 0, 1)
    t["prim_id"] = np.arange(4)
    r = np.zeros(3, vg.RAY)
    r["ori"], r["tmax"] = (2.0 ** -27, 0, 0.25), FLT_MAX
    r["dir"] = ((0, 2.0 ** -40, 0), (2.0 ** -80, 2.0 ** -40, 0), (0, 1, 0))
    want = assert_quads_equal_pairs(t, r)
    assert (want["prim_id"] == 0).all()


def test_scenes_of_different_size_in_a_batch():
    """The scenes of a batch take the smallest cells from their own trees: frames of thin
    strips beside scenes 2^30 times their size and of one triangle equal the persistent
    kernel's over the node pairs."""
    import torch
    from visionaray_gb300.types import CAMERA, MATERIAL, MATTE, PT_PARAMS
    parts = [thin_strips(1.0, 2.0 ** -60, 3), thin_strips(2.0 ** 30, 2.0 ** -60, 4), scenes.soup(1, seed=1),
             thin_strips(2.0 ** -20, 2.0 ** -40, 5)]
    batch = vg.Batch(np.concatenate([[0], np.cumsum([len(p) for p in parts])]), vg.Context(0))
    cams, params = np.zeros(4, CAMERA), np.zeros(4, PT_PARAMS)
    for s, scale in enumerate((1.0, 2.0 ** 30, 1.0, 2.0 ** -20)):
        cams[s] = scenes.box_camera((0.0, -3.0 * scale, 0.0), (0.0, 0.0, 0.0), (0.0, 0.0, 1.0), 40.0)
        params[s] = scenes.pt_params(33, 64, 2, num_bounces=3, frame_id=1, ambient=(1.0, 1.0, 1.0))
    mats = np.zeros(1, MATERIAL)
    mats["kind"], mats["color"], mats["scale"] = MATTE, 0.7, 1.0
    batch.set_frames(cams, params, mats)
    batch.build(vg.as_device_bytes(np.concatenate(parts)))
    images = []
    for stack in (64, 32):
        batch.launch = (128, 32, stack, 0)
        images.append(batch.pathtrace(batch.new_images()).clone())
    batch.ctx.synchronize()
    assert torch.equal(images[0].view(torch.int32), images[1].view(torch.int32))


def turned_plane(k, seed, noise):
    """k x k squares (two triangles each) in a plane turned at random, vertices off by noise."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(k + 1), np.arange(k + 1), indexing="ij")
    g = np.stack([x, y, np.zeros_like(x)], 2) / k @ np.linalg.qr(rng.normal(size=(3, 3)))[0].T
    g = (g + rng.normal(size=g.shape) * noise).astype(np.float32)
    a, b, c, d = g[:-1, :-1], g[1:, :-1], g[1:, 1:], g[:-1, 1:]
    t = np.zeros(2 * k * k, vg.TRIANGLE)
    for h, (p, q, r) in enumerate(((a, b, d), (c, d, b))):
        t["v1"][h::2], t["e1"][h::2] = p.reshape(-1, 3), (q - p).reshape(-1, 3)
        t["e2"][h::2] = (r - p).reshape(-1, 3)
    t["prim_id"] = np.arange(len(t))
    return t


@pytest.mark.parametrize("builder", ["lbvh", "ploc"])
@pytest.mark.parametrize("noise", [0.0, 1e-8, 1e-7])
@pytest.mark.parametrize("k", [16, 64])
def test_rays_in_a_turned_plane(k, noise, builder):
    """Rays between two points of the plane, from the first one and from outside."""
    n = 400_000
    t = turned_plane(k, 3, noise)
    rng = np.random.default_rng(k)

    def points():
        s = t[rng.integers(0, len(t), n)]
        w = rng.dirichlet((1, 1, 1), n)
        return s["v1"].astype(float) + s["e1"] * w[:, 1:2] + s["e2"] * w[:, 2:3]

    p, q = points(), points()
    d = (q - p) / np.linalg.norm(q - p, axis=1, keepdims=True)
    r = np.zeros(n, vg.RAY)
    r["ori"], r["dir"], r["tmax"] = p, d, FLT_MAX
    r["ori"][::2] -= 2.0 * d[::2].astype(np.float32)
    want = assert_quads_equal_pairs(t, r, builder)
    assert (want["prim_id"] != 0xFFFFFFFF).sum() > n // 2
