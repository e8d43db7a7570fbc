"""Long ray queries are shared by a counter between the warps that fit the GPU, 32 rays at a
time: at and around the line where that starts (32 rays for each of the resident warps, 36
per multiprocessor), one ray more, a partial last chunk and several chunks per warp, sorted
and in input order, every ray gets the node pairs' answer, byte for byte, and the hits past
the last ray stay untouched; any-hit queries likewise on both sides of 2^23 rays, where the
keys of their order change."""
import numpy as np
import pytest
import torch

import visionaray_gb300 as vg
from visionaray_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sort", [0, 1])
@pytest.mark.parametrize("extra", [-1, 0, 1, 31, 33, 160_000, 800_001])
def test_shared_queries_equal_pairs(extra, sort):
    resident = torch.cuda.get_device_properties(0).multi_processor_count * 36
    n = 32 * resident + extra
    ctx = vg.Context(0)
    ctx.set_trace_flags(sort)
    tris = scenes.soup(3000, seed=2, offset=0.05)
    bvh = vg.lbvh_builder(ctx).build(vg.as_device_bytes(tris))
    nodes, idx = bvh.export_bvh2()
    pairs = vg.IndexBVH.upload(nodes, idx, tris, ctx)
    rng = np.random.default_rng(7)
    rays = np.zeros(n, vg.RAY)
    rays["ori"] = rng.uniform(-0.2, 1.2, (n, 3))
    rays["dir"] = rng.normal(size=(n, 3))
    rays["tmax"] = np.finfo(np.float32).max
    d = vg.device_rays(rays)
    for query in (vg.closest_hit, vg.any_hit):
        got = torch.full((n + 64, 4), -7.0, dtype=torch.float32, device="cuda")
        want = torch.full((n + 64, 4), -7.0, dtype=torch.float32, device="cuda")
        query(d, bvh, out=got[:n])
        query(d, pairs, out=want[:n])
        ctx.synchronize()
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("n", [1 << 23, (1 << 23) + 1])
def test_the_finer_order_of_many_any_hit_rays(n):
    ctx = vg.Context(0)
    ctx.set_trace_flags(vg.Context.TRACE_SORT_RAYS)
    tris = scenes.soup(500, seed=4, offset=0.05)
    bvh = vg.lbvh_builder(ctx).build(vg.as_device_bytes(tris))
    nodes, idx = bvh.export_bvh2()
    pairs = vg.IndexBVH.upload(nodes, idx, tris, ctx)
    g = torch.Generator(device="cuda").manual_seed(3)
    rays = torch.rand((n, 8), generator=g, device="cuda") - 0.5
    rays[:, :3] += 0.5
    rays[:, 6], rays[:, 7] = 0.0, 3e38
    assert torch.equal(vg.any_hit(rays, bvh).view(torch.int32), vg.any_hit(rays, pairs).view(torch.int32))
    ctx.synchronize()
