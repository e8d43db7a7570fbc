"""Calls on several streams and in captured graphs: what a call enqueues does not depend on
what the context's other calls do to its memory later or at the same time."""
import contextlib

import numpy as np
import pytest
import torch

import visionaray_gb300 as vg
from visionaray_gb300 import scenes

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def on_stream(ctx, stream):
    """The context's calls go to `stream` inside."""
    ctx.check(ctx.lib.gbrt_context_set_stream(ctx.h, stream.cuda_stream))
    yield
    ctx.check(ctx.lib.gbrt_context_set_stream(ctx.h, torch.cuda.current_stream().cuda_stream))


def capture(ctx, call):
    """A graph of what call() enqueues on the context's stream."""
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream), on_stream(ctx, stream):
        call()
    return graph


def random_rays(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rays = torch.rand((n, 8), generator=g, device="cuda") - 0.5
    rays[:, :3] += 0.5
    rays[:, 6], rays[:, 7] = 0.0, 3e38
    return rays


@pytest.fixture
def soup_tree():
    ctx = vg.Context(0)
    return ctx, vg.lbvh_builder(ctx).build(vg.as_device_bytes(scenes.soup(20000, seed=2, offset=0.05)))


def sorted_query(ctx, bvh, rays):
    ctx.set_trace_flags(vg.Context.TRACE_SORT_RAYS)
    vg.closest_hit(rays, bvh)
    ctx.synchronize()
    ctx.set_trace_flags(0)


def test_queries_in_input_order_on_two_streams(soup_tree):
    """Long queries in input order, on a context that has traced sorted rays, in turn on
    two streams without a synchronisation between them."""
    ctx, bvh = soup_tree
    rays = [random_rays(1_000_000 + 7 * k, k) for k in range(2)]
    want = [vg.closest_hit(r, bvh) for r in rays]
    sorted_query(ctx, bvh, rays[1])
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[torch.full_like(w, -7.0) for w in want] for _ in range(4)]
    torch.cuda.synchronize()
    for pair in got:
        for k in range(2):
            with on_stream(ctx, streams[k]):
                vg.closest_hit(rays[k], bvh, out=pair[k])
    torch.cuda.synchronize()
    for pair in got:
        for k in range(2):
            assert torch.equal(pair[k].view(torch.int32), want[k].view(torch.int32))
    ctx.synchronize()


def test_a_captured_query_outlives_a_larger_sorted_one(soup_tree):
    ctx, bvh = soup_tree
    rays = random_rays(400_001, 3)
    want = vg.closest_hit(rays, bvh)
    sorted_query(ctx, bvh, rays)
    out = torch.full_like(want, -7.0)
    graph = capture(ctx, lambda: vg.closest_hit(rays, bvh, out=out))
    sorted_query(ctx, bvh, random_rays(3_000_000, 4))
    for _ in range(2):
        out.fill_(-7.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))
    ctx.synchronize()


@pytest.mark.parametrize("extra", [-1, 1, 33, 160_000])
def test_host_queries_in_input_order_share_their_rays(soup_tree, extra):
    """Host-buffer queries in input order take their rays off the counter in each slot's
    scratch: chunks of more rays than the line where that starts."""
    ctx, bvh = soup_tree
    resident = torch.cuda.get_device_properties(0).multi_processor_count * 36
    n = 4 * (32 * resident + extra)   # one chunk is a quarter, a half and a quarter
    rays = random_rays(n, 5)
    want = vg.closest_hit(rays, bvh).cpu().numpy()
    got = vg.closest_hit(rays.cpu().numpy().view(vg.RAY).reshape(-1), bvh)
    assert got.tobytes() == want.tobytes()
