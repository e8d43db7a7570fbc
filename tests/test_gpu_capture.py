"""Calls on several streams, in captured graphs and with little memory: what a call enqueues
does not depend on what the context's other calls do to its memory later or at the same
time, and the memory that a context keeps to be faster is not asked for where there is none."""
import contextlib

import numpy as np
import pytest
import torch

import visionaray_gb300 as vg
from visionaray_gb300 import scenes
from visionaray_gb300.types import CAMERA, MATERIAL, MATTE, PT_PARAMS, PT_SORT_QUEUES

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
    with on_stream(ctx, stream), torch.cuda.graph(graph, stream=stream):
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


class Box:
    """A path-traced box with per-slot parameters."""

    def __init__(self, width, height):
        tris, mats, lights = scenes.box_scene(n_blobs=3, subdiv=3, seed=4)
        self.ctx = vg.Context(0)
        self.bvh = vg.lbvh_builder(self.ctx).build(vg.as_device_bytes(tris))
        self.scene = vg.PTScene(self.bvh, mats, lights)
        self.width, self.height = width, height
        rng = np.random.default_rng(1)
        self.albedo = torch.from_numpy(rng.uniform(0.3, 0.7, (len(mats), 3)).astype(np.float32)).cuda()
        self.emission = torch.from_numpy(np.ascontiguousarray(mats["color"])).cuda()
        self.adjoint = torch.from_numpy(rng.uniform(-1, 1, (height, width, 4)).astype(np.float32)).cuda()
        self.ctx.synchronize()

    def params(self, spp, depth, flags=0):
        return scenes.pt_params(self.width, self.height, spp, num_bounces=depth, frame_id=3, flags=flags,
                                ambient=(0.1, 0.2, 0.3))

    def frame(self, spp, depth, flags=0, out=None):
        out = torch.zeros((self.height, self.width, 4), device="cuda") if out is None else out
        return vg.pathtrace_frame(self.scene, scenes.box_camera(), self.params(spp, depth, flags), out)

    def backward(self, spp, depth, grads=None):
        grads = grads or (torch.zeros_like(self.albedo), torch.zeros_like(self.emission))
        return vg.pathtrace_backward(self.scene, scenes.box_camera(), self.params(spp, depth, 3), self.albedo,
                                     self.emission, self.adjoint, *grads)


def assert_close(got, want, scale=1.0):
    """FP32 atomics: the sums' rounding depends on the order (relative L2 1e-4)."""
    for g, w in zip(got, want):
        w = scale * w.double()
        assert float((g.double() - w).norm()) <= 1e-4 * float(w.norm())


def test_a_first_backward_call_can_be_captured():
    box = Box(64, 48)
    grads = torch.zeros_like(box.albedo), torch.zeros_like(box.emission)
    graph = capture(box.ctx, lambda: box.backward(5, 6, grads))
    want = box.backward(5, 6)
    box.frame(16, 8)             # the context's own buffers come and go
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert_close(grads, want, 3.0)
    box.ctx.synchronize()


def test_backward_calls_overlap_frames_and_each_other():
    box = Box(256, 200)
    image = box.frame(8, 5).clone()
    want = box.backward(8, 5)
    streams = [torch.cuda.Stream() for _ in range(3)]
    images = [torch.zeros_like(image) for _ in range(6)]
    grads = [(torch.zeros_like(box.albedo), torch.zeros_like(box.emission)) for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(6):
        with on_stream(box.ctx, streams[0]):
            box.frame(8, 5, out=images[k])
        for j in range(2):
            with on_stream(box.ctx, streams[1 + j]):
                box.backward(8, 5, grads[j])
    torch.cuda.synchronize()
    for got in images:
        assert torch.equal(got.view(torch.int32), image.view(torch.int32))
    for got in grads:
        assert_close(got, want, 6.0)
    box.ctx.synchronize()


@contextlib.contextmanager
def little_memory(free_bytes):
    """Leaves about free_bytes of the device's memory to others."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(max(1, torch.cuda.mem_get_info()[0] - free_bytes), dtype=torch.uint8, device="cuda")
    yield
    torch.cuda.synchronize()
    del hog
    torch.cuda.empty_cache()


def test_a_backward_call_with_little_memory():
    box = Box(512, 512)
    box.backward(1, 1)
    grads = torch.zeros_like(box.albedo), torch.zeros_like(box.emission)
    with little_memory(1 << 30):   # the passes would take 2.9 GB
        box.backward(16, 6, grads)
    assert_close(grads, box.backward(16, 6))
    box.ctx.synchronize()


@pytest.mark.parametrize("spp,depth,flags", [(1, 4, 0), (9, 4, 0), (1, 60, 0), (3, 4, PT_SORT_QUEUES)])
def test_a_frame_is_captured_after_another_of_its_size(spp, depth, flags):
    """Whatever its samples, bounces and queue order; the graph stays valid when later
    frames need larger buffers, captured or not."""
    box = Box(96, 70)
    box.frame(1, 4)
    out = torch.zeros((box.height, box.width, 4), device="cuda")
    graph = capture(box.ctx, lambda: box.frame(spp, depth, flags, out))
    want = box.frame(spp, depth, flags).clone()
    box.frame(300, 2)
    other = Box(96, 70)
    for k in range(3):
        out.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))
        more = torch.zeros_like(out)
        second = capture(box.ctx, lambda: box.frame(400 + k, 2, 0, more))
        second.replay()
        assert torch.equal(more.view(torch.int32), other.frame(400 + k, 2).view(torch.int32))
    box.ctx.synchronize()


def test_a_frame_with_little_memory():
    box, other = Box(1024, 513), Box(1024, 513)
    want = other.frame(9, 3).clone()
    other.ctx.synchronize()
    got = [torch.zeros_like(want) for _ in range(2)]
    with little_memory(300 << 20):   # the passes would take 500 MB
        for image in got:
            box.frame(9, 3, out=image)
    for image in got:
        assert torch.equal(image.view(torch.int32), want.view(torch.int32))
    box.ctx.synchronize()


def make_batch(side, spp, depth, scenes_n=2):
    parts = [scenes.soup(500 + 300 * k, seed=k, offset=0.05) for k in range(scenes_n)]
    batch = vg.Batch(np.concatenate([[0], np.cumsum([len(t) for t in parts])]), vg.Context(0))
    set_frames(batch, scenes_n, side, spp, depth)
    batch.build(vg.as_device_bytes(np.concatenate(parts)))
    batch.ctx.synchronize()
    return batch


def set_frames(batch, scenes_n, side, spp, depth):
    cams, params = np.zeros(scenes_n, CAMERA), np.zeros(scenes_n, PT_PARAMS)
    for k in range(scenes_n):
        cams[k] = scenes.box_camera((0.5, 0.5, 2.0), (0.5, 0.5, 0.5), (0.0, 1.0, 0.0), 50.0)
        params[k] = scenes.pt_params(side, side, spp, num_bounces=depth, frame_id=1, ambient=(1.0, 1.0, 1.0))
    mats = np.zeros(1, MATERIAL)
    mats["kind"], mats["color"], mats["scale"] = MATTE, 0.7, 1.0
    batch.set_frames(cams, params, mats)


def test_a_first_batch_frame_can_be_captured():
    """And its graph renders whatever frames are set later, as the frame itself does."""
    batch = make_batch(32, 2, 3)
    out = batch.new_images()
    graph = capture(batch.ctx, lambda: batch.pathtrace(out))
    for spp, depth in ((2, 3), (40, 5), (1, 1)):
        set_frames(batch, 2, 32, spp, depth)
        want = batch.pathtrace(batch.new_images())
        out.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))
    batch.ctx.synchronize()


def test_a_batch_frame_with_little_memory():
    batch, other = make_batch(1024, 2, 3), make_batch(1024, 2, 3)
    want, got = other.pathtrace(other.new_images()), batch.new_images()
    other.ctx.synchronize()
    with little_memory(300 << 20):   # the passes would take 800 MB
        batch.pathtrace(got)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert torch.equal(batch.pathtrace(batch.new_images()).view(torch.int32), want.view(torch.int32))
    batch.ctx.synchronize()


def test_captured_queries_and_frames_over_a_rebuilt_tree():
    """Replays after rebuilds and refits, among them one with triangles beyond what the quad
    nodes cover, give what the calls give then."""
    tris, mats, lights = scenes.box_scene(n_blobs=3, subdiv=3, seed=4)
    ctx = vg.Context(0)
    bvh = vg.lbvh_builder(ctx).build(vg.as_device_bytes(tris))
    scene = vg.PTScene(bvh, mats, lights)
    rays = random_rays(20000, 6)
    params = scenes.pt_params(48, 36, 1, num_bounces=4, frame_id=3)
    hits, image = torch.zeros((20000, 4), device="cuda"), torch.zeros((36, 48, 4), device="cuda")
    vg.pathtrace_frame(scene, scenes.box_camera(), params, image)

    def calls(hits, image):
        vg.closest_hit(rays, bvh, out=hits)
        vg.pathtrace_frame(scene, scenes.box_camera(), params, image)

    graph = capture(ctx, lambda: calls(hits, image))
    far = tris.copy()
    far["v1"][::40] = 3e38
    moved = tris.copy()
    moved["v1"] += np.float32(0.01)
    for geometry in (tris, far, moved):
        for change in (bvh.rebuild, bvh.refit):
            change(vg.as_device_bytes(geometry))
            want = torch.zeros_like(hits), torch.zeros_like(image)
            calls(*want)
            hits.fill_(-1.0)
            image.fill_(-1.0)
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(hits.view(torch.int32), want[0].view(torch.int32))
            assert torch.equal(image.view(torch.int32), want[1].view(torch.int32))
    ctx.synchronize()


@pytest.mark.parametrize("trees", [1, 2])
def test_a_tree_is_destroyed_during_a_relaxed_capture(trees):
    """A context's first tree and a later one: the capture goes on."""
    ctx = vg.Context(0)
    tris = vg.as_device_bytes(scenes.soup(5000, seed=1))
    built = [vg.lbvh_builder(ctx).build(tris) for _ in range(trees)]
    x = torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        x.add_(1)
        built[-1].close()
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 2.0


def test_a_destroyed_tree_is_not_reused_under_queued_queries():
    """Trees built into the memory of one whose queries are still queued."""
    ctx = vg.Context(0)
    tris = [scenes.soup(50000, seed=k, offset=0.05) for k in range(2)]
    d = [vg.as_device_bytes(t) for t in tris]
    keep = vg.lbvh_builder(ctx).build(d[0])
    rays = random_rays(400_000, 8)
    want = vg.closest_hit(rays, keep)
    out = [torch.zeros_like(want) for _ in range(4)]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for k in range(4):
        tree = vg.lbvh_builder(ctx).build(d[0])
        with on_stream(ctx, side):
            for _ in range(20):
                vg.closest_hit(rays, tree, out=out[k])
        tree.close()
        vg.lbvh_builder(ctx).build(d[1]).close()
    torch.cuda.synchronize()
    for got in out:
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    ctx.synchronize()


def test_a_tree_with_little_memory():
    """A tree without its quad nodes: built, rebuilt and refitted, traced as with them."""
    ctx = vg.Context(0)
    tris = scenes.heightfield(707, seed=1)
    d, rays = vg.as_device_bytes(tris), random_rays(100_000, 9)
    rays[:, 1] += 0.5
    rays[:, 4] = -0.5
    first = vg.lbvh_builder(ctx).build(d)
    want = vg.closest_hit(rays, first)
    nodes, idx = first.export_bvh2()
    first.close()
    with little_memory(150 << 20):   # the tree takes 184 MB, 120 without the quads
        tree = vg.lbvh_builder(ctx).build(d)
        got = [vg.closest_hit(rays, tree)]
        tree.rebuild(d)
        got.append(vg.closest_hit(rays, tree))
        tree.refit(d)
        got.append(vg.closest_hit(rays, tree))
    for hits in got:
        assert torch.equal(hits.view(torch.int32), want.view(torch.int32))
    again, indices = tree.export_bvh2()
    assert again.tobytes() == nodes.tobytes() and indices.tobytes() == idx.tobytes()
    assert int((want.view(torch.int32)[:, 0] != -1).sum()) > 10_000
    ctx.synchronize()


def test_what_the_pool_keeps_is_given_back():
    """A sorted query's scratch (134 MB) fits once the pool's freed trees are given back."""
    ctx = vg.Context(0)
    d, rays = vg.as_device_bytes(scenes.heightfield(707, seed=1)), random_rays(8_000_000, 9)
    keep = vg.lbvh_builder(ctx).build(d)
    want = vg.closest_hit(rays, keep)
    out = torch.zeros_like(want)
    vg.lbvh_builder(ctx).build(d).close()
    with little_memory(50 << 20):
        ctx.set_trace_flags(vg.Context.TRACE_SORT_RAYS)
        vg.closest_hit(rays, keep, out=out)
        ctx.synchronize()
    assert torch.equal(out.view(torch.int32), want.view(torch.int32))


def test_frames_after_a_replayed_graph():
    """A frame on the stream after a replay renders the replay's trees, which quad nodes made
    before it do not hold."""
    parts = [scenes.soup(800, seed=k, offset=0.05) for k in range(2)]
    batch = vg.Batch(np.array([0, 800]), vg.Context(0))
    set_frames(batch, 1, 32, 1, 3)
    d = [vg.as_device_bytes(t) for t in parts]
    want = []
    for k in range(2):
        batch.build(d[k])
        want.append(batch.pathtrace(batch.new_images()).clone())
    images = batch.new_images()
    batch.run_graph(d[0], images)
    assert torch.equal(images, want[0])
    batch.build(d[1])
    assert torch.equal(batch.pathtrace(batch.new_images()), want[1])
    batch.run_graph(d[0], images)
    assert torch.equal(images, want[0])
    assert torch.equal(batch.pathtrace(batch.new_images()), want[0])
    assert not torch.equal(want[0], want[1])
    batch.ctx.synchronize()
