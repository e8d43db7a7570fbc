"""The wavefront frame's passes of several samples per pixel: the image equals the
megakernel's bit for bit (one thread per pixel, its samples in order) for one pixel, odd
sizes, sample counts that split evenly and unevenly over passes (2^22 paths each), and
blended frames."""
import numpy as np
import pytest
import torch

import visionaray_gb300 as vg
from visionaray_gb300 import scenes
from visionaray_gb300.types import PT_MEGAKERNEL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp,depth", [
    (1, 1, 1, 1), (1, 1, 70, 4), (33, 7, 3, 5), (64, 64, 16, 0),
    (1024, 513, 9, 2),     # two passes, of 5 and 4 samples
    (2049, 2048, 2, 1),    # more than 2^22 pixels: one sample per pass
])
def test_passes_equal_the_megakernel(width, height, spp, depth):
    tris, mats, lights = scenes.box_scene(n_blobs=3, subdiv=3, seed=4)
    bvh = vg.lbvh_builder().build(vg.as_device_bytes(tris))
    scene = vg.PTScene(bvh, mats, lights)
    images = []
    for flags in (0, PT_MEGAKERNEL):
        accum = torch.full((height, width, 4), 0.25, dtype=torch.float32, device="cuda")
        for frame, (sf, df) in enumerate(((1.0, 0.0), (0.5, 0.5))):
            params = scenes.pt_params(width, height, spp, num_bounces=depth, frame_id=frame, sfactor=sf, dfactor=df,
                                      ambient=(0.1, 0.2, 0.3), flags=flags)
            vg.pathtrace_frame(scene, scenes.box_camera(), params, accum)
        bvh.ctx.synchronize()
        images.append(accum.cpu().numpy())
    assert np.isfinite(images[1]).all()
    assert images[0].tobytes() == images[1].tobytes()


@pytest.mark.parametrize("width,height,spp,depth", [(1, 1, 1, 1), (33, 7, 3, 5), (40, 30, 5, 16),
                                                    (1024, 513, 9, 2)])   # the last: several passes
def test_replay_passes_sum_to_the_gradient(width, height, spp, depth):
    """The gradient is linear in the image adjoint: the adjoint's left and right halves,
    alone, add up to it, whatever the passes (FP32 atomics: relative L2 1e-4).  The values
    are pinned by test_gpu_adjoint.py."""
    tris, mats, lights = scenes.box_scene(n_blobs=3, subdiv=1, seed=4)
    bvh = vg.lbvh_builder().build(vg.as_device_bytes(tris))
    scene = vg.PTScene(bvh, mats, lights)
    flags = 3   # shadow-range fix, no roulette
    params = scenes.pt_params(width, height, spp, num_bounces=depth, frame_id=5, flags=flags)
    rng = np.random.default_rng(1)
    albedo = torch.from_numpy(rng.uniform(0.3, 0.7, (len(mats), 3)).astype(np.float32)).cuda()
    emission = torch.from_numpy(np.ascontiguousarray(mats["color"])).cuda()
    adj = torch.from_numpy(rng.uniform(-1, 1, (height, width, 4)).astype(np.float32)).cuda()
    cam = scenes.box_camera()
    ga, ge = vg.pathtrace_backward(scene, cam, params, albedo, emission, adj)
    half = adj.clone()
    half[:, width // 2:] = 0
    pa, pe = vg.pathtrace_backward(scene, cam, params, albedo, emission, half)
    pa, pe = vg.pathtrace_backward(scene, cam, params, albedo, emission, adj - half, pa, pe)
    bvh.ctx.synchronize()
    for got, want in ((ga, pa), (ge, pe)):
        n = float(want.double().norm())
        assert float((got.double() - want.double()).norm()) <= 1e-4 * n + 1e-12
    assert float(ga.abs().sum()) > 0 or width * height == 1
