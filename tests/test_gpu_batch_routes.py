"""Batch frames go through the wavefront queues or the persistent kernel by the number of
pixels, samples, bounces and triangles: on both sides of each line the images equal those
of the persistent kernel (its stack of 32 entries asks for it), for any number of bounces."""
import numpy as np
import pytest
import torch

import visionaray_gb300 as vg
from visionaray_gb300 import scenes
from visionaray_gb300.types import CAMERA, MATERIAL, MATTE, PT_PARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,side,spps,bounces", [
    ([300, 300], 24, [1, 1], [8, 8]), ([300, 300], 24, [1, 1], [9, 2]), ([300, 300], 24, [2, 1], [16, 3]),
    ([300, 300], 24, [2, 1], [3, 17]), ([300], 16, [1], [1000]), ([300], 16, [3], [0xFFFFFFFF]),
    ([128, 128], 32, [1, 1], [3, 3]), ([127, 128], 32, [1, 1], [3, 3]), ([20, 1, 0, 30], 32, [4, 1, 2, 5], [4, 4, 4, 4]),
    ([2048], 725, [1], [1]), ([2047], 725, [1], [1]), ([1024], 725, [1], [2]), ([1023], 725, [1], [2]),
    ([256], 725, [1], [12]), ([255], 725, [2], [3]), ([256], 725, [1], [13]),
    ([300, 300], 24, [1, 70], [3, 3]),
])
def test_both_routes_give_the_same_images(counts, side, spps, bounces):
    n = len(counts)
    parts = [scenes.soup(max(c, 1), seed=k + 1, offset=0.05)[:c] for k, c in enumerate(counts)]
    batch = vg.Batch(np.concatenate([[0], np.cumsum(counts)]), vg.Context(0))
    cams, params = np.zeros(n, CAMERA), np.zeros(n, PT_PARAMS)
    for k in range(n):
        cams[k] = scenes.box_camera((0.5, 0.5, 2.0), (0.5, 0.5, 0.5), (0.0, 1.0, 0.0), 50.0)
        params[k] = scenes.pt_params(side, side, spps[k], num_bounces=bounces[k], frame_id=1, ambient=(1.0, 1.0, 1.0))
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
    # the sky is seen from the second bounce on
    assert bounces == [1] or float(images[1][..., :3].abs().sum()) > 0
