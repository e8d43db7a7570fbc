"""The bottom-up LBVH build at the edges of its blocks (512 leaves): trees equal the
oracle's restatement of the reference GPU builder, with distinct codes, with one code for
all triangles (the index alone decides every split) and with few codes; rebuilds and
refits run the same kernels on used scratch memory; batches put several scenes, empty and
one-triangle ones among them, into one block and across blocks."""
import numpy as np
import pytest

import visionaray_gb300 as vg
from visionaray_gb300 import scenes

pytestmark = pytest.mark.gpu


def make(n, kind):
    tris = scenes.soup(n, seed=n + 7)
    if kind == "same":
        tris[["v1", "e1", "e2"]] = tris[["v1", "e1", "e2"]][0]
    elif kind == "few":
        tris["v1"] = np.round(tris["v1"] * 2) / 2
        tris["e1"], tris["e2"] = (0.01, 0, 0), (0, 0.01, 0)
    return tris


def check(bvh, tris, oracle):
    nodes, idx = bvh.export_bvh2()
    want = oracle.build_karras(tris)
    assert np.array_equal(nodes["first"], want.nodes["first"])
    assert np.array_equal(nodes["num_prims"], want.nodes["num_prims"])
    assert (nodes["bbox_min"] == want.nodes["bbox_min"]).all() and (nodes["bbox_max"] == want.nodes["bbox_max"]).all()
    assert np.array_equal(idx, np.arange(len(tris)))


@pytest.mark.parametrize("kind", ["soup", "same", "few"])
@pytest.mark.parametrize("n", [2, 3, 511, 512, 513, 1024, 1025, 5003, 70001])
def test_trees_at_block_edges(oracle, n, kind):
    if kind == "same" and n > 5003:
        pytest.skip("covered by the smaller sizes")
    tris = make(n, kind)
    d = vg.as_device_bytes(tris)
    bvh = vg.lbvh_builder().build(d)
    check(bvh, tris, oracle)
    bvh.rebuild(d)
    check(bvh, tris, oracle)
    bvh.refit(d)
    check(bvh, tris, oracle)


@pytest.mark.parametrize("sizes", [[0, 1, 2, 509, 0, 1], [511, 1, 512, 513], [1], [3, 1021, 1, 700]])
def test_batches_at_block_edges(oracle, sizes):
    parts = [scenes.soup(n, seed=40 + k) for k, n in enumerate(sizes)]
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    batch = vg.Batch(offsets)
    d = vg.as_device_bytes(np.concatenate(parts))
    for _ in range(2):
        batch.build(d)
        for s, tris in enumerate(parts):
            if not len(tris):
                continue
            nodes, idx = batch.export_bvh2(s)
            want = oracle.build_karras(tris)
            assert np.array_equal(nodes["first"], want.nodes["first"])
            assert (nodes["bbox_min"] == want.nodes["bbox_min"]).all()
            assert (nodes["bbox_max"] == want.nodes["bbox_max"]).all()
            assert np.array_equal(idx, np.arange(len(tris)))
