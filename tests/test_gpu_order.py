"""The Morton order of a build, alone and in a batch, at the edges of its sizes: one block holds up to 8,192
triangles (1, 2, 4 or 8 per thread), and the radix sort scans its digit table inside the
scatter for up to 256 tiles of 4,096 keys.  Codes and trees equal the oracle's, which sorts
with std::stable_sort; equal codes keep their input order, and triangles that are not
finite stay out of the centroid bounds."""
import numpy as np
import pytest

import visionaray_gb300 as vg
from visionaray_gb300 import scenes

pytestmark = pytest.mark.gpu


def make(n, kind):
    tris = scenes.soup(n, seed=n + 3)
    if kind == "few":   # 27 codes: long runs of equal keys
        tris["v1"] = np.round(tris["v1"] * 2) / 2
    elif kind == "flat":
        tris["v1"][:, 1] = 0.25
        tris["e1"][:, 1] = tris["e2"][:, 1] = 0.0
    return tris


def check(bvh, tris, oracle):
    assert np.array_equal(bvh.morton_codes(), oracle.morton_codes(tris))
    nodes, _ = bvh.export_bvh2()
    want = oracle.build_karras(tris)
    assert np.array_equal(nodes["first"], want.nodes["first"])
    assert (nodes["bbox_min"] == want.nodes["bbox_min"]).all() and (nodes["bbox_max"] == want.nodes["bbox_max"]).all()


@pytest.mark.parametrize("kind", ["soup", "few", "flat"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 256, 257, 287, 1023, 1024, 1025, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 12289])
def test_one_block_and_few_tiles(oracle, n, kind):
    tris = make(n, kind)
    d = vg.as_device_bytes(tris)
    bvh = vg.lbvh_builder().build(d)
    check(bvh, tris, oracle)
    bvh.rebuild(d)
    check(bvh, tris, oracle)


@pytest.mark.parametrize("n", [256 * 4096, 256 * 4096 + 1])
def test_table_scan_inside_and_outside_the_scatter(oracle, n):
    tris = make(n, "few")
    check(vg.lbvh_builder().build(vg.as_device_bytes(tris)), tris, oracle)


@pytest.mark.parametrize("n", [700, 3000, 9000])
def test_triangles_that_are_not_finite(oracle, n):
    tris = make(n, "soup")
    tris["v1"][n // 3] = (np.inf, 0, 0)
    tris["v1"][n // 2] = (0, -np.inf, 0)
    tris["v1"][n - 1] = (0, 0, np.nan)
    bvh = vg.lbvh_builder().build(vg.as_device_bytes(tris))
    assert np.array_equal(bvh.morton_codes(), oracle.morton_codes(tris))


@pytest.mark.parametrize("sizes", [[256, 256], [31, 1, 224, 1, 255], [255, 0, 2, 512, 33], [1] * 70, [8192, 3, 300]])
def test_batches_across_runs_of_triangles(oracle, sizes):
    # a warp folds the centroid bounds of 256 triangles, 32 at a time
    parts = [make(n, "soup") for n in sizes]
    for k, p in enumerate(parts):
        p["v1"] += np.float32(k)
    batch = vg.Batch(np.concatenate([[0], np.cumsum(sizes)]))
    batch.build(vg.as_device_bytes(np.concatenate(parts)))
    for s, tris in enumerate(parts):
        if not len(tris):
            continue
        nodes, _ = batch.export_bvh2(s)
        want = oracle.build_karras(tris)
        assert np.array_equal(nodes["first"], want.nodes["first"])
        assert (nodes["bbox_min"] == want.nodes["bbox_min"]).all()
        assert (nodes["bbox_max"] == want.nodes["bbox_max"]).all()
