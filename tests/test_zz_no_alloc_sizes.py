"""gbrt_bvh_build_lbvh_noalloc takes every size up to its limit: sizes on both sides of the
bottom-up build's blocks of 256 leaves, where the share of its waiting lists in the fixed
array is tightest, equal the allocating build's tree."""
import pytest

import visionaray_gb300 as vg
from tests.test_zz_no_alloc import MAX_PRIMS, allocating_build, assert_same, noalloc_build
from visionaray_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 8191, 8193, 8448, 8449, 8703, 8704, 10000, 33000, 65281,
                               MAX_PRIMS - 1])
def test_noalloc_build_at_the_edges_of_its_blocks(n):
    ctx = vg.Context(0)
    tris = scenes.soup(n, seed=50 + n)
    assert_same(noalloc_build(ctx, tris), allocating_build(ctx, tris))


@pytest.mark.parametrize("n", [255, 256, 257, 767, 769])
def test_trees_at_the_edges_of_blocks_equal_the_oracle(oracle, n):
    tris = scenes.soup(n, seed=n)
    nodes, idx = allocating_build(vg.Context(0), tris)
    want = oracle.build_karras(tris)
    assert_same((nodes, idx), (want.nodes, idx))
    assert idx.tolist() == list(range(n))
