"""The clustering steps of the PLOC build against a plain restatement, at the edges of its
tiles (608 clusters), of a group of tiles (64), of the block that finishes (2,048 clusters,
two per thread above 1,024) and of the smallest trees.  Coordinates are multiples of 2^-10
below 2, so every box area is exact in float32 whatever the order of its operations, and
ties between neighbours are frequent."""
import numpy as np
import pytest

import visionaray_gb300 as vg

pytestmark = pytest.mark.gpu

RADIUS = 16


def make(n):
    rng = np.random.default_rng(n)
    tris = np.zeros(n, vg.TRIANGLE)
    tris["v1"] = rng.integers(0, 1024, (n, 3)) / 1024
    tris["e1"] = rng.integers(-16, 17, (n, 3)) / 1024
    tris["e2"] = rng.integers(-16, 17, (n, 3)) / 1024
    tris["prim_id"] = np.arange(n)
    return tris


def cluster(tris, order):
    """(lo, hi, left, right, root): boxes and children of the pairs, leaves as ~position."""
    v = np.stack([tris["v1"], tris["v1"] + tris["e1"], tris["v1"] + tris["e2"]])[:, order]
    lo, hi, ids = v.min(0), v.max(0), ~np.arange(len(tris))
    pairs = []
    while len(ids) > 1:
        m = len(ids)
        best, nearest = np.full(m, np.inf), np.full(m, -1)
        for d in list(range(-RADIUS, 0)) + list(range(1, RADIUS + 1)):
            i = np.arange(max(0, -d), min(m, m - d))
            e = np.maximum(hi[i], hi[i + d]) - np.minimum(lo[i], lo[i + d])
            area = e[:, 0] * e[:, 1] + e[:, 1] * e[:, 2] + e[:, 2] * e[:, 0]
            i = i[area < best[i]]
            area = area[area < best[np.arange(max(0, -d), min(m, m - d))]]
            best[i], nearest[i] = area, i + d
        i = np.arange(m)
        mutual = nearest[nearest] == i
        merges, gone = mutual & (i < nearest), mutual & (i > nearest)
        a, b = i[merges], nearest[merges]
        made = len(pairs) + np.arange(len(a))
        pairs += [(lo[x].copy(), hi[x].copy(), ids[x], lo[y].copy(), hi[y].copy(), ids[y]) for x, y in zip(a, b)]
        lo[a], hi[a] = np.minimum(lo[a], lo[b]), np.maximum(hi[a], hi[b])
        ids[a] = made
        lo, hi, ids = lo[~gone], hi[~gone], ids[~gone]
    return pairs, lo[0], hi[0], ids[0]


@pytest.mark.parametrize("n", [2, 3, 33, 1024, 1025, 2047, 2048, 2049, 2432, 2433, 64 * 608, 64 * 608 + 1, 90001])
def test_trees_equal_the_restated_clustering(oracle, n):
    tris = make(n)
    bvh = vg.ploc_builder().build(vg.as_device_bytes(tris))
    nodes, _ = bvh.export_bvh2()
    order = np.argsort(oracle.morton_codes(tris), kind="stable")
    pairs, lo, hi, root = cluster(tris, order)
    assert len(pairs) == n - 1 and root == n - 2
    assert (nodes["bbox_min"][0] == lo).all() and (nodes["bbox_max"][0] == hi).all()
    # breadth first, the two children of a node adjacent
    queue, at = [root], 1
    for node in queue:
        alo, ahi, a, blo, bhi, b = pairs[node]
        for clo, chi, c in ((alo, ahi, a), (blo, bhi, b)):
            got = nodes[at]
            assert (got["bbox_min"] == clo).all() and (got["bbox_max"] == chi).all()
            assert got["num_prims"] == (1 if c < 0 else 0)
            if c < 0:
                assert got["first"] == order[~c]
            else:
                queue.append(c)
            at += 1
