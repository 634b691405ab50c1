"""Queries answered by groups of lanes (one search for a warp's 32 kNN
queries, eight lanes for a triangle query) at the sizes where they can go
wrong, against the kernels that answer one query per thread."""
import numpy as np
import pytest
import torch

from cubql_b200 import workloads as W
from tests.helpers import boxes_np

pytestmark = pytest.mark.gpu


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


# sizes around a warp; radii from none to all; k around the list sizes; leaves of one and of many prims
@pytest.mark.parametrize("nq", [2, 31, 32, 33, 4097])
@pytest.mark.parametrize("k", [1, 4, 5, 16, 17, 32])
@pytest.mark.parametrize("n,leaf", [(1, 1), (3, 1), (40, 8), (20000, 1), (20000, 40)])
def test_knn_shared_search_equals_one_thread_per_query(bq, nq, k, n, leaf):
    pts, qs = W.uniform_points(n), W.uniform_points(nq, W.SEED_QUERIES, -0.1, 1.1)
    tp, tq = _cuda(pts), _cuda(qs)
    bvh = bq.cuda.radixBuilder(_cuda(boxes_np(pts)), bq.BuildConfig(makeLeafThreshold=leaf))
    for r in (float("inf"), 0.01, 0.0):
        a = bq.points.findKNN(bvh, tp, tq, k, maxSqrDist=r)
        b = bq.points.findKNN(bvh, tp, tq, k, maxSqrDist=r, qcfg=bq.query_config(reorder=0))
        assert _same(a, b), f"radius {r}"
    bvh.free()


def test_knn_shared_search_on_duplicates_and_clusters(bq):
    """Copies of points (ids decide) and tight clusters that uniform queries
    are far from (their warps give the shared search up)."""
    rng = np.random.default_rng(3)
    dup = np.repeat(W.uniform_points(300), 40, axis=0)
    clu = (W.uniform_points(8, 5)[rng.integers(0, 8, 30000)] + 0.002 * rng.standard_normal((30000, 3))).astype(np.float32)
    for pts, qs in ((dup, np.concatenate([dup[::7], W.uniform_points(3000, 9)])), (clu, W.uniform_points(20000, 9))):
        bvh = bq.gpuBuilder(_cuda(boxes_np(pts)), bq.BuildConfig(makeLeafThreshold=4))
        for k in (1, 8, 20):
            a = bq.points.findKNN(bvh, _cuda(pts), _cuda(qs), k)
            b = bq.points.findKNN(bvh, _cuda(pts), _cuda(qs), k, qcfg=bq.query_config(reorder=0))
            assert _same(a, b), f"k {k}"


def test_knn_shared_search_leaves_out_unusable_queries(bq):
    """NaN, infinite and overflowing queries share a warp with ordinary ones."""
    pts = W.uniform_points(5000)
    qs = W.uniform_points(500, 4)
    qs[::9, 0] = np.nan
    qs[4::9, 1] = np.inf
    qs[5::9, 2] = 1e30
    qs[6::9] = -np.inf
    bvh = bq.cuda.radixBuilder(_cuda(boxes_np(pts)))
    a = bq.points.findKNN(bvh, _cuda(pts), _cuda(qs), 6)
    b = bq.points.findKNN(bvh, _cuda(pts), _cuda(qs), 6, qcfg=bq.query_config(reorder=0))
    assert _same(a, b)


def test_batched_knn_warps_that_span_clouds(bq):
    """Clouds with fewer than 32 queries, empty ones and one of one point."""
    sizes, nqs = [1, 500, 0, 3, 4000, 17], [5, 40, 3, 1, 300, 31]
    pts, qs = W.uniform_points(sum(sizes)), W.uniform_points(sum(nqs), 6)
    off, qoff = np.concatenate([[0], np.cumsum(sizes)]), np.concatenate([[0], np.cumsum(nqs)])
    tp, tq = _cuda(pts), _cuda(qs)
    batch = bq.Batch(_cuda(boxes_np(pts)), _cuda(off))
    for k in (1, 8, 20):
        a = bq.batched_knn(batch, tp, _cuda(off), tq, _cuda(qoff), k)
        b = bq.batched_knn(batch, tp, _cuda(off), tq, _cuda(qoff), k, qcfg=bq.query_config(reorder=0))
        assert _same(a, b), f"k {k}"
