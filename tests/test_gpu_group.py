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


def _phases(bq, call):
    """(result, names of the phases that ran)"""
    with bq.profile() as prof:
        r = call()
    return r, set(prof.table)


def _knn_both_ways(bq, bvh, tp, tq, k, shared, **kw):
    """The search as it is chosen (and that it is the shared one, or not), and with a thread a query in the given
    order; they have to be the same."""
    a, ran = _phases(bq, lambda: bq.points.findKNN(bvh, tp, tq, k, **kw))
    b, ran0 = _phases(bq, lambda: bq.points.findKNN(bvh, tp, tq, k, qcfg=bq.query_config(reorder=0), **kw))
    assert "query.knn_shared" not in ran0 and ("query.knn_shared" in ran) == shared, (ran, ran0)
    assert _same(a, b), (k, kw)
    return a


# batches whose last warp is whole, one query, all but one; radii from none to all; k around the list sizes; leaves of
# one and of many prims
@pytest.mark.parametrize("extra", [0, 1, 31, 33])
@pytest.mark.parametrize("k", [2, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n,leaf", [(32, 1), (1024, 1), (1024, 40), (3000, 8)])
def test_knn_shared_search_equals_one_thread_per_query(bq, extra, k, n, leaf):
    nq = (24064 if k <= 4 else 6016 if k <= 16 else 1504) + extra
    pts, qs = W.uniform_points(n), W.uniform_points(nq, W.SEED_QUERIES, -0.1, 1.1)
    tp, tq = _cuda(pts), _cuda(qs)
    bvh = bq.cuda.radixBuilder(_cuda(boxes_np(pts)), bq.BuildConfig(makeLeafThreshold=leaf))
    for r in (float("inf"), 0.3, 0.01, 0.0):
        _knn_both_ways(bq, bvh, tp, tq, k, n >= 1024 or k > 4, maxSqrDist=r)
    bvh.free()


# either side of each line that decides between the shared search and a thread a query
@pytest.mark.parametrize("n,nq,k,shared", [
    (8192, 32768, 1, True), (8192, 32767, 1, False), (8191, 40000, 1, False),
    (16384, 32768, 4, True), (16384, 32767, 4, False), (20000, 39999, 2, False), (1000, 8000, 3, True),
    (1000, 7999, 3, False), (256, 5000, 2, True), (255, 5000, 4, False),
    (6000, 6000, 5, True), (6000, 5999, 16, False), (1 << 20, 1 << 19, 9, True), (1 << 20, (1 << 19) - 1, 9, False),
    (32, 5000, 16, True), (31, 5000, 16, False), (4000, 2000, 17, True), (4000, 1999, 32, False),
    (2000, 4096, 8, True), (2000, 4095, 8, False), (5000, 9000, 33, False)])
def test_knn_where_the_shared_search_begins(bq, n, nq, k, shared):
    pts = W.uniform_points(n)
    bvh = bq.cuda.radixBuilder(_cuda(boxes_np(pts)))
    _knn_both_ways(bq, bvh, _cuda(pts), _cuda(W.uniform_points(nq, 3)), k, shared)
    bvh.free()


@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("k", [1, 2, 3, 5, 6])
@pytest.mark.parametrize("leaf", [1, 8])
def test_knn_plain_and_in_step_match_oracle(bq, oracle, tie, k, leaf):
    """A thread a query, on its own (short lists over short leaves) and with
    the warp in step."""
    pts, qs = W.uniform_points(5000), W.uniform_points(333, 5, -0.1, 1.1)
    bvh = bq.cuda.radixBuilder(_cuda(boxes_np(pts)), bq.BuildConfig(makeLeafThreshold=leaf))
    assert (bvh.numPrims // 2 >= bvh.numNodes) == (leaf == 8)
    n, pr = bvh.to_host()
    want = oracle.knn(n, pr, pts, qs, k, tie_mode=tie)
    cfg = bq.query_config(tieMode=tie, reorder=0)
    got = bq.points.findKNN(bvh, _cuda(pts), _cuda(qs), k, qcfg=cfg)
    for a, b in zip(got, want):
        assert np.array_equal(a.cpu().numpy(), b)
    many = _cuda(np.resize(qs, (65536 + 33, 3)))  # the size from which lists of three to five are plain
    for nq in (65535, 65536, len(many)):
        for a, b in zip(bq.points.findKNN(bvh, _cuda(pts), many[:nq], k, qcfg=cfg), got):
            assert np.array_equal(a.cpu().numpy(), np.resize(b.cpu().numpy(), (nq,) + b.shape[1:]))


def test_knn_shared_search_on_duplicates_and_clusters(bq):
    """Copies of points (ids decide); tight clusters, planes and lines that
    the queries are far from, and queries far outside: their warps give the
    shared search up."""
    rng = np.random.default_rng(3)
    u = W.uniform_points(20000, 9)
    dup = np.repeat(W.uniform_points(300), 40, axis=0)
    clu = W.uniform_points(8, 5)[rng.integers(0, 8, 20000)]
    clu = (clu + 0.002 * rng.standard_normal((20000, 3))).astype(np.float32)
    for pts, qs in ((dup, np.concatenate([dup[::2], W.uniform_points(9000, 9)])), (clu, u),
                    (u * np.float32([1, 1, 0]), u), (u * np.float32([1, 0, 0]), u), (u, 3 * u - 1),
                    (np.repeat(u[:1], 40, axis=0), u)):
        bvh = bq.gpuBuilder(_cuda(boxes_np(pts)), bq.BuildConfig(makeLeafThreshold=4))
        for k in (5, 16, 20):
            _knn_both_ways(bq, bvh, _cuda(pts), _cuda(qs), k, True)
        bvh.free()


def test_knn_shared_search_leaves_out_unusable_queries(bq):
    """NaN, infinite and overflowing queries share a warp with ordinary ones."""
    pts = W.uniform_points(5000)
    qs = W.uniform_points(6000, 4)
    qs[::9, 0] = np.nan
    qs[4::9, 1] = np.inf
    qs[5::9, 2] = 1e30
    qs[6::9] = -np.inf
    bvh = bq.cuda.radixBuilder(_cuda(boxes_np(pts)))
    for k in (6, 20):
        ids, _, found = _knn_both_ways(bq, bvh, _cuda(pts), _cuda(qs), k, True)
        ok = torch.from_numpy(np.abs(qs).max(1) <= 1).cuda()
        assert bool((found[ok] == k).all()) and bool((ids[~ok] == -1).all())


def test_batched_knn_warps_that_span_clouds(bq):
    """Clouds with fewer than 32 queries, empty ones, one of one point, some
    with enough queries a prim to share the search and some without."""
    sizes, nqs = [1, 500, 0, 3, 400, 17, 60, 32, 2000, 33], [5, 40, 3, 1, 1000, 31, 77, 45, 1999, 700]
    pts, qs = W.uniform_points(sum(sizes)), W.uniform_points(sum(nqs), 6)
    qs[::50] = np.nan
    off, qoff = np.concatenate([[0], np.cumsum(sizes)]), np.concatenate([[0], np.cumsum(nqs)])
    tp, tq = _cuda(pts), _cuda(qs)
    batch = bq.Batch(_cuda(boxes_np(pts)), _cuda(off))
    for k in (1, 4, 5, 8, 16, 20, 32, 33):
        for r in (float("inf"), 0.01):
            a, ran = _phases(bq, lambda: bq.batched_knn(batch, tp, _cuda(off), tq, _cuda(qoff), k, maxSqrDist=r))
            b = bq.batched_knn(batch, tp, _cuda(off), tq, _cuda(qoff), k, maxSqrDist=r, qcfg=bq.query_config(reorder=0))
            assert ("batch.knn_shared" in ran) == (4 < k <= 32)
            assert _same(a, b), f"k {k} radius {r}"


def _mesh(level, n=None):
    verts, tris = W.icosphere(level)
    return _cuda(verts), _cuda(tris[:n])


# sizes around a group of eight and a block's sixteen groups
@pytest.mark.parametrize("nq", [1, 7, 8, 9, 129])
@pytest.mark.parametrize("n", [1, 2, 80, 20480])
def test_triangle_groups_do_not_depend_on_batch_or_tree(bq, n, nq):
    """A query's answer is the same alone, among many (corners copied into
    leaf order or fetched through the index), on a tree of another shape and
    in a batch; and no farther than under the reference's rule."""
    tv, tt = _mesh(5, n)
    qs = _cuda(W.uniform_points(40000, W.SEED_QUERIES, -1.5, 1.5))  # enough to be sorted, too few for threads first
    boxes = bq.triangles.boxes(tt, tv)
    bvh, sah = bq.cuda.radixBuilder(boxes), bq.cuda.sahBuilder(boxes, bq.BuildConfig(makeLeafThreshold=3))
    for r in (float("inf"), 0.05):
        many = bq.triangles.findClosest(bvh, tt, tv, qs, maxSqrDist=r)
        few = bq.triangles.findClosest(bvh, tt, tv, qs[:nq], maxSqrDist=r)
        assert _same(few, [x[:nq] for x in many])
        assert _same(bq.triangles.findClosest(sah, tt, tv, qs[:nq], maxSqrDist=r)[:2], few[:2])
        ref = bq.triangles.findClosest(bvh, tt, tv, qs, maxSqrDist=r, qcfg=bq.query_config(tieMode=1))
        assert bool((many[1] <= ref[1]).all()) and float((many[1] == ref[1]).float().mean()) > 0.99
        off, qoff = _cuda(np.array([0, n, n])), _cuda(np.array([0, 40000, 40000]))
        batch = bq.Batch(boxes, off)
        for reorder in (0, 1):
            got = bq.batched_tri_closest(batch, tt, tv, qs, qoff, maxSqrDist=r, qcfg=bq.query_config(reorder=reorder))
            assert _same(got, many), f"batch, reorder {reorder}"


def _corners(n, rng):
    """n fans of three unit triangles, each around a corner that is extreme in its mesh's box."""
    verts, tris = [], []
    for _ in range(n):
        a = rng.uniform(0, 2 * np.pi) + np.arange(3) * 2 * np.pi / 3 + rng.uniform(-0.4, 0.4, 3)
        apex, b = rng.uniform(-3, 3, 3), len(verts)
        verts += [apex] + list(apex + np.stack([np.cos(a), np.sin(a), -rng.uniform(0.2, 1.0, 3)], 1))
        tris += [[b, b + 1, b + 2], [b, b + 2, b + 3], [b, b + 3, b + 1]]
    return np.array(verts, np.float32), np.array(tris, np.int32)


def _near_queries(verts, tris, nq, rng):
    """Queries 0.001 to 0.03 from random points of the triangles, most of them near a corner."""
    w = rng.random((nq, 3)) ** 3
    p = (verts[tris[rng.integers(0, len(tris), nq)]] * (w / w.sum(1, keepdims=True))[:, :, None]).sum(1)
    u = rng.standard_normal((nq, 3))
    return (p + u / np.linalg.norm(u, axis=1, keepdims=True) * rng.uniform(0.001, 0.03, (nq, 1))).astype(np.float32)


@pytest.mark.parametrize("fans", [1, 4, 64])
def test_triangle_rounded_below_its_box_does_not_depend_on_batch_or_tree(bq, fans):
    """Near unit triangles a computed distance can lie below the distance of
    the triangle's own box; the answer still is a function of query and mesh."""
    rng = np.random.default_rng(fans)
    verts, tris = _corners(fans, rng)
    tv, tt, tq = _cuda(verts), _cuda(tris), _cuda(_near_queries(verts, tris, 1_000_000, rng))
    boxes = bq.triangles.boxes(tt, tv)
    bvh, sah = bq.cuda.radixBuilder(boxes), bq.cuda.sahBuilder(boxes, bq.BuildConfig(makeLeafThreshold=3))
    many = bq.triangles.findClosest(bvh, tt, tv, tq)
    few = [torch.cat(x) for x in zip(*[bq.triangles.findClosest(bvh, tt, tv, q) for q in tq.split(20_000)])]
    assert _same(few, many), "split"
    assert _same(bq.triangles.findClosest(bvh, tt, tv, tq, qcfg=bq.query_config(reorder=0)), many), "as given"
    assert _same(bq.triangles.findClosest(sah, tt, tv, tq), many), "another tree"
    batch, off = bq.Batch(boxes, _cuda(np.array([0, len(tris)]))), _cuda(np.array([0, len(tq)]))
    assert _same(bq.batched_tri_closest(batch, tt, tv, tq, off), many), "batch"
    assert bool((many[1] <= bq.triangles.findClosest(bvh, tt, tv, tq, qcfg=bq.query_config(tieMode=1))[1]).all())


def test_triangle_slivers_do_not_depend_on_batch_or_tree(bq):
    """The plane of a sliver is known to few digits: its computed distance
    can be far from its box's, and it is still met in every order."""
    rng = np.random.default_rng(9)
    c = rng.uniform(-1, 1, (3000, 1, 3))
    e = rng.standard_normal((3000, 1, 3)) * 0.3
    v = c + e * np.array([0.0, 0.5, 1.0])[None, :, None]  # three points on a line, moved by 1e-8 to 1e-2
    v += rng.standard_normal((3000, 3, 3)) * 10.0 ** rng.uniform(-8, -2, (3000, 1, 1))
    verts, tris = v.reshape(-1, 3).astype(np.float32), np.arange(9000, dtype=np.int32).reshape(-1, 3)
    tv, tt, tq = _cuda(verts), _cuda(tris), _cuda(_near_queries(verts, tris, 400_000, rng))
    boxes = bq.triangles.boxes(tt, tv)
    bvh, sah = bq.cuda.radixBuilder(boxes), bq.cuda.sahBuilder(boxes, bq.BuildConfig(makeLeafThreshold=3))
    many = bq.triangles.findClosest(bvh, tt, tv, tq)
    few = [torch.cat(x) for x in zip(*[bq.triangles.findClosest(bvh, tt, tv, q) for q in tq.split(20_000)])]
    assert bool((many[0] >= 0).all())
    assert _same(few, many), "split"
    assert _same(bq.triangles.findClosest(sah, tt, tv, tq), many), "another tree"


# the smallest batch a thread a query goes first in, and the next number of rounds; the largest tree and the one after
@pytest.mark.parametrize("nq", [65535, 65536, 262143, 262144 + 33])
@pytest.mark.parametrize("n", [1, 1280, 131072, 131073])
def test_triangle_threads_before_groups(bq, n, nq):
    """Answered by threads, by groups after them, or by groups alone: the same."""
    tv, tt = _mesh(7 if n > 1280 else 3, n)
    g = np.random.default_rng(n)
    qs = W.uniform_points(nq, 4, -1.5, 1.5)
    c = tv.cpu().numpy()[tt.cpu().numpy()[g.integers(0, n, nq // 2)]].mean(1)
    qs[::2][:nq // 2] = c + 0.01 * g.standard_normal(c.shape)  # half of them near the surface
    qs[7::501] = np.nan
    tq, bvh = _cuda(qs), bq.cuda.radixBuilder(bq.triangles.boxes(tt, tv))
    for r in (float("inf"), 0.01):
        many = bq.triangles.findClosest(bvh, tt, tv, tq, maxSqrDist=r)
        few = [bq.triangles.findClosest(bvh, tt, tv, q, maxSqrDist=r) for q in tq.split(30_000)]
        few = [torch.cat(x) for x in zip(*few)]
        assert _same(few, many), f"radius {r}"


@pytest.mark.parametrize("leaf", [1, 40])
@pytest.mark.parametrize("builder", ["gpuBuilder", "sahBuilder", "radixBuilder"])
def test_triangles_without_a_box_are_not_read(bq, builder, leaf):
    """Removed triangles (an empty box, indices that point nowhere) are listed
    after the others by some builders; a tree handed in need not say how many
    prims it has.  The corners of neither are copied."""
    tv, tt = _mesh(4)
    tq = _cuda(W.uniform_points(3000, 4, -1.5, 1.5))
    boxes = bq.triangles.boxes(tt, tv)
    build = bq.gpuBuilder if builder == "gpuBuilder" else getattr(bq.cuda, builder)
    bvh = build(boxes, bq.BuildConfig(makeLeafThreshold=leaf))
    want = bq.triangles.findClosest(bvh, tt, tv, tq)
    n = bvh.c.numPrims
    for fewer in (n - 7, 1, 0):
        bvh.c.numPrims = fewer
        assert _same(bq.triangles.findClosest(bvh, tt, tv, tq), want), fewer
    bvh.c.numPrims = n
    bvh.free()
    gone = torch.rand(len(tt), generator=torch.Generator().manual_seed(1)) < 0.3
    tt2 = tt.clone()
    tt2[gone.cuda()] = -(1 << 30)
    empty = boxes.clone()
    empty[gone.cuda()] = torch.tensor([np.inf] * 3 + [-np.inf] * 3, device="cuda", dtype=torch.float32)
    bvh = build(empty, bq.BuildConfig(makeLeafThreshold=leaf))
    kept = build(boxes[~gone.cuda()].contiguous(), bq.BuildConfig(makeLeafThreshold=leaf))
    ids, d, p = bq.triangles.findClosest(bvh, tt2, tv, tq)
    wi, wd, wp = bq.triangles.findClosest(kept, tt[~gone.cuda()].contiguous(), tv, tq)
    assert _same((d, p), (wd, wp)) and torch.equal(ids.cpu(), torch.nonzero(~gone)[:, 0].int()[wi.cpu().long()])


@pytest.mark.parametrize("nq", [300_000, 1_100_000])
def test_batched_triangles_sorted_and_seeded(bq, oracle, nq):
    """Meshes too large for a thread a query (its groups start from their
    neighbour's triangle, and drop it where the mesh changes), small ones and
    empty ones, in one sorted batch: as their queries in small calls, and as
    an FP64 brute force."""
    rng = np.random.default_rng(nq)
    meshes = [W.icosphere(3), None, W.icosphere(7), W.icosphere(1), None, W.icosphere(7, amp=0.2), W.icosphere(4)]
    verts, tris, sizes, base = [], [], [], 0
    for m in meshes:
        if m is not None:
            verts.append(m[0])
            tris.append(m[1] + base)
            base += len(m[0])
        sizes.append(0 if m is None else len(m[1]))
    verts, tris = np.concatenate(verts), np.concatenate(tris).astype(np.int32)
    cuts = np.sort(rng.integers(0, nq, len(meshes) - 1))
    off, qoff = np.concatenate([[0], np.cumsum(sizes)]), np.concatenate([[0], cuts, [nq]])
    qs = W.uniform_points(nq, 11, -1.5, 1.5)
    qs[::2] /= np.linalg.norm(qs[::2], axis=1, keepdims=True)  # half of them near the surfaces
    tv, tt, tq = _cuda(verts), _cuda(tris), _cuda(qs)
    batch = bq.Batch(bq.triangles.boxes(tt, tv), _cuda(off))
    for r in (float("inf"), 0.02):
        many = bq.batched_tri_closest(batch, tt, tv, tq, _cuda(qoff), maxSqrDist=r)
        few = []
        for a in range(0, nq, 30_000):
            part = np.clip(qoff - a, 0, min(30_000, nq - a))
            few.append(bq.batched_tri_closest(batch, tt, tv, tq[a:a + 30_000], _cuda(part), maxSqrDist=r))
        assert _same([torch.cat(x) for x in zip(*few)], many), f"radius {r}"
    ids, d = (x.cpu().numpy() for x in bq.batched_tri_closest(batch, tt, tv, tq, _cuda(qoff))[:2])
    for s, n in enumerate(sizes):
        assert (ids[qoff[s]:qoff[s + 1]] >= 0).all() == (n > 0) or qoff[s] == qoff[s + 1]
        if n:
            at = rng.integers(qoff[s], qoff[s + 1], 20) if qoff[s] < qoff[s + 1] else []
            for i in at:
                assert off[s] <= ids[i] < off[s + 1]
            d64, _ = oracle.tri_brute_f64(tris[off[s]:off[s + 1]], verts, qs[at])
            # within the distance's rounding: 2^-20 of the coordinates at hand
            assert np.all(np.abs(np.sqrt(d[at].astype(np.float64)) - np.sqrt(d64)) <= 2.0 ** -20 * 3)


def _limited_allocator(bq, limit):
    """Blocks from torch, `limit` bytes (a list of one number) of them at a time."""
    class Limited(bq.TorchAllocator):
        def _malloc(self, ctx, out, size, stream):
            if sum(t.numel() for t in self.live.values()) + size > limit[0]:
                return 1
            return super()._malloc(ctx, out, size, stream)

    a = Limited()
    a.c.scratchFromPool = 0
    return a


def test_triangle_queries_need_no_more_scratch_than_a_thread_a_query(bq):
    """With room for the overflow list and the deep stacks alone (and, for one tree, the sort), the answers are the
    same as with room for the order, the list of heavy queries and the copy of the corners."""
    tv, tt = _mesh(4)
    boxes = bq.triangles.boxes(tt, tv)
    tq = _cuda(W.uniform_points(100_000, 4, -1.5, 1.5))
    least = 4 * len(tq) + 2048 * 1024 * 8 + 4096
    off, qoff = _cuda(np.array([0, 2000, 2000, len(tt)])), _cuda(np.array([0, 40_000, 40_100, len(tq)]))
    batch = bq.Batch(boxes, off)
    want = bq.batched_tri_closest(batch, tt, tv, tq, qoff)
    limit = [1 << 40]
    alloc = _limited_allocator(bq, limit)
    for extra in (0, 4, 12, 16, 20):  # bytes a query
        limit[0] = least + extra * len(tq)
        assert _same(bq.batched_tri_closest(batch, tt, tv, tq, qoff, allocator=alloc), want), extra
    limit[0] = 1 << 40
    bvh = bq.cuda.radixBuilder(boxes, None, alloc)
    want = bq.triangles.findClosest(bvh, tt, tv, tq)
    tree = sum(t.numel() for t in alloc.live.values())
    for extra, reorder in ((0, 0), (4, 0), (24, 1)):
        limit[0] = tree + least + extra * len(tq)
        got = bq.triangles.findClosest(bvh, tt, tv, tq, qcfg=bq.query_config(reorder=reorder))
        assert _same(got, want), (extra, reorder)
    bvh.free()


def test_triangle_groups_heavy_queries(bq):
    """Queries around the middle of a sphere of equal radius visit most of its
    tree and go to the second launch; NaN and infinite ones find nothing."""
    verts, tris = W.icosphere(6, amp=0.0)
    tv, tt = _cuda(verts), _cuda(tris)
    qs = W.uniform_points(300, 2, -0.02, 0.02)
    qs[::17, 0] = np.nan
    qs[5::17, 1] = np.inf
    bvh = bq.cuda.radixBuilder(bq.triangles.boxes(tt, tv))
    ids, d, p = (x.cpu().numpy() for x in bq.triangles.findClosest(bvh, tt, tv, _cuda(qs)))
    ok = np.isfinite(qs).all(1)
    assert (ids[~ok] == -1).all() and np.isinf(d[~ok]).all()
    c = verts.astype(np.float64)[tris]
    nrm = np.cross(c[:, 1] - c[:, 0], c[:, 2] - c[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    for i in np.nonzero(ok)[0]:  # near the middle the closest point lies inside its triangle, on the nearest plane
        h = np.abs((c[:, 0] * nrm).sum(1) - nrm @ qs[i].astype(np.float64)) ** 2
        assert abs(d[i] - h.min()) <= 1e-6, i
    assert np.allclose(((p[ok] - qs[ok]) ** 2).sum(1), d[ok], rtol=1e-5)


# below four queries each lane is on its own; one warp, parts of one, more than one; above 16,384 queries are sorted.
# A row of 3 ids sends most queries to the second traversal.
@pytest.mark.parametrize("nq", [1, 3, 4, 31, 33, 129, 16385])
@pytest.mark.parametrize("leaf", [1, 8])
def test_box_queries_of_partial_warps_match_oracle(bq, oracle, nq, leaf):
    pts = W.uniform_points(6000)
    boxes = boxes_np(pts)
    c = W.uniform_points(nq, 4, -0.1, 1.1)
    h = np.float32(0.02) + np.float32(0.06) * W.uniform_points(nq, 5)
    q = np.concatenate([c - h, c + h], 1)
    bvh = bq.cuda.radixBuilder(_cuda(boxes), bq.BuildConfig(makeLeafThreshold=leaf))
    n, pr = bvh.to_host()
    ooff, oids = oracle.box_query(n, pr, boxes, q)
    for cap in (None, 3, 0):
        off, ids = bq.fixedBoxQuery.findPrims(bvh, _cuda(boxes), _cuda(q), slabCap=cap)
        assert np.array_equal(off.cpu().numpy(), ooff) and np.array_equal(ids.cpu().numpy(), oids), f"slab {cap}"
    assert np.array_equal(bq.fixedBoxQuery.count(bvh, _cuda(boxes), _cuda(q)).cpu().numpy(), np.diff(ooff))


@pytest.mark.parametrize("tie", [0, 1])
@pytest.mark.parametrize("leaf", [1, 8, 60])
def test_closest_point_where_sorting_begins(bq, tie, leaf):
    """The last batch taken as given and the first ones sorted, with leaves
    that are processed at once and in step."""
    pts = W.uniform_points(30000)
    tp = _cuda(pts)
    qs = _cuda(W.uniform_points(196609, W.SEED_QUERIES, -0.1, 1.1))
    bvh = bq.gpuBuilder(_cuda(boxes_np(pts)), bq.BuildConfig(makeLeafThreshold=leaf))
    b = bq.points.findClosest(bvh, tp, qs, qcfg=bq.query_config(tieMode=tie, reorder=0))
    for nq in (1, 33, 196607, 196608, 196609):
        a, ran = _phases(bq, lambda: bq.points.findClosest(bvh, tp, qs[:nq], qcfg=bq.query_config(tieMode=tie)))
        assert _same(a, [x[:nq] for x in b]) and ("query.keys" in ran) == (nq >= 196608), nq


def test_closest_point_over_many_nodes_is_sorted_sooner(bq):
    g = torch.Generator(device="cuda").manual_seed(2)
    tp = torch.rand((5_000_000, 3), generator=g, device="cuda")
    bvh = bq.cuda.radixBuilder(bq.points_to_boxes(tp))
    first = -(-1_700_000_000_000 // bvh.numNodes)
    assert 1 << 16 < first < 3 << 16
    qs = torch.rand((first, 3), generator=g, device="cuda")
    b = bq.points.findClosest(bvh, tp, qs, qcfg=bq.query_config(reorder=0))
    for nq in (first - 1, first):
        a, ran = _phases(bq, lambda: bq.points.findClosest(bvh, tp, qs[:nq]))
        assert _same(a, [x[:nq] for x in b]) and ("query.keys" in ran) == (nq == first), nq
    bvh.free()


# just below and above the pairs a vertex at which four lanes sum them, and a warp, and many more
@pytest.mark.parametrize("nq", [250, 863, 864, 3455, 3456, 40000])
def test_vertex_gradients_by_thread_by_four_lanes_and_by_warp(bq, oracle, nq):
    verts, tris = W.icosphere(2)  # 162 vertices (16 pairs each from 864 queries on, 64 from 3,456)
    qs = W.uniform_points(nq, 3, -1.5, 1.5)
    g = (0.5 + W.uniform_points(nq, 8)[:, 0]).astype(np.float32)
    tv, tt, tq = _cuda(verts), _cuda(tris), _cuda(qs)
    ids, _, _ = bq.triangles.findClosest(bq.cuda.radixBuilder(bq.triangles.boxes(tt, tv)), tt, tv, tq)
    gq, gv = bq.triangles.distanceBackward(tt, tv, tq, ids, _cuda(g))
    assert _same((gq, gv), bq.triangles.distanceBackward(tt, tv, tq, ids, _cuda(g)))
    rq, rv = oracle.tri_grad_f64(tris, verts, qs, ids.cpu().numpy(), g)
    # the bound the adjoint is held to elsewhere: 1e-5 of the norm
    assert np.linalg.norm(gv.cpu().numpy() - rv) <= 1e-5 * np.linalg.norm(rv)
