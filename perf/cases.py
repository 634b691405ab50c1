"""The work a user of the library has it do, as cases that can be timed.

A case is a dict of plain values.  Its "kind" says which public calls one
pass makes:

  refresh  build a tree over a moved point set and match queries against it
  build    one tree from prim boxes
  closest  closest point of every query, over a tree the program keeps
  knn      k nearest points of every query, over a tree the program keeps
  boxes    all prims overlapping every query box
  mesh     point-to-mesh distance, forward and adjoint
  clouds   many uneven point clouds: one batched build, one batched kNN
  fit      one step of fitting many meshes: boxes, refit, distance, adjoint,
           vertex update

Data: "uniform" is U[0,1]^3; "gmm" is a mixture of 64 Gaussians, sigma
log-uniform in [1e-4, 1e-1], shifted by 1e5 so that tight clusters collapse
into exact duplicates (queries over it use the reference's tie rule, which is
what a program uses on such data); meshes are icospheres with every vertex
moved radially by up to 5%.
"""
import functools
import math

import numpy as np
import torch

import cubql_b200 as bq
from cubql_b200 import workloads

BUILDERS = ("morton", "median", "sah", "rebin")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one iteration of a registration loop on a small scan: rebuild, match; launches and latency count
        {"name": "refresh_5k", "kind": "refresh", "n": 5003, "nq": 5003, "leaf": 1},
        # the headline build: a large scene, one prim a leaf
        {"name": "build_morton_10m", "kind": "build", "builder": "morton", "n": 10_000_000, "leaf": 1,
         "data": "uniform"},
        # the default builder on clustered data far from the origin, leaves of eight
        {"name": "build_median_gmm_3m", "kind": "build", "builder": "median", "n": 3_000_017, "leaf": 8,
         "data": "gmm"},
        # the quality builder over a triangle mesh (1,310,720 triangles)
        {"name": "build_sah_mesh_1m3", "kind": "build", "builder": "sah", "n": 1_310_720, "leaf": 1, "data": "mesh"},
        # an ordinary query batch: a million points, a million queries, leaves of eight
        {"name": "closest_1m", "kind": "closest", "builder": "median", "n": 1_000_000, "nq": 1_000_000, "leaf": 8,
         "data": "uniform"},
        # the large query batch of the benchmark
        {"name": "closest_10m", "kind": "closest", "builder": "morton", "n": 10_000_000, "nq": 10_000_000, "leaf": 1,
         "data": "uniform"},
        # neighbourhoods for normals, densities and graphs, large
        {"name": "knn16_10m", "kind": "knn", "builder": "morton", "n": 10_000_000, "nq": 10_000_000, "leaf": 1,
         "k": 16, "data": "uniform"},
        # neighbourhoods on clustered data with duplicates, under the reference's tie rule
        {"name": "knn16_gmm_2m", "kind": "knn", "builder": "morton", "n": 2_000_003, "nq": 1_000_001, "leaf": 1,
         "k": 16, "data": "gmm"},
        # range search: a million small boxes, about sixteen points in each
        {"name": "boxes_1m", "kind": "boxes", "builder": "morton", "n": 10_000_000, "nq": 1_000_000, "leaf": 1,
         "per_box": 16},
        # differentiable point-to-mesh distance over a fine mesh
        {"name": "mesh_4m", "kind": "mesh", "n": 1_310_720, "nq": 4_000_000},
        # many uneven clouds at once
        {"name": "clouds_512", "kind": "clouds", "segs": 512, "lo": 1000, "hi": 200_000, "nq": 50_000, "k": 16},
        # one step of fitting many meshes at once
        {"name": "fit_128", "kind": "fit", "segs": 128, "lo": 2000, "hi": 100_000, "nq": 50_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("refresh", "build", "build", "closest", "closest", "knn", "knn", "boxes", "mesh", "clouds",
                       "fit"))
    if kind == "refresh":
        return {"kind": kind, "n": _log(rng, 1000, 300_000), "nq": _log(rng, 1000, 300_000),
                "leaf": rng.choice((1, 4, 8))}
    if kind == "build":
        builder = rng.choice(BUILDERS)
        data = rng.choice(("uniform", "gmm", "mesh"))
        hi = 1_310_720 if data == "mesh" else 10_000_000
        return {"kind": kind, "builder": builder, "n": _log(rng, 1000, hi), "leaf": rng.choice((1, 4, 8)),
                "data": data}
    if kind == "closest":
        return {"kind": kind, "builder": rng.choice(BUILDERS[:2]), "n": _log(rng, 1000, 10_000_000),
                "nq": _log(rng, 1000, 10_000_000), "leaf": rng.choice((1, 4, 8)),
                "data": rng.choice(("uniform", "uniform", "gmm"))}
    if kind == "knn":
        k = rng.choice((1, 4, 8, 16, 20, 32))
        return {"kind": kind, "builder": rng.choice(BUILDERS[:2]), "n": _log(rng, 1000, 10_000_000),
                "nq": _log(rng, 1000, 10_000_000 if k <= 16 else 3_000_000), "leaf": rng.choice((1, 4, 8)), "k": k,
                "data": rng.choice(("uniform", "uniform", "gmm"))}
    if kind == "boxes":
        return {"kind": kind, "builder": rng.choice(BUILDERS[:2]), "n": _log(rng, 1000, 10_000_000),
                "nq": _log(rng, 1000, 1_000_000), "leaf": rng.choice((1, 4, 8)), "per_box": rng.choice((2, 16, 40))}
    if kind == "mesh":
        return {"kind": kind, "n": _log(rng, 1000, 1_310_720), "nq": _log(rng, 1000, 4_000_000)}
    if kind == "clouds":
        return {"kind": kind, "segs": _log(rng, 2, 400), "lo": 1000, "hi": _log(rng, 20_000, 200_000),
                "nq": _log(rng, 500, 50_000), "k": rng.choice((1, 8, 16))}
    return {"kind": kind, "segs": _log(rng, 2, 100), "lo": 2000, "hi": _log(rng, 10_000, 100_000),
            "nq": _log(rng, 500, 50_000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed, what):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1_000_003 + what) & 0x7FFFFFFFFFFF)


def _uniform(n, g, lo=0.0, hi=1.0):
    return torch.rand((n, 3), generator=g, device="cuda") * (hi - lo) + lo


def _gmm(n, g, mix):
    c = torch.rand((64, 4), generator=mix, device="cuda", dtype=torch.float64)
    sigma = 1e-4 * (1e-1 / 1e-4) ** c[:, 3:]
    which = torch.randint(0, 64, (n,), generator=g, device="cuda")
    x = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return (c[which, :3] + sigma[which] * x + 1e5).float()


def _points(case, seed):
    if case.get("data") == "gmm":
        return _gmm(case["n"], _gen(seed, 1), _gen(seed, 3))
    return _uniform(case["n"], _gen(seed, 1))


def _queries(case, seed):
    if case.get("data") == "gmm":  # fresh samples of the same mixture
        return _gmm(case["nq"], _gen(seed, 2), _gen(seed, 3))
    if case["kind"] == "closest":  # some queries outside the cloud
        return _uniform(case["nq"], _gen(seed, 2), -0.1, 1.1)
    return _uniform(case["nq"], _gen(seed, 2))


@functools.lru_cache(maxsize=None)
def _sphere(level):
    """Unit icosphere of a level, on the host: (vertices, triangles)."""
    return workloads.icosphere(level, amp=0.0)


def _mesh(n, g):
    """(verts, tris): the first n triangles of the smallest icosphere that has as many."""
    level = 0
    while 20 * 4 ** level < n:
        level += 1
    v, t = _sphere(level)
    v = torch.from_numpy(v).cuda()
    v = v * (1.0 + 0.05 * (2.0 * torch.rand((v.shape[0], 1), generator=g, device="cuda") - 1.0))
    return v, torch.from_numpy(t[:n]).cuda().int()


def _sizes(case):
    """Sizes of the clouds or meshes of a batch, spread over the logarithm of [lo, hi]."""
    s = case["segs"]
    return [int(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / s)) for i in range(s)]


def _offsets(sizes):
    return torch.tensor(np.concatenate([[0], np.cumsum(sizes)]), dtype=torch.int32, device="cuda")


def _cloud_batch(case, seed):
    sizes = _sizes(case)
    g = _gen(seed, 1)
    order = np.random.RandomState(seed % (1 << 31)).permutation(len(sizes))
    sizes = [sizes[i] for i in order]
    clouds = []
    for i, n in enumerate(sizes):
        p = _uniform(n, g)
        if i % 2:  # every other cloud: eight clusters
            centres = _uniform(8, g)
            which = torch.randint(0, 8, (n,), generator=g, device="cuda")
            p = centres[which] + 0.02 * torch.randn((n, 3), generator=g, device="cuda")
        clouds.append(p)
    nq = case["nq"]
    return (torch.cat(clouds), _offsets(sizes), _uniform(nq * len(sizes), _gen(seed, 2)),
            _offsets([nq] * len(sizes)))


def _mesh_batch(case, seed):
    sizes = _sizes(case)
    g = _gen(seed, 1)
    verts, tris, base = [], [], 0
    for n in sizes:
        v, t = _mesh(n, g)
        verts.append(v)
        tris.append(t + base)
        base += v.shape[0]
    nq = case["nq"]
    return (torch.cat(verts), torch.cat(tris).int(), _offsets(sizes),
            _uniform(nq * len(sizes), _gen(seed, 2), -1.5, 1.5), _offsets([nq] * len(sizes)))


class _Tree:
    """A tree a program keeps; given back when the program drops it."""

    def __init__(self, bvh):
        self.bvh = bvh

    def __del__(self):
        self.bvh.free()


class _Buffers(bq.TorchAllocator):
    """Blocks that a program which rebuilds again and again keeps for its trees: what a build asks for comes out of
    them.  Their size does not depend on how many nodes a tree turns out to have."""

    def __init__(self, n):
        super().__init__()
        # prim ids (a builder may ask for two and give one back), nodes
        self.blocks = [torch.zeros(size, dtype=torch.uint8, device="cuda") for size in (4 * n, 4 * n, 64 * n + 128)]

    def _malloc(self, ctx, out, size, stream):
        block = next((b for b in self.blocks if b.data_ptr() not in self.live and size <= b.numel()), None)
        if block is None:
            return 1
        self.live[block.data_ptr()] = block
        out[0] = block.data_ptr()
        return 0


def _builder(name):
    return {"morton": bq.cuda.radixBuilder, "median": bq.gpuBuilder, "sah": bq.cuda.sahBuilder,
            "rebin": bq.cuda.rebinRadixBuilder}[name]


def _config(case):
    return bq.BuildConfig(makeLeafThreshold=case["leaf"])


def _query_config(case):
    return bq.query_config(tieMode=bq.TIES_REFERENCE if case.get("data") == "gmm" else bq.TIES_LOWEST_ID)


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("build", "refresh"):
        s["buffers"] = _Buffers(case["n"])
    if kind == "build":
        if case["data"] == "mesh":
            v, t = _mesh(case["n"], _gen(seed, 1))
            s["boxes"] = bq.triangles.boxes(t, v)
        else:
            s["boxes"] = bq.points_to_boxes(_points(case, seed))
    elif kind in ("refresh", "closest", "knn", "boxes"):
        s["points"] = _points(case, seed)
        if kind == "boxes":
            # half sizes around the one that holds `per_box` points on average, about a factor of two between boxes
            c = _uniform(case["nq"], _gen(seed, 2))
            h = 0.5 * (case["per_box"] / case["n"]) ** (1.0 / 3.0)
            h = h * (0.7 + 0.6 * torch.rand((case["nq"], 3), generator=_gen(seed, 4), device="cuda"))
            s["query_boxes"] = torch.cat([c - h, c + h], 1).contiguous()
            # where the program keeps the prims it is given, query after query
            s["found"] = torch.zeros(case["nq"] * (2 * case["per_box"] + 30), dtype=torch.int32, device="cuda")
        else:
            s["queries"] = _queries(case, seed)
        if kind != "refresh":
            s["boxes"] = bq.points_to_boxes(s["points"])
            s["tree"] = _Tree(_builder(case["builder"])(s["boxes"], _config(case)))
    elif kind == "mesh":
        s["verts"], s["tris"] = _mesh(case["n"], _gen(seed, 1))
        s["queries"] = _uniform(case["nq"], _gen(seed, 2), -1.5, 1.5)
        s["weights"] = torch.rand((case["nq"],), generator=_gen(seed, 4), device="cuda")
        s["tree"] = _Tree(bq.cuda.radixBuilder(bq.triangles.boxes(s["tris"], s["verts"])))
    elif kind == "clouds":
        s["points"], s["offsets"], s["queries"], s["query_offsets"] = _cloud_batch(case, seed)
        s["boxes"] = bq.points_to_boxes(s["points"])
    else:
        v, s["tris"], s["offsets"], s["queries"], s["query_offsets"] = _mesh_batch(case, seed)
        s["batch"] = bq.Batch(bq.triangles.boxes(s["tris"], v), s["offsets"])
        # the vertices after an update: the trees are refitted to them
        s["verts"] = v * (1.0 + 0.01 * (2.0 * torch.rand((v.shape[0], 1), generator=_gen(seed, 5), device="cuda") - 1))
        s["weights"] = torch.rand((s["queries"].shape[0],), generator=_gen(seed, 4), device="cuda")
    return s


def _take_tree(bvh, n):
    """A built tree as words: how many nodes, the root, the nodes after the unused one (up to the most that n prims can
    have), the prim ids; its blocks are free for the next build."""
    nodes = bvh.allocator.view(bvh.c.nodes, torch.int32, 16 * n).view(-1, 8)
    tree = {"count": bvh.numNodes, "root": nodes[:1], "nodes": nodes[2:], "prims": bvh.primids_tensor()}
    bvh.free()
    return tree


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "build":
        bvh = _builder(case["builder"])(s["boxes"], _config(case), s["buffers"])
        return _take_tree(bvh, case["n"])
    if kind == "refresh":
        bvh = bq.cuda.radixBuilder(bq.points_to_boxes(s["points"]), _config(case), s["buffers"])
        ids, d = bq.points.findClosest(bvh, s["points"], s["queries"])
        return {"ids": ids, "d": d, "tree": _take_tree(bvh, case["n"])}
    if kind == "closest":
        ids, d = bq.points.findClosest(s["tree"].bvh, s["points"], s["queries"], qcfg=_query_config(case))
        return {"ids": ids, "d": d}
    if kind == "knn":
        ids, d, found = bq.points.findKNN(s["tree"].bvh, s["points"], s["queries"], case["k"],
                                          qcfg=_query_config(case))
        return {"ids": ids, "d": d, "found": found}
    if kind == "boxes":
        offsets, ids = bq.fixedBoxQuery.findPrims(s["tree"].bvh, s["boxes"], s["query_boxes"])
        s["found"][:ids.shape[0]] = ids
        return {"offsets": offsets, "ids": s["found"]}
    if kind == "mesh":
        ids, d, p = bq.triangles.findClosest(s["tree"].bvh, s["tris"], s["verts"], s["queries"])
        gq, gv = bq.triangles.distanceBackward(s["tris"], s["verts"], s["queries"], ids, s["weights"])
        return {"ids": ids, "d": d, "p": p, "grad_queries": gq, "grad_verts": gv}
    if kind == "clouds":
        batch = bq.Batch(s["boxes"], s["offsets"])
        ids, d, found = bq.batched_knn(batch, s["points"], s["offsets"], s["queries"], s["query_offsets"], case["k"])
        return {"prims": batch.primIDs, "ids": ids, "d": d, "found": found}
    bq.batched_refit(s["batch"], bq.triangles.boxes(s["tris"], s["verts"]))
    ids, d, p = bq.batched_tri_closest(s["batch"], s["tris"], s["verts"], s["queries"], s["query_offsets"])
    gq, gv = bq.triangles.distanceBackward(s["tris"], s["verts"], s["queries"], ids, s["weights"])
    return {"ids": ids, "d": d, "p": p, "grad_queries": gq, "grad_verts": gv, "verts": s["verts"] - 1e-4 * gv}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _tree_bytes(n, leaf):
    """Nodes and prim ids of a tree of n prims, about 0.7 * leaf prims in a leaf."""
    return 64 * n / max(1.0, 0.7 * leaf) + 4 * n


def work(case):
    kind = case["kind"]
    if kind in ("clouds", "fit"):
        n, nq = sum(_sizes(case)), case["nq"] * case["segs"]
    else:
        n, nq = case["n"], case.get("nq", 0)
    leaf = case.get("leaf", 1)
    if kind == "build":
        return {"bytes": 24 * n + _tree_bytes(n, leaf), "flops": 12 * n}
    if kind == "refresh":
        return {"bytes": 12 * n + _tree_bytes(n, leaf) + 12 * nq + 8 * nq, "flops": 12 * n + 8 * nq}
    if kind == "closest":
        return {"bytes": _tree_bytes(n, leaf) + 12 * n + 12 * nq + 8 * nq, "flops": 8 * nq}
    if kind == "knn":
        return {"bytes": _tree_bytes(n, leaf) + 12 * n + 12 * nq + (8 * case["k"] + 4) * nq,
                "flops": 8 * case["k"] * nq}
    if kind == "boxes":
        found = case["per_box"] * nq
        return {"bytes": _tree_bytes(n, leaf) + 24 * n + 24 * nq + 8 * nq + 4 * found, "flops": 6 * found}
    if kind == "clouds":
        return {"bytes": 36 * n + _tree_bytes(n, 1) + 12 * nq + (8 * case["k"] + 4) * nq,
                "flops": 12 * n + 8 * case["k"] * nq}
    # meshes: triangles, about half as many vertices, the tree; queries and weights; ids, distances, points and the
    # two gradients
    verts = 6 * n + 6 * n
    mesh = 12 * n + verts + _tree_bytes(n, 1) + (16 + 20 + 12) * nq
    if kind == "mesh":
        return {"bytes": mesh, "flops": 200 * nq}
    return {"bytes": mesh + 64 * n + 6 * n, "flops": 200 * nq + 12 * n}


def tolerance(case):
    # Whole numbers: trees, ids and counts are determined by the inputs (lowest id among equal distances, or the
    # reference's visiting order), and a distance is one fixed expression of one pair.
    if case["kind"] not in ("mesh", "fit"):
        return "exact"
    # Gradients are 32-bit sums, up to some thousand terms a vertex: with the queries in another order they move by
    # 3.1e-6 (largest 1.0e-5) over 1,000 triangles and 4M queries, by less elsewhere.
    return {"rel": 1.2e-5, "max": 4e-5, "differ": 0.0}


# ---------------------------------------------------------------------------
# the same in 64 bits, by brute force
# ---------------------------------------------------------------------------
PAIRS = 1e11  # point pairs that take some seconds


def _nearest(points, queries, k):
    """(nq, k) squared distances in 64 bits, ascending."""
    p, q = points.double(), queries.double()
    out = torch.full((q.shape[0], k), math.inf, dtype=torch.float64, device="cuda")
    kk = min(k, p.shape[0])
    step = max(1, int(2e8) // p.shape[0])
    for a in range(0, q.shape[0], step):
        b = q[a:a + step]
        d = (b[:, None, 0] - p[None, :, 0]).square_()
        for j in (1, 2):
            d += (b[:, None, j] - p[None, :, j]).square_()
        out[a:a + step, :kk] = d.amin(1, keepdim=True) if kk == 1 else torch.topk(d, kk, 1, largest=False)[0]
    return out


def _triangle_points(tri, q):
    """Closest point of every triangle (t,3,3) to every query (b,3): weights (b,t,3) and squared distances (b,t)."""
    a, ab, ac = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    d00, d01, d11 = (ab * ab).sum(-1), (ab * ac).sum(-1), (ac * ac).sum(-1)
    aq = q[:, None, :] - a[None]
    e0, e1, qq = (aq * ab).sum(-1), (aq * ac).sum(-1), (aq * aq).sum(-1)

    def dist(v, w):
        return qq - 2 * (v * e0 + w * e1) + v * v * d00 + 2 * v * w * d01 + w * w * d11

    det = d00 * d11 - d01 * d01
    v, w = (d11 * e0 - d01 * e1) / det, (d00 * e1 - d01 * e0) / det
    inside = (v >= 0) & (w >= 0) & (v + w <= 1)
    best_v, best_w = torch.where(inside, v, 0.0), torch.where(inside, w, 0.0)
    best = torch.where(inside, dist(v, w), math.inf)
    t = (e0 / d00).clamp(0, 1)  # edge ab, edge ac, edge bc
    u = (e1 / d11).clamp(0, 1)
    s = ((e1 - e0 - d01 + d00) / (d00 - 2 * d01 + d11)).clamp(0, 1)
    for cv, cw in ((t, torch.zeros_like(t)), (torch.zeros_like(u), u), (1 - s, s)):
        d = dist(cv, cw)
        nearer = d < best
        best, best_v, best_w = torch.where(nearer, d, best), torch.where(nearer, cv, best_v), torch.where(
            nearer, cw, best_w)
    return torch.stack([1 - best_v - best_w, best_v, best_w], -1), best


def _mesh_exact(verts, tris, offsets, queries, query_offsets, weights):
    v, q, w = verts.double(), queries.double(), weights.double()
    d, p = torch.empty(q.shape[0], dtype=torch.float64, device="cuda"), torch.empty_like(q)
    gv = torch.zeros_like(v)
    for s in range(len(offsets) - 1):
        ts = tris[offsets[s]:offsets[s + 1]].long()
        tri = v[ts]
        step = max(1, int(1e7) // max(1, ts.shape[0]))
        for a in range(query_offsets[s], query_offsets[s + 1], step):
            b = min(a + step, query_offsets[s + 1])
            bary, dd = _triangle_points(tri, q[a:b])
            at = dd.argmin(1)
            bary = bary[torch.arange(b - a, device="cuda"), at]
            x = (bary[:, :, None] * tri[at]).sum(1)
            p[a:b], d[a:b] = x, (q[a:b] - x).square().sum(1)
            g = -2.0 * bary[:, :, None] * (q[a:b] - x)[:, None, :] * w[a:b, None, None]
            gv.index_add_(0, ts[at].reshape(-1), g.reshape(-1, 3))
    return {"ids": None, "d": d, "p": p, "grad_queries": 2.0 * (q - p) * w[:, None], "grad_verts": gv}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("refresh", "closest", "knn"):
        if 1.0 * case["n"] * case["nq"] > PAIRS:
            return None
        k = case.get("k", 1)
        d = _nearest(_points(case, seed), _queries(case, seed), k)
        if kind == "knn":
            return {"ids": None, "d": d, "found": None}
        if kind == "closest":
            return {"ids": None, "d": d[:, 0]}
        return {"ids": None, "d": d[:, 0], "tree": {"count": None, "root": None, "nodes": None, "prims": None}}
    if kind == "clouds":
        if 1.0 * sum(_sizes(case)) * case["nq"] > PAIRS:
            return None
        pts, off, qs, qoff = _cloud_batch(case, seed)
        off, qoff = off.tolist(), qoff.tolist()
        d = [_nearest(pts[off[i]:off[i + 1]], qs[qoff[i]:qoff[i + 1]], case["k"]) for i in range(case["segs"])]
        return {"prims": None, "ids": None, "d": torch.cat(d), "found": None}
    if kind == "mesh":
        if 1.0 * case["n"] * case["nq"] > PAIRS / 20:
            return None
        v, t = _mesh(case["n"], _gen(seed, 1))
        return _mesh_exact(v, t, [0, case["n"]], _uniform(case["nq"], _gen(seed, 2), -1.5, 1.5), [0, case["nq"]],
                           torch.rand((case["nq"],), generator=_gen(seed, 4), device="cuda"))
    if kind == "fit":
        if 1.0 * sum(_sizes(case)) * case["nq"] > PAIRS / 20:
            return None
        v, t, off, qs, qoff = _mesh_batch(case, seed)
        v = v * (1.0 + 0.01 * (2.0 * torch.rand((v.shape[0], 1), generator=_gen(seed, 5), device="cuda") - 1))
        w = torch.rand((qs.shape[0],), generator=_gen(seed, 4), device="cuda")
        out = _mesh_exact(v, t, off.tolist(), qs, qoff.tolist(), w)
        out["verts"] = v.double() - 1e-4 * out["grad_verts"]
        return out
    return None  # trees and box queries return whole numbers only
