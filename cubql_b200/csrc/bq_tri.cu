// bq_tri.cu -- point-to-triangle closest point (forward) and its adjoint.
//
// Forward: cuBQL::triangles::findClosest (cuBQL/queries/triangles/
// findClosest.h:132-152) over an indexed mesh, batched like the point
// queries (Hilbert-ordered and eight lanes a query under the lowest-id rule, see
// bq_tri.cuh; Morton-ordered and a thread each under the reference's;
// deep-stack fallback).  The
// per-triangle arithmetic follows findClosest.h:56-122 expression for
// expression (edge projections with clamped t, the three edge-plane tests,
// the normalised plane distance), so nvcc contracts it as it does the
// reference's.
//
// Adjoint (no counterpart in the reference): for the closest point
// X = sum_k w_k v_k with barycentric weights w on the fixed simplex, the
// envelope theorem gives
//     d sqrDist / d q   =  2 (q - X)
//     d sqrDist / d v_k = -2 w_k (q - X).
// Per query the three vertex contributions become (vertexID, pair index)
// records; a stable radix sort by vertex id groups them and one thread (four or
// 32 of many pairs) per vertex sums its group in a fixed order.  No float
// atomics: the result is bitwise reproducible.
#include <algorithm>

#include "bq_query.cuh"
#include "bq_tri.cuh"

namespace bq {
namespace {

// stack entries a triangle-query thread keeps in shared memory (the top of
// its traversal stack); the rest of the stack is in local memory.  Measured
// on the 4M-query, 1.31M-triangle workload: 45.0 ms with none, 46.4 with 8,
// 44.8 with 16 -- the kernel waits on its node and vertex loads, not on the
// stack -- so none.
constexpr int TRI_SMEM_STACK = 0;
// Pairs a vertex (on average) from which four lanes, and from which a warp,
// sum them.  The whole adjoint, ms by one thread, four lanes and a warp a
// vertex, pairs spread evenly and as the closest triangles of queries in a
// cube around the mesh: 10 (2.2M queries, 655,362 vertices) 0.53 0.55 0.99 and
// 1.16 0.62 0.98; 18 (4M) 0.88 0.86 1.29 and 2.16 1.02 1.30; 64 (14M) 3.57
// 2.73 2.96 and 7.76 3.13 2.97; 1,852 (100,000 queries, 162 vertices) 1.64
// 0.21 0.11 and 2.15 0.25 0.11.
constexpr uint32_t BWD_QUAD_PAIRS = 16, BWD_WARP_PAIRS = 64;

template <int TIE, typename Stack>
__device__ __forceinline__ bool run_tri(const Node *nodes, const uint32_t *primIDs, const int32_t *tris,
                                        const float *verts, const float *queries, uint32_t qi, float maxSqr,
                                        Stack &st, int32_t *outIds, float *outD, float *outP)
{
  TriLeaf<TIE> leaf(primIDs, tris, verts, queries + 3ull * qi, maxSqr);
  if (!traverse<TIE>(nodes, leaf.q.x, leaf.q.y, leaf.q.z, leaf.cull(), st, leaf)) return false;
  outIds[qi] = leaf.id;
  outD[qi] = leaf.d;
  if (outP) {
    outP[3ull * qi + 0] = leaf.P.x;
    outP[3ull * qi + 1] = leaf.P.y;
    outP[3ull * qi + 2] = leaf.P.z;
  }
  return true;
}

template <int TIE, int STACK>
__global__ void __launch_bounds__(128) k_tri(const Node *__restrict__ nodes, const uint32_t *__restrict__ primIDs,
                                             const int32_t *__restrict__ tris, const float *__restrict__ verts,
                                             const float *__restrict__ queries, const uint32_t *__restrict__ order,
                                             uint32_t nq, float maxSqr, int32_t *__restrict__ outIds,
                                             float *__restrict__ outD, float *__restrict__ outP,
                                             uint32_t *__restrict__ ovfList, uint32_t *ovfCount)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nq) return;
  const uint32_t qi = order ? __ldg(order + t) : t;
  extern __shared__ StackEntry sStack[];
  HybridStack<TRI_SMEM_STACK, STACK> st(sStack);
  if (!run_tri<TIE>(nodes, primIDs, tris, verts, queries, qi, maxSqr, st, outIds, outD, outP))
    ovfList[atomicAdd(ovfCount, 1u)] = qi;
}

template <int TIE>
__global__ void k_tri_deep(const Node *__restrict__ nodes, const uint32_t *__restrict__ primIDs,
                           const int32_t *__restrict__ tris, const float *__restrict__ verts,
                           const float *__restrict__ queries, float maxSqr, int32_t *__restrict__ outIds,
                           float *__restrict__ outD, float *__restrict__ outP, const uint32_t *ovfList,
                           const uint32_t *ovfCount, StackEntry *stacks, uint32_t *err)
{
  griddep_wait();
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t cnt = *ovfCount;
  for (uint32_t w = tid; w < cnt; w += gridDim.x * blockDim.x) {
    const uint32_t qi = ovfList[w];
    GlobalStack st{stacks + (size_t)tid * DEEP_STACK, DEEP_STACK, 0};
    if (!run_tri<TIE>(nodes, primIDs, tris, verts, queries, qi, maxSqr, st, outIds, outD, outP)) {
      outIds[qi] = -1;
      outD[qi] = INFINITY;
      atomicOr(err, DEV_ERR_STACK);
    }
  }
}

// visit counts of the triangle traversal (measurement pass of the forward's
// roofline): node pairs loaded, admin loads, triangles tested
template <int TIE>
__global__ void __launch_bounds__(128) k_tri_visit_count(const Node *__restrict__ nodes,
                                                         const uint32_t *__restrict__ primIDs,
                                                         const int32_t *__restrict__ tris,
                                                         const float *__restrict__ verts,
                                                         const float *__restrict__ queries, uint32_t nq, float maxSqr,
                                                         unsigned long long *out)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  VisitCount vc;
  uint32_t prims = 0;
  if (t < nq) {  // no early return: every lane takes part in the warp sum below
    TriLeaf<TIE> leaf(primIDs, tris, verts, queries + 3ull * t, maxSqr);
    CountingLeaf<TriLeaf<TIE>> cl{leaf};
    LocalStack<128> st;
    traverse_counted<TIE>(nodes, leaf.q.x, leaf.q.y, leaf.q.z, leaf.cull(), st, cl, vc);
    prims = cl.prims;
  }
  add_visit_counts(vc.pairs, vc.admins, prims, out);
}

__global__ void k_tri_fill_empty(uint32_t nq, int32_t *ids, float *d, float *P)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nq) return;
  ids[t] = -1;
  d[t] = INFINITY;
  if (P) P[3ull * t] = P[3ull * t + 1] = P[3ull * t + 2] = 0.f;
}

// ------------------------------------------------------------------
// adjoint
// ------------------------------------------------------------------
__global__ void k_tri_bwd_pairs(const int32_t *__restrict__ tris, const float *__restrict__ verts,
                                const float *__restrict__ queries, uint32_t nq, const int32_t *__restrict__ ids,
                                const float *__restrict__ gradSqr, float *__restrict__ gradQ,
                                uint32_t *__restrict__ keys, uint32_t *__restrict__ vals,
                                float *__restrict__ contrib)
{
  const uint32_t qi = blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= nq) return;
  const int32_t id = ids[qi];
  const float *qp = queries + 3ull * qi;
  const V3 q = V3{qp[0], qp[1], qp[2]};
  float r[3] = {0.f, 0.f, 0.f}, w[3] = {0.f, 0.f, 0.f};
  int32_t vi[3] = {-1, -1, -1};
  if (id >= 0) {
    const int32_t *t = tris + 3ll * id;
    vi[0] = t[0]; vi[1] = t[1]; vi[2] = t[2];
    const V3 a = ldv(verts, vi[0]), b = ldv(verts, vi[1]), c = ldv(verts, vi[2]);
    const TriHit h = tri_cp(a, b, c, q);
    if (h.region == 0) {
      // barycentric weights of the projection of q (the off-plane part of
      // q - a drops out of both triple products)
      const V3 N = v3cross(v3sub(b, a), v3sub(c, a));
      const float nn = v3dot(N, N);
      const V3 qa = v3sub(q, a);
      const float u = v3dot(v3cross(qa, v3sub(c, a)), N) / nn;
      const float v = v3dot(v3cross(v3sub(b, a), qa), N) / nn;
      w[0] = 1.f - u - v; w[1] = u; w[2] = v;
    } else if (h.region == 1) {
      w[0] = 1.f - h.t; w[1] = h.t;
    } else if (h.region == 2) {
      w[1] = 1.f - h.t; w[2] = h.t;
    } else if (h.region == 3) {
      w[2] = 1.f - h.t; w[0] = h.t;
    }
    const float g = 2.f * gradSqr[qi];
    r[0] = (q.x - h.P.x) * g;
    r[1] = (q.y - h.P.y) * g;
    r[2] = (q.z - h.P.z) * g;
  }
  gradQ[3ull * qi + 0] = r[0];
  gradQ[3ull * qi + 1] = r[1];
  gradQ[3ull * qi + 2] = r[2];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const uint64_t pi = 3ull * qi + k;
    keys[pi] = vi[k] >= 0 ? (uint32_t)vi[k] : 0xffffffffu;
    vals[pi] = (uint32_t)pi;
    contrib[3 * pi + 0] = -w[k] * r[0];
    contrib[3 * pi + 1] = -w[k] * r[1];
    contrib[3 * pi + 2] = -w[k] * r[2];
  }
}

// first pair with key >= v
__device__ __forceinline__ uint32_t first_pair(const uint32_t *__restrict__ sortedKeys, uint32_t numPairs, uint32_t v)
{
  uint32_t lo = 0, hi = numPairs;
  while (lo < hi) {
    const uint32_t m = lo + ((hi - lo) >> 1);
    if (sortedKeys[m] < v) lo = m + 1; else hi = m;
  }
  return lo;
}

// L lanes per vertex: lane l adds its pairs l, l + L, ... in sorted order, then
// the lanes are added pairwise; reproducible like the other, and with shorter
// chains of additions.  For meshes with many queries a vertex, where one
// thread's chain of dependent gathers is what takes the time.
template <int L>
__global__ void k_tri_bwd_reduce_lanes(const uint32_t *__restrict__ sortedKeys,
                                       const uint32_t *__restrict__ sortedVals, uint32_t numPairs,
                                       const float *__restrict__ contrib, uint32_t numVerts, float *__restrict__ gradV)
{
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & (L - 1);
  const bool mine = t / L < numVerts;
  const uint32_t v = mine ? (uint32_t)(t / L) : numVerts - 1;
  const uint32_t lo = first_pair(sortedKeys, numPairs, v), hi = first_pair(sortedKeys, numPairs, v + 1);
  float sx = 0.f, sy = 0.f, sz = 0.f;
  for (uint32_t j = lo + lane; j < hi; j += L) {
    const uint32_t p = sortedVals[j];
    sx += contrib[3ull * p + 0];
    sy += contrib[3ull * p + 1];
    sz += contrib[3ull * p + 2];
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) {
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    sy += __shfl_xor_sync(0xffffffffu, sy, o);
    sz += __shfl_xor_sync(0xffffffffu, sz, o);
  }
  if (mine && lane == 0) {
    gradV[3ull * v + 0] = sx;
    gradV[3ull * v + 1] = sy;
    gradV[3ull * v + 2] = sz;
  }
}

__global__ void k_tri_bwd_reduce(const uint32_t *__restrict__ sortedKeys, const uint32_t *__restrict__ sortedVals,
                                 uint32_t numPairs, const float *__restrict__ contrib, uint32_t numVerts,
                                 float *__restrict__ gradV)
{
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= numVerts) return;
  const uint32_t lo = first_pair(sortedKeys, numPairs, v);
  float sx = 0.f, sy = 0.f, sz = 0.f;
  for (uint32_t j = lo; j < numPairs && sortedKeys[j] == v; j++) {
    const uint32_t p = sortedVals[j];
    sx += contrib[3ull * p + 0];
    sy += contrib[3ull * p + 1];
    sz += contrib[3ull * p + 2];
  }
  gradV[3ull * v + 0] = sx;
  gradV[3ull * v + 1] = sy;
  gradV[3ull * v + 2] = sz;
}

// Triangle::bounds() (cuBQL/queries/triangles/Triangle.h:40-41)
__global__ void k_tri_boxes(const int32_t *__restrict__ tris, const float *__restrict__ verts, uint32_t nt,
                            bq_box3f *__restrict__ boxes)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const int32_t *ix = tris + 3ull * t;
  const V3 a = ldv(verts, ix[0]), b = ldv(verts, ix[1]), c = ldv(verts, ix[2]);
  bq_box3f bx;
  bx.lower[0] = fminf(fminf(fminf(INFINITY, a.x), b.x), c.x);
  bx.lower[1] = fminf(fminf(fminf(INFINITY, a.y), b.y), c.y);
  bx.lower[2] = fminf(fminf(fminf(INFINITY, a.z), b.z), c.z);
  bx.upper[0] = fmaxf(fmaxf(fmaxf(-INFINITY, a.x), b.x), c.x);
  bx.upper[1] = fmaxf(fmaxf(fmaxf(-INFINITY, a.y), b.y), c.y);
  bx.upper[2] = fmaxf(fmaxf(fmaxf(-INFINITY, a.z), b.z), c.z);
  boxes[t] = bx;
}

} // namespace

int query_config(const bq_query_config *q, bq_query_config &out);

int tri_closest(const bq_bvh3f *bvh, const int32_t *tris, const float *verts, const float *queries, uint32_t nq,
                float maxSqr, const bq_query_config *qcfg, int32_t *ids, float *d, float *P, Alloc &al)
{
  bq_query_config c;
  BQ_TRY(query_config(qcfg, c));
  if (nq == 0) return BQ_OK;
  if (bvh->numNodes == 0) {
    k_tri_fill_empty<<<div_up(nq, 256), 256, 0, al.s>>>(nq, ids, d, P);
    BQ_CUDA(cudaGetLastError());
    return BQ_OK;
  }
  TempSet tmp(al);
  uint32_t *ovfList = nullptr, *ovfCount = nullptr, *order = nullptr, *heavy = nullptr;
  StackEntry *deep = nullptr;
  BQ_TRY(tmp.get(&ovfList, nq));
  BQ_TRY(tmp.get(&ovfCount, 4));  // overflow count, error word, heavy count, count left by the first launch
  BQ_TRY(tmp.get(&deep, (size_t)DEEP_THREADS * DEEP_STACK));
  BQ_CUDA(cudaMemsetAsync(ovfCount, 0, 16, al.s));
  uint32_t *err = ovfCount + 1;
  const Node *nodes = (const Node *)bvh->nodes;
  if (c.reorder && nq >= TRI_ORDER_MIN) {
    uint32_t *keys[2], *idx[2];
    BQ_TRY(tmp.get(&keys[0], nq));
    BQ_TRY(tmp.get(&keys[1], nq));
    BQ_TRY(tmp.get(&idx[0], nq));
    BQ_TRY(tmp.get(&idx[1], nq));
    {
      // a thread a query is no faster along a Hilbert curve, and heavy queries
      // then share their warps (33,000 queries over 20,480 triangles under the
      // reference's rule 1.7 ms along a Morton curve, 2.5 along a Hilbert curve)
      ProfScope ps("tri.keys", al.s);
      query_keys((const float *)nodes, queries, nq, c.tieMode == BQ_TIES_LOWEST_ID, keys[0], idx[0], al.s);
    }
    BQ_CUDA(cudaGetLastError());
    int sel = 0;
    BQ_TRY(onesweep_sort_u32(keys, idx, nq, nullptr, 6, 30, nullptr, &sel, err, al));  // order only: top 24 bits
    order = idx[sel];
    heavy = keys[sel];  // the sorted keys are of no further use
  }
  const int b = c.blockSize;
  auto status_of = [](uint32_t herr) -> int {
    if (herr & DEV_ERR_STACK) return set_error(BQ_ERR_STACK_OVERFLOW, "query exceeded the deep fallback stack");
    if (herr & DEV_ERR_TIMEOUT) return set_error(BQ_ERR_TIMEOUT, "query reordering sort timed out");
    return BQ_OK;
  };
#define BQ_TRI_LAUNCH(TIE, ST)                                                                                     \
  ProfScope ps("tri.closest", al.s, 2);                                                                            \
  k_tri<TIE, ST><<<div_up(nq, b), b, TRI_SMEM_STACK * sizeof(StackEntry) * b, al.s>>>(                           \
      nodes, bvh->primIDs, tris, verts, queries, order, nq, maxSqr, ids,                                           \
                                                d, P, ovfList, ovfCount);                                          \
  k_tri_deep<TIE><<<DEEP_THREADS / 128, 128, 0, al.s>>>(nodes, bvh->primIDs, tris, verts, queries, maxSqr, ids, d, \
                                                        P, ovfList, ovfCount, deep, err)
  if (c.tieMode == BQ_TIES_REFERENCE) {
    if (c.stackDepth == 32) { BQ_TRI_LAUNCH(TIE_REFERENCE, 32); }
    else if (c.stackDepth == 64) { BQ_TRI_LAUNCH(TIE_REFERENCE, 64); }
    else { BQ_TRI_LAUNCH(TIE_REFERENCE, 128); }
  } else {
    if (!heavy && tmp.get(&heavy, nq) != BQ_OK) {
      heavy = nullptr;
      cudaGetLastError();
    }
    // a query tests some twenty triangles: the copy pays from about a
    // twentieth as many queries as triangles
    float4 *packed = nullptr;
    if (bvh->numPrims && (uint64_t)nq * 16 >= bvh->numPrims) {
      if (tmp.get(&packed, 3ull * bvh->numPrims) != BQ_OK) {
        packed = nullptr;  // no room for the copy: corners through the index
        cudaGetLastError();
      } else {
        ProfScope ps("tri.pack", al.s);
        launch_pdl(k_tri_pack, dim3(div_up(bvh->numNodes, 256)), dim3(256), 0, al.s, nodes, bvh->numNodes, bvh->primIDs,
                   bvh->numPrims, tris, verts, packed, err);
      }
    }
    auto search = [&](const float4 *corners) {
      const TriMesh m{nodes, bvh->primIDs, nullptr, nullptr, nullptr, 0, corners, tris, verts};
      launch_tri_group(m, bvh->numPrims, queries, order, nq, maxSqr, ids, d, P, heavy, ovfList, ovfCount, ovfCount + 2,
                       ovfCount + 3, corners ? err : nullptr, al.s);
      ProfScope ps("tri.deep", al.s);
      launch_pdl(k_tri_deep<TIE_LOWEST>, dim3(DEEP_THREADS / 128), dim3(128), 0, al.s, nodes, bvh->primIDs, tris, verts,
                 queries, maxSqr, ids, d, P, ovfList, ovfCount, deep, err);
    };
    search(packed);
    uint32_t herr = 0;
    BQ_CUDA(cudaGetLastError());
    BQ_CUDA(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, al.s));
    BQ_CUDA(cudaStreamSynchronize(al.s));
    if (!(herr & DEV_ERR_RANGE)) return status_of(herr);
    // the tree has leaves past the number of prims it was given with
    BQ_CUDA(cudaMemsetAsync(ovfCount, 0, 16, al.s));
    search(nullptr);
  }
#undef BQ_TRI_LAUNCH
  BQ_CUDA(cudaGetLastError());
  uint32_t herr = 0;
  BQ_CUDA(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, al.s));
  BQ_CUDA(cudaStreamSynchronize(al.s));
  return status_of(herr);
}

int tri_distance_bwd(const int32_t *tris, const float *verts, uint32_t numVerts, const float *queries, uint32_t nq,
                     const int32_t *ids, const float *gradSqr, float *gradQ, float *gradV, Alloc &al)
{
  if (numVerts > 0x7fffffffu) return set_error(BQ_ERR_INVALID_ARGUMENT, "too many vertices");
  if (nq == 0) {
    if (numVerts) BQ_CUDA(cudaMemsetAsync(gradV, 0, sizeof(float) * 3ull * numVerts, al.s));
    return BQ_OK;
  }
  if ((uint64_t)nq * 3 >= (1ull << 30)) return set_error(BQ_ERR_INVALID_ARGUMENT, "too many queries for one call");
  const uint32_t np = nq * 3;
  TempSet tmp(al);
  uint32_t *keys[2], *vals[2], *err = nullptr;
  float *contrib = nullptr;
  BQ_TRY(tmp.get(&keys[0], np));
  BQ_TRY(tmp.get(&keys[1], np));
  BQ_TRY(tmp.get(&vals[0], np));
  BQ_TRY(tmp.get(&vals[1], np));
  BQ_TRY(tmp.get(&contrib, 3ull * np));
  BQ_TRY(tmp.get(&err, 1));
  BQ_CUDA(cudaMemsetAsync(err, 0, 4, al.s));
  ProfScope ps("tri.backward", al.s, 5);
  k_tri_bwd_pairs<<<div_up(nq, 128), 128, 0, al.s>>>(tris, verts, queries, nq, ids, gradSqr, gradQ, keys[0], vals[0],
                                                     contrib);
  BQ_CUDA(cudaGetLastError());
  // enough key bits that the "no vertex" key 0xffffffff sorts after every id
  int bits = 1;
  while (bits < 32 && (1ull << bits) <= numVerts) bits++;
  int sel = 0;
  BQ_TRY(onesweep_sort_u32(keys, vals, np, nullptr, 0, bits, nullptr, &sel, err, al));
  if (numVerts && np / BWD_WARP_PAIRS >= numVerts)
    k_tri_bwd_reduce_lanes<32><<<div_up(32ull * numVerts, 256), 256, 0, al.s>>>(keys[sel], vals[sel], np, contrib,
                                                                                numVerts, gradV);
  else if (numVerts && np / BWD_QUAD_PAIRS >= numVerts)
    k_tri_bwd_reduce_lanes<4><<<div_up(4ull * numVerts, 256), 256, 0, al.s>>>(keys[sel], vals[sel], np, contrib,
                                                                              numVerts, gradV);
  else if (numVerts)
    k_tri_bwd_reduce<<<div_up(numVerts, 256), 256, 0, al.s>>>(keys[sel], vals[sel], np, contrib, numVerts, gradV);
  BQ_CUDA(cudaGetLastError());
  uint32_t herr = 0;
  BQ_CUDA(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, al.s));
  BQ_CUDA(cudaStreamSynchronize(al.s));
  if (herr & DEV_ERR_TIMEOUT) return set_error(BQ_ERR_TIMEOUT, "vertex-gradient sort timed out");
  return BQ_OK;
}

int tri_boxes(const int32_t *tris, const float *verts, uint32_t nt, bq_box3f *boxes, cudaStream_t s)
{
  if (nt == 0) return BQ_OK;
  k_tri_boxes<<<div_up(nt, 256), 256, 0, s>>>(tris, verts, nt, boxes);
  BQ_CUDA(cudaGetLastError());
  return BQ_OK;
}

int tri_visit_counts(const bq_bvh3f *bvh, const int32_t *tris, const float *verts, const float *queries, uint32_t nq,
                     float maxSqr, const bq_query_config *qcfg, uint64_t *hostCounts, Alloc &al)
{
  bq_query_config c;
  BQ_TRY(query_config(qcfg, c));
  hostCounts[0] = hostCounts[1] = hostCounts[2] = 0;
  if (nq == 0 || bvh->numNodes == 0) return BQ_OK;
  TempSet tmp(al);
  unsigned long long *out = nullptr;
  BQ_TRY(tmp.get(&out, 3));
  BQ_CUDA(cudaMemsetAsync(out, 0, 3 * sizeof(unsigned long long), al.s));
  const Node *nodes = (const Node *)bvh->nodes;
  if (c.tieMode == BQ_TIES_REFERENCE)
    k_tri_visit_count<TIE_REFERENCE><<<div_up(nq, 128), 128, 0, al.s>>>(nodes, bvh->primIDs, tris, verts, queries, nq,
                                                                        maxSqr, out);
  else
    k_tri_visit_count<TIE_LOWEST><<<div_up(nq, 128), 128, 0, al.s>>>(nodes, bvh->primIDs, tris, verts, queries, nq,
                                                                     maxSqr, out);
  BQ_CUDA(cudaGetLastError());
  unsigned long long h[3];
  BQ_CUDA(cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, al.s));
  BQ_CUDA(cudaStreamSynchronize(al.s));
  for (int i = 0; i < 3; i++) hostCounts[i] = h[i];
  return BQ_OK;
}

} // namespace bq
