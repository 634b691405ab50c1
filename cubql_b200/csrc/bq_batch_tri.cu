// bq_batch_tri.cu -- batched meshes: refit of every mesh's tree and the
// closest-triangle query of every mesh's queries, each in one launch.
//
// Layout (as produced by bq_batched_build_morton63_f3 over triangle boxes):
// mesh s owns triangles tris[triOff[s] .. triOff[s+1]) (vertex indices into
// one shared vertex array), its tree's nodes sit in the block starting at
// nodes[2*triOff[s]] and its primIDs (mesh-local triangle ids) at
// primIDs[triOff[s]].  This is the per-step work of a differentiable
// fitting loop: move vertices, recompute triangle boxes, refit all trees,
// query, backpropagate (bq_tri_distance_bwd_f3 works on the shared arrays
// directly because the query returns global triangle ids).
#include <algorithm>

#include <cuda/atomic>

#include "bq_tri.cuh"

namespace bq {
int query_config(const bq_query_config *q, bq_query_config &out);

namespace {

constexpr uint32_t BR_NO_PARENT = 0xffffffffu;

// slot j of the node buffer belongs to the mesh whose block contains it;
// returns false for slots past that tree's node count
__device__ __forceinline__ bool node_slot(const bq_bvh3f *__restrict__ bvhs, const uint32_t *__restrict__ off,
                                          uint32_t numSegs, uint32_t j, uint32_t &s, uint32_t &local)
{
  s = seg_of(off, numSegs, j >> 1);
  local = j - 2 * __ldg(off + s);
  return local < bvhs[s].numNodes;
}

__global__ void k_brefit_parents(const Node *__restrict__ nodes, uint32_t numSlots, const bq_bvh3f *__restrict__ bvhs,
                                 const uint32_t *__restrict__ off, uint32_t numSegs, uint32_t *__restrict__ parent,
                                 uint32_t *__restrict__ counter)
{
  griddep_wait();
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= numSlots) return;
  counter[j] = 0;
  uint32_t s, local;
  if (!node_slot(bvhs, off, numSegs, j, s, local)) return;
  const uint32_t base = 2 * off[s];
  if (local == 0) parent[j] = BR_NO_PARENT;
  if (local == 1) return;
  const uint64_t a = node_admin(nodes[j]);
  if (admin_count(a) == 0) {
    const uint64_t c = base + admin_offset(a);
    parent[c] = j;
    parent[c + 1] = j;
  }
}

__global__ void k_brefit_climb(Node *nodes, uint32_t numSlots, const bq_bvh3f *__restrict__ bvhs,
                               const uint32_t *__restrict__ off, uint32_t numSegs, const uint32_t *__restrict__ primIDs,
                               const bq_box3f *__restrict__ boxes, const uint32_t *__restrict__ parent,
                               uint32_t *counter)
{
  griddep_wait();
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= numSlots) return;
  uint32_t s, local;
  if (!node_slot(bvhs, off, numSegs, j, s, local) || local == 1) return;
  const uint64_t a = node_admin(nodes[j]);
  const uint32_t cnt = admin_count(a);
  if (cnt == 0) return;
  const uint32_t pbase = off[s], base = 2 * pbase;
  const uint64_t o = admin_offset(a);
  float lx = INFINITY, ly = INFINITY, lz = INFINITY, hx = -INFINITY, hy = -INFINITY, hz = -INFINITY;
  for (uint32_t q = 0; q < cnt; q++) {
    const bq_box3f b = boxes[pbase + primIDs[pbase + o + q]];
    lx = fminf(lx, b.lower[0]); ly = fminf(ly, b.lower[1]); lz = fminf(lz, b.lower[2]);
    hx = fmaxf(hx, b.upper[0]); hy = fmaxf(hy, b.upper[1]); hz = fmaxf(hz, b.upper[2]);
  }
  nodes[j] = make_node(lx, ly, lz, hx, hy, hz, a);
  while (true) {
    const uint32_t p = parent[j];
    if (p == BR_NO_PARENT) return;
    // device-scope release of this node's box / acquire of the sibling's
    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> arrived(counter[p]);
    if (arrived.fetch_add(1u, cuda::memory_order_acq_rel) == 0) return;  // the sibling finishes this parent
    const float4 pb = __ldcg(&nodes[p].b);  // from L2: the box half of this word is being written
    const uint64_t pa = ((uint64_t)__float_as_uint(pb.w) << 32) | __float_as_uint(pb.z);
    const uint64_t c0 = base + admin_offset(pa);
    const Node sib = ldcg_node(nodes + (c0 == j ? c0 + 1 : c0));
    if (c0 == j) {  // union in child order (left, right)
      lx = fminf(lx, sib.a.x); ly = fminf(ly, sib.a.y); lz = fminf(lz, sib.a.z);
      hx = fmaxf(hx, sib.a.w); hy = fmaxf(hy, sib.b.x); hz = fmaxf(hz, sib.b.y);
    } else {
      lx = fminf(sib.a.x, lx); ly = fminf(sib.a.y, ly); lz = fminf(sib.a.z, lz);
      hx = fmaxf(sib.a.w, hx); hy = fmaxf(sib.b.x, hy); hz = fmaxf(sib.b.y, hz);
    }
    nodes[p] = make_node(lx, ly, lz, hx, hy, hz, pa);
    j = p;
  }
}

// ------------------------------------------------------------------
// batched closest triangle
// ------------------------------------------------------------------
template <int TIE, typename Stack>
__device__ __forceinline__ bool run_btri(const bq_bvh3f &d, const uint32_t triBase, const int32_t *tris,
                                         const float *verts, const float *queries, uint32_t qi, float maxSqr,
                                         Stack &st, int32_t *outIds, float *outD, float *outP)
{
  TriLeaf<TIE> leaf(d.primIDs, tris + 3ull * triBase, verts, queries + 3ull * qi, maxSqr);
  if (d.numNodes && !traverse<TIE>((const Node *)d.nodes, leaf.q.x, leaf.q.y, leaf.q.z, leaf.cull(), st, leaf))
    return false;
  outIds[qi] = leaf.id >= 0 ? (int32_t)(triBase + leaf.id) : -1;
  outD[qi] = leaf.d;
  if (outP) {
    outP[3ull * qi] = leaf.P.x;
    outP[3ull * qi + 1] = leaf.P.y;
    outP[3ull * qi + 2] = leaf.P.z;
  }
  return true;
}

template <int TIE, int STACK>
__global__ void __launch_bounds__(128) k_btri(const bq_bvh3f *__restrict__ bvhs, const uint32_t *__restrict__ triOff,
                                              const uint32_t *__restrict__ qoff, uint32_t numSegs,
                                              const int32_t *__restrict__ tris, const float *__restrict__ verts,
                                              const float *__restrict__ queries, uint32_t nq, float maxSqr,
                                              int32_t *__restrict__ outIds, float *__restrict__ outD,
                                              float *__restrict__ outP, uint32_t *__restrict__ ovfList,
                                              uint32_t *ovfCount)
{
  griddep_wait();
  const uint32_t qi = blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= nq) return;
  const uint32_t s = seg_of(qoff, numSegs, qi);
  const bq_bvh3f d = bvhs[s];
  LocalStack<STACK> st;
  if (!run_btri<TIE>(d, __ldg(triOff + s), tris, verts, queries, qi, maxSqr, st, outIds, outD, outP))
    ovfList[atomicAdd(ovfCount, 1u)] = qi;
}

template <int TIE>
__global__ void k_btri_deep(const bq_bvh3f *__restrict__ bvhs, const uint32_t *__restrict__ triOff,
                            const uint32_t *__restrict__ qoff, uint32_t numSegs, const int32_t *__restrict__ tris,
                            const float *__restrict__ verts, const float *__restrict__ queries, float maxSqr,
                            int32_t *__restrict__ outIds, float *__restrict__ outD, float *__restrict__ outP,
                            const uint32_t *ovfList, const uint32_t *ovfCount, StackEntry *stacks, uint32_t *err)
{
  griddep_wait();
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t cnt = *ovfCount;
  for (uint32_t w = tid; w < cnt; w += gridDim.x * blockDim.x) {
    const uint32_t qi = ovfList[w];
    const uint32_t s = seg_of(qoff, numSegs, qi);
    GlobalStack st{stacks + (size_t)tid * DEEP_STACK, DEEP_STACK, 0};
    if (!run_btri<TIE>(bvhs[s], triOff[s], tris, verts, queries, qi, maxSqr, st, outIds, outD, outP)) {
      outIds[qi] = -1;
      outD[qi] = INFINITY;
      atomicOr(err, DEV_ERR_STACK);
    }
  }
}

// visiting order of the queries: mesh by mesh, along a Hilbert curve in the
// mesh's root box (as many of its top bits as the mesh index leaves)
__global__ void k_btri_keys(const bq_bvh3f *__restrict__ bvhs, const float *__restrict__ queries, uint32_t nq,
                            const uint32_t *__restrict__ qoff, uint32_t numSegs, int segBits,
                            uint32_t *__restrict__ keys, uint32_t *__restrict__ idx)
{
  griddep_wait();
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nq) return;
  const uint32_t s = seg_of(qoff, numSegs, t);
  const bq_bvh3f d = bvhs[s];
  const uint32_t h = d.numNodes ? query_order_key((const float *)d.nodes, queries + 3ull * t) : 0;
  keys[t] = (uint32_t)((((uint64_t)s << 30) | h) >> max(segBits - 2, 0));
  idx[t] = t;
}

} // namespace

int batched_refit(const bq_bvh3f *bvhs, const uint32_t *off, uint32_t numSegs, uint32_t numPrims, bq_node3f *nodes,
                  const uint32_t *primIDs, const bq_box3f *boxes, Alloc &al)
{
  if (numPrims == 0 || numSegs == 0) return BQ_OK;
  const uint32_t slots = 2 * numPrims;
  TempSet tmp(al);
  uint32_t *parent = nullptr, *counter = nullptr;
  BQ_TRY(tmp.get(&parent, slots));
  BQ_TRY(tmp.get(&counter, slots));
  ProfScope ps("batch.refit", al.s, 2);
  launch_pdl(k_brefit_parents, dim3(div_up(slots, 256)), dim3(256), 0, al.s, (const Node *)nodes, slots, bvhs, off,
             numSegs, parent, counter);
  launch_pdl(k_brefit_climb, dim3(div_up(slots, 128)), dim3(128), 0, al.s, (Node *)nodes, slots, bvhs, off, numSegs,
             primIDs, boxes, parent, counter);
  BQ_CUDA(cudaGetLastError());
  return BQ_OK;
}

int batched_tri_closest(const bq_bvh3f *bvhs, const uint32_t *triOff, const int32_t *tris, const float *verts,
                        const float *queries, const uint32_t *qoff, uint32_t numSegs, uint32_t nq, float maxSqr,
                        const bq_query_config *qcfg, int32_t *ids, float *d, float *P, uint32_t *errOut, Alloc &al)
{
  bq_query_config c;
  BQ_TRY(query_config(qcfg, c));
  if (nq == 0 || numSegs == 0) return BQ_OK;
  TempSet tmp(al);
  uint32_t *ovfList = nullptr, *ctl = nullptr;
  StackEntry *deep = nullptr;
  BQ_TRY(tmp.get(&ovfList, nq));
  BQ_TRY(tmp.get(&ctl, 4));  // overflow count, error word, heavy count, count left by the first launch
  BQ_TRY(tmp.get(&deep, (size_t)DEEP_THREADS * DEEP_STACK));
  BQ_CUDA(cudaMemsetAsync(ctl, 0, 16, al.s));
  uint32_t *err = errOut ? errOut : ctl + 1;
  const int b = c.blockSize;
  if (c.tieMode == BQ_TIES_LOWEST_ID) {
    // The order and the list of heavy queries save time only: without room for
    // them the queries are taken as given, and each by a thread.
    uint32_t *heavy = nullptr;
    const uint32_t *order = nullptr;
    int segBits = 0;
    while (segBits < 32 && (1ull << segBits) < numSegs) segBits++;
    // with few queries a mesh, order within a mesh saves less than it costs
    // (5,000 meshes of 320 triangles, 20 queries each: 0.366 and 0.296 ms)
    if (c.reorder && nq >= TRI_ORDER_MIN && nq / 256 >= numSegs) {
      const int kept = tmp.n;
      const int status = [&]() -> int {
        uint32_t *keys[2], *idx[2];
        BQ_TRY(tmp.get(&keys[0], nq));
        BQ_TRY(tmp.get(&keys[1], nq));
        BQ_TRY(tmp.get(&idx[0], nq));
        BQ_TRY(tmp.get(&idx[1], nq));
        ProfScope ps("batch.query_keys", al.s);
        launch_pdl(k_btri_keys, dim3(div_up(nq, 256)), dim3(256), 0, al.s, bvhs, queries, nq, qoff, numSegs, segBits,
                   keys[0], idx[0]);
        int sel = 0;
        // order only: 24 bits (3 passes) while they leave the curve at least 16
        BQ_TRY(onesweep_sort_u32(keys, idx, nq, nullptr, segBits <= 8 ? 8 - std::max(2 - segBits, 0) : 0,
                                 std::min(32, 30 + segBits), nullptr, &sel, err, al));
        order = idx[sel];
        heavy = keys[sel];  // the sorted keys are of no further use
        return BQ_OK;
      }();
      if (status == BQ_ERR_ALLOC) {
        tmp.release(kept);
        cudaGetLastError();
      } else {
        BQ_TRY(status);
      }
    }
    if (!heavy && tmp.get(&heavy, nq) != BQ_OK) {
      heavy = nullptr;
      cudaGetLastError();
    }
    const TriMesh m{nullptr, nullptr, bvhs, triOff, qoff, numSegs, nullptr, tris, verts};
    launch_tri_group(m, 0, queries, order, nq, maxSqr, ids, d, P, heavy, ovfList, ctl, ctl + 2, ctl + 3, nullptr, al.s);
    ProfScope ps("tri.deep", al.s);
    launch_pdl(k_btri_deep<TIE_LOWEST>, dim3(DEEP_THREADS / 128), dim3(128), 0, al.s, bvhs, triOff, qoff, numSegs, tris,
               verts, queries, maxSqr, ids, d, P, ovfList, ctl, deep, err);
    BQ_CUDA(cudaGetLastError());
    return BQ_OK;
  }
  ProfScope ps("batch.tri", al.s, 2);
#define BQ_BTRI(TIE, ST)                                                                                           \
  k_btri<TIE, ST><<<div_up(nq, b), b, 0, al.s>>>(bvhs, triOff, qoff, numSegs, tris, verts, queries, nq, maxSqr, ids, \
                                                 d, P, ovfList, ctl);                                              \
  k_btri_deep<TIE><<<DEEP_THREADS / 128, 128, 0, al.s>>>(bvhs, triOff, qoff, numSegs, tris, verts, queries, maxSqr,  \
                                                         ids, d, P, ovfList, ctl, deep, err)
  if (c.stackDepth == 32) { BQ_BTRI(TIE_REFERENCE, 32); }
  else if (c.stackDepth == 64) { BQ_BTRI(TIE_REFERENCE, 64); }
  else { BQ_BTRI(TIE_REFERENCE, 128); }
#undef BQ_BTRI
  BQ_CUDA(cudaGetLastError());
  return BQ_OK;
}

} // namespace bq
