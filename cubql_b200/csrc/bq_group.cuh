// bq_group.cuh -- nearest-neighbour search of a warp's 32 queries at once.
//
// The queries of a warp are neighbours (they come sorted along a Hilbert
// curve), so they want nearly the same prims.  Instead of 32 traversals
// that diverge, the warp makes one: its lanes take 32 NODES at a time off a
// stack in shared memory and keep those within reach of the box around the
// 32 queries (reach: the largest k-th best distance so far).  The prims
// found are gathered 32 at a time into shared memory, and every lane tests
// all of them against its own query.  Node loads and point gathers are
// spread over the lanes and the distance tests run without divergence.
//
// What it costs, 10M uniform points and queries, k = 16, per warp: 55 steps
// down the tree (25 of them before every lane has k prims), 481 prims
// tested, 64 of them wanted by a lane, 8 merges.  One thread per query had 5
// of 32 lanes active and 76,000 instructions a warp, waiting on dependent
// loads: 32.7 ms; this takes 15.0 ms, bound by issue slots and the L1 data
// pipe (67% of its wavefronts).  What made the difference, ms: inserting
// each prim into the sorted list as it is met 53, merging 16 at a time 15.7,
// registers capped for five blocks an SM 15.0.  The Hilbert order instead of
// Morton: 2M points, 1M queries, k = 32: 10.9 -> 5.2 before the merges, as a
// run of a Morton curve jumps and its box is then large.
//
// The answer does not depend on the order in which prims are met: the list
// keeps the k smallest (distance, id) pairs, so this serves the lowest-id
// tie rule only; the reference's rule keeps the traversal of
// bq_traverse.cuh.
#pragma once

#include "bq_traverse.cuh"

namespace bq {

constexpr int GROUP_STACK = 320;  // nodes on a warp's stack
constexpr int GROUP_QUEUE = 64;   // prim slots waiting for a batch of 32

// What a lane has found but not yet merged into its list: up to P keys are
// merged at once, and a chunk of C prims is tested between two looks at
// whether a merge is due.
template <int K>
struct GroupShape {
  static constexpr int P = K < 16 ? K : 16;
  static constexpr int C = K < 8 ? 4 : 8;
  static constexpr int BLOCKS = K < 8 ? 8 : K < 16 ? 6 : K < 32 ? 5 : 4;  // of 128 threads an SM
};

template <int K>
struct GroupShared {
  uint64_t pend[GroupShape<K>::P + GroupShape<K>::C][32];
  float4 cand[32];  // x y z, prim id
  StackEntry stack[GROUP_STACK];
  uint32_t queue[GROUP_QUEUE];
};

__device__ __forceinline__ void key_exchange(uint64_t &a, uint64_t &b)
{
  const bool s = b < a;
  const uint64_t t = s ? b : a;
  b = s ? a : b;
  a = t;
}

// the smallest K of the list (sorted) and P more keys (any order), sorted:
// the keys are sorted by Batcher's odd-even merge sort, the K smallest of
// both are a bitonic sequence, which log2 K rounds of exchanges sort
template <int K, int P>
__device__ __forceinline__ void merge_keys(uint64_t (&L)[K], uint64_t (&k)[P])
{
#pragma unroll
  for (int p = 1; p < P; p *= 2)
#pragma unroll
    for (int q = p; q >= 1; q /= 2)
#pragma unroll
      for (int j = q % p; j <= P - 1 - q; j += 2 * q)
#pragma unroll
        for (int i = 0; i < q; i++)
          if (i + j + q < P && (i + j) / (2 * p) == (i + j + q) / (2 * p)) key_exchange(k[i + j], k[i + j + q]);
#pragma unroll
  for (int i = K - P; i < K; i++) L[i] = k[K - 1 - i] < L[i] ? k[K - 1 - i] : L[i];
#pragma unroll
  for (int q = K / 2; q >= 1; q /= 2)
#pragma unroll
    for (int i = 0; i < K; i++)
      if ((i & q) == 0) key_exchange(L[i], L[i + q]);
}

// squared distance between a node's box and the queries' box
__device__ __forceinline__ float sqr_boxbox(const Node &n, float lx, float ly, float lz, float hx, float hy, float hz)
{
  const float gx = fmaxf(fmaxf(n.a.x - hx, lx - n.a.w), 0.f);
  const float gy = fmaxf(fmaxf(n.a.y - hy, ly - n.b.x), 0.f);
  const float gz = fmaxf(fmaxf(n.a.z - hz, lz - n.b.y), 0.f);
  return gx * gx + gy * gy + gz * gz;
}

__device__ __forceinline__ float warp_min_f(float x) { return dec_f(__reduce_min_sync(0xffffffffu, enc_f(x))); }
__device__ __forceinline__ float warp_max_f(float x) { return dec_f(__reduce_max_sync(0xffffffffu, enc_f(x))); }

// Whole warp; `in`: this lane's query takes part.  Returns whether the
// search was finished (the same for all lanes): false if the stack was full
// or the queries turned out too far apart; the lists then hold a subset of
// the candidates, so their k-th best are upper bounds.
template <int K>
__device__ __forceinline__ bool group_search(const Node *__restrict__ nodes, const uint32_t *__restrict__ primIDs,
                                             const float *__restrict__ points, bool in, float qx, float qy, float qz,
                                             float maxSqr, KnnList<K, TIE_LOWEST> &list, GroupShared<K> &sh)
{
  constexpr int P = GroupShape<K>::P, C = GroupShape<K>::C;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t abovePair = 0xfffffffcu << (lane & ~1u);  // lanes of the pairs after this one's
  const uint32_t below = (1u << lane) - 1u;
  const float lx = warp_min_f(in ? qx : INFINITY), ly = warp_min_f(in ? qy : INFINITY),
              lz = warp_min_f(in ? qz : INFINITY);
  const float hx = warp_max_f(in ? qx : -INFINITY), hy = warp_max_f(in ? qy : -INFINITY),
              hz = warp_max_f(in ? qz : -INFINITY);
  // a prim is wanted at up to `mine`: below the radius, and no farther than
  // the k-th best (at the same distance its id decides)
  const float limit = maxSqr > 0.f ? __uint_as_float(__float_as_uint(maxSqr) - 1) : -1.f;
  float mine = in ? fminf(limit, list.worst()) : -1.f;
  auto warp_reach = [&]() {
    return lowest_slack(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(mine, 0.f)))));
  };
  float reach = warp_reach();
  bool bounded = reach < 3e38f;
  uint32_t np = 0;  // keys pending
  auto merge_pending = [&]() {
    uint64_t k[P];
#pragma unroll
    for (int i = 0; i < P; i++) k[i] = (uint32_t)i < np ? sh.pend[np - 1 - i][lane] : KNN_KEY_EMPTY;
    np -= min(np, (uint32_t)P);
    merge_keys<K, P>(list.L, k);
    if (in) mine = fminf(limit, list.worst());
  };
  uint32_t sp = 0, nq = 0, tested = 0, wanted = 0;
  uint32_t off = 0, cnt = 0;  // the leaf this lane found
  {
    const uint64_t admin = ldg_admin(nodes);
    if (admin_count(admin) == 0) {
      if (lane == 0) sh.stack[0] = StackEntry{(uint32_t)admin_offset(admin), 0.f};
      sp = 1;
    } else if (lane == 0) {
      off = (uint32_t)admin_offset(admin);
      cnt = admin_count(admin);
    }
  }
  __syncwarp();
  while (true) {
    // queue the prims of the leaves found, one of each leaf at a time; a
    // batch of 32 (the rest, once nothing is left to visit) is tested
    while (true) {
      const bool has = cnt != 0;
      const uint32_t m = __ballot_sync(0xffffffffu, has);
      if (m) {
        if (has) {
          sh.queue[nq + __popc(m & below)] = off++;
          cnt--;
        }
        nq += __popc(m);
        __syncwarp();
      }
      if (nq < 32 && (m || sp || nq == 0)) {
        if (m) continue;
        break;
      }
      // test a batch
      const uint32_t nb = min(nq, 32u);
      if (lane < nb) {
        const uint32_t pid = __ldg(primIDs + sh.queue[lane]);
        const float *p = points + 3ull * pid;
        sh.cand[lane] = make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __uint_as_float(pid));
      } else {
        sh.cand[lane] = make_float4(NAN, NAN, NAN, 0.f);  // never within reach
      }
      const uint32_t rest = 32 + lane < nq ? sh.queue[32 + lane] : 0;
      __syncwarp();
      if (32 + lane < nq) sh.queue[lane] = rest;
      nq -= nb;
      const uint32_t before = np;
      uint32_t merged = 0;
#pragma unroll 1
      for (int c0 = 0; c0 < 32; c0 += C) {
#pragma unroll
        for (int c = c0; c < c0 + C; c++) {
          const float4 p = sh.cand[c];
          const float d = sqr_pp(p.x, p.y, p.z, qx, qy, qz);
          if (d <= mine) {
            sh.pend[np][lane] = ((uint64_t)__float_as_uint(d) << 32) | __float_as_uint(p.w);
            np++;
          }
        }
        if (__any_sync(0xffffffffu, np > P)) {
          merged += min(np, (uint32_t)P);
          merge_pending();
        }
      }
      tested += nb;
      wanted += __reduce_add_sync(0xffffffffu, np + merged - before);
      reach = warp_reach();
      bounded = reach < 3e38f;
      __syncwarp();
    }
    if (sp == 0) break;  // the queue is empty too
    // The queries are too far apart for one search when fewer than one lane
    // wanted each prim that was tested, or far more prims were tested than a
    // compact warp needs and not nearly every lane wanted them (copies of one
    // point are wanted by all).  Queries far from the prims they look for are
    // the case: without the second limit a warp tests thousands of prims.
    // 2 clouds, one of them clusters: 1.22 ms with both, 2.76 with the first
    // alone, 1.42 one thread per query; 512 clouds 69.8, 75.9, 83.8.
    if (tested > 512 + 16 * K && wanted < (tested > 512 + 64 * K ? 8 : 1) * tested) return false;
    // Until k prims are known to every lane nothing can be left out: a
    // narrow front then keeps the stack short on the way down.
    const uint32_t w = min(min(bounded ? 16u : 4u, sp), (uint32_t)GROUP_STACK - sp);
    if (w == 0) return false;
    sp -= w;
    StackEntry e{0, 0.f};
    bool act = lane / 2 < w;
    if (act) e = sh.stack[sp + w - 1 - lane / 2];  // lanes 0 and 1: the top
    act = act && e.dist <= reach;
    __syncwarp();  // the entries read are overwritten below
    if (!__any_sync(0xffffffffu, act)) continue;
    float d = INFINITY;
    uint64_t admin = 0;
    if (act) {
      const Node n = ldg_node(nodes + e.idx + (lane & 1));
      d = sqr_boxbox(n, lx, ly, lz, hx, hy, hz);
      admin = node_admin(n);
    }
    const float sibling = __shfl_xor_sync(0xffffffffu, d, 1);
    const bool hit = act && d <= reach;
    const bool push = hit && admin_count(admin) == 0;
    const uint32_t mp = __ballot_sync(0xffffffffu, push);
    if (push) {  // the nearer child above the other, lane 0's above all
      const bool nearer = d < sibling || (d == sibling && !(lane & 1));
      const uint32_t to = sp + __popc(mp & abovePair) + (nearer ? mp >> (lane ^ 1) & 1 : 0);
      sh.stack[to] = StackEntry{(uint32_t)admin_offset(admin), d};
    }
    sp += __popc(mp);
    if (hit && !push) {
      off = (uint32_t)admin_offset(admin);
      cnt = admin_count(admin);
    }
    __syncwarp();
  }
  while (__any_sync(0xffffffffu, np != 0)) merge_pending();
  return true;
}

// Whether the queries are dense enough among the prims for a warp's 32 to
// share a search (a warp whose queries are not gives up by itself).  Below
// this the box of 32 queries holds hundreds of prims that no lane wants:
// 200,000 queries over 3M points, k = 16, take 1.95 ms shared and 1.0 ms one
// thread each; 3,000 over 5M 4.3 and 0.32 ms; 1M over 2M, k = 32, 3.7 and
// 10.5 ms.
__host__ __device__ inline bool group_pays(uint32_t numQueries, uint32_t numPrims)
{
  return (uint64_t)numQueries * 8 >= numPrims;
}

// whether a query can take part: it is finite and its distance to the tree
// does not overflow (such a query would keep the reach infinite)
__device__ __forceinline__ bool group_can_search(const Node *nodes, float qx, float qy, float qz)
{
  const Node r = ldg_node(nodes);
  const float d = sqr_pbox(qx, qy, qz, r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y);
  return d < 1e37f && fabsf(qx) < 1e37f && fabsf(qy) < 1e37f && fabsf(qz) < 1e37f;
}

} // namespace bq
