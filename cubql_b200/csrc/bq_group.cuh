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
// loads: 32.7 ms, 25 with the warp's traversals in step; this takes 15.2 ms
// with 30 lanes active.  Of 2M over 2M (3.2 ms): issue slots 51% busy, L1 data
// pipe 56% of its wavefronts, 17 warps an SM (shared memory and registers)
// that wait on loads and on the list code, whose 16 keys lie in local memory.
// What made the difference, ms: inserting
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
                                             float maxSqr, uint32_t numQueries, uint32_t numPrims,
                                             KnnList<K, TIE_LOWEST> &list, GroupShared<K> &sh)
{
  constexpr int P = GroupShape<K>::P, C = GroupShape<K>::C;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t abovePair = 0xfffffffcu << (lane & ~1u);  // lanes of the pairs after this one's
  const uint32_t below = (1u << lane) - 1u;
  const float lx = warp_min_f(in ? qx : INFINITY), ly = warp_min_f(in ? qy : INFINITY),
              lz = warp_min_f(in ? qz : INFINITY);
  const float hx = warp_max_f(in ? qx : -INFINITY), hy = warp_max_f(in ? qy : -INFINITY),
              hz = warp_max_f(in ? qz : -INFINITY);
  const float diag2 = (hx - lx) * (hx - lx) + (hy - ly) * (hy - ly) + (hz - lz) * (hz - lz);
  {
    // Queries far from their neighbours on the curve, as those outside the
    // root's box are (the curve ends there): spread over 1,024 times the
    // space of 32 queries.  1M queries of which 1 in 27 is inside, 2M points,
    // k = 16: 4.3 ms without this, 3.4 with it, 3.6 one thread per query.
    const Node root = ldg_node(nodes);
    const float ext = fmaxf(fmaxf(root.a.w - root.a.x, root.b.x - root.a.y), root.b.y - root.a.z);
    if (diag2 * sqrtf(diag2) * (float)numQueries > 32.f * 1024.f * ext * ext * ext) return false;
  }
  // (dense queries: the box is small against the prims' spacing)
  const float far = (uint64_t)numQueries < 4ull * numPrims ? 4.f * diag2 : INFINITY;
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
    // The queries have too little in common for one search when their prims
    // are farther away than twice the size of their box (the shell between
    // the nearest and the farthest lane's reach holds thousands of prims),
    // when fewer than one lane wanted each prim that was tested, or when far
    // more prims were tested than a compact warp needs and not nearly every
    // lane wanted them (copies of one point are wanted by all).  500,000
    // queries in a cube, 1M points on a plane in it, k = 32: 7.2 ms without
    // the first, 3.8 with it, 4.4 one thread per query before; 300,000 points
    // on a line, k = 16: 37, 10 and 7.6 (the last limit: 13 without it).  The
    // limits on prims, 2 clouds, one of them clusters: 1.22 ms with 512 + 16 K
    // and 512 + 64 K, 2.76 with the first alone, 1.42 one thread per query.
    if (bounded && reach > far) return false;
    if (tested > 512 + 16 * K &&
        wanted < (tested > 2048 + 128 * K ? 16 : tested > 512 + 64 * K ? 8 : 1) * tested)
      return false;
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
// share a search.  Fewer queries have wide boxes that hold many prims no lane
// wants, and short lists are found sooner by a thread.  Uniform points, ms
// shared and a thread a query (k <= 5 plain, above in step), by queries a
// prim.  2M points: k = 1 at 1 1.27 and 1.01, at 4 2.81 and 3.26; k = 4 at 1
// 1.51 and 1.84 (but clustered data lose), at 2 2.12 and 3.23; k = 8 at 1/4
// 1.06 and 0.98, at 1 2.00 and 3.01; k = 16 at 1/4 1.82 and 1.58, at 1 3.55
// and 5.08; k = 32 at 1/4 2.88 and 3.21, at 1/2 3.78 and 5.77.  200,000
// points: k = 16 at 1/2 0.52 and 0.41, at 1 0.48 and 0.66.  20,000: k = 8 at 1
// 0.22 and 0.20, at 2 0.16 and 0.21; k = 16 at 1/2 0.37 and 0.24 (too few
// warps to hide the steps).  A handful of points is found at once by a thread:
// 1M queries, k = 1, 2,306 points 0.27 and 0.25, 10,000 0.29 and 0.31; k = 2,
// 100 points 0.25 and 0.21, 300 0.26 and 0.25 (20,000 queries 0.12 and 0.13).
__host__ __device__ inline bool group_pays(uint32_t numQueries, uint32_t numPrims, int k)
{
  const uint64_t q = numQueries, p = numPrims;
  if (k == 1) return q >= 4 * p && p >= 8192;
  if (k <= 4) return ((q >= 2 * p && q >= 32768) || q >= 8 * p) && p >= 256;
  if (k <= 16) return (q >= p || (2 * q >= p && q >= (1u << 19))) && p >= 32;
  return 2 * q >= p && p >= 32;
}

// Whether a ball of a finite radius can be expected to hold half the k prims
// that are looked for (were they spread evenly over the root's box).
__device__ __forceinline__ bool group_radius_pays(const Node *nodes, uint32_t numPrims, float maxSqr, int k)
{
  if (!(maxSqr < INFINITY)) return true;
  const Node n = ldg_node(nodes);
  const float r = sqrtf(fmaxf(maxSqr, 0.f));
  const float vx = fmaxf(n.a.w - n.a.x, r), vy = fmaxf(n.b.x - n.a.y, r), vz = fmaxf(n.b.y - n.a.z, r);
  return 8.f * r / vx * r / vy * r / vz * (float)numPrims >= (float)k;
}

// Blocks of 128 threads for the queries that the shared search has left: one
// for every 128 queries of the call, though most find nothing, as those left
// take very different times.  512 clouds: 58.9 ms with 64 blocks an SM that go
// through the list, 57.5 so.
inline int knn_left_blocks(uint32_t nq) { return div_up(nq, 128); }

// whether a query can take part: it is finite and its distance to the tree
// does not overflow (such a query would keep the reach infinite)
__device__ __forceinline__ bool group_can_search(const Node *nodes, float qx, float qy, float qz)
{
  const Node r = ldg_node(nodes);
  const float d = sqr_pbox(qx, qy, qz, r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y);
  return d < 1e37f && fabsf(qx) < 1e37f && fabsf(qy) < 1e37f && fabsf(qz) < 1e37f;
}

} // namespace bq
