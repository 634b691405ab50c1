// bq_tri.cuh -- closest triangle of a query by a group of lanes.
//
// A triangle query visits hundreds of nodes (inside a closed mesh most of
// the surface is nearly equidistant) and tests few triangles, and
// neighbouring queries need different numbers of steps: with one thread per
// query five of a warp's 32 lanes were active on average, and the few
// queries near the middle of a mesh kept their warps alive long after the
// rest had finished.  Here G lanes share one query: they take G nodes at a
// time off a stack in shared memory, push the children within the best
// distance so far, and test up to G queued triangles at once.  A group goes
// on to its next query as soon as one is answered, and starts it with the
// triangle that the last one found (a neighbour's answer is nearly always
// close), so culling works from the first step.  A query that takes more
// than TRI_STEP_LIMIT steps is left to a second launch with a whole warp each.
//
// Eight lanes are wasted on a query that needs few steps: one near the surface
// of a small mesh, or any over a handful of triangles.  Large batches over
// meshes of up to TRI_NEAR_PRIMS triangles therefore start with a thread a
// query, the warps in step, for some rounds; the groups get what is left, each
// query with the triangle found so far (figures at TRI_NEAR_PRIMS).
//
// 4M queries over 1.31M triangles: 46-50 ms with one thread per query (the
// last warps ran alone for 20 ms), 23.0 so: 20.9 for the first launch, bound by
// the L1 data pipe (90% of its wavefronts), 2.1 for the second.
// Four lanes a query 23.5 ms, sixteen 32.9; one lane a child instead of a
// pair of children 19.1 + 4.7 ms.  5,001 queries over the same mesh: 14.5
// -> 0.9 ms.  A batch of 128 meshes, 6.4M queries: 19.3 -> 14.6 ms by groups
// alone, 11.8 with threads first (sorting the queries, which it did not do
// before, takes 0.6 of it).
//
// The answer, the lowest id among equal distances, is a function of the query
// and the triangles alone, not of the tree, the batch or the visiting order
// (tri_reach, tri_key); the reference's tie rule keeps the per-thread
// traversal.
#pragma once

#include <algorithm>

#include "bq_traverse.cuh"

namespace bq {

// fewer queries are taken in the given order: sorting costs more than it
// saves (20,480 triangles, forward and adjoint, ms sorted and not: 5,003
// queries 0.579 and 0.500, 16,001 0.607 and 0.526, 50,001 0.736 and 0.701,
// 150,001 1.15 and 1.19; 1.31M triangles 1.11 and 1.10, 1.32 and 1.19, equal,
// 2.05 and 2.19)
constexpr uint32_t TRI_ORDER_MIN = 32768;

struct V3 {
  float x, y, z;
};
__device__ __forceinline__ V3 v3sub(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
// dot as the reference's accumulating loop (cuBQL/math/vec.h:459-466)
__device__ __forceinline__ float v3dot(V3 a, V3 b)
{
  float r = 0.f;
  r += a.x * b.x;
  r += a.y * b.y;
  r += a.z * b.z;
  return r;
}
// cuBQL/math/vec.h:232-237
__device__ __forceinline__ V3 v3cross(V3 a, V3 b)
{
  return V3{a.y * b.z - b.y * a.z, a.z * b.x - b.z * a.x, a.x * b.y - b.x * a.y};
}
__device__ __forceinline__ V3 ldv(const float *verts, int32_t i)
{
  const float *p = verts + 3ll * i;
  return V3{__ldg(p), __ldg(p + 1), __ldg(p + 2)};
}

// closest point on one triangle; region: 0 = inside (plane distance),
// 1 = edge ab, 2 = edge bc, 3 = edge ca; t = parameter along that edge
struct TriHit {
  float d;
  V3 P;
  int region;
  float t;
};

// Edge::closestPoint (findClosest.h:74-88)
__device__ __forceinline__ void edge_cp(TriHit &h, V3 a, V3 b, V3 p, int region)
{
  const V3 ba = v3sub(b, a);
  float t = v3dot(v3sub(p, a), ba) / v3dot(ba, ba);
  t = fminf(fmaxf(t, 0.f), 1.f);
  const V3 cp = V3{a.x + t * ba.x, a.y + t * ba.y, a.z + t * ba.z};
  const V3 dv = v3sub(cp, p);
  const float sd = v3dot(dv, dv);
  if (sd >= h.d) return;
  h.d = sd;
  h.P = cp;
  h.region = region;
  h.t = t;
}

// closestPoint(result, triangle, qp) (findClosest.h:93-122), evaluated
// against a running best starting at +inf
__device__ __forceinline__ TriHit tri_cp(V3 a, V3 b, V3 c, V3 qp)
{
  TriHit h;
  h.d = INFINITY;
  h.P = V3{0.f, 0.f, 0.f};
  h.region = -1;
  h.t = 0.f;
  V3 N = v3cross(v3sub(b, a), v3sub(c, a));
  const bool outside = (N.x == 0.f && N.y == 0.f && N.z == 0.f) ||
                       (v3dot(v3sub(qp, a), v3cross(v3sub(b, a), N)) >= 0.f) ||
                       (v3dot(v3sub(qp, b), v3cross(v3sub(c, b), N)) >= 0.f) ||
                       (v3dot(v3sub(qp, c), v3cross(v3sub(a, c), N)) >= 0.f);
  if (outside) {
    edge_cp(h, a, b, qp, 1);
    edge_cp(h, b, c, qp, 2);
    edge_cp(h, c, a, qp, 3);
    return h;
  }
  const float inv = 1.f / sqrtf(v3dot(N, N));
  N = V3{N.x * inv, N.y * inv, N.z * inv};
  const float sd = v3dot(v3sub(qp, a), N);
  h.d = sd * sd;
  h.P = V3{qp.x - sd * N.x, qp.y - sd * N.y, qp.z - sd * N.z};
  h.region = 0;
  return h;
}

// Lowest-id rule: culling that rounding cannot upset.  A closest point is
// computed as a + t * (b - a), off its triangle by up to sqrt(3) * 2^-24 *
// (|point| + |b - a|) in distance, and a plane distance carries the error of
// the normal, so a triangle can be nearer, as computed, than its own box.
// With the relative slack of the point queries its node was then visited or
// not according to what had been found before: of 1M queries 0.001 to 0.03
// from corners of unit triangles up to 56 changed their triangle with the
// batch.  So (1) nodes are visited up to the best distance plus TRI_ROUND of
// the coordinates at hand (query and distance), which covers edges up to some
// eight times as long; (2) a triangle that is nearer than its box by more
// than that (a sliver's plane) competes at the least distance at which its
// box is visited, and still reports its own.  Every box around a triangle is
// then visited while the triangle could win, whatever came first:
// tri_reach(tri_key(d, b)) >= b, and boxes of ancestors are no farther.
constexpr float TRI_ROUND = 0x1p-20f;

__device__ __forceinline__ float abs_max(V3 q) { return fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fabsf(q.z)); }

// squared distance up to which nodes are visited; qmax: abs_max(query)
__device__ __forceinline__ float tri_reach(float best, float qmax)
{
  const float r = sqrtf(fmaxf(best, 0.f));
  const float s = __fmaf_rn(TRI_ROUND, qmax + r, r);
  return lowest_slack(s * s);
}

// squared distance at which a triangle competes that is computed to be at d
// and whose box is at boxD
__device__ __forceinline__ float tri_key(float d, float boxD, float qmax)
{
  if (!(d < boxD)) return d;  // NaN stays NaN
  const float r = fmaxf(__fmaf_rn(-TRI_ROUND, qmax, sqrtf(boxD)), 0.f) * (1.f / (1.f + TRI_ROUND));
  return fmaxf(d, r * r);
}

__device__ __forceinline__ float tri_key(const TriHit &h, V3 a, V3 b, V3 c, V3 q, float qmax)
{
  const float boxD = sqr_pbox(q.x, q.y, q.z, fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y),
                              fminf(fminf(a.z, b.z), c.z), fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y),
                              fmaxf(fmaxf(a.z, b.z), c.z));
  return tri_key(h.d, boxD, qmax);
}

// leaf functor of the per-thread traversals over one tree
template <int TIE>
struct TriLeaf {
  const uint32_t *__restrict__ primIDs;
  const int32_t *__restrict__ tris;  // the tree's first triangle
  const float *__restrict__ verts;
  V3 q;
  float best;  // of the triangles met so far (lowest-id rule: tri_key's)
  int32_t id = -1;
  V3 P = V3{0.f, 0.f, 0.f};
  float d = INFINITY;  // distance of triangle `id`
  float qmax = 0.f;
  __device__ __forceinline__ TriLeaf(const uint32_t *p, const int32_t *t, const float *v, const float *qp, float maxSqr)
      : primIDs(p), tris(t), verts(v), q(V3{__ldg(qp), __ldg(qp + 1), __ldg(qp + 2)}), best(maxSqr)
  {
    if (TIE != TIE_REFERENCE) qmax = abs_max(q);
  }
  __device__ __forceinline__ float cull() const { return TIE == TIE_REFERENCE ? best : tri_reach(best, qmax); }
  __device__ __forceinline__ float operator()(uint64_t off, uint32_t cnt)
  {
    for (uint32_t j = 0; j < cnt; j++) {
      const uint32_t pid = __ldg(primIDs + off + j);
      const int32_t *t = tris + 3ull * pid;
      const V3 a = ldv(verts, __ldg(t)), b = ldv(verts, __ldg(t + 1)), c = ldv(verts, __ldg(t + 2));
      const TriHit h = tri_cp(a, b, c, q);
      const float key = TIE == TIE_REFERENCE ? h.d : tri_key(h, a, b, c, q, qmax);
      const bool take = (TIE == TIE_REFERENCE) ? (key < best)
                                               : (key < best || (key == best && id >= 0 && (int32_t)pid < id));
      if (take) {
        best = key;
        d = h.d;
        id = (int32_t)pid;
        P = h.P;
      }
    }
    return cull();
  }
};

namespace {
// ------------------------------------------------------------------
// closest triangle, G lanes per query
// ------------------------------------------------------------------
constexpr int TRI_GROUP = 8;           // lanes of a query in the first launch
constexpr int TRI_GROUP_STACK = 96;    // nodes on its stack
constexpr int TRI_HEAVY_STACK = 1024;  // on a whole warp's, in the second
// steps of the first launch; 4M queries, ms: 64 35.4, 192 25.4, 1024 27.2
// (forward and adjoint); 5,001 queries: 1.10, 1.10, 1.51
constexpr uint32_t TRI_STEP_LIMIT = 192;
// Where a thread a query goes first, and for how many rounds.  1M queries, ms
// by a thread alone, by groups alone, and with 256 rounds before the groups:
// within 0.01 of the surface of 80 triangles 0.22 0.72 0.24, of 20,480 0.68
// 1.59 0.59, of 81,920 1.37 2.03 1.05, of 327,680 3.28 2.90 2.24; in a cube
// around the mesh 0.46 0.90 0.42, 7.1 3.43 3.25, 8.1 3.71 4.12, 14.1 4.64
// 5.65.  So up to 2^17 triangles.  100,000 queries, 20,480 triangles, near
// 0.25 0.30 0.22, around 4.2 0.55 0.68 (0.64 with 128 rounds).  128 meshes of
// 2,000 to 100,000 triangles, a fitting step: groups alone 17.6, 128 rounds
// 16.5, 256 14.2.
constexpr uint32_t TRI_NEAR_PRIMS = 1u << 17;
constexpr uint32_t TRI_NEAR_MIN = 1u << 16;
inline uint32_t tri_near_rounds(uint32_t nq) { return nq < (1u << 18) ? 128 : 256; }
constexpr int TRI_NEAR_STACK = 64;     // entries of a thread's stack in the first of them

// One tree, or a batch of them.  `packed`: three float4 per triangle in leaf
// order (the corners; the first one's w holds the id), or null, and corners
// are fetched through the prim ids and index triples.
struct TriMesh {
  const Node *nodes;  // one tree
  const uint32_t *primIDs;
  const bq_bvh3f *bvhs;  // a batch (null: one tree)
  const uint32_t *triOff, *queryOff;
  uint32_t numSegs;
  const float4 *packed;
  const int32_t *tris;
  const float *verts;
};

// the triangle at leaf position `slot` of a tree whose first triangle is
// `base`; key: where it competes
__device__ __forceinline__ TriHit tri_test(const TriMesh &m, const uint32_t *primIDs, uint32_t base, uint32_t slot,
                                           V3 q, float qmax, int32_t &id, float &key)
{
  V3 a, b, c;
  if (m.packed) {
    const float4 *t = m.packed + 3ull * slot;
    const float4 ta = __ldg(t), tb = __ldg(t + 1), tc = __ldg(t + 2);
    a = V3{ta.x, ta.y, ta.z};
    b = V3{tb.x, tb.y, tb.z};
    c = V3{tc.x, tc.y, tc.z};
    id = __float_as_int(ta.w);
  } else {
    id = (int32_t)(base + __ldg(primIDs + slot));
    const int32_t *t = m.tris + 3ull * id;
    a = ldv(m.verts, __ldg(t));
    b = ldv(m.verts, __ldg(t + 1));
    c = ldv(m.verts, __ldg(t + 2));
  }
  const TriHit h = tri_cp(a, b, c, q);
  key = tri_key(h, a, b, c, q, qmax);
  return h;
}

template <int G, int CAP>
struct TriGroupShared {
  StackEntry stack[CAP];
  uint32_t queue[2 * G];
};

// leaf functor of a thread that answers a query by itself
struct TriNear {
  const TriMesh &m;
  const uint32_t *primIDs;
  uint32_t base;
  V3 q;
  float qmax, best;
  int32_t id = -1;
  uint32_t slot = 0;
  V3 P{0.f, 0.f, 0.f};
  float d = INFINITY;
  __device__ __forceinline__ TriNear(const TriMesh &m_, const uint32_t *p, uint32_t b, V3 q_, float maxSqr)
      : m(m_), primIDs(p), base(b), q(q_), qmax(abs_max(q_)), best(maxSqr)
  {
  }
  __device__ __forceinline__ float cull() const { return tri_reach(best, qmax); }
  __device__ __forceinline__ float operator()(uint64_t off, uint32_t cnt)
  {
    for (uint32_t j = 0; j < cnt; j++) {
      int32_t tid;
      float key;
      const TriHit h = tri_test(m, primIDs, base, (uint32_t)off + j, q, qmax, tid, key);
      if (key < best || (key == best && id >= 0 && tid < id)) {
        best = key;
        d = h.d;
        id = tid;
        P = h.P;
        slot = (uint32_t)off + j;
      }
    }
    return cull();
  }
};

// The warp's 32 / G groups answer queries at, at + stride, .. of `order`.
// SEEDED: they come from the list of an earlier launch, each with the place
// of the triangle it had found so far in outIds.  LIMIT: steps after which a
// query is left (0: none).
template <int G, int CAP, bool SEEDED, uint32_t LIMIT>
__device__ __forceinline__ void tri_group(const TriMesh &m, const float *__restrict__ queries,
                                          const uint32_t *__restrict__ order, uint32_t at, uint32_t end,
                                          uint32_t stride, float maxSqr, int32_t *outIds, float *outD, float *outP,
                                          uint32_t *leftList, uint32_t *leftCount, TriGroupShared<G, CAP> &sh)
{
  const uint32_t gl = threadIdx.x & (G - 1);                  // lane of the group
  const uint32_t shift = threadIdx.x & 31 & ~(uint32_t)(G - 1);  // the group's first lane
  const uint32_t ones = G == 32 ? 0xffffffffu : (1u << G) - 1u;
  const uint32_t below = (1u << gl) - 1u, above = (0xfffffffeu << gl) & ones;
  auto ballot = [&](bool p) { return (__ballot_sync(0xffffffffu, p) >> shift) & ones; };
  bool busy = false;
  uint32_t qi = 0, sp = 0, qn = 0, steps = 0;
  const Node *nodes = m.nodes;
  const uint32_t *primIDs = m.primIDs;
  uint32_t base = 0, seg = 0xffffffffu;
  V3 q{0.f, 0.f, 0.f};
  float best = 0.f, reach = 0.f, qmax = 0.f;
  int32_t id = -1;                 // best triangle of the group
  uint32_t slot = 0;               // where it is
  V3 P{0.f, 0.f, 0.f};             // the lane that tested it: its point and distance
  float ownD = -1.f;               // (negative: another lane did)
  uint32_t off0 = 0, cnt0 = 0, off1 = 0, cnt1 = 0;  // the leaves this lane found: nearer child, farther child
  while (true) {
    if (!busy && at < end) {
      qi = order ? __ldg(order + at) : at;
      at += stride;
      const float *p = queries + 3ull * qi;
      q = V3{__ldg(p), __ldg(p + 1), __ldg(p + 2)};
      qmax = abs_max(q);
      bool seeded = id >= 0;
      if (m.bvhs) {
        const uint32_t s = seg_of(m.queryOff, m.numSegs, qi);
        seeded = seeded && s == seg;
        seg = s;
        const bq_bvh3f d = m.bvhs[s];
        nodes = (const Node *)d.nodes;
        primIDs = d.primIDs;
        base = __ldg(m.triOff + s);
        busy = d.numNodes != 0;
      } else {
        busy = true;
      }
      best = maxSqr;
      id = -1;
      ownD = -1.f;
      steps = 0;
      // the last query's triangle and (odd lanes) the one found before
      uint32_t cand = slot;
      if (SEEDED && (gl & 1)) {
        cand = (uint32_t)outIds[qi];
        seeded = cand != 0xffffffffu;
      }
      TriHit h;
      float key = INFINITY;
      int32_t sid = 0x7fffffff;
      if (seeded) {
        h = tri_test(m, primIDs, base, cand, q, qmax, sid, key);
        if (!(key < best)) {
          key = INFINITY;
          sid = 0x7fffffff;
        }
      }
      bool owner = gl == 0;
      if (SEEDED) {
        const float okey = __shfl_xor_sync(ones << shift, key, 1);
        const int32_t osid = __shfl_xor_sync(ones << shift, sid, 1);
        const uint32_t ocand = __shfl_xor_sync(ones << shift, cand, 1);
        const bool mine = key < okey || (key == okey && (gl & 1 ? sid < osid : sid <= osid));
        owner = gl < 2 && mine;
        if (!mine) {
          key = okey;
          sid = osid;
          cand = ocand;
        }
      }
      if (sid != 0x7fffffff) {
        best = key;
        id = sid;
        slot = cand;
        if (owner) {
          P = h.P;
          ownD = h.d;
        }
      }
      reach = tri_reach(best, qmax);
      if (busy) {
        const uint64_t admin = ldg_admin(nodes);
        if (admin_count(admin) == 0) {
          if (gl == 0) sh.stack[0] = StackEntry{(uint32_t)admin_offset(admin), 0.f};
          sp = 1;
        } else if (gl == 0) {
          off0 = (uint32_t)admin_offset(admin);
          cnt0 = admin_count(admin);
        }
      } else if (gl == 0) {  // an empty tree
        outIds[qi] = -1;
        outD[qi] = INFINITY;
        if (outP) outP[3ull * qi] = outP[3ull * qi + 1] = outP[3ull * qi + 2] = 0.f;
      }
    }
    if (!__any_sync(0xffffffffu, busy || at < end)) return;
    __syncwarp();
    // take nodes; until a triangle is known nothing can be left out, so a
    // narrow front keeps the stack short on the way down
    const uint32_t w = min(min(id >= 0 || best < 3e38f ? (uint32_t)G : 2u, sp), (uint32_t)CAP - sp);
    const bool left = busy && sp != 0 && (w == 0 || (LIMIT && ++steps > LIMIT));
    bool act = busy && gl < w;
    sp -= w;
    StackEntry e{0, 0.f};
    if (act) e = sh.stack[sp + w - 1 - gl];  // lane 0: the top
    act = act && e.dist <= reach;
    __syncwarp();  // the entries read are overwritten below
    bool pushNear = false, pushFar = false;
    StackEntry nearE{0, 0.f}, farE{0, 0.f};
    if (act) {
      const Node n0 = ldg_node(nodes + e.idx), n1 = ldg_node(nodes + e.idx + 1);
      const float d0 = sqr_pbox(q.x, q.y, q.z, n0.a.x, n0.a.y, n0.a.z, n0.a.w, n0.b.x, n0.b.y);
      const float d1 = sqr_pbox(q.x, q.y, q.z, n1.a.x, n1.a.y, n1.a.z, n1.a.w, n1.b.x, n1.b.y);
      const uint64_t a0 = node_admin(n0), a1 = node_admin(n1);
      const bool swap = d1 < d0;
      const float dn = swap ? d1 : d0, df = swap ? d0 : d1;
      const uint64_t an = swap ? a1 : a0, af = swap ? a0 : a1;
      nearE = StackEntry{(uint32_t)admin_offset(an), dn};
      farE = StackEntry{(uint32_t)admin_offset(af), df};
      cnt0 = dn <= reach ? admin_count(an) : 0;
      cnt1 = df <= reach ? admin_count(af) : 0;
      pushNear = dn <= reach && cnt0 == 0;
      pushFar = df <= reach && cnt1 == 0;
      off0 = nearE.idx;
      off1 = farE.idx;
    }
    const uint32_t mn = ballot(pushNear), mf = ballot(pushFar);
    uint32_t to = sp + __popc(mn & above) + __popc(mf & above);
    if (pushFar) sh.stack[to++] = farE;
    if (pushNear) sh.stack[to] = nearE;
    sp += __popc(mn) + __popc(mf);
    // queue the triangles of the leaves found and test them: G at a time,
    // or what there is when the group has nothing else to do or no bound
    bool more = __any_sync(0xffffffffu, (cnt0 | cnt1) != 0 || (sp == 0 && qn != 0));
    while (more) {
      const bool has = (cnt0 | cnt1) != 0 && qn < G;
      const uint32_t mh = ballot(has);
      if (has) {
        sh.queue[qn + __popc(mh & below)] = cnt0 ? off0 : off1;
        if (cnt0) { off0++; cnt0--; }
        else { off1++; cnt1--; }
      }
      qn += __popc(mh);
      __syncwarp();
      const uint32_t waiting = ballot((cnt0 | cnt1) != 0);
      const bool due = qn >= G || (qn != 0 && waiting == 0 && (sp == 0 || id < 0));
      if (__any_sync(0xffffffffu, due)) {
        float td = INFINITY;
        int32_t tid = 0x7fffffff;
        TriHit h;
        uint32_t sl = 0;
        const uint32_t nb = min(qn, (uint32_t)G);
        if (gl < nb) {
          sl = sh.queue[gl];
          float key;
          h = tri_test(m, primIDs, base, sl, q, qmax, tid, key);
          // below the best, or as near with a lower id
          if (key < best || (key == best && id >= 0 && tid < id)) td = key;
          else tid = 0x7fffffff;
        }
        const uint32_t rest = G + gl < qn ? sh.queue[G + gl] : 0;
        float bd = td;
        int32_t bi = tid;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
          const float od = __shfl_xor_sync(0xffffffffu, bd, o);
          const int32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (od < bd || (od == bd && oi < bi)) { bd = od; bi = oi; }
        }
        if (bi != 0x7fffffff) {
          best = bd;
          reach = tri_reach(bd, qmax);
          id = bi;
          ownD = -1.f;
          if (tid == bi) {
            P = h.P;
            ownD = h.d;
          }
        }
        const uint32_t from = __ffs(ballot(tid == bi)) - 1;  // the lane that tested it
        const uint32_t ns = __shfl_sync(0xffffffffu, sl, from & (G - 1), G);
        if (bi != 0x7fffffff) slot = ns;
        __syncwarp();
        if (G + gl < qn) sh.queue[gl] = rest;
        qn -= nb;
        __syncwarp();
      }
      more = __any_sync(0xffffffffu, (cnt0 | cnt1) != 0 || (sp == 0 && qn != 0));
    }
    if (busy && (left || sp == 0)) {
      if (left && sp != 0) {
        if (gl == 0) {
          outIds[qi] = id >= 0 ? (int32_t)slot : -1;
          leftList[atomicAdd(leftCount, 1u)] = qi;
        }
        // triangles still queued are found again
      } else if (id >= 0 ? ownD >= 0.f : gl == 0) {
        outIds[qi] = id;
        outD[qi] = id >= 0 ? ownD : INFINITY;
        if (outP) {
          outP[3ull * qi] = id >= 0 ? P.x : 0.f;
          outP[3ull * qi + 1] = id >= 0 ? P.y : 0.f;
          outP[3ull * qi + 2] = id >= 0 ? P.z : 0.f;
        }
      }
      busy = false;
      sp = 0;
      qn = 0;
    }
  }
}

// A thread a query, the warps in step, for `rounds` rounds (TRI_ALL: to the
// end; in a batch, none for warps whose meshes are all too large); what is not
// answered then goes on a list, with the place of the triangle found so far in
// outIds.
constexpr uint32_t TRI_ALL = 0xffffffffu;
__global__ void __launch_bounds__(128) k_tri_near(TriMesh m, const float *__restrict__ queries,
                                                  const uint32_t *__restrict__ order, uint32_t nq, uint32_t rounds,
                                                  float maxSqr, int32_t *outIds, float *outD, float *outP,
                                                  uint32_t *leftList, uint32_t *leftCount, const uint32_t *stop)
{
  griddep_wait();
  if (stop && (*stop & DEV_ERR_RANGE)) return;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, tt = min(t, nq - 1);
  const uint32_t qi = order ? __ldg(order + tt) : tt;
  const float *p = queries + 3ull * qi;
  const V3 q{__ldg(p), __ldg(p + 1), __ldg(p + 2)};
  const Node *nodes = m.nodes;
  const uint32_t *primIDs = m.primIDs;
  uint32_t base = 0;
  bool tree = true;
  if (m.bvhs) {
    const uint32_t s = seg_of(m.queryOff, m.numSegs, qi);
    const bq_bvh3f d = m.bvhs[s];
    if (__all_sync(0xffffffffu, d.numPrims > TRI_NEAR_PRIMS) && rounds != TRI_ALL) rounds = 0;
    nodes = (const Node *)d.nodes;
    primIDs = d.primIDs;
    base = __ldg(m.triOff + s);
    tree = d.numNodes != 0;
  }
  TriNear leaf(m, primIDs, base, q, maxSqr);
  LocalStack<TRI_NEAR_STACK> st;
  const bool ok = traverse_warp<TIE_LOWEST, true>(nodes, q.x, q.y, q.z, leaf.cull(), st, leaf, t < nq && tree, rounds);
  if (t < nq) {
    if (ok) {
      outIds[qi] = leaf.id;
      outD[qi] = leaf.d;
      if (outP) {
        outP[3ull * qi] = leaf.P.x;
        outP[3ull * qi + 1] = leaf.P.y;
        outP[3ull * qi + 2] = leaf.P.z;
      }
    } else {
      outIds[qi] = leaf.id >= 0 ? (int32_t)leaf.slot : -1;
    }
  }
  list_append(t < nq && !ok, qi, leftList, leftCount);
}

// the queries of that list, by groups, each `run` next to each other
__global__ void __launch_bounds__(128, 8) k_tri_left(TriMesh m, const float *__restrict__ queries, uint32_t run,
                                                     float maxSqr, int32_t *outIds, float *outD, float *outP,
                                                     const uint32_t *__restrict__ list, const uint32_t *listCount,
                                                     uint32_t *leftList, uint32_t *leftCount)
{
  griddep_wait();
  __shared__ TriGroupShared<TRI_GROUP, TRI_GROUP_STACK> sh[128 / TRI_GROUP];
  const uint32_t g = threadIdx.x / TRI_GROUP, nq = *listCount;
  const uint64_t at = ((uint64_t)blockIdx.x * (128 / TRI_GROUP) + g) * run;
  const uint32_t b = (uint32_t)min(at, (uint64_t)nq), e = (uint32_t)min(at + run, (uint64_t)nq);
  tri_group<TRI_GROUP, TRI_GROUP_STACK, true, TRI_STEP_LIMIT>(m, queries, list, b, e, 1, maxSqr, outIds, outD, outP,
                                                              leftList, leftCount, sh[g]);
}

// each group answers `run` queries next to each other in the visiting order
__global__ void __launch_bounds__(128, 8) k_tri_group(TriMesh m, const float *__restrict__ queries,
                                                   const uint32_t *__restrict__ order, uint32_t nq, uint32_t run,
                                                   float maxSqr, int32_t *outIds, float *outD, float *outP,
                                                   uint32_t *leftList, uint32_t *leftCount, const uint32_t *stop)
{
  griddep_wait();
  if (stop && (*stop & DEV_ERR_RANGE)) return;
  __shared__ TriGroupShared<TRI_GROUP, TRI_GROUP_STACK> sh[128 / TRI_GROUP];
  const uint32_t g = threadIdx.x / TRI_GROUP;
  const uint64_t at = ((uint64_t)blockIdx.x * (128 / TRI_GROUP) + g) * run;
  const uint32_t b = (uint32_t)min(at, (uint64_t)nq), e = (uint32_t)min(at + run, (uint64_t)nq);
  tri_group<TRI_GROUP, TRI_GROUP_STACK, false, TRI_STEP_LIMIT>(m, queries, order, b, e, 1, maxSqr, outIds, outD, outP,
                                                               leftList, leftCount, sh[g]);
}

__global__ void __launch_bounds__(128) k_tri_heavy(TriMesh m, const float *__restrict__ queries, float maxSqr,
                                                   int32_t *outIds, float *outD, float *outP,
                                                   const uint32_t *__restrict__ list, const uint32_t *listCount,
                                                   uint32_t *leftList, uint32_t *leftCount)
{
  griddep_wait();
  __shared__ TriGroupShared<32, TRI_HEAVY_STACK> sh[4];
  const uint32_t warp = threadIdx.x >> 5;
  tri_group<32, TRI_HEAVY_STACK, true, 0>(m, queries, list, blockIdx.x * 4 + warp, *listCount, gridDim.x * 4, maxSqr,
                                       outIds, outD, outP, leftList, leftCount, sh[warp]);
}

// queries a group answers one after the other: each but the first starts
// from its neighbour's triangle, while every SM still gets its groups
inline uint32_t tri_run(uint32_t nq) { return std::min(8u, std::max(1u, nq >> 17)); }

__device__ __forceinline__ void pack_corners(uint32_t j, const uint32_t *__restrict__ primIDs,
                                             const int32_t *__restrict__ tris, const float *__restrict__ verts,
                                             float4 *__restrict__ packed)
{
  const uint32_t id = __ldg(primIDs + j);
  const int32_t *t = tris + 3ull * id;
  const V3 a = ldv(verts, __ldg(t)), b = ldv(verts, __ldg(t + 1)), c = ldv(verts, __ldg(t + 2));
  packed[3ull * j] = make_float4(a.x, a.y, a.z, __uint_as_float(id));
  packed[3ull * j + 1] = make_float4(b.x, b.y, b.z, 0.f);
  packed[3ull * j + 2] = make_float4(c.x, c.y, c.z, 0.f);
}

// Corners of the triangles in leaf order.  Leaf by leaf, a thread a node: the
// list of prim ids may go on after the last leaf with prims that have no box,
// and their index triples need not be usable.  Long leaves are shared by the
// warp.  A leaf that goes past numPrims sets DEV_ERR_RANGE, and the search that
// would use the copy does not start (`stop`).
__global__ void k_tri_pack(const Node *__restrict__ nodes, uint32_t numNodes, const uint32_t *__restrict__ primIDs,
                           uint32_t numPrims, const int32_t *__restrict__ tris, const float *__restrict__ verts,
                           float4 *__restrict__ packed, uint32_t *err)
{
  griddep_wait();
  constexpr uint32_t SHORT = 4;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  uint32_t off = 0, cnt = 0;
  if (t < numNodes && t != 1) {  // node 1 is unused
    const uint64_t admin = ldg_admin(nodes + t);
    off = (uint32_t)admin_offset(admin);
    cnt = admin_count(admin);
    if (cnt && (uint64_t)off + cnt > numPrims) {
      atomicOr(err, DEV_ERR_RANGE);
      cnt = 0;
    }
  }
  if (cnt <= SHORT)
    for (uint32_t j = 0; j < cnt; j++) pack_corners(off + j, primIDs, tris, verts, packed);
  for (uint32_t m = __ballot_sync(0xffffffffu, cnt > SHORT); m; m &= m - 1) {
    const uint32_t from = __ffs(m) - 1;
    const uint32_t o = __shfl_sync(0xffffffffu, off, from), n = __shfl_sync(0xffffffffu, cnt, from);
    for (uint32_t j = lane; j < n; j += 32) pack_corners(o + j, primIDs, tris, verts, packed);
  }
}

// The launches; queries that none finished are on ovfList.  numPrims: of the
// tree (0 for a batch: k_tri_near looks at each).  heavy: a list of nq words, or
// null when there is no room for one: each query is then answered by a thread.
// The counts are zeroed.  stop: the word in which k_tri_pack reports, or null.
inline void launch_tri_group(const TriMesh &m, uint32_t numPrims, const float *queries, const uint32_t *order,
                             uint32_t nq, float maxSqr, int32_t *ids, float *d, float *P, uint32_t *heavy,
                             uint32_t *ovfList, uint32_t *ovfCount, uint32_t *heavyCount, uint32_t *nearCount,
                             const uint32_t *stop, cudaStream_t s)
{
  const uint32_t run = tri_run(nq);
  if (!heavy) {
    ProfScope ps("tri.near", s);
    launch_pdl(k_tri_near, dim3(div_up(nq, 128)), dim3(128), 0, s, m, queries, order, nq, TRI_ALL, maxSqr, ids, d, P,
               ovfList, ovfCount, stop);
    return;
  }
  if (nq >= TRI_NEAR_MIN && numPrims <= TRI_NEAR_PRIMS) {
    {
      ProfScope ps("tri.near", s);
      launch_pdl(k_tri_near, dim3(div_up(nq, 128)), dim3(128), 0, s, m, queries, order, nq,
                 tri_near_rounds(nq), maxSqr, ids, d, P, ovfList, nearCount, stop);
    }
    ProfScope ps("tri.group", s);
    launch_pdl(k_tri_left, dim3(div_up((uint64_t)div_up(nq, run) * TRI_GROUP, 128)), dim3(128), 0, s, m, queries, run,
               maxSqr, ids, d, P, (const uint32_t *)ovfList, (const uint32_t *)nearCount, heavy, heavyCount);
  } else {
    ProfScope ps("tri.group", s);
    launch_pdl(k_tri_group, dim3(div_up((uint64_t)div_up(nq, run) * TRI_GROUP, 128)), dim3(128), 0, s, m, queries,
               order, nq, run, maxSqr, ids, d, P, heavy, heavyCount, stop);
  }
  ProfScope ps("tri.heavy", s);
  launch_pdl(k_tri_heavy, dim3(4 * num_sms()), dim3(128), 0, s, m, queries, maxSqr, ids, d, P,
             (const uint32_t *)heavy, (const uint32_t *)heavyCount, ovfList, ovfCount);
}
} // namespace
} // namespace bq
