// The fast exact kNN / FCP traversal of one query over a float or int32 tree
// (D = 2..4, k <= 128): the body of knn_fast_kernel (fast_kernel.cuh) and of
// the learned path's fused kernel (learned.cu).  Why the answer is the
// reference's, whatever the visiting order, is argued in fast.cu's header.
#pragma once

#include "common.cuh"
#include "fast.cuh"

namespace ckb {
namespace fast {

// Coordinate arithmetic.  `sq` and `add` give the float distance bound L the
// traversal works with; `exact` the squared distance the answer is made of.
// Floats: L is the exact distance (the reference's rounding, no FMA
// contraction).  Ints: every step rounds down, so L never exceeds the exact
// int64 distance and falls short of it by less than (D + 2) 2^-23 of it (a
// rounding each for the difference, which the square doubles, the square and
// the additions); L grows
// with every |coordinate difference|, so a box's L (of its closest point)
// never exceeds the L of a point inside.
template <int SC> struct Num;
template <> struct Num<0> {
  using T = float;
  using E = float;  // squared distances of the answer
  __device__ static float sq(T a, T b)
  {
    const float d = __fsub_rn(a, b);
    return __fmul_rn(d, d);
  }
  __device__ static float add(float a, float b) { return __fadd_rn(a, b); }
  __device__ static E exact_sq(T a, T b) { return sq(a, b); }
  __device__ static E exact_add(E a, E b) { return __fadd_rn(a, b); }
  // bits of a float at or below / at or above a distance of the answer
  __device__ static uint32_t below(E e) { return __float_as_uint(e); }
  __device__ static uint32_t above(E e) { return __float_as_uint(e); }
  __device__ static E farthest() { return __uint_as_float(0x7f800000u); }
  __device__ static E cutoff(const query::QArgs &a) { return __fmul_rn(a.cutoff, a.cutoff); }
  __device__ static E seeded(E r2, float radius, float scale)
  {
    const float rr = __fmul_rn(radius, scale);
    const float rb = __fmul_rn(rr, rr);
    return rb < r2 ? rb : r2;
  }
  __device__ static bool usable(E r2) { return r2 >= 0.f; }  // not NaN
};
template <> struct Num<1> {
  using T = int32_t;
  using E = long long;
  __device__ static float sq(T a, T b)
  {
    const uint32_t d = a > b ? uint32_t(a) - uint32_t(b) : uint32_t(b) - uint32_t(a);
    const float f = __uint2float_rd(d);
    return __fmul_rd(f, f);
  }
  __device__ static float add(float a, float b) { return __fadd_rd(a, b); }
  __device__ static E exact_sq(T a, T b)
  {
    const long long d = (long long)a - (long long)b;
    return d * d;
  }
  __device__ static E exact_add(E a, E b) { return a + b; }
  __device__ static uint32_t below(E e) { return __float_as_uint(__ll2float_rd(e)); }
  __device__ static uint32_t above(E e) { return __float_as_uint(__ll2float_ru(e)); }
  __device__ static E farthest() { return 0x7fffffffffffffffll; }
  __device__ static E cutoff(const query::QArgs &a) { return a.cutoff_d2; }
  __device__ static E seeded(E r2, float radius, float scale)
  {
    // any bound is exact (the answer is checked); only the number of
    // fallbacks depends on it
    const double rr = double(radius) * double(scale);
    const double rb = ceil(rr * rr);
    const long long s = rb >= 9.0e18 ? 0x7fffffffffffffffll : (long long)rb;
    return s < r2 ? s : r2;
  }
  __device__ static bool usable(E r2) { return r2 >= 0; }
};

// Reads a node's point, its split dim, or both.  VEC: the point is one
// vector load (8 bytes for D = 2, 16 for D = 3 and 4; for D = 3 with
// explicit dims the fourth word holds the dim).
template <int SC, int D, bool EXPL, bool VEC>
struct Nodes {
  using T = typename Num<SC>::T;
  const uint8_t *tree;
  int stride, poff, doff, dshift;
  uint32_t dmask;
  __device__ __forceinline__ Nodes(const query::QArgs &a, const uint8_t *t)
      : tree(t), stride(a.stride), poff(a.poff), doff(a.doff), dshift(a.dshift), dmask(a.dmask)
  {
  }
  __device__ __forceinline__ static T word(uint32_t w)
  {
    T v;
    memcpy(&v, &w, 4);
    return v;
  }
  __device__ __forceinline__ int dim_of(int node) const
  {
    if (!EXPL) return level_of(node) % D;
    return int((__ldg((const uint32_t *)(tree + int64_t(node) * stride + doff)) >> dshift) & dmask);
  }
  __device__ __forceinline__ int load(int node, T (&p)[D]) const  // point and dim
  {
    if (VEC && D == 3) {
      const uint4 v = __ldg((const uint4 *)(tree + int64_t(node) * stride + poff));
      p[0] = word(v.x);
      p[1] = word(v.y);
      if (D > 2) p[D > 2 ? 2 : 0] = word(v.z);
      return EXPL ? int((v.w >> dshift) & dmask) : level_of(node) % D;
    }
    point(node, p);
    return dim_of(node);
  }
  // the same for a node whose level is known
  __device__ __forceinline__ int load_at(int node, int lvl, T (&p)[D]) const
  {
    if (EXPL) return load(node, p);
    point(node, p);
    return lvl % D;
  }
  __device__ __forceinline__ void point(int node, T (&p)[D]) const
  {
    const uint8_t *c = tree + int64_t(node) * stride + poff;
    if (VEC && D == 2) {
      const uint2 v = __ldg((const uint2 *)c);
      p[0] = word(v.x);
      p[1] = word(v.y);
    } else if (VEC) {
      const uint4 v = __ldg((const uint4 *)c);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int d = 0; d < D; d++) p[d] = word(w[d]);
    } else {
#pragma unroll
      for (int d = 0; d < D; d++) p[d] = __ldg((const T *)c + d);
    }
  }
  // the split coordinate of a node at level lvl
  __device__ __forceinline__ T split(int node, int lvl, int *dim) const
  {
    if (VEC && D == 3 && EXPL) {
      T p[D];
      const int dd = load(node, p);
      T c = p[0];
#pragma unroll
      for (int d = 1; d < D; d++) c = d == dd ? p[d] : c;
      *dim = dd;
      return c;
    }
    const int dd = EXPL ? dim_of(node) : lvl % D;
    *dim = dd;
    // (a record whose dim is none of the point's reads as if it were the first)
    return __ldg((const T *)(tree + int64_t(node) * stride + poff) + (uint32_t(dd) < D ? dd : 0));
  }
};

template <int SC, int D>
__device__ __forceinline__ typename Num<SC>::E exact_d2(const typename Num<SC>::T (&a)[D],
                                                        const typename Num<SC>::T (&b)[D])
{
  using N = Num<SC>;
  typename N::E s = N::exact_sq(a[0], b[0]);
#pragma unroll
  for (int d = 1; d < D; d++) s = N::exact_add(s, N::exact_sq(a[d], b[d]));
  return s;
}

// Which side of a split the traversal `method` takes first: the left one for a
// query strictly left of the plane (stack-based, cct) or not right of it
// (stack-free).
template <class T> __device__ __forceinline__ bool left_first(int method, T qc, T c)
{
  return method == CUKD_STACK_FREE ? !(qc > c) : qc < c;
}

// Whether the reference's traversal `method` visits `node` whatever its
// candidate list holds meanwhile, X being the final k-th distance: its list's
// cull distance never drops below X, and it skips a child only on the far
// side, when the child's plane (cct: box) distance is not below the cull
// distance.  So a node is visited for sure when every far-side step on its
// path has a distance below X.
//
// For a single candidate (FCP, k = 1) the cull distance is above X until the
// first point at distance X is visited, and X from then on.  With that point
// in `first`, a far side at distance X is entered exactly when it holds
// `first`, and the outcome is exact: the node is visited, or it is not.
template <int SC, int D, bool EXPL, bool VEC>
__device__ __forceinline__ bool surely_visited(const FastArgs &fa, const Nodes<SC, D, EXPL, VEC> &nd,
                               const typename Num<SC>::T (&q)[D], const void *bounds, int node,
                               typename Num<SC>::E X, int first = -1)
{
  using N = Num<SC>;
  using T = typename N::T;
  T close[D];
#pragma unroll
  for (int d = 0; d < D; d++) {
    close[d] = q[d];
    if (fa.method == CUKD_CCT) {
      const T lo = __ldg((const T *)bounds + d), hi = __ldg((const T *)bounds + D + d);
      T v = q[d];
      v = v < lo ? lo : v;
      v = hi < v ? hi : v;
      close[d] = v;
    }
  }
  const int depth = level_of(node), firstDepth = first < 0 ? -1 : level_of(first);
#pragma unroll 1
  for (int lvl = 0; lvl < depth; lvl++) {
    const int a = ((node + 1) >> (depth - lvl)) - 1;
    const int child = (node + 1) >> (depth - lvl - 1);  // (+ 1)
    int dim;
    const T c = nd.split(a, lvl, &dim);
    T qc = q[0];
#pragma unroll
    for (int d = 1; d < D; d++) qc = d == dim ? q[d] : qc;
    if (((child & 1) == 0) == left_first(fa.method, qc, c)) continue;  // the near side
    bool in;
    if (fa.method == CUKD_CCT) {
#pragma unroll
      for (int d = 0; d < D; d++) close[d] = d == dim ? c : close[d];
      in = exact_d2<SC, D>(close, q) < X;
    } else {
      in = N::exact_sq(qc, c) < X;
    }
    if (!in && (firstDepth <= lvl || ((first + 1) >> (firstDepth - lvl - 1)) != child)) return false;
  }
  return true;
}

// The rare end of a query: candidates that the truncated keys left in the
// wrong order, or an exact distance tie at the k-th boundary.  Sorts the
// query's row of ids (already written) and the (k+1)-th candidate yid by
// (d2, id) and settles the answer where that can be done without the
// reference's visiting order: a tie is settled when every candidate taken
// at the tied distance is surely visited by the reference (it keeps the
// smallest (d2, id) keys among the nodes it visits).  false: the query has
// to be re-run.
template <int SC, int D, bool EXPL, bool VEC>
__device__ __forceinline__ bool settle_row(const FastArgs &fa, int64_t myq, typename Num<SC>::E r2,
                                        uint32_t safe, bool hasSeed, int yid)
{
  using N = Num<SC>;
  using T = typename N::T;
  using E = typename N::E;
  const query::QArgs &a = fa.q;
  const query::TreeView tv = query::tree_of<D, 4>(a, myq);
  const Nodes<SC, D, EXPL, VEC> nd(a, tv.tree);
  const int k = fa.kk;
  T q[D];
#pragma unroll
  for (int d = 0; d < D; d++) q[d] = __ldg((const T *)a.queries + myq * D + d);
  int32_t *row = a.out_ids + myq * k;
  auto dist = [&](int id) {
    T p[D];
    nd.point(id, p);
    return exact_d2<SC, D>(p, q);
  };
  int m = 0;  // real candidates: the row's, then yid
  while (m < k && row[m] >= 0) m++;
  if (m == k && yid >= 0) m++;
#pragma unroll 1
  for (int i = 1; i < m; i++) {
    const int id = i < k ? row[i] : yid;
    const E d = dist(id);
    int j = i;
#pragma unroll 1
    for (; j > 0; j--) {
      const int pid = row[j - 1];
      const E pd = dist(pid);
      if (pd < d || (pd == d && pid < id)) break;
      if (j < k)
        row[j] = pid;
      else
        yid = pid;
    }
    if (j < k)
      row[j] = id;
    else
      yid = id;
  }
  if (m < k) {
    if (hasSeed) return false;
    if (m > 0 && !(dist(row[m - 1]) < r2)) return false;
    if (a.out_max) ((E *)a.out_max)[myq] = r2;
  } else {
    const E X = dist(row[k - 1]);
    if (!(X < r2) || !(N::above(X) < safe)) return false;
    if (m > k && dist(yid) == X) {
      if (fa.fcp || (fa.method == CUKD_STACK_FREE && a.eps != 0.f) ||
          (fa.method == CUKD_CCT && !tv.bounds))
        return false;
#pragma unroll 1
      for (int j = k - 1; j >= 0 && dist(row[j]) == X; j--)
        if (!surely_visited<SC, D, EXPL, VEC>(fa, nd, q, tv.bounds, row[j], X)) return false;
    }
    if (a.out_max) ((E *)a.out_max)[myq] = X;
  }
  if (a.out_d2)
#pragma unroll 1
    for (int j = 0; j < k && j < m; j++) ((E *)a.out_d2)[myq * k + j] = dist(row[j]);
  return true;
}

__device__ __forceinline__ void store4(float *p, const float (&v)[4])
{
  *(float4 *)p = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store4(long long *p, const long long (&v)[4])
{
  *(longlong2 *)p = make_longlong2(v[0], v[1]);
  *(longlong2 *)(p + 2) = make_longlong2(v[2], v[3]);
}

// full levels of the home subtree (see knn_fast_one), which has to hold k + 1
// nodes for the traversal to start with a bound.  At k = 16 (10M points and
// queries) 31 nodes or more: 10.27 ms, 63 or more: 10.19 ms.
__host__ __device__ constexpr int home_levels(int kc)
{
  int h = 2;
  while ((1 << h) - 1 < kc) h++;
  return h;
}
__host__ __device__ constexpr int slot_bits(int kc)
{
  int b = 1;
  while ((1 << b) < kc) b++;
  return b;
}

// One thread per query (queries in Morton order).
//
// Candidate list: the k+1 nearest so far in KC >= k+1 registers, each a
// 32-bit key: the distance bound L as float bits with the low slot_bits(KC)
// bits replaced by a slot number.  Keys compare like the truncated
// distances; inserting one is a min and a max per register and needs no
// second register for the node, which is stored in shared memory at
// ids[slot * idStride] (the evicted key's slot is reused).  Slots below
// KC - (k+1) hold 0 and never move.  At the end the exact distances of the
// k+1 candidates are recomputed from their nodes, and the answer stands only
// if no other point can be as near as the k-th (`safe`, below).
//
// Home subtree: a descent to the node whose subtree of about k+1 nodes
// surrounds the query, and that subtree's nodes first, as one run per level,
// fill the list while all lanes of the warp are active and give a cull
// distance close to the final one; the traversal from the root then skips
// that subtree.  Far children are pushed only when within that distance.
//
// Culling uses the closest-corner distance of each subtree's domain box, the
// bound of traverse_cct (traverse-cct.h:25-99): the far child's box differs
// from its parent's only in the split dim, so its closest point to the query
// is the parent's with that coordinate set to the split value.  The traversal
// keeps the squared offsets of that closest point per dimension, off[d]; the
// box distance is their sum in dimension order, which never exceeds the L of
// a point inside.  A box is entered while its distance is at or below the
// top of the last key's truncation bucket, so every point whose truncated L
// is at or below the final (k+1)-th key's is seen.
//
// myq: the query's index; hasSeed / seedR: a per-query initial cull radius
// (learned proposal, before fa.radius_scale) or none.
template <int SC, int D, bool EXPL, bool VEC, int KC>
__device__ __forceinline__ void knn_fast_one(const FastArgs &fa, int64_t myq, bool hasSeed,
                                             float seedR, uint32_t *ids, int idStride)
{
  using N = Num<SC>;
  using T = typename N::T;
  using E = typename N::E;
  constexpr uint32_t MASK = (1u << slot_bits(KC)) - 1u;
  constexpr int H = home_levels(KC);
  const query::QArgs &a = fa.q;
  const query::TreeView tv = query::tree_of<D, 4>(a, myq);
  const int n = int(tv.n);
  const int k = fa.kk;  // live slots: k+1, right-aligned
  const Nodes<SC, D, EXPL, VEC> nd(a, tv.tree);

  T q[D];
  {
    const T *qp = (const T *)a.queries + myq * D;
#pragma unroll
    for (int d = 0; d < D; d++) q[d] = __ldg(qp + d);
  }
  E r2 = N::cutoff(a);
  if (hasSeed) r2 = N::seeded(r2, seedR, fa.radius_scale);
  const bool usable = N::usable(r2);
  // unfilled slots: the bucket above the cut-off's, so that every point
  // within the cut-off is listed (those of its own bucket that are not are
  // found out at the end)
  const uint32_t unfilled = (N::below(usable ? r2 : E(0)) & ~MASK) + (MASK + 1u);
  uint32_t e[KC];
#pragma unroll
  for (int j = 0; j < KC; j++) {
    const int s = j - (KC - (k + 1));
    e[j] = s < 0 ? 0u : unfilled | uint32_t(s);
  }
  uint32_t dropped = ~0u;  // smallest key that is not in the list
  int visits = 0;

  auto bound = [&](const T (&p)[D]) {
    float s = N::sq(p[0], q[0]);
#pragma unroll
    for (int d = 1; d < D; d++) s = N::add(s, N::sq(p[d], q[d]));
    return __float_as_uint(s);
  };
  auto sum = [](const float (&o)[D]) {
    float s = o[0];
#pragma unroll
    for (int d = 1; d < D; d++) s = N::add(s, o[d]);
    return __float_as_uint(s);
  };
  auto offer = [&](uint32_t l, int node) {
    const uint32_t last = e[KC - 1];
    const uint32_t key = (l & ~MASK) | (last & MASK);
    dropped = umin(dropped, umax(key, last));
    if (key < last) {
      ids[(last & MASK) * idStride] = uint32_t(node);
#pragma unroll
      for (int j = KC - 1; j > 0; j--) e[j] = umin(e[j], umax(e[j - 1], key));
      e[0] = umin(e[0], key);
    }
  };

  // ---- the home subtree
  int home = -1;
  if (n > 0 && usable) {
    home = 0;
    // down while the child's subtree has H full levels (2^H - 1 nodes or
    // more): its last node on the H-th one is ((child + 2) << (H - 1)) - 2
    const int lim = ((n + 1) >> (H - 1)) - 2;
    int lvl = 0;
#pragma unroll 1
    for (;;) {
      int dim;
      const T c = nd.split(home, lvl, &dim);
      T qc = q[0];
#pragma unroll
      for (int d = 1; d < D; d++) qc = d == dim ? q[d] : qc;
      const int child = 2 * home + (qc < c ? 1 : 2);
      if (child > lim) break;
      home = child;
      lvl++;
    }
    // its nodes level by level (nodes of a level are consecutive, and the
    // first one beyond the tree ends them all); the next point is loaded
    // before the current one is inserted
    T p[D];
    nd.point(home, p);
    int node = home;
#pragma unroll 1
    for (uint32_t y = 2; node < n; y++) {
      const int t = 31 - __clz(y);
      const uint32_t next = ((uint32_t(home) + 1u) << t) - 1u + (y - (1u << t));
      const uint32_t l = bound(p);
      if (next < uint32_t(n)) nd.point(int(next), p);
      visits++;
      offer(l, node);
      node = int(next < uint32_t(n) ? next : uint32_t(n));
    }
  }

  // ---- the rest of the tree
  // squared offsets of the root box's closest point (the world bounds, or
  // all of space)
  float off[D];
  const T *bnd = (const T *)tv.bounds;
#pragma unroll
  for (int d = 0; d < D; d++) {
    T v = q[d];
    if (bnd) {
      const T lo = __ldg(bnd + d), hi = __ldg(bnd + D + d);
      v = v < lo ? lo : v;
      v = hi < v ? hi : v;
    }
    off[d] = N::sq(v, q[d]);
  }
  // Pending far children are one word each on the stack: their squared
  // offsets in fractions of the bound after the home subtree, FB bits per
  // dimension, rounded down (a popped box can only look nearer than it is);
  // `trail` has a bit per level with a pending far child, which is the
  // sibling of the current path's node on that level.  (Against the node and
  // its offsets as bf16 in three words: a third of the local-memory traffic,
  // whose lanes' words lie in different sectors; 11.67 -> 10.85 ms.)
  constexpr int FB = D == 2 ? 16 : (D == 3 ? 10 : 8);
  constexpr uint32_t FM = (1u << FB) - 1u;
  uint32_t offSt[32];
  uint32_t trail = 0;
  int sp = 0;
  const uint32_t topBits = e[KC - 1] | MASK;
  // The unit is a power of two, so products with it are exact and a smaller
  // bound (a seeded search's) only refines the grid.  A list that the home
  // subtree did not fill has no bound to scale by (and a tiny one no finite
  // scale): its offsets round to 0, nothing is culled by them.
  const bool scaled = topBits < 0x7f800000u && topBits > 0x0da24260u;  // > 1e-30
  const uint32_t topExp = topBits >> 23;
  const float scale = scaled ? __uint_as_float((253u + FB - topExp) << 23) : 0.f;
  const float unit = scaled ? __uint_as_float((topExp + 1u - FB) << 23) : 0.f;
  int curr = (home >= 0 && sum(off) <= topBits) ? 0 : n;
  for (;;) {
    if (curr >= n || curr == home) {
      bool found = false;
      while (trail) {
        const uint32_t w = offSt[--sp];
        const int lvl = 31 - __clz(trail);
        trail ^= 1u << lvl;
        float o[D];
#pragma unroll
        for (int d = 0; d < D; d++) o[d] = float((w >> (FB * d)) & FM) * unit;
        if (sum(o) <= (e[KC - 1] | MASK)) {
#pragma unroll
          for (int d = 0; d < D; d++) off[d] = o[d];
          const int c1 = curr + 1;
          curr = ((c1 >> (31 - __clz(c1) - lvl)) ^ 1) - 1;
          found = true;
          break;
        }
      }
      if (!found) break;
    }
    T p[D];
    const int dim = nd.load(curr, p);
    visits++;
    offer(bound(p), curr);
    T nodeC = p[0], queryC = q[0];
#pragma unroll
    for (int d = 1; d < D; d++)
      if (d == dim) {
        nodeC = p[d];
        queryC = q[d];
      }
    const bool leftIsClose = queryC < nodeC;
    const int lChild = 2 * curr + 1;
    const int farChild = leftIsClose ? lChild + 1 : lChild;
    if (farChild < n) {
      float fo[D];
      const float split = N::sq(nodeC, queryC);
#pragma unroll
      for (int d = 0; d < D; d++) fo[d] = d == dim ? split : off[d];
      if (sum(fo) <= (e[KC - 1] | MASK)) {
        // 2^23 + x holds floor(x) in its low mantissa bits
        uint32_t w = 0;
#pragma unroll
        for (int d = 0; d < D; d++)
          w |= (__float_as_uint(__fadd_rz(__fmul_rz(fo[d], scale), 8388608.f)) & FM) << (FB * d);
        offSt[sp++] = w;
        trail |= 2u << (31 - __clz(curr + 1));
      }
    }
    curr = leftIsClose ? lChild : lChild + 1;
  }

  // ---- exact distances, written in key order (a query that is not settled
  // here is written again by its re-run)
  if (a.visits) a.visits[myq] += visits;  // accumulated over chained passes
  // the exact distance of a point that is not in the list is at least the
  // float with these bits: it was dropped, or lies in a box beyond the last
  // key's bucket
  const uint32_t safe = umin(dropped & ~MASK, (e[KC - 1] | MASK) + 1u);
  int32_t *oid = a.out_ids ? a.out_ids + myq * k : nullptr;
  E *od = a.out_d2 ? (E *)a.out_d2 + myq * k : nullptr;
  E prev = E(0), X = r2, Y = r2;
  int prevId = -1, xid = -1, yid = -1;
  bool sorted = true;
  // (with k = KC - 1 the k entries of a row are registers 0..k-1)
  const bool vec = KC >= 5 && k == KC - 1 &&
                   ((reinterpret_cast<uintptr_t>(oid) | reinterpret_cast<uintptr_t>(od)) & 15u) == 0;
  int idBuf[4];
  E dBuf[4];
#pragma unroll
  for (int j = 0; j < KC; j++) {
    const int pos = j - (KC - 1 - k);
    if (pos < 0) continue;
    const bool real = e[j] < unfilled;
    int id = -1;
    E d = r2;
    if (real) {
      id = int(ids[(e[j] & MASK) * idStride]);
      T p[D];
      nd.point(id, p);
      d = exact_d2<SC, D>(p, q);
      sorted = sorted && (prev < d || (prev == d && prevId < id));
      prev = d;
      prevId = id;
    }
    if (pos < k) {
      if (!vec) {
        if (oid) oid[pos] = id;
        if (od) od[pos] = d;
      } else {
        // full rows of an aligned array: 16 bytes at a time
        idBuf[j & 3] = id;
        dBuf[j & 3] = d;
        if ((j & 3) == 3) {
          if (oid) *(int4 *)(oid + j - 3) = make_int4(idBuf[0], idBuf[1], idBuf[2], idBuf[3]);
          if (od) store4(od + j - 3, dBuf);
        }
      }
      X = d;
      xid = id;
    } else {
      Y = d;
      yid = id;
    }
  }
  bool ok = usable && sorted;
  if (xid >= 0)
    ok = ok && X < r2 && N::above(X) < safe && (yid < 0 || X < Y);
  else
    ok = ok && !hasSeed && (prevId < 0 || prev < r2);
  if (ok && a.out_max) ((E *)a.out_max)[myq] = X;
  if (!ok && usable && (!sorted || (xid >= 0 && yid >= 0)))
    ok = settle_row<SC, D, EXPL, VEC>(fa, myq, r2, safe, hasSeed, yid);
  if (!ok) {
    const int slot = atomicAdd(fa.fb_count, 1);
    fa.fb_list[slot] = int32_t(myq);
  }
  if (fa.status) fa.status[myq] = ok ? 0 : 1;
}

// FCP and k = 1 of one query: the same search (home subtree, one-word stack
// entries, corner culling) for a single candidate in registers, with the
// reference's answer at ties:
//   - FCP keeps the first visited of the points at the smallest distance X.
//     Until then the reference's cull distance is above X, so that point is
//     the first in the traversal's preorder (near side before far side).
//     This search leaves preorder only for the home subtree: that lies on the
//     near path, so its points and the path's above it come before all others
//     and are compared by preorder; later ones have to be strictly nearer.
//   - k = 1 keeps the smallest id of the points at distance X that the
//     reference visits: the smallest seen here, if `surely_visited` (exact,
//     given the first one in preorder) says so; else the query is queued.
//     Far sides that the reference cannot enter are not entered.
// Boxes beyond `top` are culled, which is the bound of the candidate's
// distance (rounded up for ints, whose bound L is rounded down); boxes at it
// only where a point there can matter, so a group of points at the nearest
// distance costs a path (FCP), or what the reference itself visits of it.
//
// Whole calls of 1M float3 queries, us, stack-based reference order (sorted) ->
// FCP here / k = 1 here (B200): 1M uniform points 619 -> 394 / 413; with ties,
// cell centres of a 100^3 lattice 762 -> 498 / 658 and its half steps
// 704 -> 423 / 668, 500K points twice each 212 -> 140 / 160, 15K points 64
// times each from elsewhere 4780 -> 3060 / 3390 (these five, when ties were
// left to the reference order after this search: -, 1508, 1163, 312, 6750).
template <int SC, int D, bool EXPL, bool VEC, bool FCP>
__device__ __forceinline__ void fcp_fast_one(const FastArgs &fa, int64_t myq)
{
  using N = Num<SC>;
  using T = typename N::T;
  using E = typename N::E;
  constexpr int H = 3;
  const query::QArgs &a = fa.q;
  const query::TreeView tv = query::tree_of<D, 4>(a, myq);
  const int n = int(tv.n);
  const Nodes<SC, D, EXPL, VEC> nd(a, tv.tree);
  T q[D];
#pragma unroll
  for (int d = 0; d < D; d++) q[d] = __ldg((const T *)a.queries + myq * D + d);
  // the nearest distance so far (at first the cut-off, at which k = 1 still
  // takes points and FCP does not), the first point at it in preorder, and
  // (k = 1) the smallest id seen at it
  E bestD = N::cutoff(a);
  uint32_t top = N::above(bestD);
  int first = -1, least = -1;
  auto bound = [&](const T (&p)[D]) {
    float s = N::sq(p[0], q[0]);
#pragma unroll
    for (int d = 1; d < D; d++) s = N::add(s, N::sq(p[d], q[d]));
    return __float_as_uint(s);
  };
  auto sum = [](const float (&o)[D]) {
    float s = o[0];
#pragma unroll
    for (int d = 1; d < D; d++) s = N::add(s, o[d]);
    return __float_as_uint(s);
  };
  auto coord = [&](int dim) {
    T qc = q[0];
#pragma unroll
    for (int d = 1; d < D; d++) qc = d == dim ? q[d] : qc;
    return qc;
  };
  auto precedes = [&](int x, int y) {  // in preorder, x != y
    const int lx = level_of(x), ly = level_of(y), m = lx < ly ? lx : ly;
    const uint32_t ax = uint32_t(x + 1) >> (lx - m), ay = uint32_t(y + 1) >> (ly - m);
    if (ax == ay) return lx < ly;
    const int s = 32 - __clz(ax ^ ay);  // up to their last common ancestor
    int dim;
    const T c = nd.split(int(ax >> s) - 1, m - s, &dim);
    return (((ax >> (s - 1)) & 1u) == 0) == left_first(fa.method, coord(dim), c);
  };
  // early: in the home subtree or on the path to it
  auto offer = [&](const T (&p)[D], int node, bool early) {
    const uint32_t l = bound(p);
    if (SC == 0 && FCP) {  // l is the distance: no branch but at early ties
      const bool tie = early && l == top;
      const bool nearer = l < top;
      top = nearer ? l : top;
      first = nearer ? node : first;
      if (tie && first >= 0 && precedes(node, first)) first = node;
    } else if (l <= top) {
      const E d = exact_d2<SC, D>(p, q);
      if (d < bestD) {
        bestD = d;
        top = N::above(d);
        first = least = node;
      } else if (d == bestD && (early || !FCP)) {
        if (early && first >= 0 && precedes(node, first)) first = node;
        least = int(umin(uint32_t(least), uint32_t(node)));
      }
    }
  };
  int home = -1;
  if (n > 0) {
    home = 0;
    const int lim = ((n + 1) >> (H - 1)) - 2;
    int lvl = 0;
#pragma unroll 1
    for (;;) {
      int dim;
      const T c = nd.split(home, lvl, &dim);
      const int child = 2 * home + (left_first(fa.method, coord(dim), c) ? 1 : 2);
      if (child > lim) break;
      home = child;
      lvl++;
    }
    T p[D];
    nd.point(home, p);
    int node = home;
#pragma unroll 1
    for (uint32_t y = 2; node < n; y++) {
      const int t = 31 - __clz(y);
      const uint32_t next = ((uint32_t(home) + 1u) << t) - 1u + (y - (1u << t));
      T c[D];
#pragma unroll
      for (int d = 0; d < D; d++) c[d] = p[d];
      if (next < uint32_t(n)) nd.point(int(next), p);
      offer(c, node, true);
      node = int(next < uint32_t(n) ? next : uint32_t(n));
    }
  }
  float off[D];
  const T *bnd = (const T *)tv.bounds;
#pragma unroll
  for (int d = 0; d < D; d++) {
    T v = q[d];
    if (bnd) {
      const T lo = __ldg(bnd + d), hi = __ldg(bnd + D + d);
      v = v < lo ? lo : v;
      v = hi < v ? hi : v;
    }
    off[d] = N::sq(v, q[d]);
  }
  // (stack entries as in knn_fast_one)
  constexpr int FB = D == 2 ? 16 : (D == 3 ? 10 : 8);
  constexpr uint32_t FM = (1u << FB) - 1u;
  uint32_t offSt[32];
  uint32_t trail = 0;
  int sp = 0;
  const bool scaled = top < 0x7f800000u && top > 0x0da24260u;  // > 1e-30
  const uint32_t topExp = top >> 23;
  const float scale = scaled ? __uint_as_float((253u + FB - topExp) << 23) : 0.f;
  const float unit = scaled ? __uint_as_float((topExp + 1u - FB) << 23) : 0.f;
  int curr = 0;
  auto step = [&](bool early) {  // visits curr and goes on to its near child
    T p[D];
    const int dim = nd.load(curr, p);
    offer(p, curr, early);
    T nodeC = p[0], queryC = q[0];
#pragma unroll
    for (int d = 1; d < D; d++)
      if (d == dim) {
        nodeC = p[d];
        queryC = q[d];
      }
    const bool leftIsClose = left_first(fa.method, queryC, nodeC);
    const int lChild = 2 * curr + 1;
    const int farChild = leftIsClose ? lChild + 1 : lChild;
    if (farChild < n) {
      float fo[D];
      const float split = N::sq(nodeC, queryC);
#pragma unroll
      for (int d = 0; d < D; d++) fo[d] = d == dim ? split : off[d];
      // (k = 1: a box at `top` may hold a point that counts, if the
      // reference enters it, which cct does by the box, the others by the plane)
      const uint32_t box = sum(fo);
      if (FCP ? box < top : box <= top) {
        const bool enter = FCP || box < top ||
                           (fa.method != CUKD_CCT && __float_as_uint(split) < top);
        uint32_t w = 0;
#pragma unroll
        for (int d = 0; d < D; d++)
          w |= (__float_as_uint(__fadd_rz(__fmul_rz(fo[d], scale), 8388608.f)) & FM) << (FB * d);
        offSt[sp] = w;
        sp += int(enter);
        trail |= (enter ? 2u : 0u) << (31 - __clz(curr + 1));
      }
    }
    curr = leftIsClose ? lChild : lChild + 1;
  };
  auto pop = [&]() {  // curr: the last pending far child that still matters
    while (trail) {
      const uint32_t w = offSt[--sp];
      const int lvl = 31 - __clz(trail);
      trail ^= 1u << lvl;
      float o[D];
#pragma unroll
      for (int d = 0; d < D; d++) o[d] = float((w >> (FB * d)) & FM) * unit;
      if (FCP ? sum(o) < top : sum(o) <= top) {
#pragma unroll
        for (int d = 0; d < D; d++) off[d] = o[d];
        const int c1 = curr + 1;
        curr = ((c1 >> (31 - __clz(c1) - lvl)) ^ 1) - 1;
        return true;
      }
    }
    return false;
  };
  if (n > 0 && sum(off) <= top) {
    // the path to the home subtree, then what is pending
    while (curr < home) step(true);
    bool more = pop();
    while (more) {
      step(false);
      if (curr >= n) more = pop();
    }
  }
  if (SC == 0 && FCP) {  // (of the same four bytes)
    const float d = __uint_as_float(top);
    memcpy(&bestD, &d, 4);
  }
  if (!FCP && least != first &&
      !surely_visited<SC, D, EXPL, VEC>(fa, nd, q, tv.bounds, least, bestD, first)) {
    fa.fb_list[atomicAdd(fa.fb_count, 1)] = int32_t(myq);
    return;
  }
  if (a.out_ids) a.out_ids[myq] = FCP ? first : least;
  if (a.out_d2) ((E *)a.out_d2)[myq] = bestD;
  if (a.out_max) ((E *)a.out_max)[myq] = bestD;
}

}  // namespace fast
}  // namespace ckb
