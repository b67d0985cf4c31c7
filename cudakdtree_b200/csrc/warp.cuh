// kNN / FCP with a warp per query (instantiated in warp_float.cu and
// warp_int.cu): for calls of few queries, and for the queries that the
// thread-per-query kernels queued.
//
// What bounds those is latency, not throughput: a thread-per-query traversal
// is a chain of a hundred and more dependent loads, whatever the number of
// queries (777 queries, k = 8, 100K points: 104 us, after 70 us of sorting
// the queries; a queued query far from every point, whose reference-order
// traversal culls little: 12 ms and more).  Here a warp loads a whole
// five-level subtree (31 nodes, a lane each) per step and looks at subtrees
// in order of their distance, so the chain is a dozen steps.
//
// The candidate list is exact: the k smallest (d2, id) keys, spread over the
// lanes in order.  Boxes are culled by closest-corner distance with "<=", so
// every point at or below the final k-th distance X is seen, and the list is
// the reference's answer when the reference surely visits each listed point
// at distance X (fast.cu's header; otherwise the query is queued for the
// reference-order kernel).
#pragma once

#include <algorithm>

#include "common.cuh"
#include "fast.cuh"
#include "fast_one.cuh"
#include "query.cuh"

namespace ckb {
namespace fast {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarpsPerBlock = 4;
constexpr int kTreelet = 5;     // levels a warp takes in one step
// Pending subtrees are taken nearest first while there are at most
// kBestFirst of them, else last in first out: every step then adds at most
// 31, and a path has at most 7 steps (30 levels).
constexpr int kBestFirst = 128;
constexpr int kPending = kBestFirst + 32 * 7;

template <int SC, int KL> struct WarpList;
// row i of lane l holds the (32 i + l)-th smallest key
template <int KL> struct WarpList<0, KL> {
  unsigned long long key[KL];
  __device__ void init(float r2)
  {
#pragma unroll
    for (int i = 0; i < KL; i++)
      key[i] = ((unsigned long long)__float_as_uint(r2) << 32) | 0xffffffffull;
  }
  __device__ static unsigned long long make(float d, int id)
  {
    return ((unsigned long long)__float_as_uint(d) << 32) | uint32_t(id);
  }
  __device__ static bool less(unsigned long long a, unsigned long long b) { return a < b; }
  __device__ static unsigned long long shfl(unsigned long long k, int l)
  {
    return __shfl_sync(kFull, k, l);
  }
  __device__ static unsigned long long up(unsigned long long k)
  {
    return __shfl_up_sync(kFull, k, 1);
  }
  __device__ static float d2(unsigned long long k) { return __uint_as_float(uint32_t(k >> 32)); }
  __device__ static int id(unsigned long long k) { return int(uint32_t(k)); }
};
template <int KL> struct WarpList<1, KL> {
  using K = query::IKey;
  K key[KL];
  __device__ void init(long long r2)
  {
#pragma unroll
    for (int i = 0; i < KL; i++) key[i] = K{r2, 0xffffffffu};
  }
  __device__ static K make(long long d, int id) { return K{d, uint32_t(id)}; }
  __device__ static bool less(K a, K b) { return a.d < b.d || (a.d == b.d && a.id < b.id); }
  __device__ static K shfl(K k, int l)
  {
    return K{__shfl_sync(kFull, k.d, l), __shfl_sync(kFull, k.id, l)};
  }
  __device__ static K up(K k)
  {
    return K{__shfl_up_sync(kFull, k.d, 1), __shfl_up_sync(kFull, k.id, 1)};
  }
  __device__ static long long d2(K k) { return k.d; }
  __device__ static int id(K k) { return int(k.id); }
};

template <int D> struct Pending {
  uint32_t dist[kPending];  // box distance (float bits)
  int node[kPending];
  float off[D][kPending];   // squared offsets of the box's closest point
};

// LIST: k >= 2 without eps (compiled apart: the others' bookkeeping costs it
// 4% of a 27 us call)
template <int SC, int D, bool EXPL, bool VEC, int KL, bool LIST>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
    knn_warp_kernel(const __grid_constant__ WarpArgs wa)
{
  using N = Num<SC>;
  using T = typename N::T;
  using E = typename N::E;
  using L = WarpList<SC, KL>;
  extern __shared__ uint32_t sh[];
  const FastArgs &fa = wa.f;
  const query::QArgs &a = fa.q;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  Pending<D> &st = reinterpret_cast<Pending<D> *>(sh)[wid];
  int64_t limit = a.nq;
  if (a.count_ptr) {
    limit = *a.count_ptr;
    if (limit > wa.queue_limit) {
      if (!wa.hand_over) return;
      // (behind what is queued there already: each block takes its share)
      for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < limit;
           i += int64_t(gridDim.x) * blockDim.x)
        fa.fb_list[atomicAdd(fa.fb_count, 1)] = a.order[i];
      return;
    }
  }
  const int k = fa.kk;
  // keys that count; for FCP and k = 1 the second tells a tie, and once there
  // are two, boxes at the second's distance are of use only to k = 1, to find
  // the smallest id of the tied points (while they are at most kTied: a group
  // of equal points may be the whole tree)
  constexpr int kTied = 32;
  const bool single = !LIST && k == 1;
  const int K = single ? 2 : k;
  // a stack-free list with eps is its traversal's at ties, else the exact one:
  // the smallest distance left out tells (`beyond`)
  const bool eps = !LIST && !single && fa.method == CUKD_STACK_FREE && a.eps != 0.f;
  // this lane's place in a treelet (lane 31 has none)
  const int t = 31 - __clz(lane + 1);
  for (int64_t w = blockIdx.x * int64_t(kWarpsPerBlock) + wid; w < limit;
       w += int64_t(gridDim.x) * kWarpsPerBlock) {
    const int64_t myq = a.order ? int64_t(a.order[w]) : w;
    const query::TreeView tv = query::tree_of<D, 4>(a, myq);
    const int n = int(tv.n);
    const Nodes<SC, D, EXPL, VEC> nd(a, tv.tree);
    T q[D];
#pragma unroll
    for (int d = 0; d < D; d++) q[d] = __ldg((const T *)a.queries + myq * D + d);
    const E r2 = N::cutoff(a);
    const bool usable = N::usable(r2);
    L list;
    list.init(r2);
    auto kth = list.key[0];
    int tied = 0;  // points seen at the first key's distance
    uint32_t cull = N::above(r2) + 1u;  // boxes at this distance and more are skipped
    auto refresh = [&]() {
#pragma unroll
      for (int i = 0; i < KL; i++) {
        const auto v = L::shfl(list.key[i], (K - 1) & 31);
        if (i == (K - 1) >> 5) kth = v;
      }
      const bool exclusive = single && L::id(kth) != -1 && (fa.fcp || tied > kTied);
      cull = N::above(L::d2(kth)) + (exclusive ? 0u : 1u);
    };
    E beyond = N::farthest();  // this lane's share
    auto insert = [&](auto x) {
      if (eps && L::id(kth) != -1 && L::d2(kth) < beyond) beyond = L::d2(kth);  // pushed out
#pragma unroll
      for (int i = 0; i < KL; i++) {
        const int pos = __popc(__ballot_sync(kFull, L::less(list.key[i], x)));
        if (pos < 32) {
          const auto carry = L::shfl(list.key[i], 31);
          const auto up = L::up(list.key[i]);
          if (lane == pos) list.key[i] = x;
          if (lane > pos) list.key[i] = up;
          x = carry;
        }
      }
      refresh();
    };
    // levels: the bottom treelets have kTreelet levels (the last one partly
    // filled), the root's what remains
    const int levels = 32 - __clz(max(n, 1));
    const int bottom = max(0, levels - kTreelet);
    const int rootLevels = bottom == 0 || bottom % kTreelet == 0 ? kTreelet : bottom % kTreelet;
    float rootOff[D];
    const T *bnd = (const T *)tv.bounds;
#pragma unroll
    for (int d = 0; d < D; d++) {
      T v = q[d];
      if (bnd) {
        const T lo = __ldg(bnd + d), hi = __ldg(bnd + D + d);
        v = v < lo ? lo : v;
        v = hi < v ? hi : v;
      }
      rootOff[d] = N::sq(v, q[d]);
    }
    auto sum = [](const float (&o)[D]) {
      float s = o[0];
#pragma unroll
      for (int d = 1; d < D; d++) s = N::add(s, o[d]);
      return __float_as_uint(s);
    };

    // ---- the start subtree around the query: a bottom treelet, or for lists
    // that one may not fill (15 full nodes) the ten-level subtree above it
    int start = 0;
    if (n > 0 && usable) {
      const int startLevel = K <= 15 ? bottom : max(0, bottom - kTreelet);
      int lvl = 0;
      while (lvl < startLevel) {
        const int h = lvl == 0 ? rootLevels : kTreelet;
        const int node = ((start + 1) << t) + (lane - (1 << t));
        bool right = false;
        if (lane < (1 << h) - 1 && node < n) {
          int dim;
          const T c = nd.split(node, lvl + t, &dim);
          T qc = q[0];
#pragma unroll
          for (int d = 1; d < D; d++) qc = d == dim ? q[d] : qc;
          right = !(qc < c);
        }
        const unsigned rights = __ballot_sync(kFull, right);
        int x = 0;
        for (int s = 0; s < h; s++) x = 2 * x + 1 + int((rights >> x) & 1u);
        start = ((start + 1) << h) + (x - (1 << h));
        lvl += h;
      }
    }

    // ---- best first: the start subtree, then the tree without it
    for (int pass = 0; pass < 2; pass++) {
      if (n == 0 || !usable || (pass == 1 && start == 0)) break;
      const int skip = pass == 0 ? -1 : start;
      int cnt = 0;
      int curr = pass == 0 ? start : 0;
      float off[D];
#pragma unroll
      for (int d = 0; d < D; d++) off[d] = rootOff[d];
      if (sum(off) >= cull) break;
      for (;;) {
        const int lvl = level_of(curr);
        const int h = lvl == 0 ? rootLevels : kTreelet;
        // a node per lane: its split, then its box from its ancestors' splits
        const int node = ((curr + 1) << t) + (lane - (1 << t));
        const bool here = lane < (1 << h) - 1 && node < n;
        T p[D];
#pragma unroll
        for (int d = 0; d < D; d++) p[d] = q[d];
        int dim = 0;
        if (here) dim = nd.load_at(node, lvl + t, p);
        T c = p[0], qc = q[0];
#pragma unroll
        for (int d = 1; d < D; d++)
          if (d == dim) {
            c = p[d];
            qc = q[d];
          }
        const float plane = N::sq(c, qc);
        const bool leftIsClose = qc < c;
        const int info = dim * 2 + int(leftIsClose);
        float bo[D];
#pragma unroll
        for (int d = 0; d < D; d++) bo[d] = off[d];
#pragma unroll
        for (int s = 0; s < kTreelet - 1; s++) {
          const int up = t > s ? ((lane + 1) >> (t - s)) - 1 : 0;
          const float pa = __shfl_sync(kFull, plane, up);
          const int ia = __shfl_sync(kFull, info, up);
          const int right = t > s ? ((lane + 1) >> (t - s - 1)) & 1 : 0;
          if (t > s && right == (ia & 1)) {  // the far side
#pragma unroll
            for (int d = 0; d < D; d++) bo[d] = d == (ia >> 1) ? pa : bo[d];
          }
        }
        const uint32_t bd = sum(bo);
        const auto key = L::make(exact_d2<SC, D>(p, q), node);
        const bool seen = here && bd < cull;
        bool cand = seen && L::less(key, kth);
        unsigned m = __ballot_sync(kFull, cand);
        const E nearest = LIST ? E(0) : L::d2(L::shfl(list.key[0], 0));
        bool listed = false;
        while (m) {
          const int src = __ffs(m) - 1;
          insert(L::shfl(key, src));
          listed = listed || lane == src;
          cand = cand && lane != src && L::less(key, kth);
          m = __ballot_sync(kFull, cand);
        }
        if (eps && seen && !listed && L::d2(key) < beyond) beyond = L::d2(key);
        if (single && !fa.fcp) {
          const E now = L::d2(L::shfl(list.key[0], 0));
          tied = (now < nearest ? 0 : tied) + __popc(__ballot_sync(kFull, seen && L::d2(key) == now));
          refresh();  // (`tied` went up, or a nearer point began it anew)
        }
        // the subtrees below: far children, then near ones
        if (lvl + h < levels) {
          const bool last = here && t == h - 1 && bd < cull;
          const int lChild = 2 * node + 1;
          float fo[D];
#pragma unroll
          for (int d = 0; d < D; d++) fo[d] = d == dim ? plane : bo[d];
          const uint32_t fd = sum(fo);
#pragma unroll
          for (int side = 0; side < 2; side++) {  // 0: far, 1: near
            const int child = lChild + int(leftIsClose == (side == 0));
            const bool push = last && child < n && child != skip && (side == 1 || fd < cull);
            const unsigned pm = __ballot_sync(kFull, push);
            if (push) {
              const int at = cnt + __popc(pm & ((1u << lane) - 1u));
              st.dist[at] = side == 0 ? fd : bd;
              st.node[at] = child;
#pragma unroll
              for (int d = 0; d < D; d++) st.off[d][at] = side == 0 ? fo[d] : bo[d];
            }
            cnt += __popc(pm);
          }
        }
        __syncwarp();
        // the next subtree
        int pick = -1;
        if (cnt > kBestFirst) {
          while (cnt > 0 && pick < 0) {
            if (st.dist[cnt - 1] < cull)
              pick = cnt - 1;
            else
              cnt--;
          }
        } else if (cnt > 0) {
          uint32_t best = ~0u;
          int at = -1;
          for (int i = lane; i < cnt; i += 32) {
            const uint32_t v = st.dist[i];
            if (v <= best) {  // of equals the last one pushed
              best = v;
              at = i;
            }
          }
          const uint32_t least = __reduce_min_sync(kFull, best);
          if (least < cull) pick = __reduce_max_sync(kFull, best == least ? at : -1);
        }
        if (pick < 0) break;
        curr = st.node[pick];
#pragma unroll
        for (int d = 0; d < D; d++) off[d] = st.off[d][pick];
        __syncwarp();
        cnt--;
        if (pick != cnt && lane == 0) {
          st.dist[pick] = st.dist[cnt];
          st.node[pick] = st.node[cnt];
#pragma unroll
          for (int d = 0; d < D; d++) st.off[d][pick] = st.off[d][cnt];
        }
        __syncwarp();
      }
      __syncwarp();
    }

    // ---- the answer, or the queue
    bool ok = usable;
    const bool filled = L::id(kth) != -1;
    const E X = filled ? L::d2(kth) : r2;
    if (single) {
      const auto first = L::shfl(list.key[0], 0);
      const auto second = L::shfl(list.key[0], 1);
      const bool none = fa.fcp ? !(L::d2(first) < r2) : L::id(first) == -1;
      if (ok && !none && !(L::d2(first) < r2 &&
                           (L::id(second) == -1 || L::d2(first) < L::d2(second))))
        ok = !fa.fcp && tied <= kTied &&
             surely_visited<SC, D, EXPL, VEC>(fa, nd, q, tv.bounds, L::id(first), L::d2(first));
      if (ok && lane == 0) {
        const E d = none ? r2 : L::d2(first);
        if (a.out_ids) a.out_ids[myq] = none ? -1 : L::id(first);
        if (a.out_d2) ((E *)a.out_d2)[myq] = d;
        if (a.out_max) ((E *)a.out_max)[myq] = d;
      }
    } else {
      bool sure = !(eps && filled) || (X < r2 && X < beyond);
#pragma unroll
      for (int i = 0; i < KL; i++) {
        const int j = 32 * i + lane;
        if (ok && !(eps && filled) && j < k && L::id(list.key[i]) != -1 &&
            !(L::d2(list.key[i]) < X))
          sure = sure && !eps && !(fa.method == CUKD_CCT && !tv.bounds) &&
                 surely_visited<SC, D, EXPL, VEC>(fa, nd, q, tv.bounds, L::id(list.key[i]), X);
      }
      ok = ok && __all_sync(kFull, sure);
      if (ok) {
#pragma unroll
        for (int i = 0; i < KL; i++) {
          const int j = 32 * i + lane;
          if (j < k) {
            if (a.out_ids) a.out_ids[myq * k + j] = L::id(list.key[i]);
            if (a.out_d2) ((E *)a.out_d2)[myq * k + j] = L::d2(list.key[i]);
          }
        }
        if (a.out_max && lane == 0) ((E *)a.out_max)[myq] = X;
      }
    }
    if (!ok && lane == 0) fa.fb_list[atomicAdd(fa.fb_count, 1)] = int32_t(myq);
  }
}

template <int SC, int D, bool EXPL, bool VEC, int KL, bool LIST>
int launch_warp(const WarpArgs &wa, cudaStream_t st)
{
  // at least a block per SM's share of a queue whose length the host does
  // not know; 7 blocks' stacks fit an SM
  int64_t grid = div_up(wa.f.q.nq, kWarpsPerBlock);
  if (wa.f.q.count_ptr) grid = std::min<int64_t>(grid, int64_t(kNumSMs) * 7);
  knn_warp_kernel<SC, D, EXPL, VEC, KL, LIST>
      <<<unsigned(std::max<int64_t>(1, grid)), 32 * kWarpsPerBlock,
         sizeof(Pending<D>) * kWarpsPerBlock, st>>>(wa);
  CKB_CHECK_LAUNCH();
  return CUKD_OK;
}

template <int SC, int D>
int launch_warp_layout(const WarpArgs &wa, cudaStream_t st)
{
  const bool vec = vector_points(wa.f.q, D);
  const bool one = wa.f.kk <= 32;
  const bool list = wa.f.kk > 1 && !(wa.f.method == CUKD_STACK_FREE && wa.f.q.eps != 0.f);
#define CKB_WARP(EXPL_, VEC_)                                                       \
  return list ? (one ? launch_warp<SC, D, EXPL_, VEC_, 1, true>(wa, st)             \
                     : launch_warp<SC, D, EXPL_, VEC_, 4, true>(wa, st))            \
              : (one ? launch_warp<SC, D, EXPL_, VEC_, 1, false>(wa, st)            \
                     : launch_warp<SC, D, EXPL_, VEC_, 4, false>(wa, st))
  if (wa.f.q.doff >= 0) {
    if (vec) CKB_WARP(true, true);
    CKB_WARP(true, false);
  }
  if (vec) CKB_WARP(false, true);
  CKB_WARP(false, false);
#undef CKB_WARP
}

template <int SC> int run_warp_scalar(const WarpArgs &wa, int D, cudaStream_t st)
{
  if (D == 2) return launch_warp_layout<SC, 2>(wa, st);
  if (D == 3) return launch_warp_layout<SC, 3>(wa, st);
  if (D == 4) return launch_warp_layout<SC, 4>(wa, st);
  return CUKD_ERR_UNSUPPORTED;
}

}  // namespace fast
}  // namespace ckb
