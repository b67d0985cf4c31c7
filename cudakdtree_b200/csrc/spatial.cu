// Spatial k-d tree (reference: cukd/spatial-kdtree.h) -- builder and
// traversals, sm_100a.
//
// Builder.  The reference grows the tree one level per pass: every open node
// either becomes a leaf (at most makeLeafThreshold prims, default 8) or is
// split at the centre of its prims' bounding box along the widest extent
// (first widest dim wins; a split whose centre rounds onto the box boundary
// is "degenerate" and alternates prims between the children), then every
// prim moves to a child (coord >= pos goes right) and the children's boxes
// grow atomically (:316-436).  Two of its choices depend on atomic order: the
// children's node ids (atomicAdd on a counter, :385) and which prims of a
// degenerate split go left (atomicAdd on an uninitialised counter, :424-427).
// This builder makes both canonical -- children are numbered in the order of
// their parents' ids, and the i-th prim (by prim id) of a degenerate node
// goes to side i&1 -- and otherwise follows the reference: same split rule,
// same leaf rule, node 1 kept as the reference's empty dummy, leaf prim lists
// in node-id order with prims in prim-id order (the reference's radix sort
// on node id is stable over the prim array, :577-585), bounds kept in the
// reference's int32 order-preserving float encoding (:177-192).
//
// Data layout.  Prims are kept in segments, one per open node, in prim-id
// order; a level stably partitions each split node's segment into its two
// children's segments, so every node's prims stay contiguous and ordered.
//
// Two phases.  Nodes of more than kSub prims are split level by level by
// all CTAs (three launches a level: side bits with their prefix sums, the
// nodes' children, the move with the children's boxes); what is left at
// kSub prims or fewer becomes the root of a subtree that one CTA finishes in
// shared memory.  Neither phase numbers nodes: a split node is stored under
// the boundary between its children's prims, a leaf under its first prim,
// which are unique, and in which nodes of one level stand in the order of
// their numbers.  Sorting those places by level (stably) numbers the nodes.
// The host reads back twice, plus once per four levels beyond the expected.
//
// Before, every level of the tree (27 for 1M mixture points) ran twelve
// launches and a device->host read of its split count: 2.6 ms for 1M points
// (B200), of which the kernels took 2.1 ms, against 1.0 ms now (20 levels
// 0.63 ms, bound by their launches and scattered moves; subtrees 0.18 ms).
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "query.cuh"
#include "scan.cuh"
#include "sort.cuh"

namespace ckb {
namespace spatial {

using Node = cukd_spatial_node;

// AtomicBox encoding (spatial-kdtree.h:177-192)
__host__ __device__ inline int32_t enc(float f)
{
#ifdef __CUDA_ARCH__
  int32_t b = __float_as_int(f);
#else
  int32_t b;
  memcpy(&b, &f, 4);
#endif
  if (b & int32_t(0x80000000)) b ^= 0x7fffffff;
  return b;
}
__host__ __device__ inline float dec(int32_t b)
{
  if (b & int32_t(0x80000000)) b ^= 0x7fffffff;
#ifdef __CUDA_ARCH__
  return __int_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}

constexpr uint32_t kSub = 1024;       // prims of a subtree that one CTA finishes
constexpr uint32_t kDone = 0xffffffffu;  // position not in an open node of the level phase
constexpr int kSideTile = 1024;  // positions of a CTA of side_kernel
constexpr int kSideWords = kSideTile / 8 / 32;  // per warp

struct SubRoot {
  uint32_t begin, count, level;
  uint32_t link;    // parent's boundary * 2 + (this is its left child); kDone: none
  uint32_t parity;  // buffer that holds its prims
};

struct BuildState {  // device-side counters
  uint32_t open[2];  // open nodes of the level phase, by parity of the level
  uint32_t subRoots, leaves, maxLevel, ticket;
};

struct BuildBufs {
  BuildState *st;
  // open nodes of the level phase, by parity
  uint32_t *begin[2], *count[2], *link[2];
  int32_t *lo[2], *hi[2];  // [node][D], encoded
  uint4 *move;             // per open node: first position, left prims before it,
                           // left prims, (unused)
  uint2 *codes;            // its children's open nodes of the next level, or kDone
  // side bits of a level's prims: words, their prefix within a tile, tile sums
  uint32_t *bits, *wordPre, *tileBase;
  SubRoot *roots;
  // the tree by place: splits under their boundary, leaves under their first
  // prim; key[2 * first] / key[2 * boundary - 1] holds the node's level
  uint32_t *key, *splitChild, *leaf;  // leaf: prim count, buffer in bit 31
  float *splitPos;
  uint8_t *splitDim;
  // per prim position, by parity
  uint32_t *prim[2], *nodeOf[2];
  float *coord[2][4];  // the prim's coordinates, moved with it (SoA per dim)
  const uint8_t *data;
  int stride, poff;
};

template <int D>
__device__ inline void load_point(const BuildBufs &b, uint32_t prim, float *p)
{
  const float *c = (const float *)(b.data + int64_t(prim) * b.stride + b.poff);
#pragma unroll
  for (int d = 0; d < D; d++) p[d] = __ldg(c + d);
}

template <int D>
__device__ inline void warp_grow(int32_t *lo, int32_t *hi, uint32_t node, bool valid,
                                 const float *p)
{
  // one atomic per (warp, node): lanes holding prims of the same node reduce
  // their encoded coordinates together
  const unsigned active = __ballot_sync(0xffffffffu, valid);
  if (!valid) return;
  const unsigned peers = __match_any_sync(active, node);
  const int leader = __ffs(peers) - 1;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 0; d < D; d++) {
    const int32_t e = enc(p[d]);
    const int32_t l = __reduce_min_sync(peers, e);
    const int32_t h = __reduce_max_sync(peers, e);
    if (lane == leader) {
      atomicMin(&lo[int64_t(node) * D + d], l);
      atomicMax(&hi[int64_t(node) * D + d], h);
    }
  }
}

// Grows the boxes of the nodes that this CTA's valid lanes carry prims to.
// When those nodes' numbers span fewer than kGrowSlots (always near the root,
// where every warp would otherwise hit the same few boxes), the warps' partial
// boxes are merged in shared memory first and the CTA issues one global atomic
// per (node, dim, bound); otherwise each warp issues its own (warp_grow).
// Deeper levels are mostly the latter: a level's nodes are numbered in the
// order in which their parents' threads come to a counter, so those of one CTA
// may lie far apart.
constexpr int kGrowSlots = 64;
template <int D>
__device__ inline void block_grow(int32_t *lo, int32_t *hi, uint32_t node, bool valid,
                                  const float *p)
{
  __shared__ uint32_t nmin, nmax;
  __shared__ int32_t slo[kGrowSlots][D], shi[kGrowSlots][D];
  if (threadIdx.x == 0) {
    nmin = 0xffffffffu;
    nmax = 0u;
  }
  __syncthreads();
  if (valid) {
    atomicMin(&nmin, node);
    atomicMax(&nmax, node);
  }
  __syncthreads();
  const uint32_t n0 = nmin, n1 = nmax;
  if (n0 > n1) return;  // no valid lane in the CTA (uniform)
  if (n1 - n0 >= uint32_t(kGrowSlots)) {  // uniform
    warp_grow<D>(lo, hi, node, valid, p);
    return;
  }
  const int slots = int(n1 - n0) + 1;
  for (int i = threadIdx.x; i < slots * D; i += blockDim.x) {
    (&slo[0][0])[i] = enc(+FLT_MAX);
    (&shi[0][0])[i] = enc(-FLT_MAX);
  }
  __syncthreads();
  const unsigned active = __ballot_sync(0xffffffffu, valid);
  if (valid) {
    const unsigned peers = __match_any_sync(active, node);
    const int leader = __ffs(peers) - 1;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 0; d < D; d++) {
      const int32_t e = enc(p[d]);
      const int32_t l = __reduce_min_sync(peers, e);
      const int32_t h = __reduce_max_sync(peers, e);
      if (lane == leader) {
        atomicMin(&slo[node - n0][d], l);
        atomicMax(&shi[node - n0][d], h);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < slots * D; i += blockDim.x) {
    const int sl = i / D, d = i % D;
    const int32_t l = slo[sl][d], h = shi[sl][d];
    if (l <= h) {  // the slot's node received prims
      atomicMin(&lo[int64_t(n0 + sl) * D + d], l);
      atomicMax(&hi[int64_t(n0 + sl) * D + d], h);
    }
  }
}

template <int D>
__global__ void init_kernel(BuildBufs b, int64_t n)
{
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const bool valid = i < n;
  float p[D];
  if (valid) {
    load_point<D>(b, uint32_t(i), p);
    b.prim[0][i] = uint32_t(i);
    b.nodeOf[0][i] = 0;
#pragma unroll
    for (int d = 0; d < D; d++) b.coord[0][d][i] = p[d];
  } else {
#pragma unroll
    for (int d = 0; d < D; d++) p[d] = 0.f;
  }
  block_grow<D>(b.lo[0], b.hi[0], 0, valid, p);
}

__device__ inline void note_leaf(const BuildBufs &b, uint32_t begin, uint32_t count,
                                 uint32_t level, uint32_t parity, uint32_t link)
{
  b.key[2 * size_t(begin)] = level;
  b.leaf[begin] = count | (parity << 31);
  if (link != kDone && (link & 1)) b.splitChild[link >> 1] = 2 * begin;
}
__device__ inline void note_split(const BuildBufs &b, uint32_t boundary, int dim, float pos,
                                  uint32_t level, uint32_t link)
{
  b.key[2 * size_t(boundary) - 1] = level;
  b.splitPos[boundary] = pos;
  b.splitDim[boundary] = uint8_t(dim < 0 ? 0 : dim);
  if (link != kDone && (link & 1)) b.splitChild[link >> 1] = 2 * boundary - 1;
}

// the root: a leaf, a subtree, or the first open node
__global__ void root_kernel(BuildBufs b, uint32_t n, uint32_t threshold)
{
  BuildState s = {};
  if (n <= threshold) {
    note_leaf(b, 0, n, 0, 0, kDone);
    s.leaves = 1;
  } else if (n <= kSub) {
    b.roots[0] = SubRoot{0, n, 0, kDone, 0};
    s.subRoots = 1;
  } else {
    b.begin[0][0] = 0;
    b.count[0][0] = n;
    b.link[0][0] = kDone;
    s.open[0] = 1;
  }
  *b.st = s;
}

// selectSplits (:316-396): the widest extent's centre; dim -1: degenerate.
// Degenerate is every centre that is not inside its box: one that rounds onto
// a face, and the infinite or NaN centre of a box whose l + h overflows or
// that holds infinities of both signs or a NaN.  Such a centre leaves one side
// empty and the other as it was, level after level; the alternating split
// halves the prims instead, so both children of every split hold some.
template <int D>
__device__ inline int decide(const int32_t *lo, const int32_t *hi, float *pos)
{
  float widestWidth = 0.f, at = 0.f;
  int dim = -1;
#pragma unroll
  for (int d = 0; d < D; d++) {
    const float l = dec(lo[d]), h = dec(hi[d]);
    const float width = __fsub_rn(h, l);
    if (width <= widestWidth) continue;
    widestWidth = width;
    dim = d;
    at = __fmul_rn(0.5f, __fadd_rn(l, h));
    if (!(at > l && at < h)) dim = -2 - d;
  }
  if (dim < 0) {
    dim = -1;
    at = dec(lo[0]);
  }
  *pos = at;
  return dim;
}

// Left-side prims at positions below p (the level's side bits).
__device__ inline uint32_t left_before(const BuildBufs &b, uint32_t p)
{
  const uint32_t t = b.tileBase[p / kSideTile];
  if ((p & (kSideTile - 1)) == 0) return t;
  const uint32_t w = p >> 5;
  return t + b.wordPre[w] + __popc(b.bits[w] & ((1u << (p & 31)) - 1u));
}

// updatePrims (:398-436): a bit per prim of an open node that goes left, the
// bits' prefix sums within kSideTile-prim tiles, and (the last CTA) over tiles.
// Every prim decides its node's split itself: the box is in L1, and a launch
// of its own would cost more.
template <int D>
__global__ void __launch_bounds__(256) side_kernel(BuildBufs b, int64_t n, int par, int tiles)
{
  __shared__ uint32_t warpSum[8];
  __shared__ bool last;
  // (also without open nodes: the next level must find none either)
  if (blockIdx.x == 0 && threadIdx.x == 0) b.st->open[par ^ 1] = 0;
  if (b.st->open[par] == 0) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t base = int64_t(blockIdx.x) * kSideTile + wid * (32 * kSideWords);
  uint32_t word = 0;
#pragma unroll
  for (int j = 0; j < kSideWords; j++) {
    const int64_t p = base + 32 * j + lane;
    bool left = false;
    if (p < n) {
      const uint32_t node = b.nodeOf[par][p];
      if (node != kDone) {
        float pos;
        const int dim = decide<D>(b.lo[par] + int64_t(node) * D, b.hi[par] + int64_t(node) * D,
                                  &pos);
        left = dim < 0 ? ((uint32_t(p) - b.begin[par][node]) & 1u) == 0
                       : !(b.coord[par][dim][p] >= pos);
      }
    }
    const uint32_t w = __ballot_sync(0xffffffffu, left);
    if (lane == j) word = w;
  }
  const uint32_t c = lane < kSideWords ? __popc(word) : 0;
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < kSideWords; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == kSideWords - 1) warpSum[wid] = incl;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < 8; w++) {
    before += w < wid ? warpSum[w] : 0;
    total += warpSum[w];
  }
  if (lane < kSideWords) {
    b.bits[(base >> 5) + lane] = word;
    b.wordPre[(base >> 5) + lane] = before + incl - c;
  }
  if (threadIdx.x == 0) {
    b.tileBase[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(&b.st->ticket, 1u) + 1 == gridDim.x;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // exclusive scan of the tile sums, [tiles] = their total
  uint32_t carry = 0;
  for (int off = 0; off < tiles; off += 1024) {
    uint32_t v[4], s = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = off + threadIdx.x * 4 + j;
      v[j] = i < tiles ? __ldcg(b.tileBase + i) : 0u;
      s += v[j];
    }
    uint32_t in = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, in, o);
      if (lane >= o) in += t;
    }
    __syncthreads();
    if (lane == 31) warpSum[wid] = in;
    __syncthreads();
    uint32_t run = carry + in - s;
#pragma unroll
    for (int w = 0; w < 8; w++) {
      run += w < wid ? warpSum[w] : 0;
      carry += warpSum[w];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = off + threadIdx.x * 4 + j;
      if (i < tiles) b.tileBase[i] = run;
      run += v[j];
    }
  }
  if (threadIdx.x == 0) {
    b.tileBase[tiles] = carry;
    b.st->ticket = 0;
  }
}

// The open nodes' split records and children: leaves, subtree roots, or open
// nodes of the next level (empty boxes).
template <int D>
__global__ void __launch_bounds__(128) children_kernel(BuildBufs b, int par, uint32_t level,
                                                       uint32_t threshold)
{
  const uint32_t m = b.st->open[par];
  const int nxt = par ^ 1;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const uint32_t begin = b.begin[par][i], count = b.count[par][i];
    float pos;
    const int dim = decide<D>(b.lo[par] + int64_t(i) * D, b.hi[par] + int64_t(i) * D, &pos);
    const uint32_t pre = left_before(b, begin);
    const uint32_t nl = left_before(b, begin + count) - pre;
    const uint32_t boundary = begin + nl;
    note_split(b, boundary, dim, pos, level, b.link[par][i]);
    uint32_t code[2];
    for (int s = 0; s < 2; s++) {
      const uint32_t cb = s == 0 ? begin : boundary, cc = s == 0 ? nl : count - nl;
      const uint32_t link = boundary * 2 + (s == 0);
      code[s] = kDone;
      if (cc <= threshold) {
        note_leaf(b, cb, cc, level + 1, nxt, link);
        atomicAdd(&b.st->leaves, 1u);
        atomicMax(&b.st->maxLevel, level + 1);
      } else if (cc <= kSub) {
        b.roots[atomicAdd(&b.st->subRoots, 1u)] = SubRoot{cb, cc, level + 1, link, uint32_t(nxt)};
      } else {
        const uint32_t c = atomicAdd(&b.st->open[nxt], 1u);
        code[s] = c;
        b.begin[nxt][c] = cb;
        b.count[nxt][c] = cc;
        b.link[nxt][c] = link;
        for (int d = 0; d < D; d++) {
          b.lo[nxt][int64_t(c) * D + d] = enc(+FLT_MAX);
          b.hi[nxt][int64_t(c) * D + d] = enc(-FLT_MAX);
        }
      }
    }
    b.move[i] = make_uint4(begin, pre, nl, 0u);
    b.codes[i] = make_uint2(code[0], code[1]);
  }
}

// Every prim of an open node to its place in its child's segment; boxes of
// the children that stay open.
template <int D>
__global__ void __launch_bounds__(256) move_kernel(BuildBufs b, int64_t n, int par)
{
  if (b.st->open[par] == 0) return;
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int nxt = par ^ 1;
  uint32_t code = kDone;
  float pt[D];
#pragma unroll
  for (int d = 0; d < D; d++) pt[d] = 0.f;
  if (p < n) {
    const uint32_t node = b.nodeOf[par][p];
    if (node == kDone) {
      b.nodeOf[nxt][p] = kDone;
    } else {
      const uint4 mv = b.move[node];
      const uint2 cd = b.codes[node];
      const uint32_t before = left_before(b, uint32_t(p)) - mv.y;
      const bool isL = (b.bits[p >> 5] >> (p & 31)) & 1u;
      // a prim of a split node goes left or right: its right-side rank is its
      // rank in the segment minus its left-side rank
      const uint32_t dst = isL ? mv.x + before : mv.x + mv.z + (uint32_t(p) - mv.x - before);
      code = isL ? cd.x : cd.y;
      b.prim[nxt][dst] = b.prim[par][p];
      b.nodeOf[nxt][dst] = code;
#pragma unroll
      for (int d = 0; d < D; d++) {
        pt[d] = b.coord[par][d][p];
        b.coord[nxt][d][dst] = pt[d];
      }
    }
  }
  block_grow<D>(b.lo[nxt], b.hi[nxt], code, code != kDone, pt);
}

// ---------------------------------------------------------------------------
// one CTA finishes a subtree of at most kSub prims
// ---------------------------------------------------------------------------
constexpr int kSubThreads = 256;
constexpr int kSubPer = kSub / kSubThreads;
constexpr int kSubOpen = kSub / 2;  // open nodes hold at least two prims

template <int D> struct SubtreeSmem {
  float co[D][kSub];      // by input position
  uint32_t pid[kSub];
  int32_t lo[kSubOpen][D], hi[kSubOpen][D];
  uint32_t link[2][kSubOpen];
  uint16_t begin[2][kSubOpen], count[2][kSubOpen];
  float pos[kSubOpen];
  uint16_t pre[kSubOpen], nl[kSubOpen], code[kSubOpen][2];
  int8_t dim[kSubOpen];
  uint16_t ix[kSub], node[kSub];  // by position: input position, open node
  uint32_t bits[kSub / 32], wordPre[kSub / 32 + 1];
  uint32_t open[2], leaves, deepest;
};

template <int D>
__global__ void __launch_bounds__(kSubThreads) subtree_kernel(BuildBufs b, uint32_t threshold)
{
  extern __shared__ __align__(16) unsigned char raw[];
  SubtreeSmem<D> &s = *reinterpret_cast<SubtreeSmem<D> *>(raw);
  const SubRoot r = b.roots[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n = int(r.count);
  constexpr uint16_t kLeaf = 0xffff;
  for (int p = tid; p < n; p += kSubThreads) {
#pragma unroll
    for (int d = 0; d < D; d++) s.co[d][p] = b.coord[r.parity][d][r.begin + p];
    s.pid[p] = b.prim[r.parity][r.begin + p];
    s.ix[p] = uint16_t(p);
    s.node[p] = 0;
  }
  if (tid == 0) {
    s.begin[0][0] = 0;
    s.count[0][0] = uint16_t(n);
    s.link[0][0] = r.link;
    s.open[0] = 1;
    s.leaves = 0;
    s.deepest = r.level;
  }
  __syncthreads();
  uint32_t level = r.level;
  for (int par = 0;; par ^= 1, level++) {
    const int m = int(s.open[par]);
    if (m == 0) break;
    for (int i = tid; i < m * D; i += kSubThreads) {
      (&s.lo[0][0])[i] = enc(+FLT_MAX);
      (&s.hi[0][0])[i] = enc(-FLT_MAX);
    }
    if (tid == 0) s.open[par ^ 1] = 0;
    __syncthreads();
    // positions p = (4 wid + j) * 32 + lane: a warp's are consecutive
    uint16_t ix[kSubPer], nd[kSubPer];
#pragma unroll
    for (int j = 0; j < kSubPer; j++) {
      const int p = (kSubPer * wid + j) * 32 + lane;
      nd[j] = p < n ? s.node[p] : kLeaf;
      ix[j] = p < n ? s.ix[p] : 0;
      const uint32_t first = __shfl_sync(0xffffffffu, uint32_t(nd[j]), 0);
      if (__all_sync(0xffffffffu, nd[j] == first)) {  // one node: reduced first
        if (first != kLeaf) {
#pragma unroll
          for (int d = 0; d < D; d++) {
            const int32_t e = enc(s.co[d][ix[j]]);
            const int32_t l = __reduce_min_sync(0xffffffffu, e);
            const int32_t h = __reduce_max_sync(0xffffffffu, e);
            if (lane == 0) {
              atomicMin(&s.lo[first][d], l);
              atomicMax(&s.hi[first][d], h);
            }
          }
        }
      } else if (nd[j] != kLeaf) {
#pragma unroll
        for (int d = 0; d < D; d++) {
          const int32_t e = enc(s.co[d][ix[j]]);
          atomicMin(&s.lo[nd[j]][d], e);
          atomicMax(&s.hi[nd[j]][d], e);
        }
      }
    }
    __syncthreads();
    for (int i = tid; i < m; i += kSubThreads) {
      float pos;
      s.dim[i] = int8_t(decide<D>(s.lo[i], s.hi[i], &pos));
      s.pos[i] = pos;
    }
    __syncthreads();
    bool left[kSubPer];
#pragma unroll
    for (int j = 0; j < kSubPer; j++) {
      const int p = (kSubPer * wid + j) * 32 + lane;
      left[j] = false;
      if (nd[j] != kLeaf) {
        const int dim = s.dim[nd[j]];
        left[j] = dim < 0 ? ((p - s.begin[par][nd[j]]) & 1) == 0
                          : !(s.co[dim][ix[j]] >= s.pos[nd[j]]);
      }
      const uint32_t w = __ballot_sync(0xffffffffu, left[j]);
      if (lane == 0) s.bits[kSubPer * wid + j] = w;
    }
    __syncthreads();
    if (wid == 0) {
      const uint32_t c = __popc(s.bits[lane]);
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      s.wordPre[lane] = incl - c;
      if (lane == 31) s.wordPre[32] = incl;
    }
    __syncthreads();
    auto before = [&](int p) -> uint32_t {
      return p == int(kSub) ? s.wordPre[32]
                            : s.wordPre[p >> 5] + __popc(s.bits[p >> 5] & ((1u << (p & 31)) - 1u));
    };
    for (int i = tid; i < m; i += kSubThreads) {
      const uint32_t begin = s.begin[par][i], count = s.count[par][i];
      const uint32_t pre = before(int(begin)), nl = before(int(begin + count)) - pre;
      const uint32_t boundary = r.begin + begin + nl;
      note_split(b, boundary, s.dim[i], s.pos[i], level, s.link[par][i]);
      s.pre[i] = uint16_t(pre);
      s.nl[i] = uint16_t(nl);
      for (int side = 0; side < 2; side++) {
        const uint32_t cb = side == 0 ? begin : begin + nl, cc = side == 0 ? nl : count - nl;
        const uint32_t link = boundary * 2 + (side == 0);
        if (cc <= threshold) {
          note_leaf(b, r.begin + cb, cc, level + 1, r.parity, link);
          s.code[i][side] = kLeaf;
          atomicAdd(&s.leaves, 1u);
          s.deepest = level + 1;
        } else {
          const uint32_t c = atomicAdd(&s.open[par ^ 1], 1u);
          s.begin[par ^ 1][c] = uint16_t(cb);
          s.count[par ^ 1][c] = uint16_t(cc);
          s.link[par ^ 1][c] = link;
          s.code[i][side] = uint16_t(c);
        }
      }
    }
    __syncthreads();
    // every thread holds its positions' prims in registers: moved in place
#pragma unroll
    for (int j = 0; j < kSubPer; j++) {
      const int p = (kSubPer * wid + j) * 32 + lane;
      if (nd[j] == kLeaf) continue;
      const int i = nd[j];
      const int begin = s.begin[par][i];
      const int bf = int(before(p)) - int(s.pre[i]);
      const int dst = left[j] ? begin + bf : begin + int(s.nl[i]) + (p - begin - bf);
      s.ix[dst] = ix[j];
      s.node[dst] = s.code[i][left[j] ? 0 : 1];
    }
    __syncthreads();
  }
  for (int p = tid; p < n; p += kSubThreads)
    b.prim[r.parity][r.begin + p] = s.pid[s.ix[p]];
  if (tid == 0) {
    atomicAdd(&b.st->leaves, s.leaves);
    atomicMax(&b.st->maxLevel, s.deepest);
  }
}

// ---------------------------------------------------------------------------
// numbering
// ---------------------------------------------------------------------------
__global__ void iota_kernel(uint32_t *v, int64_t n)
{
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    v[i] = uint32_t(i);
}

// node 1 is the reference's empty dummy (initState, :276-290)
__device__ inline uint32_t node_id(uint32_t rank) { return rank == 0 ? 0u : rank + 1u; }

// each place's node number, and the prims of the leaves by node number
__global__ void number_kernel(BuildBufs b, const uint32_t *__restrict__ place, uint32_t nodes,
                              uint32_t *id, uint32_t *leafPrims)
{
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nodes) return;
  const uint32_t p = place[r];
  id[p] = node_id(r);
  leafPrims[node_id(r)] = (p & 1) ? 0u : b.leaf[p >> 1] & 0x7fffffffu;
  if (r == 0) leafPrims[1] = 0;
}

// node records and the leaves' prim lists (a leaf of more than 16 prims by
// its whole warp)
__global__ void __launch_bounds__(256) write_kernel(BuildBufs b,
                                                    const uint32_t *__restrict__ place,
                                                    uint32_t nodes,
                                                    const uint32_t *__restrict__ id,
                                                    const uint32_t *__restrict__ offset,
                                                    Node *out, uint32_t *primIDs)
{
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t count = 0, first = 0, to = 0, parity = 0;
  if (r < nodes) {
    const uint32_t p = place[r];
    Node o;
    if (p & 1) {
      const uint32_t boundary = (p + 1) >> 1;
      o.pos = b.splitPos[boundary];
      o.offset = id[b.splitChild[boundary]];
      o.count = 0;
      o.dim = int16_t(b.splitDim[boundary]);
    } else {
      first = p >> 1;
      count = b.leaf[first] & 0x7fffffffu;
      parity = b.leaf[first] >> 31;
      to = offset[node_id(r)];
      o.pos = 0.f;
      o.offset = to;
      o.count = uint16_t(count);
      o.dim = 0;
    }
    out[node_id(r)] = o;
    if (r == 0) out[1] = Node{0.f, 0u, 0, 0};
  }
  if (count <= 16)
    for (uint32_t j = 0; j < count; j++) primIDs[to + j] = b.prim[parity][first + j];
  for (unsigned big = __ballot_sync(0xffffffffu, count > 16); big; big &= big - 1) {
    const int l = __ffs(big) - 1;
    const uint32_t c = __shfl_sync(0xffffffffu, count, l);
    const uint32_t f = __shfl_sync(0xffffffffu, first, l);
    const uint32_t t = __shfl_sync(0xffffffffu, to, l);
    const uint32_t *src = b.prim[__shfl_sync(0xffffffffu, parity, l)];
    for (uint32_t j = threadIdx.x & 31; j < c; j += 32) primIDs[t + j] = src[f + j];
  }
}

static int alloc_out(const cukd_mem_resource *mem, cudaStream_t st, void **p, size_t bytes)
{
  bytes = std::max<size_t>(bytes, 16);
  if (mem && mem->alloc) {
    if (mem->alloc(mem->ctx, p, bytes, st) != 0 || !*p) return CUKD_ERR_OUT_OF_MEMORY;
    return CUKD_OK;
  }
  cudaError_t e = cudaMallocAsync(p, bytes, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? CUKD_ERR_OUT_OF_MEMORY : CUKD_ERR_CUDA;
  }
  return CUKD_OK;
}

template <int D>
int build_impl(const void *pts, int64_t n, const Layout &L, int threshold,
               cukd_spatial_tree *tree, cudaStream_t st, const cukd_mem_resource *mem)
{
  if (threshold == 0) threshold = 8;  // spatial-kdtree.h:505-506
  if (threshold < 1 || threshold > 65535) return CUKD_ERR_INVALID_ARGUMENT;
  TempArena arena(st, mem);
  BuildBufs b = {};
  b.data = (const uint8_t *)pts;
  b.stride = L.stride;
  b.poff = L.poff;
  // open nodes hold more than kSub prims each
  const int64_t cap = std::max<int64_t>(1, n / kSub + 1);
  const int tiles = int(std::max<int64_t>(1, div_up(n, kSideTile)));
  const int64_t np = std::max<int64_t>(n, 1);
  uint32_t *key2 = nullptr, *place = nullptr, *place2 = nullptr;
  CKB_TRY(arena.alloc(&b.st, 1));
  for (int x = 0; x < 2; x++) {
    CKB_TRY(arena.alloc(&b.begin[x], cap));
    CKB_TRY(arena.alloc(&b.count[x], cap));
    CKB_TRY(arena.alloc(&b.link[x], cap));
    CKB_TRY(arena.alloc(&b.lo[x], cap * D));
    CKB_TRY(arena.alloc(&b.hi[x], cap * D));
    CKB_TRY(arena.alloc(&b.prim[x], np));
    CKB_TRY(arena.alloc(&b.nodeOf[x], np));
    for (int d = 0; d < D; d++) CKB_TRY(arena.alloc(&b.coord[x][d], np));
  }
  CKB_TRY(arena.alloc(&b.move, cap));
  CKB_TRY(arena.alloc(&b.codes, cap));
  CKB_TRY(arena.alloc(&b.bits, int64_t(tiles) * (kSideTile / 32)));
  CKB_TRY(arena.alloc(&b.wordPre, int64_t(tiles) * (kSideTile / 32)));
  CKB_TRY(arena.alloc(&b.tileBase, tiles + 1));
  CKB_TRY(arena.alloc(&b.roots, np / 2 + 1));  // at least two prims each
  CKB_TRY(arena.alloc(&b.key, 2 * np));
  CKB_TRY(arena.alloc(&key2, 2 * np));
  CKB_TRY(arena.alloc(&place, 2 * np));
  CKB_TRY(arena.alloc(&place2, 2 * np));
  CKB_TRY(arena.alloc(&b.splitChild, np));
  CKB_TRY(arena.alloc(&b.splitPos, np));
  CKB_TRY(arena.alloc(&b.splitDim, np));
  CKB_TRY(arena.alloc(&b.leaf, np));
  // root: empty box, then grown by every prim (initPrims, :300-314)
  {
    int32_t box[2 * D];
    for (int d = 0; d < D; d++) {
      box[d] = enc(+FLT_MAX);
      box[D + d] = enc(-FLT_MAX);
    }
    CKB_CUDA(cudaMemcpyAsync(b.lo[0], box, sizeof(int32_t) * D, cudaMemcpyHostToDevice, st));
    CKB_CUDA(cudaMemcpyAsync(b.hi[0], box + D, sizeof(int32_t) * D, cudaMemcpyHostToDevice, st));
  }
  // places without a node sort behind every level
  CKB_CUDA(cudaMemsetAsync(b.key, 0xff, sizeof(uint32_t) * 2 * np, st));
  const unsigned nb = unsigned(div_up(np, 256));
  init_kernel<D><<<nb, 256, 0, st>>>(b, n);
  CKB_CHECK_LAUNCH();
  // the root's box is the tree's: kept before its buffer is used again
  int32_t *box = nullptr;
  CKB_TRY(arena.alloc(&box, 2 * D));
  CKB_CUDA(cudaMemcpyAsync(box, b.lo[0], sizeof(int32_t) * D, cudaMemcpyDeviceToDevice, st));
  CKB_CUDA(cudaMemcpyAsync(box + D, b.hi[0], sizeof(int32_t) * D, cudaMemcpyDeviceToDevice, st));
  root_kernel<<<1, 1, 0, st>>>(b, uint32_t(n), uint32_t(threshold));
  CKB_CHECK_LAUNCH();

  // ---- the level phase: the levels a balanced tree would need, two more,
  // then four at a time until no open node is left (a launch without open
  // nodes returns at once)
  uint32_t subRoots = n <= threshold ? 0 : 1;
  const int64_t big = std::max<int64_t>(kSub, threshold);
  if (n > big) {
    int batch = 2;
    for (int64_t c = n; c > big; c = div_up(c, 2)) batch++;
    BuildState hs = {};
    uint32_t level = 0;
    do {
      for (int i = 0; i < batch; i++, level++) {
        const int par = int(level & 1);
        side_kernel<D><<<unsigned(tiles), 256, 0, st>>>(b, n, par, tiles);
        CKB_CHECK_LAUNCH();
        const int64_t open = level < 40 ? std::min<int64_t>(cap, int64_t(1) << level) : cap;
        children_kernel<D><<<unsigned(std::min<int64_t>(div_up(open, 128), kNumSMs * 8)), 128, 0,
                             st>>>(b, par, level, uint32_t(threshold));
        CKB_CHECK_LAUNCH();
        move_kernel<D><<<nb, 256, 0, st>>>(b, n, par);
        CKB_CHECK_LAUNCH();
      }
      CKB_CUDA(cudaMemcpyAsync(&hs, b.st, sizeof(hs), cudaMemcpyDeviceToHost, st));
      CKB_CUDA(cudaStreamSynchronize(st));
      batch = 4;
    } while (hs.open[level & 1] != 0);
    subRoots = hs.subRoots;
  }
  // ---- subtrees
  if (subRoots > 0) {
    constexpr int smem = int(sizeof(SubtreeSmem<D>));
    CKB_CUDA(cudaFuncSetAttribute(subtree_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  smem));
    subtree_kernel<D><<<subRoots, kSubThreads, smem, st>>>(b, uint32_t(threshold));
    CKB_CHECK_LAUNCH();
  }
  // ---- numbering: nodes by level, then from left to right
  iota_kernel<<<unsigned(std::min<int64_t>(div_up(2 * np, 256), kNumSMs * 16)), 256, 0, st>>>(
      place, 2 * np);
  CKB_CHECK_LAUNCH();
  BuildState hs = {};
  int32_t hb[2 * D];
  CKB_CUDA(cudaMemcpyAsync(&hs, b.st, sizeof(hs), cudaMemcpyDeviceToHost, st));
  CKB_CUDA(cudaMemcpyAsync(hb, box, sizeof(hb), cudaMemcpyDeviceToHost, st));
  CKB_CUDA(cudaStreamSynchronize(st));
  // (a box halves an extent per level: a depth of a few thousand at most)
  CKB_TRY(radix_sort_pairs(b.key, place, key2, place2, 2 * np, hs.maxLevel < 255 ? 8 : 16, st,
                           &arena));
  const uint32_t count = n > 0 ? 2 * hs.leaves - 1 : 1;
  const uint32_t numNodes = count + 1;
  uint32_t *id = key2, *off = nullptr;
  CKB_TRY(arena.alloc(&off, numNodes + 1));
  const unsigned tb = unsigned(div_up(count, 256));
  number_kernel<<<tb, 256, 0, st>>>(b, place, count, id, off);
  CKB_CHECK_LAUNCH();
  CKB_TRY(exclusive_scan_u32(off, off, numNodes, nullptr, st, &arena));

  void *nodes = nullptr, *prims = nullptr;
  CKB_TRY(alloc_out(mem, st, &nodes, sizeof(Node) * numNodes));
  const int rcP = alloc_out(mem, st, &prims, sizeof(uint32_t) * np);
  if (rcP != CUKD_OK) {
    if (mem && mem->release) mem->release(mem->ctx, nodes, st); else cudaFreeAsync(nodes, st);
    return rcP;
  }
  write_kernel<<<tb, 256, 0, st>>>(b, place, count, id, off, (Node *)nodes, (uint32_t *)prims);
  CKB_CHECK_LAUNCH();
  tree->nodes = (Node *)nodes;
  tree->prim_ids = (uint32_t *)prims;
  tree->data = pts;
  tree->num_prims = int32_t(n);
  tree->num_nodes = int32_t(numNodes);
  tree->num_dims = D;
  for (int i = 0; i < 8; i++) tree->bounds[i] = 0.f;
  for (int d = 0; d < D; d++) {
    tree->bounds[d] = dec(hb[d]);
    tree->bounds[4 + d] = dec(hb[D + d]);
  }
  return CUKD_OK;
}

// ---------------------------------------------------------------------------
// traversals (fcp.h:256-427, knn.h:566-646 cct / 680-752 stackBased), one
// thread per query, 50-entry stack like the reference
// ---------------------------------------------------------------------------
struct SArgs {
  query::QArgs q;
  const Node *nodes;
  const uint32_t *primIDs;
  const uint8_t *data;
  int stride, poff;
  int numPrims;
  float lo[4], hi[4];
};

template <int D, int METHOD, class Res>
__global__ void __launch_bounds__(128) spatial_query_kernel(SArgs s)
{
  const query::QArgs &a = s.q;
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= a.nq) return;
  const int64_t qi = a.order ? int64_t(a.order[i]) : i;
  float q[D];
#pragma unroll
  for (int d = 0; d < D; d++) q[d] = __ldg((const float *)a.queries + qi * D + d);
  Res res(a);
  auto d2of = [&](const float *c) {
    float sum = __fmul_rn(__fsub_rn(c[0], q[0]), __fsub_rn(c[0], q[0]));
#pragma unroll
    for (int d = 1; d < D; d++)
      sum = __fadd_rn(sum, __fmul_rn(__fsub_rn(c[d], q[d]), __fsub_rn(c[d], q[d])));
    return sum;
  };
  if (s.numPrims > 0) {
    constexpr int kDepth = 50;
    int nodeSt[kDepth];
    float distSt[kDepth];
    float cornerSt[METHOD == CUKD_CCT ? kDepth : 1][D];
    int sp = 0;
    float cullDist = res.init();
    float closest[D];
    bool run = true;
    if (METHOD == CUKD_CCT) {
#pragma unroll
      for (int d = 0; d < D; d++) {
        float v = q[d];
        v = v < s.lo[d] ? s.lo[d] : v;
        v = s.hi[d] < v ? s.hi[d] : v;
        closest[d] = v;
      }
      if (d2of(closest) > cullDist) run = false;
    }
    int nodeID = 0;
    bool overflow = false;
    while (run) {
      Node node;
      for (;;) {
        node = s.nodes[nodeID];
        if (node.count) break;
        float qc = q[0];
#pragma unroll
        for (int d = 1; d < D; d++)
          if (d == node.dim) qc = q[d];
        const bool leftIsClose = qc < node.pos;
        const int lChild = int(node.offset), rChild = lChild + 1;
        const int closeChild = leftIsClose ? lChild : rChild;
        const int farChild = leftIsClose ? rChild : lChild;
        bool push;
        float fc[D];
        if (METHOD == CUKD_CCT) {
#pragma unroll
          for (int d = 0; d < D; d++) fc[d] = d == node.dim ? node.pos : closest[d];
          push = d2of(fc) < cullDist;
        } else {
          const float diff = __fsub_rn(qc, node.pos);
          const float pd2 = __fmul_rn(diff, diff);
          push = pd2 < cullDist;
          fc[0] = pd2;
        }
        if (push) {
          nodeSt[sp] = farChild;
          if (METHOD == CUKD_CCT) {
#pragma unroll
            for (int d = 0; d < D; d++) cornerSt[sp][d] = fc[d];
          } else {
            distSt[sp] = fc[0];
          }
          ++sp;
          if (sp >= kDepth) {  // the reference prints STACK OVERFLOW and returns -1
            overflow = true;
            run = false;
            break;
          }
        }
        nodeID = closeChild;
      }
      if (!run) break;
      for (int j = 0; j < node.count; j++) {
        const uint32_t primID = __ldg(s.primIDs + node.offset + j);
        float p[D];
        const float *c = (const float *)(s.data + int64_t(primID) * s.stride + s.poff);
#pragma unroll
        for (int d = 0; d < D; d++) p[d] = __ldg(c + d);
        cullDist = res.process(int32_t(primID), d2of(p));
      }
      for (;;) {
        if (sp == 0) {
          run = false;
          break;
        }
        --sp;
        if (METHOD == CUKD_CCT) {
#pragma unroll
          for (int d = 0; d < D; d++) closest[d] = cornerSt[sp][d];
          if (d2of(closest) >= cullDist) continue;
        } else {
          if (distSt[sp] >= cullDist) continue;
        }
        nodeID = nodeSt[sp];
        break;
      }
    }
    if (overflow) res.overflow();
  }
  res.write(a, qi);
}

template <class Res> struct WithOverflow : Res {
  __device__ WithOverflow(const query::QArgs &a) : Res(a) {}
  __device__ void overflow() {}
};
struct FcpOverflow : query::FcpRes<0> {
  __device__ FcpOverflow(const query::QArgs &a) : query::FcpRes<0>(a) {}
  __device__ void overflow() { id = -1; }
};

template <int D, int METHOD>
int launch_method(const SArgs &s, int kind, cudaStream_t st)
{
  using namespace query;
  const unsigned grid = unsigned(div_up(s.q.nq, 128));
#define CKB_L(...) spatial_query_kernel<D, METHOD, __VA_ARGS__><<<grid, 128, 0, st>>>(s)
  switch (kind) {
    case RES_FCP: CKB_L(FcpOverflow); break;
    case RES_FIX4: CKB_L(WithOverflow<FixedRes<0, 4>>); break;
    case RES_FIX8: CKB_L(WithOverflow<FixedRes<0, 8>>); break;
    case RES_FIX16: CKB_L(WithOverflow<FixedRes<0, 16>>); break;
    case RES_FIX32: CKB_L(WithOverflow<FixedRes<0, 32>>); break;
    case RES_HEAP128: CKB_L(WithOverflow<HeapRes<0, 128>>); break;
    case RES_HEAP1024: CKB_L(WithOverflow<HeapRes<0, 1024>>); break;
    default: return CUKD_ERR_UNSUPPORTED;
  }
#undef CKB_L
  CKB_CHECK_LAUNCH();
  return CUKD_OK;
}

template <int D>
int query_impl(const SArgs &s, int method, int kind, cudaStream_t st)
{
  if (method == CUKD_CCT) return launch_method<D, CUKD_CCT>(s, kind, st);
  if (method == CUKD_STACK_BASED) return launch_method<D, CUKD_STACK_BASED>(s, kind, st);
  return CUKD_ERR_UNSUPPORTED;  // the reference has no stack-free spatial traversal
}

}  // namespace spatial

int query_order(const void *queries, int64_t n, int scalar, int D, const void *d_bounds,
                const float *lo, const float *hi, const int32_t **order, cudaStream_t st,
                TempArena *arena);

static int spatial_query(const cukd_spatial_tree *tree, const cukd_layout *layout,
                         const void *d_queries, int64_t nq, const cukd_query_params *p,
                         bool knn, int32_t *ids, void *d2, cudaStream_t st,
                         const cukd_mem_resource *mem)
{
  using namespace query;
  Layout L;
  if (!tree || !p || !make_layout(layout, &L) || L.scalar != CUKD_FLOAT32)
    return CUKD_ERR_INVALID_ARGUMENT;
  if (L.D != tree->num_dims) return CUKD_ERR_INVALID_ARGUMENT;
  if (nq < 0) return CUKD_ERR_INVALID_ARGUMENT;
  if (nq == 0) return CUKD_OK;
  if (!d_queries || !ids) return CUKD_ERR_INVALID_ARGUMENT;
  int kind = RES_FCP;
  if (knn) {
    const int k = p->k;
    if (k < 1 || k > 1024) return CUKD_ERR_INVALID_ARGUMENT;
    const bool heap = (p->flags & (CUKD_QUERY_FORCE_HEAP | CUKD_QUERY_HEAP_ORDER)) || k > 32;
    kind = heap ? (k <= 128 ? RES_HEAP128 : RES_HEAP1024)
                : (k <= 4 ? RES_FIX4 : (k <= 8 ? RES_FIX8 : (k <= 16 ? RES_FIX16 : RES_FIX32)));
  }
  spatial::SArgs s = {};
  s.q.nq = nq;
  s.q.queries = d_queries;
  s.q.k = knn ? p->k : 1;
  s.q.cutoff = p->cutoff_radius;
  s.q.heap_order = (p->flags & CUKD_QUERY_HEAP_ORDER) != 0;
  s.q.out_ids = ids;
  s.q.out_d2 = d2;
  s.nodes = tree->nodes;
  s.primIDs = tree->prim_ids;
  s.data = (const uint8_t *)tree->data;
  s.stride = L.stride;
  s.poff = L.poff;
  s.numPrims = tree->num_prims;
  for (int d = 0; d < 4; d++) {
    s.lo[d] = tree->bounds[d];
    s.hi[d] = tree->bounds[4 + d];
  }
  TempArena arena(st, mem);
  if ((p->flags & CUKD_QUERY_MORTON) && nq > 1) {
    CKB_TRY(query_order(d_queries, nq, CUKD_FLOAT32, L.D, nullptr, s.lo, s.hi, &s.q.order, st,
                        &arena));
  }
  if (L.D == 2) return spatial::query_impl<2>(s, p->method, kind, st);
  if (L.D == 3) return spatial::query_impl<3>(s, p->method, kind, st);
  if (L.D == 4) return spatial::query_impl<4>(s, p->method, kind, st);
  return CUKD_ERR_UNSUPPORTED;
}

}  // namespace ckb

extern "C" {

int cukd_spatial_build(const void *d_points, int64_t n, const cukd_layout *layout,
                       int leaf_threshold, cukd_spatial_tree *out_tree, cudaStream_t stream,
                       const cukd_mem_resource *mem)
{
  ckb::Layout L;
  if (!out_tree || !ckb::make_layout(layout, &L)) return CUKD_ERR_INVALID_ARGUMENT;
  if (L.scalar != CUKD_FLOAT32) return CUKD_ERR_UNSUPPORTED;
  if (n < 0 || n > (int64_t(1) << 30)) return CUKD_ERR_INVALID_ARGUMENT;
  if (n > 0 && !d_points) return CUKD_ERR_INVALID_ARGUMENT;
  if (L.D == 2) return ckb::spatial::build_impl<2>(d_points, n, L, leaf_threshold, out_tree, stream, mem);
  if (L.D == 3) return ckb::spatial::build_impl<3>(d_points, n, L, leaf_threshold, out_tree, stream, mem);
  if (L.D == 4) return ckb::spatial::build_impl<4>(d_points, n, L, leaf_threshold, out_tree, stream, mem);
  return CUKD_ERR_UNSUPPORTED;
}

int cukd_spatial_free(cukd_spatial_tree *tree, cudaStream_t stream, const cukd_mem_resource *mem)
{
  if (!tree) return CUKD_ERR_INVALID_ARGUMENT;
  for (void *p : {(void *)tree->nodes, (void *)tree->prim_ids}) {
    if (!p) continue;
    if (mem && mem->release)
      mem->release(mem->ctx, p, stream);
    else
      cudaFreeAsync(p, stream);
  }
  tree->nodes = nullptr;
  tree->prim_ids = nullptr;
  tree->num_nodes = 0;
  tree->num_prims = 0;
  return CUKD_OK;
}

int cukd_spatial_fcp(const cukd_spatial_tree *tree, const cukd_layout *layout,
                     const void *d_queries, int64_t nq, const cukd_query_params *params,
                     int32_t *d_out_ids, void *d_out_d2, cudaStream_t stream,
                     const cukd_mem_resource *mem)
{
  return ckb::spatial_query(tree, layout, d_queries, nq, params, false, d_out_ids, d_out_d2,
                            stream, mem);
}

int cukd_spatial_knn(const cukd_spatial_tree *tree, const cukd_layout *layout,
                     const void *d_queries, int64_t nq, const cukd_query_params *params,
                     int32_t *d_out_ids, void *d_out_d2, cudaStream_t stream,
                     const cukd_mem_resource *mem)
{
  return ckb::spatial_query(tree, layout, d_queries, nq, params, true, d_out_ids, d_out_d2,
                            stream, mem);
}

}  // extern "C"
