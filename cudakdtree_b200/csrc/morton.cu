// Morton (Z-order) query reordering and the stable LSD radix sort it uses.
//
// The reference has no query reordering: callers launch one thread per
// query in input order (sample.cu:49-74).  Sorting queries along a Morton
// curve makes the 32 traversals of a warp walk nearly the same tree path,
// which cuts divergence and raises L1/L2 hit rates.  It never changes a
// result: every query is still answered by its own traversal, and the
// answers are scattered back to the caller's order.
#include <algorithm>

#include "common.cuh"
#include "sort.cuh"

namespace ckb {

namespace {

__device__ inline uint32_t expand_bits(uint32_t v, int D)
{
  // spread the low bits of v so that consecutive bits land D apart
  uint32_t r = 0;
  const int bits = 30 / D;
  for (int b = 0; b < bits; b++) r |= ((v >> b) & 1u) << (b * D);
  return r;
}

__global__ void query_bounds_kernel(const float *__restrict__ pts, int64_t n, int D,
                                    uint32_t *kmin, uint32_t *kmax)
{
  uint32_t lo[4] = {~0u, ~0u, ~0u, ~0u}, hi[4] = {0, 0, 0, 0};
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    for (int d = 0; d < D; d++) {
      const uint32_t k = float_key(pts[i * D + d]);
      lo[d] = min(lo[d], k);
      hi[d] = max(hi[d], k);
    }
  }
  for (int d = 0; d < D; d++) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[d] = min(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = max(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
    if ((threadIdx.x & 31) == 0 && lo[d] <= hi[d]) {
      atomicMin(&kmin[d], lo[d]);
      atomicMax(&kmax[d], hi[d]);
    }
  }
}

__global__ void morton_code_kernel(const float *__restrict__ pts, int64_t n, int D,
                                   const uint32_t *kmin, const uint32_t *kmax,
                                   const float *bounds, uint32_t *codes, uint32_t *vals)
{
  const int bits = 30 / D;
  const float cells = float(1u << bits);
  float lo[4], scale[4];
  for (int d = 0; d < D; d++) {
    const float l = bounds ? bounds[d] : key_float(kmin[d]);
    const float h = bounds ? bounds[D + d] : key_float(kmax[d]);
    lo[d] = l;
    scale[d] = h > l ? cells / (h - l) : 0.f;
  }
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    uint32_t code = 0;
    for (int d = 0; d < D; d++) {
      const float x = (pts[i * D + d] - lo[d]) * scale[d];
      const uint32_t c = x >= 0.f ? (x < cells ? uint32_t(x) : (1u << bits) - 1u) : 0u;
      code |= expand_bits(c, D) << (D - 1 - d);
    }
    codes[i] = code;
    vals[i] = uint32_t(i);
  }
}

// Codes of query_order: TOTAL / D bits per dimension over a box; the first
// digit's tile counts of the sort come with them.
struct OrderBox {
  const void *bounds;  // device: lower[D], upper[D] of the scalar type; or null
  float lo[4], hi[4];  // else these
};
template <int SC, int D, int TOTAL>
__global__ void __launch_bounds__(256) order_code_kernel(const uint32_t *__restrict__ pts,
                                                         int64_t n, OrderBox box, int numTiles,
                                                         uint32_t *codes, uint32_t *counts)
{
  constexpr int BITS = TOTAL / D;
  constexpr float CELLS = float(1 << BITS);
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  auto coord = [](uint32_t w) { return SC == 0 ? __uint_as_float(w) : float(int32_t(w)); };
  float lo[D], scale[D];
#pragma unroll
  for (int d = 0; d < D; d++) {
    const uint32_t *bw = (const uint32_t *)box.bounds;
    const float l = bw ? coord(__ldg(bw + d)) : box.lo[d];
    const float u = bw ? coord(__ldg(bw + D + d)) : box.hi[d];
    lo[d] = l;
    scale[d] = u > l ? CELLS / (u - l) : 0.f;
  }
  __syncthreads();
  const int64_t base = int64_t(blockIdx.x) * kSortTile;
#pragma unroll 4
  for (int j = 0; j < kSortTile / 256; j++) {
    const int64_t i = base + j * 256 + threadIdx.x;
    if (i >= n) break;
    uint32_t code = 0;
#pragma unroll
    for (int d = 0; d < D; d++) {
      const float x = (coord(__ldg(pts + i * D + d)) - lo[d]) * scale[d];
      const uint32_t c = x >= 0.f ? (x < CELLS ? uint32_t(x) : (1u << BITS) - 1u) : 0u;
#pragma unroll
      for (int b = 0; b < BITS; b++) code |= ((c >> b) & 1u) << (b * D + D - 1 - d);
    }
    codes[i] = code;
    atomicAdd(&h[code & 255u], 1u);
  }
  __syncthreads();
  counts[int64_t(threadIdx.x) * numTiles + blockIdx.x] = h[threadIdx.x];
}

}  // namespace

int morton_order_impl(const float *pts, int64_t n, int D, const float *bounds, int32_t *perm,
                      cudaStream_t st, const cukd_mem_resource *mem)
{
  if (n <= 0) return CUKD_OK;
  if (D < 1 || D > 4) return CUKD_ERR_INVALID_ARGUMENT;
  TempArena arena(st, mem);
  uint32_t *codes = nullptr, *codes2 = nullptr, *vals2 = nullptr, *kb = nullptr;
  CKB_TRY(arena.alloc(&codes, n));
  CKB_TRY(arena.alloc(&codes2, n));
  CKB_TRY(arena.alloc(&vals2, n));
  CKB_TRY(arena.alloc(&kb, 8));
  const int blocks = int(std::max<int64_t>(1, std::min<int64_t>(div_up(n, 256), kNumSMs * 8)));
  if (!bounds) {
    CKB_CUDA(cudaMemsetAsync(kb, 0xff, 16, st));
    CKB_CUDA(cudaMemsetAsync(kb + 4, 0, 16, st));
    query_bounds_kernel<<<blocks, 256, 0, st>>>(pts, n, D, kb, kb + 4);
    CKB_CHECK_LAUNCH();
  }
  morton_code_kernel<<<blocks, 256, 0, st>>>(pts, n, D, kb, kb + 4, bounds, codes,
                                             (uint32_t *)perm);
  CKB_CHECK_LAUNCH();
  const int bits = (30 / D) * D;
  return radix_sort_pairs(codes, (uint32_t *)perm, codes2, vals2, n, bits, st, &arena);
}

// The order in which a call visits its queries: a Z-order over the tree's box,
// which only has to group them (the answers do not depend on it).  24 bits and
// three sort passes do up to 4M queries (10 launches, 32 bytes of traffic a
// query; 1M queries, k = 8: whole call 904 -> 868 us against 30 bits in four
// passes and 14 launches); above, 30 bits in four passes (10M mixture queries,
// k = 16: 10.85 ms with 24 bits, 10.7 ms with 30).  d_bounds: the tree's world
// bounds on the device, or lo / hi on the host; queries outside are clamped to
// the box's faces.
int query_order(const void *queries, int64_t n, int scalar, int D, const void *d_bounds,
                const float *lo, const float *hi, const int32_t **order, cudaStream_t st,
                TempArena *arena)
{
  uint32_t *codes = nullptr, *codes2 = nullptr, *vals = nullptr, *vals2 = nullptr,
           *counts = nullptr;
  arena->reserve(4 * TempArena::rounded(sizeof(uint32_t) * n) +
                 TempArena::rounded(sizeof(uint32_t) * radix_sort_counts(n)));
  CKB_TRY(arena->alloc(&codes, n));
  CKB_TRY(arena->alloc(&codes2, n));
  CKB_TRY(arena->alloc(&vals, n));
  CKB_TRY(arena->alloc(&vals2, n));
  CKB_TRY(arena->alloc(&counts, size_t(radix_sort_counts(n))));
  OrderBox box = {};
  box.bounds = d_bounds;
  for (int d = 0; d < D && lo; d++) {
    box.lo[d] = lo[d];
    box.hi[d] = hi[d];
  }
  const int tiles = int(div_up(n, kSortTile));
  const int passes = n <= (int64_t(1) << 22) ? 3 : 4;
#define CKB_ORDER(SC_, D_, TOTAL_)                                                       \
  if (scalar == SC_ && D == D_ && passes == (TOTAL_ == 24 ? 3 : 4)) {                    \
    order_code_kernel<SC_, D_, TOTAL_><<<unsigned(tiles), 256, 0, st>>>(                 \
        (const uint32_t *)queries, n, box, tiles, codes, counts);                        \
    CKB_CHECK_LAUNCH();                                                                  \
  }
  CKB_ORDER(0, 2, 24) CKB_ORDER(0, 3, 24) CKB_ORDER(0, 4, 24)
  CKB_ORDER(1, 2, 24) CKB_ORDER(1, 3, 24) CKB_ORDER(1, 4, 24)
  CKB_ORDER(0, 2, 30) CKB_ORDER(0, 3, 30) CKB_ORDER(0, 4, 30)
  CKB_ORDER(1, 2, 30) CKB_ORDER(1, 3, 30) CKB_ORDER(1, 4, 30)
#undef CKB_ORDER
  CKB_TRY(radix_order(codes, codes2, vals, vals2, n, passes, counts, st));
  *order = (const int32_t *)(passes & 1 ? vals2 : vals);
  return CUKD_OK;
}

}  // namespace ckb

extern "C" int cukd_morton_order(const float *d_points, int64_t n, int num_dims,
                                 const float *d_bounds, int32_t *d_out_perm,
                                 cudaStream_t stream, const cukd_mem_resource *mem)
{
  if (n < 0 || (n > 0 && (!d_points || !d_out_perm))) return CUKD_ERR_INVALID_ARGUMENT;
  return ckb::morton_order_impl(d_points, n, num_dims, d_bounds, d_out_perm, stream, mem);
}
