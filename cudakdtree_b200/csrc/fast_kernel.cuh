// The fast kNN / FCP kernel (body in fast_one.cuh) and its launch rules;
// instantiated per dimension in fast_d2.cu, fast_d3.cu and fast_d4.cu.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "fast.cuh"
#include "fast_one.cuh"

namespace ckb {
namespace fast {

// Threads per block and resident blocks per SM the kernel is compiled for,
// by list capacity: the most threads whose registers hold the list.  Lists
// of up to 17 slots: 1024 threads (64 registers; 48 registers measured the
// same, 80 and 40 slower); 33: 768 (512 threads 3.25 ms, 768 2.57 ms for 1M
// mixture queries on 4M points, 1280 5.4 ms); 65: 512 (640 and 768 spill,
// 6.7 and 12.4 ms against 6.25 for 500K record32 queries); 129: 384.
constexpr int fast_threads(int kc) { return kc <= 17 ? 512 : (kc <= 33 ? 256 : (kc <= 65 ? 128 : 64)); }
constexpr int fast_blocks(int kc) { return kc <= 17 ? 2 : (kc <= 33 ? 3 : (kc <= 65 ? 4 : 6)); }

template <int SC, int D, bool EXPL, bool VEC, int KC>
__global__ void __launch_bounds__(fast_threads(KC), fast_blocks(KC))
    knn_fast_kernel(const __grid_constant__ FastArgs fa)
{
  extern __shared__ uint32_t sh[];
  const int64_t limit = fa.q.count_ptr ? int64_t(*fa.q.count_ptr) : fa.q.nq;
  if (fa.q.count_ptr && limit <= fa.queue_min) return;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < limit;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t myq = fa.q.order ? int64_t(fa.q.order[i]) : i;
    const bool seeded = fa.radius != nullptr;
    const float r = seeded ? __ldg(fa.radius + myq) : 0.f;
    knn_fast_one<SC, D, EXPL, VEC, KC>(fa, myq, seeded, r, sh + threadIdx.x, blockDim.x);
  }
}

template <int SC, int D, bool EXPL, bool VEC, int KC>
int launch_fast(const FastArgs &fa, cudaStream_t st)
{
  const int bs = std::min(fa.q.block_size > 0 ? fa.q.block_size : 128, fast_threads(KC));
  const int qpt = fa.q.queries_per_thread > 1 ? fa.q.queries_per_thread : 1;
  int64_t grid = std::max<int64_t>(1, div_up(fa.q.nq, int64_t(bs) * qpt));
  // a queue whose length is known on the device only: most blocks of a grid
  // for its capacity would find nothing to do
  if (fa.q.count_ptr) grid = std::min<int64_t>(grid, int64_t(kNumSMs) * 16);
  prefer_shared(knn_fast_kernel<SC, D, EXPL, VEC, KC>, fast_threads(KC) * fast_blocks(KC), bs, KC);
  knn_fast_kernel<SC, D, EXPL, VEC, KC><<<unsigned(grid), bs, sizeof(uint32_t) * KC * bs, st>>>(fa);
  CKB_CHECK_LAUNCH();
  return CUKD_OK;
}

template <int SC, int D, bool EXPL, bool VEC, bool FCP>
__global__ void __launch_bounds__(128, 10) fcp_fast_kernel(const __grid_constant__ FastArgs fa)
{
  const int64_t limit = fa.q.count_ptr ? int64_t(*fa.q.count_ptr) : fa.q.nq;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < limit;
       i += int64_t(gridDim.x) * blockDim.x)
    fcp_fast_one<SC, D, EXPL, VEC, FCP>(fa, fa.q.order ? int64_t(fa.q.order[i]) : i);
}

template <int SC, int D, bool EXPL, bool VEC, bool FCP>
int launch_fcp(const FastArgs &fa, cudaStream_t st)
{
  const int bs = fa.q.block_size > 0 ? std::min(fa.q.block_size, 128) : 128;
  int64_t grid = div_up(fa.q.nq, bs);
  if (fa.q.count_ptr) grid = std::min<int64_t>(grid, int64_t(kNumSMs) * 10);
  fcp_fast_kernel<SC, D, EXPL, VEC, FCP><<<unsigned(grid), bs, 0, st>>>(fa);
  CKB_CHECK_LAUNCH();
  return CUKD_OK;
}

template <int SC, int D, bool EXPL, bool VEC>
int dispatch_kc(const FastArgs &fa, cudaStream_t st)
{
  const int slots = fa.kk + 1;
  if (slots == 2)  // without seeds
    return fa.fcp ? launch_fcp<SC, D, EXPL, VEC, true>(fa, st)
                  : launch_fcp<SC, D, EXPL, VEC, false>(fa, st);
  if (slots <= 5) return launch_fast<SC, D, EXPL, VEC, 5>(fa, st);
  if (slots <= 9) return launch_fast<SC, D, EXPL, VEC, 9>(fa, st);
  if (slots <= 17) return launch_fast<SC, D, EXPL, VEC, 17>(fa, st);
  if (slots <= 33) return launch_fast<SC, D, EXPL, VEC, 33>(fa, st);
  if (slots <= 65) return launch_fast<SC, D, EXPL, VEC, 65>(fa, st);
  if (slots <= 129) return launch_fast<SC, D, EXPL, VEC, 129>(fa, st);
  return CUKD_ERR_UNSUPPORTED;
}

template <int SC, int D>
int dispatch_layout(const FastArgs &fa, cudaStream_t st)
{
  const bool vec = vector_points(fa.q, D);
  if (fa.q.doff >= 0)
    return vec ? dispatch_kc<SC, D, true, true>(fa, st) : dispatch_kc<SC, D, true, false>(fa, st);
  return vec ? dispatch_kc<SC, D, false, true>(fa, st) : dispatch_kc<SC, D, false, false>(fa, st);
}

}  // namespace fast

template <int D> int run_fast_dim(const fast::FastArgs &fa, int scalar, cudaStream_t st)
{
  return scalar == CUKD_FLOAT32 ? fast::dispatch_layout<0, D>(fa, st)
                                : fast::dispatch_layout<1, D>(fa, st);
}

}  // namespace ckb
