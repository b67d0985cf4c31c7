// Fast exact kNN / FCP path (fast.cu): arguments and launcher.
#pragma once

#include <algorithm>

#include "query.cuh"

namespace ckb {
namespace fast {

struct FastArgs {
  query::QArgs q;       // tree / queries / outputs (ids, d2 [nq][k], max [nq])
  int kk;               // k (1 for FCP)
  bool fcp;             // FCP semantics (strict minimum, -1 beyond the cut-off)
  int method;           // the named traversal (which tied candidates it visits)
  int *fb_count;        // fallback queue length (zeroed before the launch)
  int32_t *fb_list;     // fallback queue (query indices), capacity nq
  const float *radius;  // optional per-query initial cull radius (before scaling)
  int32_t *status;      // optional per-query outcome: 0 answered, 1 queued
  float radius_scale;   // multiplies `radius`
  int queue_min;        // with q.count_ptr: a queue of at most this many is left alone
};

// the warp-per-query kernel's arguments (warp.cuh)
struct WarpArgs {
  FastArgs f;
  int queue_limit;  // with f.q.count_ptr: a longer queue is handed over, or left alone
  bool hand_over;   // copy such a queue to f.fb_list
};

}  // namespace fast

// Whether a node's point can be read as one vector load (8 bytes for D = 2,
// 16 for D = 3 and 4; for D = 3 with the split dim, if explicit, in the
// fourth word): the records' stride, the point's place in them and the
// array's address all have to be aligned.
inline bool vector_points(const query::QArgs &a, int D)
{
  const int al = D == 2 ? 8 : 16;
  if (a.stride % al || a.poff % al || reinterpret_cast<uintptr_t>(a.tree) % al) return false;
  return D != 3 || a.doff < 0 || a.doff == a.poff + 12;
}

// Asks for no more shared memory per SM than the resident blocks' candidate
// nodes take (kc words a thread): the driver's own choice leaves the stack
// and the nodes less L1 (10M queries, k = 16: 132 KB, 10.85 ms; 82 KB,
// 10.50 ms).
template <class Kernel>
inline void prefer_shared(Kernel *kernel, int threads, int block, int kc)
{
  const int bytes = threads * kc * 4 + (threads + block - 1) / block * 1024;
  const int percent = std::min(100, (bytes * 100 + 228 * 1024 - 1) / (228 * 1024));
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, percent) !=
      cudaSuccess)
    cudaGetLastError();  // a preference only
}

// Launches the fast kernel for float (scalar 0) or int32 (scalar 1) trees
// with D = 2..4 and k <= 128 (fast.cu).
int run_fast(const fast::FastArgs &fa, int scalar, int D, cudaStream_t st);
// the instantiations of one dimension (fast_d2.cu, fast_d3.cu, fast_d4.cu)
template <int D> int run_fast_dim(const fast::FastArgs &fa, int scalar, cudaStream_t st);
extern template int run_fast_dim<2>(const fast::FastArgs &, int, cudaStream_t);
extern template int run_fast_dim<3>(const fast::FastArgs &, int, cudaStream_t);
extern template int run_fast_dim<4>(const fast::FastArgs &, int, cudaStream_t);

// The same answers with a warp per query (warp.cuh): lower latency, about a
// fifth of the throughput.  All of q.nq, or a device-side queue.
int run_warp(const fast::WarpArgs &wa, int scalar, int D, cudaStream_t st);

// Calls of at most this many queries are answered a warp each; the line
// lies where the two kernels take the same time.  Whole calls, us, thread /
// warp per query (B200, uniform float3, 100K points): k = 8, 1000 queries
// 157 / 41, 16384 175 / 117, 32768 181 / 200; k = 32, 16384 257 / 206; k = 64,
// 8192 367 / 295, 16384 361 / 530; int3, 1M points, k = 16, 8192 146 / 122,
// 16384 146 / 198.  FCP and k = 1 (FCP, 500K points): 4000 queries 61 / 47,
// 8000 62 / 64, 16000 63 / 85; with ties, which the thread kernel has to
// settle after the warp kernel, 1000 64 / 92.
inline int64_t warp_queries(int scalar, int k)
{
  if (k == 1) return 6144;
  return scalar == CUKD_FLOAT32 && k <= 32 ? 16384 : 8192;
}
// and queued queries, of which the host does not know how many there are
constexpr int kWarpQueue = 8192;

// Whether visiting the queries in Z-order pays for sorting them: the sort is
// 65 us of dependent launches and 14 us a million queries, and saves a
// share of the search that grows with k, with D, and with a tree that the L2
// does not hold.  Whole calls on random queries, us, sorted / not (B200,
// float3, 10K points): FCP 500K 212 / 171; k = 4, 200K 213 / 151, 500K
// 320 / 298; k = 16, 200K 330 / 284, 500K 542 / 580; k = 64, 50K 440 / 423,
// 100K 635 / 706; record32, 4M points: FCP 500K 475 / 508, k = 16, 200K
// 900 / 993.
inline bool order_pays(int64_t nq, int k, int D, int64_t treeBytes)
{
  int64_t line = int64_t(6) << 20;
  if (D >= 4) line /= 2;
  if (treeBytes > (int64_t(96) << 20)) line /= 2;
  return nq * (k == 1 ? 4 : k + 8) >= line;
}

// The warp-cooperative traversal (packet.cu): float kNN, k = 2..32, no
// forest, no device-side query count.
int run_packet(const fast::FastArgs &fa, int D, cudaStream_t st);

}  // namespace ckb
