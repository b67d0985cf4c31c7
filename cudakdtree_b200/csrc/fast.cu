// Fast exact kNN / FCP over a left-balanced tree, with reference-order
// fallback.  (float and int32 coordinates, D = 2..4, k <= 128)
//
// Why the answer can be computed in any visiting order.  The reference's
// traversals (traverse-default-stack-based.h, traverse-stack-free.h,
// traverse-cct.h) keep the k smallest (d2, id) keys among the nodes they
// visit, and skip a subtree only when its plane/corner distance is not below
// the current cull distance (the k-th key's d2, which never drops below the
// final k-th d2 X).  A point with d2 < X is therefore always visited, and a
// point with d2 == X can only be skipped once k keys with d2 <= X are
// already in the list.  So whenever exactly k points have d2 <= X (the
// (k+1)-th smallest d2 is strictly greater than X) the reference returns
// exactly those k points, whatever its visiting order.  The same holds for
// FCP (FCPResult, fcp.h:179-207) when the smallest d2 is unique, and of
// several points at it the first in the traversal's preorder is the answer
// (fcp_fast_one, fast_one.cuh, which answers k = 1 as well).  At a tie
// (the (k+1)-th d2 equals X) the reference keeps the tied points of the
// smallest ids among those it visits; a tied point is visited for certain
// when no far-side step on its path has a plane/corner distance as large as
// X (surely_visited, fast_one.cuh), so when that holds for every tied point
// that the smallest (d2, id) keys name, those keys are the answer.
//
// The kernel (fast_one.cuh) lists the k+1 nearest candidates by truncated
// distances, culling so that every point whose truncated distance is at or
// below the (k+1)-th is seen, and keeps the smallest truncated distance that
// it left out.  At the end the listed candidates' exact distances are
// recomputed; the list holds every point at or below the exact k-th distance
// X when everything left out is above X.  Queries where that cannot be
// shown, ties that cannot be settled as above, and points at exactly the
// cut-off radius are queued and re-run by the reference-order kernel of the
// requested method, so every answer is bit-identical to the reference.
//
// Whichever traversal the caller names, subtrees are culled with the
// closest-corner bound of traverse_cct, which is far tighter than the
// split-plane bound on clustered data (the named traversal still answers
// every queued query, in its own order).
//
// What it measured (B200, against a traversal from the root with (distance,
// id) register lists up to k = 32 and local-memory heaps above and for int
// trees, which this replaced): 10M queries on 10M packed points, k = 16
// 16.75 -> 10.2 ms; 1M float3, k = 8 1.09 -> 0.77 ms; 500K queries on 4M
// points, k = 64: record32 14.2 -> 6.2 ms, int3 15.2 -> 3.5 ms.  It is bound
// by the ALU pipe (70% busy; 16 of 32 lanes active): list insertions (a min
// and a max per slot) and per-node bookkeeping under divergence.
#include "common.cuh"
#include "fast.cuh"

namespace ckb {
namespace fast {
template <int SC> int run_warp_scalar(const WarpArgs &wa, int D, cudaStream_t st);
extern template int run_warp_scalar<0>(const WarpArgs &, int, cudaStream_t);
extern template int run_warp_scalar<1>(const WarpArgs &, int, cudaStream_t);
}  // namespace fast

int run_fast(const fast::FastArgs &fa, int scalar, int D, cudaStream_t st)
{
  if (D == 2) return run_fast_dim<2>(fa, scalar, st);
  if (D == 3) return run_fast_dim<3>(fa, scalar, st);
  if (D == 4) return run_fast_dim<4>(fa, scalar, st);
  return CUKD_ERR_UNSUPPORTED;
}

int run_warp(const fast::WarpArgs &wa, int scalar, int D, cudaStream_t st)
{
  return scalar == CUKD_FLOAT32 ? fast::run_warp_scalar<0>(wa, D, st)
                                : fast::run_warp_scalar<1>(wa, D, st);
}

}  // namespace ckb
