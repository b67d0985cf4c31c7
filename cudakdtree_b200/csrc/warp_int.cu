// The warp-per-query kernel over int32 trees.
#include "warp.cuh"

namespace ckb {
namespace fast {
template int run_warp_scalar<1>(const WarpArgs &, int, cudaStream_t);
}  // namespace fast
}  // namespace ckb
