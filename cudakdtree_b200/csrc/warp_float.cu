// The warp-per-query kernel over float trees.
#include "warp.cuh"

namespace ckb {
namespace fast {
template int run_warp_scalar<0>(const WarpArgs &, int, cudaStream_t);
}  // namespace fast
}  // namespace ckb
