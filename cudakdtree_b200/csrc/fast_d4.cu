// The fast kNN / FCP kernel over trees of 4-D points.
#include "fast_kernel.cuh"

namespace ckb {
template int run_fast_dim<4>(const fast::FastArgs &, int, cudaStream_t);
}  // namespace ckb
