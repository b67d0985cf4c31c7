// The fast kNN / FCP kernel over trees of 2-D points.
#include "fast_kernel.cuh"

namespace ckb {
template int run_fast_dim<2>(const fast::FastArgs &, int, cudaStream_t);
}  // namespace ckb
