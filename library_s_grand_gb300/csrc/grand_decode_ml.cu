// grand_decode_ml.cu -- the chunk and decode kernels built with the ML (cost-ordered)
// search paths, for batches with an ML code.
#include "grand_decode.cuh"
#include "grand_front.cuh"
#include "grand_host.h"

namespace grand {

#ifndef GRAND_HOST_EMULATION
cudaError_t launch_decode_ml(const DevBatch &b, int grid, cudaStream_t s) {
  return launch_kernels<true>(b, grid, s);
}

cudaError_t decode_occupancy_ml(int *blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, decode_kernel<true>,
                                                       kDecodeWarps * 32, 0);
}
#endif

}  // namespace grand
