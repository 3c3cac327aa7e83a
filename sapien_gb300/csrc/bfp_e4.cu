// The block sweep with 4 environments per block.
#include "bfp_launch.h"

namespace sgdyn {

cudaError_t launch_bfp_step_e4(const DModel* dm, int ops, const StepArgs& a, const BlkShape& b, cudaStream_t s) {
  return launch_block(bfp_block_kernel<4>, b.blocks, b.threads, b.smem, s, dm, ops, a);
}

}  // namespace sgdyn
