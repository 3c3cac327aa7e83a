// The block sweeps with 4 environments per block.
#include "bfp_launch.h"

namespace sgdyn {

cudaError_t launch_bfp_step_e4(const DModel* dm, int ops, const StepArgs& a, const BfpRows& r, const BlkShape& b,
                                cudaStream_t s) {
  return launch_block(r.rows ? bfp_block_kernel<4, true> : bfp_block_kernel<4, false>, b.blocks, b.threads, b.smem, s, dm, ops, a, r);
}
cudaError_t launch_bfp_passive_e4(const DModel* dm, const PassiveArgs& a, const BlkShape& b, cudaStream_t s) {
  return launch_block(bfp_passive_kernel<4>, b.blocks, b.threads, b.smem, s, dm, a);
}

}  // namespace sgdyn
