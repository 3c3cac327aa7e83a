// The differentiation sweeps with 16 environments per block.
#include "bfp_diff.cuh"
#include "bfp_launch.h"

namespace sgdyn {

cudaError_t launch_bfp_diff_e16(BfpDiff what, const DModel* dm, const RolloutArgs* r, const VjpArgs* v,
                                const BlkShape& b, cudaStream_t s) {
  switch (what) {
    case BfpDiff::rollout: return launch_block(bfp_rollout_kernel<16>, b.blocks, b.threads, b.smem, s, dm, *r);
    case BfpDiff::replay: return launch_block(bfp_replay_kernel<16>, b.blocks, b.threads, b.smem, s, dm, *r);
    case BfpDiff::reverse: return launch_block(bfp_reverse_kernel<16>, b.blocks, b.threads, b.smem, s, dm, *r);
    case BfpDiff::rnea_vjp: return launch_block(bfp_rnea_vjp_kernel<16>, b.blocks, b.threads, b.smem, s, dm, *v);
    case BfpDiff::aba_vjp: return launch_block(bfp_aba_vjp_kernel<16>, b.blocks, b.threads, b.smem, s, dm, *v);
  }
  return cudaErrorInvalidValue;
}

}  // namespace sgdyn
