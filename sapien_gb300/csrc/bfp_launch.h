// Launch shape of the block sweeps.
#pragma once
#include "bfp_block.cuh"

namespace sgdyn {

struct BlkShape {
  int envs;  // environments per block, 0: the sweep cannot run
  unsigned threads, blocks;
  size_t smem;
};
BlkShape blk_shape(const BfpTree& t, bool adjoint, int64_t n);

}  // namespace sgdyn
