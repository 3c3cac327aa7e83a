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

#ifdef __CUDACC__
// Launches a kernel with `smem` bytes of dynamic shared memory.
template <class... P, class... Q>
cudaError_t launch_block(void (*kernel)(P...), dim3 blocks, unsigned threads, size_t smem, cudaStream_t s,
                         const Q&... args) {
  if (smem > 48 * 1024)
    if (cudaError_t e = allow_shared(reinterpret_cast<const void*>(kernel))) return e;
  kernel<<<blocks, threads, smem, s>>>(args...);
  return cudaGetLastError();
}
#endif

}  // namespace sgdyn
