// Which kernels serve a batch that the block sweeps could hold.
#pragma once
#include "kernels.h"
#include "model.h"

namespace sgdyn {

// Whether the FP64 kernels, which need longer for a call but less per environment of a deep tree,
// are expected to be the faster for n environments (figures at the definitions, bfp_launch.cu).
bool fp64_faster_step(const BfpTree& t, const BfpDepth& d, int ops, int64_t n);
bool fp64_faster_rollout(const BfpTree& t, const BfpDepth& d, int64_t n);
bool fp64_faster_rnea_vjp(const BfpTree& t, const BfpDepth& d, int64_t n);
bool fp64_faster_aba_vjp(const BfpTree& t, const BfpDepth& d, int64_t n);

}  // namespace sgdyn
