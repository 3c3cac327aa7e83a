// Launches of the block-floating-point sweep: environments per block.
#include "bfp_launch.h"
#include "bfp_diff.cuh"

#include <map>
#include <mutex>
#include <set>
#include <utility>

namespace sgdyn {

cudaError_t allow_shared(const void* kernel) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0, most = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({kernel, dev})) return cudaSuccess;
  cudaFuncAttributes own;
  cudaError_t e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&own, kernel);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - int(own.sharedSizeBytes));
  if (e == cudaSuccess) done.insert({kernel, dev});
  return e;
}

namespace {
int multiprocessors() {
  static std::mutex mu;
  static std::map<int, int> count;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  std::lock_guard<std::mutex> lock(mu);
  int& n = count[dev];
  if (n == 0 && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 1;
  return n;
}
}  // namespace

// Environments per block: a power of two from 4 to 32 (whole warps of one joint each at 32, the
// fewest instructions: 262144 9-DoF arms, CRBA + RNEA + forward dynamics, 1115 us against 1204
// with 16 and 1556 with 8), as many as leave room for two blocks per multiprocessor (110 KB
// each), so that one computes while the other waits at a barrier; fewer while the batch has
// less than two blocks per multiprocessor (3001 quadrupeds: 77 us with 8, 83 with 16). 0: not
// even four environments fit a block.
BlkShape blk_shape(const BfpTree& t, bool adjoint, int64_t n) {
  const bfp::BlkLayout L = bfp::blk_layout(t.nj, t.nv, t.nq, t.npairs, adjoint);
  const int nv = t.nv, tree_ints = t.tree_ints;
  int E = 32;
  while (E > 4 && (bfp::blk_bytes(L, tree_ints, E) > 110 * 1024 || E * nv > bfp::kBlkMaxThreads / 2)) E /= 2;
  while (E > 8 && (n + E - 1) / E < 2 * int64_t(multiprocessors())) E /= 2;
  BlkShape s;
  s.smem = bfp::blk_bytes(L, tree_ints, E);
  s.envs = s.smem <= 220 * 1024 && E * nv <= bfp::kBlkMaxThreads ? E : 0;
  s.threads = unsigned((E * nv + 31) / 32 * 32);
  s.blocks = unsigned((n + E - 1) / E);
  return s;
}

#define SG_STEP(E)                                                                                             \
  cudaError_t launch_bfp_step_e##E(const DModel*, int, const StepArgs&, const BfpRows&, const BlkShape&, cudaStream_t); \
  cudaError_t launch_bfp_passive_e##E(const DModel*, const PassiveArgs&, const BlkShape&, cudaStream_t);
SG_STEP(4)
SG_STEP(8)
SG_STEP(16)
SG_STEP(32)
#undef SG_STEP

bool bfp_step_fits(const BfpTree& t) { return t.nv > 0 && blk_shape(t, false, 1).envs > 0; }

cudaError_t launch_bfp_step(const DModel* dm, const BfpTree& t, int ops, const StepArgs& a, cudaStream_t s,
                            const BfpRows& r) {
  if (a.n <= 0) return cudaSuccess;
  if (t.nv <= 0) return cudaErrorNotSupported;
  const BlkShape b = blk_shape(t, false, a.n);
  switch (b.envs) {
    case 4: return launch_bfp_step_e4(dm, ops, a, r, b, s);
    case 8: return launch_bfp_step_e8(dm, ops, a, r, b, s);
    case 16: return launch_bfp_step_e16(dm, ops, a, r, b, s);
    case 32: return launch_bfp_step_e32(dm, ops, a, r, b, s);
    default: return cudaErrorNotSupported;
  }
}

cudaError_t launch_bfp_passive(const DModel* dm, const BfpTree& t, const PassiveArgs& a, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  if (t.nv <= 0) return cudaErrorNotSupported;
  const BlkShape b = blk_shape(t, false, a.n);
  switch (b.envs) {
    case 4: return launch_bfp_passive_e4(dm, a, b, s);
    case 8: return launch_bfp_passive_e8(dm, a, b, s);
    case 16: return launch_bfp_passive_e16(dm, a, b, s);
    case 32: return launch_bfp_passive_e32(dm, a, b, s);
    default: return cudaErrorNotSupported;
  }
}

#define SG_DIFF(E) \
  cudaError_t launch_bfp_diff_e##E(BfpDiff, const DModel*, const RolloutArgs*, const VjpArgs*, const BlkShape&, cudaStream_t);
SG_DIFF(4)
SG_DIFF(8)
SG_DIFF(16)
SG_DIFF(32)
#undef SG_DIFF

int64_t bfp_record_doubles(const BfpTree& t) { return bfp::blk_record_doubles(t.nv, t.nq, t.npairs); }

cudaError_t launch_bfp_diff(BfpDiff what, const DModel* dm, const BfpTree& t, const RolloutArgs* r, const VjpArgs* v,
                            cudaStream_t s) {
  const int64_t n = r ? r->n : v->n;
  if (n <= 0) return cudaSuccess;
  if (t.nv <= 0) return cudaErrorNotSupported;
  // the reverse pass takes fewer environments per block than the sweeps before it, if any: both
  // fit or neither is used
  if (blk_shape(t, true, n).envs == 0) return cudaErrorNotSupported;
  const bool adjoint = what == BfpDiff::reverse || what == BfpDiff::rnea_vjp || what == BfpDiff::aba_vjp;
  BlkShape b = blk_shape(t, adjoint, what == BfpDiff::replay ? n * r->s_cnt : n);
  b.blocks = unsigned((n + b.envs - 1) / b.envs) * unsigned(what == BfpDiff::replay ? r->s_cnt : 1);
  switch (b.envs) {
    case 4: return launch_bfp_diff_e4(what, dm, r, v, b, s);
    case 8: return launch_bfp_diff_e8(what, dm, r, v, b, s);
    case 16: return launch_bfp_diff_e16(what, dm, r, v, b, s);
    default: return launch_bfp_diff_e32(what, dm, r, v, b, s);
  }
}

}  // namespace sgdyn
