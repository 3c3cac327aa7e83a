// Launches of the block-floating-point sweep: environments per block.
#include "bfp_launch.h"
#include "bfp_diff.cuh"
#include "route.h"

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
// less than two blocks per multiprocessor. 0: not
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

// The rules below compare the block sweep with the FP64 kernels by what each takes on GB300 (device
// time, chains of 7 to 56 revolute joints, trees of 2 to 8 branches with and without a free flyer, 1024
// to 65536 environments). A block sweep's time grows with n from two blocks per multiprocessor on;
// its price per environment with the tree's depth: levels are walked one after the other, elimination
// takes steps cubic in a chain's length (the FP64 forward dynamics are linear in it), and the
// state's size leaves fewer environments resident. An FP64 kernel takes a time of its own, about
// proportional to the joints, up to a warp per scheduler and grows with n after that.
namespace {
constexpr int64_t kMany = 1 << 20;  // a batch that fills the blocks
double kilobytes(const BfpTree& t) {
  return double(bfp::blk_bytes(bfp::blk_layout(t.nj, t.nv, t.nq, t.npairs, false), 0, 1)) / 1024;
}
bool one_block(const BfpTree& t) { return blk_shape(t, true, kMany).smem > 113 * 1024; }
// microseconds per environment of forward dynamics in a large batch: chains of 20, 24, 40 and 56
// joints 0.020, 0.033, 0.12, 0.35; 35-DoF humanoid 0.029; 9 joints on each of 6 legs 0.069
double solve_cost(const BfpTree& t, const BfpDepth& d) { return 1e-5 * double(d.elimination) + 4e-4 * t.nv; }
double few_cost(const BfpTree& t, const BfpDepth& d) {
  return solve_cost(t, d) * (blk_shape(t, false, kMany).envs <= 4 ? 1.3 : 1.0);
}
}  // namespace

// Measured crossings, environments. Forward dynamics alone: chains of 24, 30, 40, 56: 11000, 3900, 2700,
// 1240 (1474 against 580 us at 4096), humanoid 23000, six legs of 9: 13400; with inverse dynamics
// 13700, 9500, 6100, 2700, none, 17500. The other sets, and all five: 24 to 28000, 16 to 20000, 10 to
// 12000, 5400 to 6100, none, none. Mass matrices without forward dynamics: none below 20000 and 1.25
// times at most.
bool fp64_faster_step(const BfpTree& t, const BfpDepth& d, int ops, int64_t n) {
  const double joints = t.nj - 1;
  if ((ops & OP_CRBA) && !(ops & OP_ABA)) return false;
  if ((ops & OP_ABA) && !(ops & OP_CRBA)) {
    const double c = few_cost(t, d);
    if (ops == OP_ABA) return double(n) * (c - 7.5e-4 * t.nv) > 7 * joints;
    return double(n) * c > 19 * joints && c > 9.5e-4 * t.nv;
  }
  // by latency: levels, times the environments that are not resident
  const double depth = d.levels * kilobytes(t);
  return double(n) * depth > 230e3 * joints && depth > 8.3 * t.nv;
}
// Crossings, forward and reverse pass: chains of 24, 30, 40, 56: 14200, 10000, 2800 to 4200, 1300 to 2800;
// 18-DoF quadruped 15500 to 16200 (32768, 10 steps: 5.9 against 4.1 ms), humanoid 11300 to 12100,
// legs 11400 to 16600; chains up to 16 and the 9-DoF arm none. More than 256 threads of 128 registers
// leave one block per multiprocessor. Up to ten environments per scheduler the FP64 kernels run
// three lanes on each.
bool fp64_faster_rollout(const BfpTree& t, const BfpDepth& d, int64_t n) {
  const double c = few_cost(t, d) * (blk_shape(t, false, kMany).threads > 256 ? 1.8 : 1.0);
  const int64_t schedulers = 4 * int64_t(multiprocessors());
  return double(n) * c > (n <= 10 * schedulers ? 10 : 21) * double(t.nj - 1) && c > 1e-3 * t.nv;
}
// Crossings: chains of 40 to 56 joints 8600 to 9300 (16384: 1.9 to 2.5 against 1.1 to 1.5 ms); else none
// but 1.1 times at 65536 for eight legs of 7.
bool fp64_faster_rnea_vjp(const BfpTree& t, const BfpDepth& d, int64_t n) {
  return n > 9000 && d.levels > 20 && one_block(t);
}
// Crossings: chains of 20, 24, 30, 40, 56: 14000, 14500, 10000, 3600, 3300 (16384 chains of 40: 6.0 against
// 1.6 ms), eight legs of 7: 10500; quadruped and humanoid about 20000 (24576: 800 against 651 us; 32768:
// 2325 against 1654); none for chains up to 11 and the 9-DoF arm (65536: 685 against 926).
bool fp64_faster_aba_vjp(const BfpTree& t, const BfpDepth& d, int64_t n) {
  const double c = 2 * solve_cost(t, d) * (one_block(t) ? 1.5 : 1.0);
  return double(n) * c > 34 * double(t.nj - 1) && c > 1.2e-3 * t.nv;
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
