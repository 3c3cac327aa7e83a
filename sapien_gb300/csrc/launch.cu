// Bucket dispatch for the fused sweep.
#include "kernels.h"

namespace sgdyn {

cudaError_t launch_step_j16(const DModel*, int, const StepArgs&, cudaStream_t);
cudaError_t launch_step_j32(const DModel*, int, const StepArgs&, cudaStream_t);
cudaError_t launch_step_j64(const DModel*, int, const StepArgs&, cudaStream_t);
cudaError_t launch_step_team_j16(const DModel*, const int*, int, int, const StepArgs&, cudaStream_t);
cudaError_t launch_step_team_j32(const DModel*, const int*, int, int, const StepArgs&, cudaStream_t);
cudaError_t launch_step_team_j64(const DModel*, const int*, int, int, const StepArgs&, cudaStream_t);

cudaError_t launch_step_team(const DModel* dm, int nj, const int* team, int lanes, int ops, const StepArgs& a,
                             cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  switch (stash_bucket(nj)) {
    case 16: return launch_step_team_j16(dm, team, lanes, ops, a, s);
    case 32: return launch_step_team_j32(dm, team, lanes, ops, a, s);
    case 64: return launch_step_team_j64(dm, team, lanes, ops, a, s);
    default: return cudaErrorInvalidValue;
  }
}

int stash_bucket(int nj) { return nj <= 16 ? 16 : nj <= 32 ? 32 : nj <= 64 ? 64 : 0; }

cudaError_t launch_step(const DModel* dm, int nj, int ops, const StepArgs& a, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  switch (stash_bucket(nj)) {
    case 16: return launch_step_j16(dm, ops, a, s);
    case 32: return launch_step_j32(dm, ops, a, s);
    case 64: return launch_step_j64(dm, ops, a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sgdyn

#include "aux_kernels.cuh"

namespace sgdyn {

#define SG_DECL(J)                                                                    \
  cudaError_t launch_link_jacobian_j##J(const DModel*, const LinkJacArgs&, cudaStream_t); \
  cudaError_t launch_coriolis_j##J(const DModel*, const CoriolisArgs&, cudaStream_t);    \
  cudaError_t launch_ik_j##J(const DModel*, const IkArgs&, bool, cudaStream_t);
SG_DECL(16)
SG_DECL(32)
SG_DECL(64)
#undef SG_DECL

cudaError_t launch_link_jacobian(const DModel* dm, int nj, const LinkJacArgs& a, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  switch (stash_bucket(nj)) {
    case 16: return launch_link_jacobian_j16(dm, a, s);
    case 32: return launch_link_jacobian_j32(dm, a, s);
    case 64: return launch_link_jacobian_j64(dm, a, s);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t launch_coriolis(const DModel* dm, int nj, const CoriolisArgs& a, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  switch (stash_bucket(nj)) {
    case 16: return launch_coriolis_j16(dm, a, s);
    case 32: return launch_coriolis_j32(dm, a, s);
    case 64: return launch_coriolis_j64(dm, a, s);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t launch_ik(const DModel* dm, int nj, const IkArgs& a, bool fixed, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  switch (stash_bucket(nj)) {
    case 16: return launch_ik_j16(dm, a, fixed, s);
    case 32: return launch_ik_j32(dm, a, fixed, s);
    case 64: return launch_ik_j64(dm, a, fixed, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sgdyn

#include "diff_kernels.cuh"

namespace sgdyn {
namespace {

// Tangent gradients to coordinate gradients, a thread per environment and joint. The chart of a
// free flyer: eps = (R^T dp, 2 vec(quat^-1 dquat)). Bound by its launch; it stands for ~45 small
// tensor operations that took 0.8 ms (values and gradients of both dynamics, 4096 18-DoF
// quadrupeds: 2.27 -> 0.66 ms).
__global__ void __launch_bounds__(128) tangent_to_coordinate_kernel(const DModel* __restrict__ model, int64_t n,
                                                                    const double* __restrict__ q,
                                                                    const double* __restrict__ g,
                                                                    double* __restrict__ out) {
  const int joints = model->nj - 1, nq = model->nq_ext, nv = model->nv;
  const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n * joints) return;
  const int64_t e = k / joints;
  const DJoint& J = model_joints(model)[1 + int(k - e * joints)];
  const double* ge = g + e * nv + J.vcol;
  double* o = out + e * nq + J.qcol;
  if (J.kind != JK_FREEFLYER) {
    o[0] = ge[0];
    return;
  }
  const double* qe = q + e * nq + J.qcol;
  const V3 v = mk(qe[3], qe[4], qe[5]), w = mk(ge[3], ge[4], ge[5]);
  const V3 p = mul(quat_to_R(v.x, v.y, v.z, qe[6]), mk(ge[0], ge[1], ge[2])), t = cross(v, w);
  o[0] = p.x; o[1] = p.y; o[2] = p.z;
  o[3] = 2 * fma(qe[6], w.x, t.x);
  o[4] = 2 * fma(qe[6], w.y, t.y);
  o[5] = 2 * fma(qe[6], w.z, t.z);
  o[6] = -2 * dot(v, w);
}

}  // namespace

cudaError_t launch_tangent_to_coordinate(const DModel* dm, int nj, int64_t n, const double* q, const double* g,
                                         double* out, cudaStream_t s) {
  if (n <= 0 || nj < 2) return cudaSuccess;
  tangent_to_coordinate_kernel<<<unsigned((n * (nj - 1) + 127) / 128), 128, 0, s>>>(dm, n, q, g, out);
  return cudaGetLastError();
}

}  // namespace sgdyn

namespace sgdyn {

#define SG_DISPATCH(kernel, Args)                                                        \
  cudaError_t launch_##kernel##_j16(const DModel*, const Args&, cudaStream_t);            \
  cudaError_t launch_##kernel##_j32(const DModel*, const Args&, cudaStream_t);            \
  cudaError_t launch_##kernel##_j64(const DModel*, const Args&, cudaStream_t);            \
  cudaError_t launch_##kernel(const DModel* dm, int nj, const Args& a, cudaStream_t s) {  \
    if (a.n <= 0) return cudaSuccess;                                                    \
    switch (stash_bucket(nj)) {                                                          \
      case 16: return launch_##kernel##_j16(dm, a, s);                                   \
      case 32: return launch_##kernel##_j32(dm, a, s);                                   \
      case 64: return launch_##kernel##_j64(dm, a, s);                                   \
      default: return cudaErrorInvalidValue;                                             \
    }                                                                                    \
  }
SG_DISPATCH(rnea_vjp, VjpArgs)
SG_DISPATCH(aba_vjp, VjpArgs)
SG_DISPATCH(fk_vjp, FkVjpArgs)
SG_DISPATCH(rnea_derivatives, DerivArgs)
SG_DISPATCH(aba_derivatives, DerivArgs)
SG_DISPATCH(rollout_forward, RolloutArgs)
SG_DISPATCH(rollout_forward3, RolloutArgs)
SG_DISPATCH(rollout_recompute, RolloutArgs)
SG_DISPATCH(rollout_reverse, RolloutArgs)
SG_DISPATCH(rollout_reverse3, RolloutArgs)
SG_DISPATCH(aba3, StepArgs)
#undef SG_DISPATCH

int64_t rollout_scratch_doubles_per_env(int nj, int nq, int nv, int K) {
  return int64_t(K) * stash_doubles_per_step(nj, nq, nv);
}

}  // namespace sgdyn
