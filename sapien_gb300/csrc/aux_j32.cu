// Instantiations of the link-Jacobian, Coriolis and IK kernels for trees of up to 32 joints.
#include "bfp_ik.cuh"

namespace sgdyn {

cudaError_t launch_link_jacobian_j32(const DModel* dm, const LinkJacArgs& a, cudaStream_t s) {
  link_jacobian_kernel<32><<<unsigned((a.n + 31) / 32), 32, 0, s>>>(dm, a);
  return cudaGetLastError();
}
cudaError_t launch_coriolis_j32(const DModel* dm, const CoriolisArgs& a, cudaStream_t s) {
  coriolis_kernel<32><<<unsigned((a.n + 31) / 32), 32, 0, s>>>(dm, a);
  return cudaGetLastError();
}
cudaError_t launch_ik_j32(const DModel* dm, const IkArgs& a, bool fixed, cudaStream_t s) {
  return fixed ? launch_bfp_ik<32>(dm, a, s) : launch_ik_kernel(ik_kernel<32>, dm, a, s);
}

}  // namespace sgdyn
