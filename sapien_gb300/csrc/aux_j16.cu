// Instantiations of the link-Jacobian, Coriolis and IK kernels for trees of up to 16 joints.
#include "bfp_ik.cuh"

namespace sgdyn {

cudaError_t launch_link_jacobian_j16(const DModel* dm, const LinkJacArgs& a, cudaStream_t s) {
  link_jacobian_kernel<16><<<unsigned((a.n + 31) / 32), 32, 0, s>>>(dm, a);
  return cudaGetLastError();
}
cudaError_t launch_coriolis_j16(const DModel* dm, const CoriolisArgs& a, cudaStream_t s) {
  coriolis_kernel<16><<<unsigned((a.n + 31) / 32), 32, 0, s>>>(dm, a);
  return cudaGetLastError();
}
cudaError_t launch_ik_j16(const DModel* dm, const IkArgs& a, bool fixed, cudaStream_t s) {
  return fixed ? launch_bfp_ik<16>(dm, a, s) : launch_ik_kernel(ik_kernel<16>, dm, a, s);
}

}  // namespace sgdyn
