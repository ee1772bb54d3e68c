// batch_round.cu -- FP64 batch kernels: tube, cone, sphere, torus.
#include "batch_launch.cuh"

namespace vgb {
template struct BatchLaunch<TubeOps<double>, TubeP>;
template struct BatchLaunch<ConeOps<double>, ConeP>;
template struct BatchLaunch<SphereOps<double>, SphereP>;
template struct BatchLaunch<TorusOps<double>, TorusP>;
}  // namespace vgb

extern "C" vgb_status vgb_refine_counts(int64_t *certified, int64_t *fallback, int32_t reset) {
  vgb::RefineCounts c = {0, 0};
  cudaError_t e = cudaMemcpyFromSymbol(&c, vgb::g_refine_counts, sizeof(c));
  if (e != cudaSuccess) return vgb::cuda_error(e, "vgb_refine_counts");
  if (certified) *certified = (int64_t)c.certified;
  if (fallback) *fallback = (int64_t)c.fallback;
  if (reset) {
    const vgb::RefineCounts z = {0, 0};
    e = cudaMemcpyToSymbol(vgb::g_refine_counts, &z, sizeof(z));
    if (e != cudaSuccess) return vgb::cuda_error(e, "vgb_refine_counts");
  }
  return VGB_OK;
}
