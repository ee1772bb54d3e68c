// nav_simple.cu -- the navigation kernels of geometries of boxes, tubes and trds (layered detectors).
#include "nav_kernels.cuh"

namespace vgb {
template struct NavLaunch<kNavMaskBoxTubeTrd>;
}  // namespace vgb
