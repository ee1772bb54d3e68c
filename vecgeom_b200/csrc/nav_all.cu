// nav_all.cu -- the navigation kernels of geometries of every shape.
#include "nav_kernels.cuh"

namespace vgb {
template struct NavLaunch<kNavMaskAll>;
}  // namespace vgb
