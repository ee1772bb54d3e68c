// batch_poly.cu -- FP64 batch kernels: polycone, polyhedron.
#include "batch_launch.cuh"

namespace vgb {
template struct BatchLaunch<PolyconeOps<double>, PolyconeP>;
template struct BatchLaunch<PolyhedronOps<double>, PolyhedronP>;
}  // namespace vgb
