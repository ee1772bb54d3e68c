// batch_simple.cu -- FP64 batch kernels: box, trd, orb, parallelepiped, paraboloid, trapezoid.
#include "batch_launch.cuh"

namespace vgb {
template struct BatchLaunch<BoxOps<double>, BoxP>;
template struct BatchLaunch<TrdOps<double>, TrdP>;
template struct BatchLaunch<OrbOps<double>, OrbP>;
template struct BatchLaunch<ParaOps<double>, ParaP>;
template struct BatchLaunch<ParaboloidOps<double>, ParaboloidP>;
template struct BatchLaunch<TrapezoidOps<double>, TrapezoidP>;
}  // namespace vgb
