// batch_boolean.cu -- FP64 batch kernels: booleans (the specialised pairs and any pair).
#include "batch_launch.cuh"

namespace vgb {
template struct BatchLaunch<BoolOps<double>, BooleanP>;
template struct BatchLaunch<BoolBoxTube<double>, BooleanP>;
template struct BatchLaunch<BoolBoxBox<double>, BooleanP>;
}  // namespace vgb
