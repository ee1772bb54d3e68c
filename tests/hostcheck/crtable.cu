// crtable.cu -- test infrastructure: compiles only where the device's sin and cos table
// is aligned for the 16-byte words it is read in.
#include "crmath.cuh"

static_assert(alignof(decltype(vgb::crm::kCrmSinCosDev)) >= 16, "read as 16-byte words");
