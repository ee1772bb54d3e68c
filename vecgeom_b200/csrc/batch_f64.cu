// batch_f64.cu -- from a placed volume to the FP64 batch kernels of its shape.
#include "dispatch.h"
#include "geometry.h"

namespace vgb {

// Boolean subtraction: compile-time components for the common pairs, the
// switch over primitive shapes for every other pair.
template <class F> static vgb_status with_boolean_ops(const BooleanP &b, F &&f) {
  const int lt = b.left.type, rt = b.right.type;
  if (lt == VGB_SHAPE_BOX && rt == VGB_SHAPE_TUBE) return f(BoolBoxTube<double>{});
  if (lt == VGB_SHAPE_BOX && rt == VGB_SHAPE_BOX) return f(BoolBoxBox<double>{});
  return f(BoolOps<double>{});
}

static BooleanP boolean_params(const vgb_geometry *g, int32_t unplaced) {
  return bind_params(*static_cast<const BooleanP *>(shape_params(g, unplaced)),
                     shape_params_dev(g, unplaced));
}

vgb_status launch_batch_f64(const vgb_geometry *g, int32_t placed, int op, const BatchIO &io0,
                            cudaStream_t s, int precision) {
  const PlacedRec &pr = g->placed[placed];
  const DXform &X = g->xforms[pr.xform];
  const int type = g->unplaced[pr.unplaced].type;
  const void *prm = shape_params(g, pr.unplaced);
  const BatchIO &io = io0;
  if (type == VGB_SHAPE_BOOLEAN) {
    const BooleanP b = boolean_params(g, pr.unplaced);
    return with_boolean_ops(
        b, [&](auto o) { return BatchLaunch<decltype(o), BooleanP>::batch(b, X, op, io, s, 0, precision); });
  }
  switch (type) {
#define VGB_SHAPE_CASE(TYPE, OPS, P) \
  case TYPE:                         \
    return BatchLaunch<OPS<double>, P>::batch(                                                     \
        bind_params(*static_cast<const P *>(prm), shape_params_dev(g, pr.unplaced)), X, op, io, s, \
        g->unplaced[pr.unplaced].param_len, precision);
    VGB_FOR_EACH_SHAPE(VGB_SHAPE_CASE)
#undef VGB_SHAPE_CASE
  default:
    return set_error(VGB_ENOTSUP, "vgb_batch: shape type %d not supported", type);
  }
}

vgb_status launch_fused_f64(const vgb_geometry *g, int32_t placed, const FusedIO &io,
                            cudaStream_t s) {
  const PlacedRec &pr = g->placed[placed];
  const DXform &X = g->xforms[pr.xform];
  const int type = g->unplaced[pr.unplaced].type;
  const void *prm = shape_params(g, pr.unplaced);
  if (type == VGB_SHAPE_BOOLEAN) {
    const BooleanP b = boolean_params(g, pr.unplaced);
    return with_boolean_ops(b, [&](auto o) { return BatchLaunch<decltype(o), BooleanP>::fused(b, X, io, s, 0); });
  }
  switch (type) {
#define VGB_SHAPE_CASE(TYPE, OPS, P) \
  case TYPE:                         \
    return BatchLaunch<OPS<double>, P>::fused(                                                   \
        bind_params(*static_cast<const P *>(prm), shape_params_dev(g, pr.unplaced)), X, io, s, \
        g->unplaced[pr.unplaced].param_len);
    VGB_FOR_EACH_SHAPE(VGB_SHAPE_CASE)
#undef VGB_SHAPE_CASE
  default:
    return set_error(VGB_ENOTSUP, "vgb_batch_fused: shape type %d not supported", type);
  }
}

}  // namespace vgb
