// navigator.cu -- navigation kernels and their C ABI (vgb_navpool_*, vgb_nav_*).
//
// One warp per track: the warp's lanes share the daughter loops of the track's
// current volume (navigation.cuh).  The kernels are instantiated for two shape
// sets, the box/tube/trd set of layered detectors and every shape, and the
// launch picks the smallest set that covers the geometry.
#include <cstring>

#include "geometry.h"
#include "nav_launch.h"

using namespace vgb;

struct vgb_navpool {
  int device = -1;
  unsigned char *dev = nullptr;
  int64_t stride = 0;
  int64_t n = 0;
  int32_t max_depth = 0;
};

namespace vgb {
namespace {

NavGeom nav_geom(const vgb_geometry *g) {
  NavGeom G;
  G.params = g->dev.params;
  G.unplaced = g->dev.unplaced;
  G.placed = g->dev.placed;
  G.xforms = g->dev.xforms;
  G.raw = g->dev.raw;
  G.logicals = g->dev.logicals;
  G.daughters = g->dev.daughters;
  G.pl_box = g->dev.pl_box;
  G.ab_box = g->dev.ab_box;
  G.ab_slot = g->dev.ab_slot;
  G.world = g->world;
  G.max_depth = g->max_depth;
  G.vols = g->dev.vols;
  G.slots = g->dev.slots;
  G.slot_box = g->dev.slot_box;
  G.grids = g->dev.grids;
  G.cell_start = g->dev.cell_start;
  G.cell_items = g->dev.cell_items;
  return G;
}

// Runs f(launchers) for the smallest shape set covering the geometry.
template <class F> vgb_status nav_launch(const vgb_geometry *g, F &&f) {
  if ((g->type_mask & ~kNavMaskBoxTubeTrd) == 0)
    f(NavLaunch<kNavMaskBoxTubeTrd>{});
  else
    f(NavLaunch<kNavMaskAll>{});
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "navigation kernel launch");
  return VGB_OK;
}

// Hits an ABBox list holds at most; volumes with more daughters fall back to the
// one-by-one walk when a ray hits more boxes.
constexpr int kAbMaxCap = 6144;

// Hit-list capacity per warp: the most daughters of any volume (so every list
// fits and is ordered as the reference orders it), rounded up to 32 and kept
// within kAbMaxCap; dynamic shared memory of a block for it.
int abbox_cap(const vgb_geometry *g) {
  int cap = (g->max_daughters + 31) / 32 * 32;
  if (cap < 32) cap = 32;
  return cap > kAbMaxCap ? kAbMaxCap : cap;
}

vgb_status check_nav_geometry(const vgb_geometry *g, const char *fn) {
  if (!g) return set_error(VGB_EINVAL, "%s: geometry is NULL", fn);
  if (!g->closed) return set_error(VGB_EINVAL, "%s: geometry is not closed", fn);
  if (g->world < 0) return set_error(VGB_EINVAL, "%s: no world volume set", fn);
  if (g->max_depth > kNavMaxLevels)
    return set_error(VGB_ENOTSUP, "%s: geometry is %d levels deep; at most %d are supported", fn,
                     g->max_depth, kNavMaxLevels);
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_error(e, fn);
  if (dev != g->device)
    return set_error(VGB_EINVAL, "%s: geometry lives on device %d, current device is %d", fn,
                     g->device, dev);
  return VGB_OK;
}

bool is_device_ptr(const void *p) {
  if (!p) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

}  // namespace
}  // namespace vgb

extern "C" {

vgb_status vgb_navpool_create(const vgb_geometry *g, int64_t n, vgb_navpool **pool) {
  if (!pool) return set_error(VGB_EINVAL, "vgb_navpool_create: pool is NULL");
  *pool = nullptr;
  vgb_status s = check_nav_geometry(g, "vgb_navpool_create");
  if (s != VGB_OK) return s;
  if (n < 0) return set_error(VGB_EINVAL, "vgb_navpool_create: n < 0");
  vgb_navpool *p = new vgb_navpool;
  p->device = g->device;
  p->max_depth = g->max_depth;
  p->stride = nav_state_stride(g->max_depth);
  p->n = n;
  const size_t bytes = (size_t)(n > 0 ? n : 1) * (size_t)p->stride;
  cudaError_t e = cudaMalloc((void **)&p->dev, bytes);
  if (e != cudaSuccess) {
    delete p;
    return cuda_error(e, "vgb_navpool_create: cudaMalloc");
  }
  e = cudaMemset(p->dev, 0, bytes);
  if (e != cudaSuccess) {
    cudaFree(p->dev);
    delete p;
    return cuda_error(e, "vgb_navpool_create: cudaMemset");
  }
  *pool = p;
  return VGB_OK;
}

vgb_status vgb_navpool_destroy(vgb_navpool *pool) {
  if (!pool) return VGB_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(pool->device);
  cudaFree(pool->dev);
  cudaSetDevice(prev);
  delete pool;
  return VGB_OK;
}

vgb_status vgb_navpool_info(const vgb_navpool *pool, void **device, int64_t *stride, int64_t *n) {
  if (!pool) return set_error(VGB_EINVAL, "vgb_navpool_info: pool is NULL");
  if (device) *device = pool->dev;
  if (stride) *stride = pool->stride;
  if (n) *n = pool->n;
  return VGB_OK;
}

vgb_status vgb_navpool_upload(vgb_navpool *pool, const void *host, int64_t n, void *stream) {
  if (!pool || (!host && n > 0)) return set_error(VGB_EINVAL, "vgb_navpool_upload: NULL argument");
  if (n < 0 || n > pool->n) return set_error(VGB_EINVAL, "vgb_navpool_upload: n out of range");
  if (n == 0) return VGB_OK;
  cudaError_t e = cudaMemcpyAsync(pool->dev, host, (size_t)(n * pool->stride),
                                  cudaMemcpyHostToDevice, (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_error(e, "vgb_navpool_upload");
  e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_error(e, "vgb_navpool_upload");
  return VGB_OK;
}

vgb_status vgb_navpool_download(const vgb_navpool *pool, void *host, int64_t n, void *stream) {
  if (!pool || (!host && n > 0))
    return set_error(VGB_EINVAL, "vgb_navpool_download: NULL argument");
  if (n < 0 || n > pool->n) return set_error(VGB_EINVAL, "vgb_navpool_download: n out of range");
  if (n == 0) return VGB_OK;
  cudaError_t e = cudaMemcpyAsync(host, pool->dev, (size_t)(n * pool->stride),
                                  cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_error(e, "vgb_navpool_download");
  e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_error(e, "vgb_navpool_download");
  return VGB_OK;
}

vgb_status vgb_nav_locate(const vgb_geometry *g, int64_t n, const double *x, const double *y,
                          const double *z, vgb_navpool *states, void *stream) {
  vgb_status s = check_nav_geometry(g, "vgb_nav_locate");
  if (s != VGB_OK) return s;
  if (!states || n < 0 || n > states->n || states->max_depth != g->max_depth)
    return set_error(VGB_EINVAL, "vgb_nav_locate: pool missing, too small or of another depth");
  if (n == 0) return VGB_OK;
  if (!is_device_ptr(x) || !is_device_ptr(y) || !is_device_ptr(z))
    return set_error(VGB_EINVAL, "vgb_nav_locate: points must be device memory");
  const NavLocateArgs a = {nav_geom(g), n, x, y, z, states->dev, states->stride, g->dev.nav_flags};
  return nav_launch(g, [&](auto k) { k.locate(a, (cudaStream_t)stream); });
}

vgb_status vgb_nav_find_next_boundary_and_step(const vgb_geometry *g, int64_t n, const double *x,
                                               const double *y, const double *z,
                                               const double *dx, const double *dy,
                                               const double *dz, const vgb_navpool *cur,
                                               vgb_navpool *next, const double *pstep,
                                               double *step, double *safety, int32_t precision,
                                               void *stream) {
  const char *fn = "vgb_nav_find_next_boundary_and_step";
  if (precision != VGB_PREC_FP64 && precision != VGB_PREC_FP32_REFINE)
    return set_error(VGB_EINVAL, "%s: unknown precision %d", fn, precision);
  vgb_status s = check_nav_geometry(g, fn);
  if (s != VGB_OK) return s;
  if (!cur || !next || cur == next || n < 0 || n > cur->n || n > next->n ||
      cur->max_depth != g->max_depth || next->max_depth != g->max_depth)
    return set_error(VGB_EINVAL, "%s: need two distinct pools of the geometry's depth", fn);
  if (n == 0) return VGB_OK;
  const void *ptrs[] = {x, y, z, dx, dy, dz, pstep, step};
  for (const void *p : ptrs)
    if (!is_device_ptr(p)) return set_error(VGB_EINVAL, "%s: arrays must be device memory", fn);
  if (safety && !is_device_ptr(safety))
    return set_error(VGB_EINVAL, "%s: safety must be device memory or NULL", fn);
  const NavStepArgs a = {nav_geom(g), n,           x,     y,    z,      dx,      dy,
                         dz,          cur->dev,    next->dev, cur->stride, pstep, step, safety,
                         nullptr,     g->dev.nav_flags};
  const bool screen = precision == VGB_PREC_FP32_REFINE;
  return nav_launch(g, [&](auto k) { k.step(a, screen, (cudaStream_t)stream); });
}

vgb_status vgb_nav_find_next_boundary_and_step_basket(
    const vgb_geometry *g, int64_t n, const double *x, const double *y, const double *z,
    const double *dx, const double *dy, const double *dz, const vgb_navpool *cur,
    vgb_navpool *next, const double *pstep, double *distance, double *safety, int32_t *nextnode,
    void *stream) {
  const char *fn = "vgb_nav_find_next_boundary_and_step_basket";
  vgb_status s = check_nav_geometry(g, fn);
  if (s != VGB_OK) return s;
  if (!cur || !next || cur == next || n < 0 || n > cur->n || n > next->n ||
      cur->max_depth != g->max_depth || next->max_depth != g->max_depth)
    return set_error(VGB_EINVAL, "%s: need two distinct pools of the geometry's depth", fn);
  if (n == 0) return VGB_OK;
  const void *ptrs[] = {x, y, z, dx, dy, dz, pstep, distance};
  for (const void *p : ptrs)
    if (!is_device_ptr(p)) return set_error(VGB_EINVAL, "%s: arrays must be device memory", fn);
  if ((safety && !is_device_ptr(safety)) || (nextnode && !is_device_ptr(nextnode)))
    return set_error(VGB_EINVAL, "%s: safety / nextnode must be device memory or NULL", fn);
  const NavStepArgs a = {nav_geom(g), n,           x,     y,    z,      dx,      dy,
                         dz,          cur->dev,    next->dev, cur->stride, pstep, distance, safety,
                         nextnode,     g->dev.nav_flags};
  return nav_launch(g, [&](auto k) { k.basket(a, (cudaStream_t)stream); });
}

vgb_status vgb_nav_trace(const vgb_geometry *g, int64_t n, const double *x, const double *y,
                         const double *z, const double *dx, const double *dy, const double *dz,
                         double pstep, int32_t max_steps, int32_t *next_ids, double *steps,
                         double *safeties, int32_t *nsteps, int32_t precision, void *stream) {
  const char *fn = "vgb_nav_trace";
  if (precision != VGB_PREC_FP64 && precision != VGB_PREC_FP32_REFINE)
    return set_error(VGB_EINVAL, "%s: unknown precision %d", fn, precision);
  vgb_status s = check_nav_geometry(g, fn);
  if (s != VGB_OK) return s;
  if (n < 0 || max_steps < 0) return set_error(VGB_EINVAL, "%s: n or max_steps < 0", fn);
  if (n == 0) return VGB_OK;
  const void *ptrs[] = {x, y, z, dx, dy, dz, nsteps};
  for (const void *p : ptrs)
    if (!is_device_ptr(p)) return set_error(VGB_EINVAL, "%s: arrays must be device memory", fn);
  const void *opt[] = {next_ids, steps, safeties};
  for (const void *p : opt)
    if (p && !is_device_ptr(p))
      return set_error(VGB_EINVAL, "%s: records must be device memory or NULL", fn);
  const NavTraceArgs a = {nav_geom(g), n,        x,     y,        z,      dx,    dy, dz,
                          pstep,       max_steps, next_ids, steps, safeties, nsteps,
                          g->dev.nav_flags};
  const bool screen = precision == VGB_PREC_FP32_REFINE;
  return nav_launch(g, [&](auto k) { k.trace(a, screen, (cudaStream_t)stream); });
}

vgb_status vgb_abbox_nav_find_next_boundary_and_step(const vgb_geometry *g, int64_t n,
                                                     const double *x, const double *y,
                                                     const double *z, const double *dx,
                                                     const double *dy, const double *dz,
                                                     const vgb_navpool *cur, vgb_navpool *next,
                                                     const double *pstep, double *step,
                                                     double *safety, void *stream) {
  const char *fn = "vgb_abbox_nav_find_next_boundary_and_step";
  vgb_status s = check_nav_geometry(g, fn);
  if (s != VGB_OK) return s;
  if (!g->abbox_ok)
    return set_error(VGB_ENOTSUP, "%s: a volume's shape has no Extent (parallelepiped), so no "
                     "aligned box", fn);
  if (!cur || !next || cur == next || n < 0 || n > cur->n || n > next->n ||
      cur->max_depth != g->max_depth || next->max_depth != g->max_depth)
    return set_error(VGB_EINVAL, "%s: need two distinct pools of the geometry's depth", fn);
  if (n == 0) return VGB_OK;
  const void *ptrs[] = {x, y, z, dx, dy, dz, pstep, step};
  for (const void *p : ptrs)
    if (!is_device_ptr(p)) return set_error(VGB_EINVAL, "%s: arrays must be device memory", fn);
  if (safety && !is_device_ptr(safety))
    return set_error(VGB_EINVAL, "%s: safety must be device memory or NULL", fn);
  const int cap = abbox_cap(g);
  const NavStepArgs a = {nav_geom(g), n,           x,     y,    z,      dx,      dy,
                         dz,          cur->dev,    next->dev, cur->stride, pstep, step, safety,
                         nullptr,     g->dev.nav_flags};
  return nav_launch(g, [&](auto k) { k.abbox_step(a, (int32_t)cap, (cudaStream_t)stream); });
}

vgb_status vgb_abbox_nav_trace(const vgb_geometry *g, int64_t n, const double *x, const double *y,
                               const double *z, const double *dx, const double *dy,
                               const double *dz, double pstep, int32_t max_steps,
                               int32_t *next_ids, double *steps, double *safeties,
                               int32_t *nsteps, void *stream) {
  const char *fn = "vgb_abbox_nav_trace";
  vgb_status s = check_nav_geometry(g, fn);
  if (s != VGB_OK) return s;
  if (!g->abbox_ok)
    return set_error(VGB_ENOTSUP, "%s: a volume's shape has no Extent (parallelepiped), so no "
                     "aligned box", fn);
  if (n < 0 || max_steps < 0) return set_error(VGB_EINVAL, "%s: n or max_steps < 0", fn);
  if (n == 0) return VGB_OK;
  const void *ptrs[] = {x, y, z, dx, dy, dz, nsteps};
  for (const void *p : ptrs)
    if (!is_device_ptr(p)) return set_error(VGB_EINVAL, "%s: arrays must be device memory", fn);
  const void *opt[] = {next_ids, steps, safeties};
  for (const void *p : opt)
    if (p && !is_device_ptr(p))
      return set_error(VGB_EINVAL, "%s: records must be device memory or NULL", fn);
  const int cap = abbox_cap(g);
  const NavTraceArgs a = {nav_geom(g), n,        x,     y,        z,      dx,    dy, dz,
                          pstep,       max_steps, next_ids, steps, safeties, nsteps,
                          g->dev.nav_flags};
  return nav_launch(g, [&](auto k) { k.abbox_trace(a, (int32_t)cap, (cudaStream_t)stream); });
}

vgb_status vgb_nav_error_flags(const vgb_geometry *g, uint32_t *flags) {
  if (!g || !flags) return set_error(VGB_EINVAL, "vgb_nav_error_flags: NULL argument");
  if (!g->closed) return set_error(VGB_EINVAL, "vgb_nav_error_flags: geometry is not closed");
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return cuda_error(e, "vgb_nav_error_flags");
  e = cudaMemcpy(flags, g->dev.nav_flags, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_error(e, "vgb_nav_error_flags");
  e = cudaMemset(g->dev.nav_flags, 0, sizeof(uint32_t));
  if (e != cudaSuccess) return cuda_error(e, "vgb_nav_error_flags");
  return VGB_OK;
}

}  // extern "C"
