// nav_launch.h -- launchers of the navigation kernels, one set per shape set
// (defined in nav_kernels.cuh, instantiated in nav_simple.cu and nav_all.cu).
#pragma once
#include "navigation.cuh"

namespace vgb {

struct NavLocateArgs {
  NavGeom G;
  int64_t n;
  const double *x, *y, *z;
  unsigned char *states;
  int64_t stride;
  uint32_t *flags;
};
struct NavStepArgs {
  NavGeom G;
  int64_t n;
  const double *x, *y, *z, *dx, *dy, *dz;
  const unsigned char *cur;
  unsigned char *next;
  int64_t stride;
  const double *pstep;
  double *step, *safety;
  int32_t *node;  // basket form only
  uint32_t *flags;
};
struct NavTraceArgs {
  NavGeom G;
  int64_t n;
  const double *x, *y, *z, *dx, *dy, *dz;
  double pstep;
  int32_t max_steps;
  int32_t *next_ids;
  double *steps, *safeties;
  int32_t *nsteps;
  uint32_t *flags;
};

template <uint32_t kMask> struct NavLaunch {
  static void locate(const NavLocateArgs &a, cudaStream_t s);
  static void step(const NavStepArgs &a, bool screen, cudaStream_t s);
  static void basket(const NavStepArgs &a, cudaStream_t s);
  static void trace(const NavTraceArgs &a, bool screen, cudaStream_t s);
  static void abbox_step(const NavStepArgs &a, int32_t cap, cudaStream_t s);
  static void abbox_trace(const NavTraceArgs &a, int32_t cap, cudaStream_t s);
};

extern template struct NavLaunch<kNavMaskBoxTubeTrd>;
extern template struct NavLaunch<kNavMaskAll>;

}  // namespace vgb
