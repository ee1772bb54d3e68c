// nav_kernels.cuh -- the navigation kernels, over the lanes that serve one track
// and the shape set of the geometry.  Each shape set is compiled in a file of its
// own (nav_simple.cu: box/tube/trd, nav_all.cu: every shape), behind the launchers
// of nav_launch.h.
#pragma once
#include <type_traits>

#include "abbox.cuh"
#include "nav_engine.cuh"
#include "nav_launch.h"

namespace vgb {

constexpr int kNavBlock = 128;
constexpr int kNavWarps = kNavBlock / 32;

// first track and track stride of the calling lanes
template <class L> VGB_D int64_t nav_first() {
  return ((int64_t)blockIdx.x * kNavBlock + threadIdx.x) / L::N;
}
template <class L> VGB_D int64_t nav_stride() { return (int64_t)gridDim.x * (kNavBlock / L::N); }

VGB_D void nav_raise(uint32_t *flags, uint32_t bits) { atomicOr(flags, bits); }

template <class L, uint32_t kMask>
__global__ void __launch_bounds__(kNavBlock) k_nav_locate(const NavGeom G, int64_t n,
                                                          const double *x, const double *y,
                                                          const double *z, unsigned char *states,
                                                          int64_t stride, uint32_t *flags) {
  using Nav = Navigator<L, kMask>;
  for (int64_t i = nav_first<L>(); i < n; i += nav_stride<L>()) {
    NavPath s;
    const V3<double> p = {x[i], y[i], z[i]};
    const bool ok = Nav::locate_from_world(G, s, p);
    if (L::lane() == 0) {
      if (!ok) {
        nav_raise(flags, VGB_NAV_ERR_DEPTH);
        s.level = 0;
      }
      nav_store(s, NavStateRef{states + i * stride}, G.max_depth);
    }
  }
}

template <class L, uint32_t kMask, bool kScreen>
__global__ void __launch_bounds__(kNavBlock)
    k_nav_step(const NavGeom G, int64_t n, const double *x, const double *y, const double *z,
               const double *dx, const double *dy, const double *dz, const unsigned char *cur,
               unsigned char *next, int64_t stride, const double *pstep, double *step_out,
               double *safety_out, uint32_t *flags) {
  using Nav = Navigator<L, kMask, kScreen>;
  for (int64_t i = nav_first<L>(); i < n; i += nav_stride<L>()) {
    NavPath c, nx;
    nav_load(c, NavStateRef{const_cast<unsigned char *>(cur) + i * stride});
    const V3<double> p = {x[i], y[i], z[i]};
    const V3<double> d = {dx[i], dy[i], dz[i]};
    double st = 0., sf = 0.;
    bool ok = true;
    nx = c;
    if (c.level > 0) {
      const DXform m = nav_top_matrix(G, c);
      const V3<double> lp = xf_point(m, p);
      const V3<double> ld = xf_dir(m, d);
      if (safety_out)
        ok = Nav::safety_and_step(G, c, nx, lp, ld, pstep[i], sf, st);
      else
        ok = Nav::step(G, c, nx, lp, ld, pstep[i], st);
    }
    if (L::lane() == 0) {
      if (!ok) nav_raise(flags, VGB_NAV_ERR_DEPTH);
      nav_store(nx, NavStateRef{next + i * stride}, G.max_depth);
      step_out[i] = st;
      if (safety_out) safety_out[i] = sf;
    }
  }
}

// basket form of the step (SimpleNavigator.h:637-743) with GetSafeties (:599-632)
template <class L, uint32_t kMask>
__global__ void __launch_bounds__(kNavBlock)
    k_nav_basket(const NavGeom G, int64_t n, const double *x, const double *y, const double *z,
                 const double *dx, const double *dy, const double *dz, const unsigned char *cur,
                 unsigned char *next, int64_t stride, const double *pstep, double *dist_out,
                 double *safety_out, int32_t *node_out, uint32_t *flags) {
  using Nav = Navigator<L, kMask>;
  for (int64_t i = nav_first<L>(); i < n; i += nav_stride<L>()) {
    NavPath c, nx;
    nav_load(c, NavStateRef{const_cast<unsigned char *>(cur) + i * stride});
    const V3<double> p = {x[i], y[i], z[i]};
    const V3<double> d = {dx[i], dy[i], dz[i]};
    double st = 0., sf = 0.;
    int32_t node = -2;
    bool ok = true;
    nx = c;
    if (c.level > 0) {
      const DXform m = nav_top_matrix(G, c);
      const V3<double> lp = xf_point(m, p);
      const V3<double> ld = xf_dir(m, d);
      ok = Nav::safety_and_step_basket(G, c, nx, lp, ld, pstep[i], safety_out != nullptr, sf, st,
                                       node);
    }
    if (L::lane() == 0) {
      if (!ok) nav_raise(flags, VGB_NAV_ERR_DEPTH);
      nav_store(nx, NavStateRef{next + i * stride}, G.max_depth);
      dist_out[i] = st;
      if (safety_out) safety_out[i] = sf;
      if (node_out) node_out[i] = node;
    }
  }
}

template <class L, uint32_t kMask, bool kScreen>
__global__ void __launch_bounds__(kNavBlock)
    k_nav_trace(const NavGeom G, int64_t n, const double *x, const double *y, const double *z,
                const double *dx, const double *dy, const double *dz, double pstep,
                int32_t max_steps, int32_t *next_ids, double *steps, double *safeties,
                int32_t *nsteps, uint32_t *flags) {
  using Nav = Navigator<L, kMask, kScreen>;
  const bool lane0 = L::lane() == 0;
  for (int64_t i = nav_first<L>(); i < n; i += nav_stride<L>()) {
    V3<double> p = {x[i], y[i], z[i]};
    const V3<double> d = {dx[i], dy[i], dz[i]};
    NavPath cur;
    bool ok = Nav::locate_from_world(G, cur, p);
    int32_t k = 0;
    while (ok && cur.level > 0 && k < max_steps) {
      const DXform m = nav_top_matrix(G, cur);
      const V3<double> lp = xf_point(m, p);
      const V3<double> ld = xf_dir(m, d);
      double sf = 0., st = 0.;
      ok = Nav::safety_and_step(G, cur, cur, lp, ld, pstep, sf, st);
      if (!ok) break;
      if (lane0) {
        const int64_t r = i * (int64_t)max_steps + k;
        if (next_ids) next_ids[r] = cur.top();
        if (steps) steps[r] = st;
        if (safeties) safeties[r] = sf;
      }
      // the client advances to the boundary: p + d * step
      p = {p.x + d.x * st, p.y + d.y * st, p.z + d.z * st};
      ++k;
    }
    if (lane0) {
      if (!ok) nav_raise(flags, VGB_NAV_ERR_DEPTH);
      nsteps[i] = ok ? k : -1;
    }
  }
}

// ABBoxNavigator kernels: the same loops with the box-culled step; each warp
// keeps its hit list in dynamic shared memory (cap hits, and the rank-sorted
// copy of a list of up to 16 beside them).  Volumes with more than kAbMaxCap
// daughters fall back to the one-by-one walk when a ray hits more boxes.
extern __shared__ AbCand vgb_ab_lists[];

template <uint32_t kMask>
__global__ void __launch_bounds__(kNavBlock)
    k_abbox_step(const NavGeom G, int32_t cap, int64_t n, const double *x, const double *y, const double *z,
                 const double *dx, const double *dy, const double *dz, const unsigned char *cur,
                 unsigned char *next, int64_t stride, const double *pstep, double *step_out,
                 double *safety_out, uint32_t *flags) {
  using Nav = ABBoxNavigator<WarpLanes, kMask>;
  AbCand *buf = vgb_ab_lists + (threadIdx.x / 32) * (cap + kAbSortThreshold);
  const int64_t warps = (int64_t)gridDim.x * kNavWarps;
  for (int64_t i = (int64_t)blockIdx.x * kNavWarps + threadIdx.x / 32; i < n; i += warps) {
    NavPath c, nx;
    nav_load(c, NavStateRef{const_cast<unsigned char *>(cur) + i * stride});
    const V3<double> p = {x[i], y[i], z[i]};
    const V3<double> d = {dx[i], dy[i], dz[i]};
    double st = 0., sf = 0.;
    bool ok = true;
    nx = c;
    if (c.level > 0) {
      const DXform m = nav_top_matrix(G, c);
      const V3<double> lp = xf_point(m, p);
      const V3<double> ld = xf_dir(m, d);
      if (safety_out) sf = Nav::safety(G, c, lp);
      ok = Nav::step(G, c, nx, lp, ld, pstep[i], st, buf, cap);
    }
    if (WarpLanes::lane() == 0) {
      if (!ok) nav_raise(flags, VGB_NAV_ERR_DEPTH);
      nav_store(nx, NavStateRef{next + i * stride}, G.max_depth);
      step_out[i] = st;
      if (safety_out) safety_out[i] = sf;
    }
  }
}

template <uint32_t kMask>
__global__ void __launch_bounds__(kNavBlock)
    k_abbox_trace(const NavGeom G, int32_t cap, int64_t n, const double *x, const double *y, const double *z,
                  const double *dx, const double *dy, const double *dz, double pstep,
                  int32_t max_steps, int32_t *next_ids, double *steps, double *safeties,
                  int32_t *nsteps, uint32_t *flags) {
  using Nav = ABBoxNavigator<WarpLanes, kMask>;
  AbCand *buf = vgb_ab_lists + (threadIdx.x / 32) * (cap + kAbSortThreshold);
  const int64_t warps = (int64_t)gridDim.x * kNavWarps;
  const bool lane0 = WarpLanes::lane() == 0;
  for (int64_t i = (int64_t)blockIdx.x * kNavWarps + threadIdx.x / 32; i < n; i += warps) {
    V3<double> p = {x[i], y[i], z[i]};
    const V3<double> d = {dx[i], dy[i], dz[i]};
    NavPath cur;
    bool ok = Navigator<WarpLanes, kMask>::locate_from_world(G, cur, p);
    int32_t k = 0;
    while (ok && cur.level > 0 && k < max_steps) {
      const DXform m = nav_top_matrix(G, cur);
      const V3<double> lp = xf_point(m, p);
      const V3<double> ld = xf_dir(m, d);
      const double sf = Nav::safety(G, cur, lp);
      double st = 0.;
      ok = Nav::step(G, cur, cur, lp, ld, pstep, st, buf, cap);
      if (!ok) break;
      if (lane0) {
        const int64_t r = i * (int64_t)max_steps + k;
        if (next_ids) next_ids[r] = cur.top();
        if (steps) steps[r] = st;
        if (safeties) safeties[r] = sf;
      }
      p = {p.x + d.x * st, p.y + d.y * st, p.z + d.z * st};
      ++k;
    }
    if (lane0) {
      if (!ok) nav_raise(flags, VGB_NAV_ERR_DEPTH);
      nsteps[i] = ok ? k : -1;
    }
  }
}


// ---------------------------------------------------------------------------
// the same calls with a thread per track (nav_engine.cuh)
// ---------------------------------------------------------------------------
// 128 registers a thread (four blocks an SM).  65,536 detector tracks, ncu: 22 of 32
// lanes active (8 without the regrouping), 160 warp instructions a track's step; the
// block's barrier, dependent loads and instruction fetch (two forms of every step)
// are what a warp waits for.
// The hit list of L's lanes: a thread's own (its volumes have at most kWideDaughters
// daughters), or the warp's part of the block's dynamic shared memory.
template <class L> struct AbList {
  AbCand own[kWideDaughters + kAbSortThreshold];
  VGB_D AbCand *get(int32_t) { return own; }
  static VGB_D int32_t cap(int32_t) { return kWideDaughters; }
};
template <> struct AbList<WarpLanes> {
  VGB_D AbCand *get(int32_t cap) {
    return vgb_ab_lists + (threadIdx.x / 32) * (cap + kAbSortThreshold);
  }
  static VGB_D int32_t cap(int32_t c) { return c; }
};
// GetSafety and the ABBox step of one track
template <class L, uint32_t kMask>
VGB_D bool abbox_safety_and_step(const NavGeom &G, NavPath &path, const V3<double> &lp,
                                 const V3<double> &ld, double pstep, bool want_s, int32_t cap,
                                 double &sf, double &st) {
  using Nav = ABBoxNavigator<L, kMask>;
  AbList<L> list;
  if (want_s) sf = Nav::safety(G, path, lp);
  return Nav::step(G, path, path, lp, ld, pstep, st, list.get(cap), list.cap(cap));
}

// kAbbox: the ABBoxNavigator's step, with cap hits a warp
template <uint32_t kMask, bool kAbbox> struct TraceClient {
  NavTraceArgs a;
  int32_t cap;
  VGB_D bool load(int64_t i, NavTrack &t) const {
    t.p = {a.x[i], a.y[i], a.z[i]};
    t.d = {a.dx[i], a.dy[i], a.dz[i]};
    t.path.level = kLevelLocate;
    t.path.boundary = false;
    t.k = t.left = 0;
    t.hash = 0;
    return true;
  }
  template <class L> VGB_D bool finish(int64_t i, const NavTrack &t, bool ok) const {
    if (L::lane() == 0) {
      if (!ok) nav_raise(a.flags, VGB_NAV_ERR_DEPTH);
      a.nsteps[i] = ok ? t.k : -1;
    }
    return false;
  }
  template <class L> VGB_D bool step(const NavGeom &G, int64_t i, NavTrack &t) const {
    using Nav = Navigator<L, kMask>;
    if (t.path.level < 0) {
      const bool ok = Nav::locate_from_world(G, t.path, t.p);
      if (!ok || t.path.level == 0 || a.max_steps == 0) return finish<L>(i, t, ok);
      return true;
    }
    const DXform m = nav_top_matrix(G, t.path);
    const V3<double> lp = xf_point(m, t.p), ld = xf_dir(m, t.d);
    double sf = 0., st = 0.;
    bool ok;
    if constexpr (kAbbox)
      ok = abbox_safety_and_step<L, kMask>(G, t.path, lp, ld, a.pstep, true, cap, sf, st);
    else
      ok = Nav::safety_and_step(G, t.path, t.path, lp, ld, a.pstep, sf, st);
    if (!ok) return finish<L>(i, t, false);
    if (L::lane() == 0) {
      const int64_t r = i * (int64_t)a.max_steps + t.k;
      if (a.next_ids) a.next_ids[r] = t.path.top();
      if (a.steps) a.steps[r] = st;
      if (a.safeties) a.safeties[r] = sf;
    }
    t.p = {t.p.x + t.d.x * st, t.p.y + t.d.y * st, t.p.z + t.d.z * st};
    ++t.k;
    if (t.path.level == 0 || t.k >= a.max_steps) return finish<L>(i, t, true);
    return true;
  }
};

enum class StepForm { kSimple, kBasket, kAbbox };
template <uint32_t kMask, StepForm kForm> struct StepClient {
  static constexpr bool kBasket = kForm == StepForm::kBasket;
  NavStepArgs a;
  int32_t cap;
  VGB_D void put(int64_t i, const NavTrack &t, double st, double sf, int32_t node) const {
    nav_store(t.path, NavStateRef{a.next + i * a.stride}, a.G.max_depth);
    a.step[i] = st;
    if (a.safety) a.safety[i] = sf;
    if (kBasket && a.node) a.node[i] = node;
  }
  VGB_D bool load(int64_t i, NavTrack &t) const {
    nav_load(t.path, NavStateRef{const_cast<unsigned char *>(a.cur) + i * a.stride});
    t.p = {a.x[i], a.y[i], a.z[i]};
    t.d = {a.dx[i], a.dy[i], a.dz[i]};
    t.k = t.left = 0;
    t.hash = 0;
    if (t.path.level > 0) return true;
    put(i, t, 0., 0., -2);
    return false;
  }
  template <class L> VGB_D bool step(const NavGeom &G, int64_t i, NavTrack &t) const {
    using Nav = Navigator<L, kMask>;
    const DXform m = nav_top_matrix(G, t.path);
    const V3<double> lp = xf_point(m, t.p), ld = xf_dir(m, t.d);
    double sf = 0., st = 0.;
    int32_t node = -2;
    bool ok;
    if constexpr (kBasket) {
      ok = Nav::safety_and_step_basket(G, t.path, t.path, lp, ld, a.pstep[i], a.safety != nullptr,
                                       sf, st, node);
    } else if constexpr (kForm == StepForm::kAbbox) {
      ok = abbox_safety_and_step<L, kMask>(G, t.path, lp, ld, a.pstep[i], a.safety != nullptr, cap,
                                           sf, st);
    } else if (a.safety) {
      ok = Nav::safety_and_step(G, t.path, t.path, lp, ld, a.pstep[i], sf, st);
    } else {
      ok = Nav::step(G, t.path, t.path, lp, ld, a.pstep[i], st);
    }
    if (L::lane() == 0) {
      if (!ok) nav_raise(a.flags, VGB_NAV_ERR_DEPTH);
      put(i, t, st, sf, node);
    }
    return false;
  }
};

template <uint32_t kMask, bool kAbbox>
__global__ void __launch_bounds__(kEngThreads, kEngBlocks)
    k_nav_trace_tracks(const NavTraceArgs a, int32_t cap) {
  nav_engine(a.G, TraceClient<kMask, kAbbox>{a, cap}, a.n);
}
template <uint32_t kMask, StepForm kForm>
__global__ void __launch_bounds__(kEngThreads, kEngBlocks)
    k_nav_step_tracks(const NavStepArgs a, int32_t cap) {
  nav_engine(a.G, StepClient<kMask, kForm>{a, cap}, a.n);
}

inline int nav_grid(int64_t n, int lanes) {
  const int64_t per = kNavBlock / lanes;
  const int64_t want = (n + per - 1) / per;
  const int64_t cap = 148 * 16;
  return (int)(want < 1 ? 1 : (want > cap ? cap : want));
}
// dynamic shared memory of an ABBox block whose warps hold cap hits each
inline size_t abbox_smem(int cap) {
  return (size_t)kNavWarps * (cap + kAbSortThreshold) * sizeof(AbCand);
}

template <uint32_t M> void NavLaunch<M>::locate(const NavLocateArgs &a, cudaStream_t s) {
  auto go = [&](auto l) {
    using L = decltype(l);
    k_nav_locate<L, M><<<nav_grid(a.n, L::N), kNavBlock, 0, s>>>(a.G, a.n, a.x, a.y, a.z, a.states,
                                                                 a.stride, a.flags);
  };
  if (nav_by_threads<M>(NavCall::kLocate, a.n))
    go(OneLane{});
  else
    go(WarpLanes{});
}
template <uint32_t M> void NavLaunch<M>::step(const NavStepArgs &a, bool screen, cudaStream_t s) {
  using L = WarpLanes;
  auto go = [&](auto scr) {
    k_nav_step<L, M, decltype(scr)::value><<<nav_grid(a.n, L::N), kNavBlock, 0, s>>>(
        a.G, a.n, a.x, a.y, a.z, a.dx, a.dy, a.dz, a.cur, a.next, a.stride, a.pstep, a.step,
        a.safety, a.flags);
  };
  if (nav_by_threads<M>(NavCall::kStep, a.n))
    k_nav_step_tracks<M, StepForm::kSimple><<<engine_grid(a.n), kEngThreads, 0, s>>>(a, 0);
  else if (screen)
    go(std::true_type{});
  else
    go(std::false_type{});
}
template <uint32_t M> void NavLaunch<M>::basket(const NavStepArgs &a, cudaStream_t s) {
  using L = WarpLanes;
  if (nav_by_threads<M>(NavCall::kStep, a.n))
    k_nav_step_tracks<M, StepForm::kBasket><<<engine_grid(a.n), kEngThreads, 0, s>>>(a, 0);
  else
    k_nav_basket<L, M><<<nav_grid(a.n, L::N), kNavBlock, 0, s>>>(
        a.G, a.n, a.x, a.y, a.z, a.dx, a.dy, a.dz, a.cur, a.next, a.stride, a.pstep, a.step,
        a.safety, a.node, a.flags);
}
template <uint32_t M> void NavLaunch<M>::trace(const NavTraceArgs &a, bool screen, cudaStream_t s) {
  using L = WarpLanes;
  auto go = [&](auto scr) {
    k_nav_trace<L, M, decltype(scr)::value><<<nav_grid(a.n, L::N), kNavBlock, 0, s>>>(
        a.G, a.n, a.x, a.y, a.z, a.dx, a.dy, a.dz, a.pstep, a.max_steps, a.next_ids, a.steps,
        a.safeties, a.nsteps, a.flags);
  };
  if (nav_by_threads<M>(NavCall::kTrace, a.n))
    k_nav_trace_tracks<M, false><<<engine_grid(a.n), kEngThreads, 0, s>>>(a, 0);
  else if (screen)
    go(std::true_type{});
  else
    go(std::false_type{});
}
template <uint32_t M>
void NavLaunch<M>::abbox_step(const NavStepArgs &a, int32_t cap, cudaStream_t s) {
  const size_t smem = abbox_smem(cap);
  if (nav_by_threads<M>(NavCall::kAbboxStep, a.n)) {
    auto k = k_nav_step_tracks<M, StepForm::kAbbox>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k<<<engine_grid(a.n), kEngThreads, smem, s>>>(a, cap);
    return;
  }
  cudaFuncSetAttribute(k_abbox_step<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_abbox_step<M><<<nav_grid(a.n, 32), kNavBlock, smem, s>>>(
      a.G, cap, a.n, a.x, a.y, a.z, a.dx, a.dy, a.dz, a.cur, a.next, a.stride, a.pstep, a.step,
      a.safety, a.flags);
}
template <uint32_t M>
void NavLaunch<M>::abbox_trace(const NavTraceArgs &a, int32_t cap, cudaStream_t s) {
  const size_t smem = abbox_smem(cap);
  if (nav_by_threads<M>(NavCall::kAbboxTrace, a.n)) {
    auto k = k_nav_trace_tracks<M, true>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k<<<engine_grid(a.n), kEngThreads, smem, s>>>(a, cap);
    return;
  }
  cudaFuncSetAttribute(k_abbox_trace<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_abbox_trace<M><<<nav_grid(a.n, 32), kNavBlock, smem, s>>>(
      a.G, cap, a.n, a.x, a.y, a.z, a.dx, a.dy, a.dz, a.pstep, a.max_steps, a.next_ids, a.steps,
      a.safeties, a.nsteps, a.flags);
}

}  // namespace vgb
