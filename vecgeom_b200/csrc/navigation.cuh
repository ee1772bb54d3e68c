// navigation.cuh -- SimpleNavigator on the device: LocatePoint, RelocatePointFromPath,
// FindNextBoundaryAndStep and GetSafety over a flat geometry image.
//
// The per-track logic follows navigation/SimpleNavigator.h:204-596 step by
// step, so the next-volume sequence, the steps and the safeties are those of the
// reference.  The daughter loops are written over a group of lanes (the Lanes
// policy): on the GPU a warp serves one track and its 32 lanes share the
// daughters of the current volume, or, in large calls, a thread serves one
// (nav_engine.cuh); the minimum over the lanes keeps the
// reference's first-index tie rule, and the containment searches keep its
// order (first daughter for LocatePoint, last for LocatePointExclVolume) through
// warp ballots.  The host build runs the same code with a single lane.
//
// A DistanceToIn candidate is evaluated with the mother's step as its step
// limit rather than the running minimum the reference passes
// (SimpleNavigator.h:396-410).  The kernels only use the limit to return
// kInfinity early for rays that cannot beat it (box: safety >= limit), and a
// larger limit only turns such an early kInfinity into a distance that is no
// smaller than the running minimum at that daughter, so the first minimum, and
// with it the chosen daughter and the step, are unchanged.
#pragma once
#include "batch.cuh"
#include "geometry.h"

namespace vgb {

constexpr int kNavMaxLevels = 16;

// Device view of the geometry tables (all indices are placed / logical ids).
struct NavGeom {
  const double *params;         // shape parameter pool
  const UnplacedRec *unplaced;  // type + record offset per unplaced shape
  const PlacedRec *placed;      // unplaced, logical, effective and raw transform ids
  const DXform *xforms;         // effective transform of each placed volume's placed ops
  const NavXform *raw;          // per Transformation3D
  const LogicalRec *logicals;   // daughter range per logical volume
  const int32_t *daughters;     // CSR over logicals
  const float *pl_box;          // per placed: enclosing box in the mother's frame (6 floats)
  const float *ab_box;          // per placed: ABBoxManager's aligned box, float (6 floats)
  const float4 *ab_slot;        // per daughter slot (CSR order): lower, upper as float4
  int32_t world;
  int32_t max_depth;            // levels of the deepest path
  const NavVol *vols = nullptr;         // per placed; nullptr (host checks): from the tables
  const NavSlot *slots = nullptr;       // per daughter slot, likewise
  const float4 *slot_box = nullptr;     // per daughter slot: its box; nullptr: not used
  const CellGrid *grids = nullptr;      // cell grids of wide volumes; nullptr: not used
  const int32_t *cell_start = nullptr;
  const int32_t *cell_items = nullptr;
};

// NavigationState in the reference's field layout (navigation/NavigationState.h:45-66,
// VecCore/inc/VariableSizeObj.h:25-31): int32 level @0, bool onBoundary @4,
// {selfAlloc:1, N:31} @8, then N path slots of 8 bytes @16.  On the device a
// slot holds the placed-volume index (int64) where the reference holds a pointer.
struct NavStateRef {
  unsigned char *p;
  VGB_HD int32_t &level() const { return *reinterpret_cast<int32_t *>(p); }
  VGB_HD uint8_t &boundary() const { return p[4]; }
  VGB_HD uint32_t &header() const { return *reinterpret_cast<uint32_t *>(p + 8); }
  VGB_HD int64_t &slot(int i) const { return reinterpret_cast<int64_t *>(p + 16)[i]; }
};
VGB_HD int64_t nav_state_stride(int max_depth) { return 16 + 8 * (int64_t)(max_depth + 1); }

// A path held in registers while a track is processed.
struct NavPath {
  int32_t level;
  bool boundary;
  int32_t v[kNavMaxLevels];
  VGB_HD int32_t top() const { return level > 0 ? v[level - 1] : -1; }
  VGB_HD void push(int32_t pv) { v[level++] = pv; }
  VGB_HD void pop() {
    if (level > 0) v[--level] = -1;
  }
};

VGB_HD void nav_load(NavPath &s, const NavStateRef &r) {
  s.level = r.level();
  s.boundary = r.boundary() != 0;
  for (int i = 0; i < kNavMaxLevels; ++i) s.v[i] = (i < s.level) ? (int32_t)r.slot(i) : -1;
}
VGB_HD void nav_store(const NavPath &s, const NavStateRef &r, int max_depth) {
  r.level() = s.level;
  r.boundary() = s.boundary ? 1 : 0;
  r.header() = (uint32_t)(max_depth + 1) << 1;
  for (int i = 0; i <= max_depth; ++i) r.slot(i) = (i < s.level) ? s.v[i] : -1;
}

// ---------------------------------------------------------------------------
// lanes: one warp per track on the GPU, one thread on the host
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
struct WarpLanes {
  static constexpr int N = 32;
  static constexpr bool kBoxes = true;  // searches the daughters' boxes (search below)
  static VGB_D int lane() { return threadIdx.x & 31; }
  static VGB_D uint32_t ballot(bool b) { return __ballot_sync(0xffffffffu, b); }
  static VGB_D double shfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
  static VGB_D int shfl_xor(int v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
  static VGB_D float shfl_xor(float v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
  static VGB_D double shfl_up(double v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
  static VGB_D uint32_t lanes_below() { return (1u << lane()) - 1u; }
  static VGB_D void sync() { __syncwarp(); }
  // 64 positions per warp of the block (blocks of up to 8 warps)
  static VGB_D int32_t *scratch() {
    __shared__ int32_t buf[8][64];
    return buf[threadIdx.x >> 5];
  }
};
#endif
struct OneLane {
  static constexpr int N = 1;
  static constexpr bool kBoxes = false;
  static VGB_HD int lane() { return 0; }
  static VGB_HD uint32_t ballot(bool b) { return b ? 1u : 0u; }
  static VGB_HD double shfl_xor(double v, int) { return v; }
  static VGB_HD int shfl_xor(int v, int) { return v; }
  static VGB_HD float shfl_xor(float v, int) { return v; }
  static VGB_HD double shfl_up(double v, int) { return v; }
  static VGB_HD uint32_t lanes_below() { return 0u; }
  static VGB_HD void sync() {}
  static VGB_HD int32_t *scratch() { return nullptr; }
};

VGB_HD int nav_lowbit(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __ffs(b) - 1;
#else
  return __builtin_ctz(b);
#endif
}
VGB_HD int nav_highbit(uint32_t b) {
#ifdef __CUDA_ARCH__
  return 31 - __clz(b);
#else
  return 31 - __builtin_clz(b);
#endif
}

VGB_HD int nav_popc(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __popc(b);
#else
  return __builtin_popcount(b);
#endif
}

// (value, index) minimum; equal values keep the lower index, NaN never wins
VGB_HD void nav_min_merge(double &v, int &i, double ov, int oi) {
  if (ov < v || (ov == v && oi < i)) {
    v = ov;
    i = oi;
  }
}
template <class L> VGB_HD void nav_min_reduce(double &v, int &i) {
  for (int m = L::N / 2; m > 0; m >>= 1) {
    const double ov = L::shfl_xor(v, m);
    const int oi = L::shfl_xor(i, m);
    nav_min_merge(v, i, ov, oi);
  }
}

// two such minima at once
template <class L> VGB_HD void nav_min_reduce2(double &v, int &i, double &w, int &j) {
  for (int m = L::N / 2; m > 0; m >>= 1) {
    const double ov = L::shfl_xor(v, m), ow = L::shfl_xor(w, m);
    const int oi = L::shfl_xor(i, m), oj = L::shfl_xor(j, m);
    nav_min_merge(v, i, ov, oi);
    nav_min_merge(w, j, ow, oj);
  }
}

// ---------------------------------------------------------------------------
// records
// ---------------------------------------------------------------------------
VGB_HD NavVol nav_vol(const NavGeom &G, int32_t pv) {
#ifdef __CUDA_ARCH__
  return G.vols[pv];
#else
  if (G.vols) return G.vols[pv];
  const PlacedRec &p = G.placed[pv];
  const UnplacedRec &u = G.unplaced[p.unplaced];
  const LogicalRec &l = G.logicals[p.logical];
  return NavVol{u.type, u.param_off, l.dfirst, l.dcount, l.wide, l.grid, p.raw_xform, p.xform};
#endif
}
// The record of daughter slot k (CSR position); `room` holds it where there is no table.
VGB_HD const NavSlot &nav_slot(const NavGeom &G, int32_t k, NavSlot &room) {
#ifdef __CUDA_ARCH__
  (void)room;
  return G.slots[k];
#else
  if (G.slots) return G.slots[k];
  const int32_t pv = G.daughters[k];
  const NavVol v = nav_vol(G, pv);
  room = NavSlot{G.xforms[v.xform], v.type, v.param_off, pv, 0};
  return room;
#endif
}
VGB_HD int32_t nav_placed(const NavGeom &G, int32_t k) {
#ifdef __CUDA_ARCH__
  return G.slots[k].placed;
#else
  return G.daughters[k];
#endif
}

// ---------------------------------------------------------------------------
// shape dispatch over the shape types a geometry holds (kMask bit = type)
// ---------------------------------------------------------------------------
constexpr uint32_t kNavMaskAll = 0x3ffeu;  // types 1..13
constexpr uint32_t kNavMaskBoxTubeTrd =
    (1u << VGB_SHAPE_BOX) | (1u << VGB_SHAPE_TUBE) | (1u << VGB_SHAPE_TRD);

template <uint32_t kMask, class Ret, class Fn>
VGB_HD Ret nav_visit(const NavGeom &G, int type, int32_t param_off, Fn fn) {
  const double *rec = G.params + param_off;
#define VGB_NAV_VISIT(T, OPS, P)                                          \
  if constexpr ((kMask >> T) & 1u) {                                      \
    if (type == T) return fn(OPS<double>{}, bind_params(*reinterpret_cast<const P *>(rec), rec)); \
  }
  VGB_FOR_EACH_SHAPE(VGB_NAV_VISIT)
#undef VGB_NAV_VISIT
  return Ret{};
}

// The shape calls on a point (and direction) in the shape's own frame.  For a
// geometry of a few simple kinds they are inline.
template <uint32_t kMask> struct NavKernels {
  using R = double;
  static VGB_HD V3<R> direction(int, const DXform &X, const V3<R> &v) { return xf_dir(X, v); }
  static VGB_HD bool contains(const NavGeom &G, int type, int32_t off, const V3<R> &l) {
    return nav_visit<kMask, bool>(G, type, off,
                                  [&](auto o, const auto &s) { return decltype(o)::contains(s, l); });
  }
  static VGB_HD R distance_to_in(const NavGeom &G, int type, int32_t off, const V3<R> &l,
                                 const V3<R> &v, R smax) {
    return nav_visit<kMask, R>(G, type, off, [&](auto o, const auto &s) {
      static_assert(!DirAsPoint<decltype(o)>::value, "the direction is moved as a direction");
      return decltype(o)::distance_to_in(s, l, v, smax);
    });
  }
  static VGB_HD R distance_to_out(const NavGeom &G, int type, int32_t off, const V3<R> &l,
                                  const V3<R> &v, R smax) {
    return nav_visit<kMask, R>(G, type, off, [&](auto o, const auto &s) {
      return decltype(o)::distance_to_out(s, l, v, smax);
    });
  }
  static VGB_HD R safety_to_in(const NavGeom &G, int type, int32_t off, const V3<R> &l) {
    return nav_visit<kMask, R>(
        G, type, off, [&](auto o, const auto &s) { return decltype(o)::safety_to_in(s, l); });
  }
  static VGB_HD R safety_to_out(const NavGeom &G, int type, int32_t off, const V3<R> &l) {
    return nav_visit<kMask, R>(
        G, type, off, [&](auto o, const auto &s) { return decltype(o)::safety_to_out(s, l); });
  }
};

// A boolean's calls, one copy of each per kernel file.
namespace navbool {
using R = double;
VGB_HD BooleanP prm(const double *rec) {
  return bind_params(*reinterpret_cast<const BooleanP *>(rec), rec);
}
VGB_HD_NOINLINE bool contains(const double *rec, V3<R> l) {
  return BoolOps<R>::contains(prm(rec), l);
}
VGB_HD_NOINLINE R distance_to_in(const double *rec, V3<R> l, V3<R> d, R smax) {
  return BoolOps<R>::distance_to_in(prm(rec), l, d, smax);
}
VGB_HD_NOINLINE R distance_to_out(const double *rec, V3<R> l, V3<R> d, R smax) {
  return BoolOps<R>::distance_to_out(prm(rec), l, d, smax);
}
VGB_HD_NOINLINE R safety_to_in(const double *rec, V3<R> l) {
  return BoolOps<R>::safety_to_in(prm(rec), l);
}
VGB_HD_NOINLINE R safety_to_out(const double *rec, V3<R> l) {
  return BoolOps<R>::safety_to_out(prm(rec), l);
}
}  // namespace navbool

// Any shape: the shape arithmetic is behind the out-of-line switches of
// boolean.cuh's any-shape component (the same calls a boolean makes), so a kernel
// holds one copy of every shape's code instead of one per call site.
template <> struct NavKernels<kNavMaskAll> {
  using R = double;
  static VGB_HD V3<R> direction(int type, const DXform &X, const V3<R> &v) {
    return anycomp::dir_as_point(type) ? xf_point(X, v) : xf_dir(X, v);
  }
  static VGB_HD bool contains(const NavGeom &G, int type, int32_t off, const V3<R> &l) {
    if (type == VGB_SHAPE_BOOLEAN) return navbool::contains(G.params + off, l);
    return anycomp::contains(type, G.params + off, l);
  }
  static VGB_HD R distance_to_in(const NavGeom &G, int type, int32_t off, const V3<R> &l,
                                 const V3<R> &v, R smax) {
    if (type == VGB_SHAPE_BOOLEAN) return navbool::distance_to_in(G.params + off, l, v, smax);
    return anycomp::distance_to_in(type, G.params + off, l, v, smax);
  }
  static VGB_HD R distance_to_out(const NavGeom &G, int type, int32_t off, const V3<R> &l,
                                  const V3<R> &v, R smax) {
    if (type == VGB_SHAPE_BOOLEAN) return navbool::distance_to_out(G.params + off, l, v, smax);
    return anycomp::distance_to_out(type, G.params + off, l, v, smax);
  }
  static VGB_HD R safety_to_in(const NavGeom &G, int type, int32_t off, const V3<R> &l) {
    if (type == VGB_SHAPE_BOOLEAN) return navbool::safety_to_in(G.params + off, l);
    return anycomp::safety_to_in(type, G.params + off, l);
  }
  static VGB_HD R safety_to_out(const NavGeom &G, int type, int32_t off, const V3<R> &l) {
    if (type == VGB_SHAPE_BOOLEAN) return navbool::safety_to_out(G.params + off, l);
    return anycomp::safety_to_out(type, G.params + off, l);
  }
};

// The calls of the navigators: a volume by its record (point in its own frame), a
// daughter by its slot (point and direction in its mother's frame).
template <uint32_t kMask> struct NavShapes {
  using R = double;
  using K = NavKernels<kMask>;
  static VGB_HD bool unplaced_contains(const NavGeom &G, int32_t pv, const V3<R> &l) {
    const NavVol v = nav_vol(G, pv);
    return K::contains(G, v.type, v.param_off, l);
  }
  static VGB_HD R distance_to_out(const NavGeom &G, const NavVol &c, const V3<R> &l,
                                  const V3<R> &v, R smax) {
    return K::distance_to_out(G, c.type, c.param_off, l, v, smax);
  }
  static VGB_HD R safety_to_out(const NavGeom &G, const NavVol &c, const V3<R> &l) {
    return K::safety_to_out(G, c.type, c.param_off, l);
  }
  // VPlacedVolume::Contains(point, localPoint) (volumes/ShapeImplementationHelper.h:163-180)
  static VGB_HD bool contains(const NavGeom &G, int32_t k, const V3<R> &p) {
    NavSlot room;
    const NavSlot &s = nav_slot(G, k, room);
    return K::contains(G, s.type, s.param_off, xf_point(s.xf, p));
  }
  static VGB_HD R distance_to_in(const NavGeom &G, int32_t k, const V3<R> &p, const V3<R> &v,
                                 R smax) {
    NavSlot room;
    const NavSlot &s = nav_slot(G, k, room);
    return K::distance_to_in(G, s.type, s.param_off, xf_point(s.xf, p),
                             K::direction(s.type, s.xf, v), smax);
  }
  static VGB_HD R safety_to_in(const NavGeom &G, int32_t k, const V3<R> &p) {
    NavSlot room;
    const NavSlot &s = nav_slot(G, k, room);
    return K::safety_to_in(G, s.type, s.param_off, xf_point(s.xf, p));
  }
  // SafetyToIn and DistanceToIn of one daughter, from one frame change
  static VGB_HD R safety_and_distance_to_in(const NavGeom &G, int32_t k, const V3<R> &p,
                                            const V3<R> &v, R smax, R &safety,
                                            bool want_distance = true) {
    NavSlot room;
    const NavSlot &s = nav_slot(G, k, room);
    const V3<R> l = xf_point(s.xf, p);
    safety = K::safety_to_in(G, s.type, s.param_off, l);
    if (!want_distance) return Lim<R>::inf();
    return K::distance_to_in(G, s.type, s.param_off, l, K::direction(s.type, s.xf, v), smax);
  }
};

// ---------------------------------------------------------------------------
// transforms
// ---------------------------------------------------------------------------
// Transformation3D::MultiplyFromRight (base/Transformation3D.h:674-743)
VGB_HD void nav_multiply_from_right(double t[3], double r[9], const NavXform &rhs) {
  if (rhs.flags & kNavIdentity) return;
  if (rhs.flags & kNavHasTrans) {
    for (int i = 0; i < 3; ++i) {
      t[i] = t[i] + r[3 * i + 0] * rhs.t[0];
      t[i] = t[i] + r[3 * i + 1] * rhs.t[1];
      t[i] = t[i] + r[3 * i + 2] * rhs.t[2];
    }
  }
  if (rhs.flags & kNavHasRot) {
    for (int i = 0; i < 3; ++i) {
      const double tx = r[3 * i + 0], ty = r[3 * i + 1], tz = r[3 * i + 2];
      r[3 * i + 0] = tx * rhs.r[0];
      r[3 * i + 1] = tx * rhs.r[1];
      r[3 * i + 2] = tx * rhs.r[2];
      r[3 * i + 0] = r[3 * i + 0] + ty * rhs.r[3];
      r[3 * i + 1] = r[3 * i + 1] + ty * rhs.r[4];
      r[3 * i + 2] = r[3 * i + 2] + ty * rhs.r[5];
      r[3 * i + 0] = r[3 * i + 0] + tz * rhs.r[6];
      r[3 * i + 1] = r[3 * i + 1] + tz * rhs.r[7];
      r[3 * i + 2] = r[3 * i + 2] + tz * rhs.r[8];
    }
  }
}

// NavigationState::TopMatrix (navigation/NavigationState.h:401-408): the product
// of the transforms of path[1..level-1], applied with Transform<kGeneric,kGeneric>.
VGB_HD DXform nav_top_matrix(const NavGeom &G, const NavPath &s) {
  DXform m;
  for (int i = 0; i < 3; ++i) m.t[i] = 0.;
  for (int i = 0; i < 9; ++i) m.r[i] = (i % 4 == 0) ? 1. : 0.;
  for (int i = 1; i < s.level; ++i) nav_multiply_from_right(m.t, m.r, G.raw[nav_vol(G, s.v[i]).raw_xform]);
  m.flags = kXfHasTrans | kXfHasRot;
  m.pad = 0;
  return m;
}

// Transform<kGeneric,kGeneric> of a raw transformation
VGB_HD V3<double> nav_generic_point(const NavXform &X, const V3<double> &p) {
  DXform d;
  for (int i = 0; i < 3; ++i) d.t[i] = X.t[i];
  for (int i = 0; i < 9; ++i) d.r[i] = X.r[i];
  d.flags = kXfHasTrans | kXfHasRot;
  d.pad = 0;
  return xf_point(d, p);
}

// InverseTransform (base/Transformation3D.h:598-632)
VGB_HD V3<double> nav_inverse_point(const NavXform &X, const V3<double> &l) {
  V3<double> m;
  m.x = X.t[0];
  m.x = m.x + l.x * X.r[0];
  m.x = m.x + l.y * X.r[1];
  m.x = m.x + l.z * X.r[2];
  m.y = X.t[1];
  m.y = m.y + l.x * X.r[3];
  m.y = m.y + l.y * X.r[4];
  m.y = m.y + l.z * X.r[5];
  m.z = X.t[2];
  m.z = m.z + l.x * X.r[6];
  m.z = m.z + l.y * X.r[7];
  m.z = m.z + l.z * X.r[8];
  return m;
}

// ---------------------------------------------------------------------------
// float screen of the FP32+refine form (ABBoxNavigator's idea, kept exact)
// ---------------------------------------------------------------------------
// A daughter's DistanceToIn is only needed when it can beat the running best, which its
// box decides (wide_meets below), and a box daughter's SafetyToIn when it can be below the
// running minimum.

// Lower bound of a box daughter's SafetyToIn (BoxImplementation.h:801-818,
// max_i |l_i| - d_i) in float, minus a margin covering the float rounding of
// the transform and the subtraction.
VGB_HD float box_safety_lower(const BoxP &b, const DXform &X, const V3<double> &p) {
  if (X.flags & kXfQuirk16A) return -3e38f;  // not the motion below
  const float ax = (float)(p.x - X.t[0]), ay = (float)(p.y - X.t[1]), az = (float)(p.z - X.t[2]);
  const bool tr = X.flags & kXfHasTrans;
  const float px = tr ? ax : (float)p.x, py = tr ? ay : (float)p.y, pz = tr ? az : (float)p.z;
  float lx = px, ly = py, lz = pz;
  if (X.flags & kXfHasRot) {
    lx = px * (float)X.r[0] + py * (float)X.r[3] + pz * (float)X.r[6];
    ly = px * (float)X.r[1] + py * (float)X.r[4] + pz * (float)X.r[7];
    lz = px * (float)X.r[2] + py * (float)X.r[5] + pz * (float)X.r[8];
  }
  float s = fabsf(lx) - (float)b.d[0];
  s = fmaxf(s, fabsf(ly) - (float)b.d[1]);
  s = fmaxf(s, fabsf(lz) - (float)b.d[2]);
  const float scale = fabsf(px) + fabsf(py) + fabsf(pz) + (float)(b.d[0] + b.d[1] + b.d[2]);
  return s - (1e-3f + 1e-5f * scale);
}

// ---------------------------------------------------------------------------
// the daughters' boxes decide which of them are evaluated
// ---------------------------------------------------------------------------
// A daughter is skipped when its box shows that its FP64 answer cannot matter; the
// rule for equal values (lowest position first) makes the outcome that of the scan
// of the whole list.  The boxes hold the daughters with a margin of 1e-3 mm + 1e-5
// of their coordinates; `e` adds the rounding of the point to float, so a test
// fails only when the exact point, or line, is outside the daughter.  A NaN skips
// nothing.
struct WidePoint {
  float p[3], e[3];
};
VGB_HD WidePoint wide_point(const V3<double> &q) {
  WidePoint t;
  const double v[3] = {q.x, q.y, q.z};
  for (int k = 0; k < 3; ++k) {
    t.p[k] = (float)v[k];
    t.e[k] = 2.5e-7f * fabsf(t.p[k]);
  }
  return t;
}
struct WideLine {
  float inv[3];
  bool flat[3];
  // The distances take the direction as a unit vector; for any other line every
  // box counts as met.
  bool all;
};
VGB_HD WideLine wide_line(const V3<double> &p, const V3<double> &d) {
  WideLine l;
  const double dd[3] = {d.x, d.y, d.z};
  for (int k = 0; k < 3; ++k) {
    l.flat[k] = fabs(dd[k]) < 1e-30;
    l.inv[k] = l.flat[k] ? 0.f : (float)(1.0 / dd[k]);
  }
  l.all = !(fabs(d.x * d.x + d.y * d.y + d.z * d.z - 1.0) < 1e-10 &&
            fabs(p.x) + fabs(p.y) + fabs(p.z) < 1e30);
  return l;
}
// Whether the line p + t d meets the box (any sign of t: a box may answer with a
// hit just behind a point on its face's plane) no farther ahead than best.
VGB_HD bool wide_meets(const float4 &lo4, const float4 &hi4, const WidePoint &t, const WideLine &l,
                       double best) {
  if (l.all) return true;
  const float lo[3] = {lo4.x, lo4.y, lo4.z}, hi[3] = {hi4.x, hi4.y, hi4.z};
  float tn = -3.0e38f, tf = 3.0e38f;
  bool out = false;
  for (int k = 0; k < 3; ++k) {
    const float a = (lo[k] - t.e[k]) - t.p[k], b = (hi[k] + t.e[k]) - t.p[k];
    const float t1 = a * l.inv[k], t2 = b * l.inv[k];
    out |= l.flat[k] && (a > 0.f || b < 0.f);
    tn = l.flat[k] ? tn : fmaxf(tn, fminf(t1, t2));
    tf = l.flat[k] ? tf : fminf(tf, fmaxf(t1, t2));
  }
  out |= tn - tf > 1e-5f * (fabsf(tn) + fabsf(tf));
  // a negative best bounds nothing: a daughter that the point is in answers -1, however
  // far behind the point its box begins (and nothing improves on a NaN)
  const float bf = fmaxf((float)best, 0.f);
  out |= tn > bf * 1.0001f + 1e-3f;
  return !out;
}
// Whether a safety, at least the distance to the box over sqrt(3), may lie below
// best.
VGB_HD bool wide_near(const float4 &lo, const float4 &hi, const WidePoint &t, double best) {
  const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
  float d2 = 0.f;
  for (int k = 0; k < 3; ++k) {
    const float a = (l[k] - t.e[k]) - t.p[k], b = t.p[k] - (h[k] + t.e[k]);
    const float g = fmaxf(fmaxf(a, b), 0.f);
    d2 += g * g;
  }
  // sqrt(3) best and a margin; where lim * lim leaves a float's range everything is near,
  // and where d2 alone does it is the larger
  const float lim = fmaxf((float)best, 0.f) * 1.7323f + 1e-3f;
  return !(d2 > lim * lim);
}

// The daughters a point may be in: the list of its cell where the volume has a
// grid (nullptr and the whole list otherwise).  A point that is not finite is in
// every box by the shapes' comparisons, so it scans the whole list.
VGB_HD const int32_t *cell_list(const NavGeom &G, const NavVol &lr, const V3<double> &p,
                                int &count) {
  count = lr.dcount;
  if (lr.grid == 0 || G.grids == nullptr) return nullptr;
  if (!(fabs(p.x) + fabs(p.y) + fabs(p.z) < 1e30)) return nullptr;
  const CellGrid c = G.grids[lr.grid - 1];
  const float v[3] = {(float)p.x, (float)p.y, (float)p.z};
  int at = 0;
  bool out = false;
  for (int k = 2; k >= 0; --k) {
    const float f = floorf((v[k] - c.org[k]) * c.inv[k]);
    out |= f < 0.f || f >= (float)c.n[k];
    at = at * c.n[k] + (int)f;
  }
  const int32_t *st = G.cell_start + c.first;
  if (out) {
    count = 0;
    return st;
  }
  const int32_t b = st[at];
  count = st[at + 1] - b;
  return G.cell_items + b;
}

// ---------------------------------------------------------------------------
// the navigator
// ---------------------------------------------------------------------------
template <class L, uint32_t kMask, bool kScreen = false> struct Navigator {
  using R = double;
  using S = NavShapes<kMask>;

  // Descends from `vol` (already pushed) through the first (kFirst) or last
  // daughter containing the point, as LocatePoint (:204-240) and
  // LocatePointExclVolume (:246-283) do.  Returns false if the path would
  // exceed kNavMaxLevels.
  template <bool kFirst>
  static VGB_HD bool descend(const NavGeom &G, NavPath &s, int32_t vol, V3<R> tmp,
                             int32_t excluded) {
    int32_t cand = vol;
    for (;;) {
      const NavVol lr = nav_vol(G, cand);
      if (lr.dcount == 0) return true;
      // positions to test, in ascending order: those of the point's cell, or all
      int count;
      const int32_t *list = cell_list(G, lr, tmp, count);
      int found = -1;
      if (kFirst) {
        for (int base = 0; base < count && found < 0; base += L::N) {
          const int j = base + L::lane();
          const int32_t k = lr.dfirst + (j < count ? (list ? list[j] : j) : 0);
          const bool hit = j < count && nav_placed(G, k) != excluded && S::contains(G, k, tmp);
          const uint32_t b = L::ballot(hit);
          if (b) found = base + nav_lowbit(b);
        }
      } else {
        for (int top = count; top > 0 && found < 0; top -= L::N) {
          const int base = top - L::N;  // lanes base..top-1, some below 0
          const int j = base + L::lane();
          const int32_t k = lr.dfirst + (j >= 0 ? (list ? list[j] : j) : 0);
          const bool hit = j >= 0 && nav_placed(G, k) != excluded && S::contains(G, k, tmp);
          const uint32_t b = L::ballot(hit);
          if (b) found = base + nav_highbit(b);
        }
      }
      if (list && found >= 0) found = list[found];
      if (found < 0) return true;
      if (s.level >= kNavMaxLevels) return false;
      NavSlot room;
      const NavSlot &sl = nav_slot(G, lr.dfirst + found, room);
      cand = sl.placed;
      s.push(cand);
      tmp = xf_point(sl.xf, tmp);
    }
  }

  // LocatePoint(world, point, path, top=true)
  static VGB_HD bool locate_from_world(const NavGeom &G, NavPath &s, const V3<R> &p) {
    s.level = 0;
    s.boundary = false;
    for (int i = 0; i < kNavMaxLevels; ++i) s.v[i] = -1;
    if (!S::unplaced_contains(G, G.world, p)) return true;
    s.push(G.world);
    return descend<true>(G, s, G.world, p, -1);
  }

  // RelocatePointFromPath (:286-318)
  static VGB_HD bool relocate_from_path(const NavGeom &G, NavPath &s, V3<R> tmp) {
    int32_t mother = s.top();
    if (mother < 0) return true;
    while (mother >= 0 && !S::unplaced_contains(G, mother, tmp)) {
      s.pop();
      tmp = nav_inverse_point(G.raw[nav_vol(G, mother).raw_xform], tmp);
      mother = s.top();
    }
    if (mother >= 0) {
      s.pop();
      s.push(mother);
      return descend<false>(G, s, mother, tmp, mother);
    }
    return true;
  }

  // Whether L's lanes search this volume's daughters through their boxes.
  static VGB_HD bool wide(const NavGeom &G, const NavVol &lr) {
    return L::kBoxes && lr.wide != 0 && G.slot_box != nullptr;
  }

  // The daughters of a wide volume, by a warp: the lanes test 32 boxes at a time and
  // queue the daughters that may lower the safety or the distance; the queue is
  // evaluated 32 at a time (the answers asked for, both from one frame change), and what
  // it finds tightens the tests that follow.  sf and best enter as the mother's values (a
  // NaN sf stays), hit is the position behind best.  Before, every daughter
  // was evaluated: traces of 16 to 1,024 detector tracks by warps 297-380 us with the
  // cells alone, 243-281 with this search.
  static VGB_HD void search_wide(const NavGeom &G, const NavVol &lr, const V3<R> &lp,
                                 const V3<R> &ld, bool want_s, bool want_d, R smax, R &sf, R &best,
                                 int &hit) {
    const int nd = lr.dcount;
    const float4 *boxes = G.slot_box + 2 * (int64_t)lr.dfirst;
    const WidePoint wp = wide_point(lp);
    const WideLine wl = wide_line(lp, ld);
    const bool bound_s = (lr.wide & kWideSafety) != 0;
    int32_t *queue = L::scratch();
    int si = -1, count = 0;
    for (int base = 0; base < nd; base += L::N) {
      const int d = base + L::lane();
      bool keep = false;
      if (d < nd) {
        const float4 lo = boxes[2 * d], hi = boxes[2 * d + 1];
        keep = (want_d && wide_meets(lo, hi, wp, wl, best)) ||
               (want_s && (!bound_s || wide_near(lo, hi, wp, sf)));
      }
      const uint32_t m = L::ballot(keep);
      if (keep) queue[count + nav_popc(m & L::lanes_below())] = d;
      count += nav_popc(m);
      const bool last = base + L::N >= nd;
      while (count >= L::N || (last && count > 0)) {
        L::sync();  // the queue is written
        const int take = count < L::N ? count : L::N;
        R t = Lim<R>::inf(), dd = Lim<R>::inf();
        int ti = 0x7fffffff, di = 0x7fffffff;
        if (L::lane() < take) {
          const int e = queue[L::lane()];
          R ts = Lim<R>::inf(), v;
          if (want_s)
            v = S::safety_and_distance_to_in(G, lr.dfirst + e, lp, ld, smax, ts, want_d);
          else
            v = S::distance_to_in(G, lr.dfirst + e, lp, ld, smax);
          if (want_s && ts == ts) {
            t = ts;
            ti = e;
          }
          if (want_d && v == v && !isinf(v)) {
            dd = v;
            di = e;
          }
        }
        int32_t rest = 0;
        if (L::lane() < count - take) rest = queue[take + L::lane()];
        L::sync();  // the queue is read
        if (L::lane() < count - take) queue[L::lane()] = rest;
        count -= take;
        if (want_s) {
          nav_min_reduce<L>(t, ti);
          if (t < sf || (t == sf && ti < si)) {
            sf = t;
            si = ti;
          }
        }
        if (want_d) {
          nav_min_reduce<L>(dd, di);
          if (dd < best || (dd == best && di < hit)) {
            best = dd;
            hit = di;
          }
        }
      }
    }
  }

  // GetSafety (:572-596) in the frame of the top volume
  static VGB_HD R safety(const NavGeom &G, const NavPath &s, const V3<R> &lp) {
    const NavVol lr = nav_vol(G, s.top());
    R best = S::safety_to_out(G, lr, lp);
    int bi = -1;
    const int32_t nd = lr.dcount;
    // std::min(safety, tmp): a daughter replaces the running value only when
    // strictly smaller; NaN never replaces and a NaN mother value stays
    if (best == best && wide(G, lr)) {
      R none = Lim<R>::inf();
      int hit = -1;
      search_wide(G, lr, lp, V3<R>{0, 0, 0}, true, false, none, best, none, hit);
    } else if (best == best) {
      R mine = best;
      int mi = -1;
      for (int d = L::lane(); d < nd; d += L::N) {
        if constexpr (kScreen && ((kMask >> VGB_SHAPE_BOX) & 1u)) {
          // a box daughter whose safety is certainly >= the running minimum
          // cannot replace it (strict <; the lane's earlier daughters hold it)
          const PlacedRec &pr = G.placed[nav_placed(G, lr.dfirst + d)];
          const UnplacedRec &ur = G.unplaced[pr.unplaced];
          if (ur.type == VGB_SHAPE_BOX &&
              (double)box_safety_lower(*reinterpret_cast<const BoxP *>(G.params + ur.param_off),
                                       G.xforms[pr.xform], lp) >= mine)
            continue;
        }
        const R t = S::safety_to_in(G, lr.dfirst + d, lp);
        if (t < mine) {
          mine = t;
          mi = d;
        }
      }
      nav_min_reduce<L>(mine, mi);
      best = mine;
      bi = mi;
    }
    (void)bi;
    return best;
  }

  // The daughters of any volume, by L's lanes: the nearest DistanceToIn and, with
  // want_s, the smallest SafetyToIn (one frame change for both answers).  sf and best
  // enter as the mother's values, hit as the position behind best.  An infinite
  // distance never wins, but for -infinity where the caller compares it (kInf).
  template <bool kInf>
  static VGB_HD void search(const NavGeom &G, const NavVol &lr, const V3<R> &lp, const V3<R> &ld,
                            bool want_s, R smax, R &sf, R &best, int &hit) {
    if (lr.dcount == 0) return;
    if (wide(G, lr)) {
      search_wide(G, lr, lp, ld, want_s && sf == sf, true, smax, sf, best, hit);
      return;
    }
    // a warp evaluating mixed shapes runs their code one after the other: the
    // DistanceToIn of a daughter whose box the ray misses is left out (27 daughters
    // of 9 kinds, 4,096 traced tracks: 2.04 -> 1.75 ms)
    const bool screen = L::kBoxes && kMask == kNavMaskAll && G.slot_box != nullptr;
    WidePoint wp;
    WideLine wl;
    if (screen) {
      wp = wide_point(lp);
      wl = wide_line(lp, ld);
    }
    int si = -1;
    for (int d = L::lane(); d < lr.dcount; d += L::N) {
      const int32_t k = lr.dfirst + d;
      const bool meets =
          !screen || wide_meets(G.slot_box[2 * k], G.slot_box[2 * k + 1], wp, wl, best);
      R t, dd = Lim<R>::inf();
      if (want_s) {
        dd = S::safety_and_distance_to_in(G, k, lp, ld, smax, t, meets);
        if (t < sf) {  // a NaN mother's safety stays
          sf = t;
          si = d;
        }
      } else if (meets) {
        dd = S::distance_to_in(G, k, lp, ld, smax);
      }
      if (dd < best && (kInf || !isinf(dd))) {
        best = dd;
        hit = d;
      }
    }
    if (want_s)
      nav_min_reduce2<L>(sf, si, best, hit);
    else
      nav_min_reduce<L>(best, hit);
  }

  // The basket form of FindNextBoundaryAndStep (:637-743) for one track, with
  // GetSafeties (:599-632) when want_s: the mother's DistanceToOut with its node
  // index (-1 leaves within pstep, -2 stays;
  // volumes/ShapeImplementationHelper.h:676-692), every daughter's
  // DistanceToInMinimize (:637-658: a strictly smaller distance takes the
  // daughter's index), then the relocation with a 1e-9 push.  Unlike the
  // single-track form there is no special case for a negative or infinite
  // distance.  The lanes share the daughters as in step().
  static VGB_HD bool safety_and_step_basket(const NavGeom &G, const NavPath &cur, NavPath &next,
                                            const V3<R> &lp, const V3<R> &ld, R pstep, bool want_s,
                                            R &safety_out, R &dist_out, int32_t &node_out) {
    const NavVol lr = nav_vol(G, cur.top());
    const R mother = S::distance_to_out(G, lr, lp, ld, pstep);
    R sf = 0;
    if (want_s) sf = S::safety_to_out(G, lr, lp);
    R best = mother;
    int hit = -1;
    search<true>(G, lr, lp, ld, want_s, mother, sf, best, hit);
    if (want_s) safety_out = sf;
    const int bi = hit >= 0 ? hit : (mother < pstep ? -1 : -2);
    dist_out = best;
    node_out = bi;
    next = cur;
    if (best > pstep) {
      dist_out = pstep;
      next.boundary = false;
      return true;
    }
    next.boundary = true;
    const R s9 = best + (R)1e-9;
    V3<R> np = {ld.x * s9, ld.y * s9, ld.z * s9};
    np = {np.x + lp.x, np.y + lp.y, np.z + lp.z};
    if (bi > -1) {
      const int32_t nv = nav_placed(G, lr.dfirst + bi);
      if (next.level >= kNavMaxLevels) return false;
      next.push(nv);
      return descend<true>(G, next, nv, nav_generic_point(G.raw[nav_vol(G, nv).raw_xform], np), -1);
    }
    return relocate_from_path(G, next, np);
  }
  static VGB_HD bool step_basket(const NavGeom &G, const NavPath &cur, NavPath &next,
                                 const V3<R> &lp, const V3<R> &ld, R pstep, R &dist_out,
                                 int32_t &node_out) {
    R none;
    return safety_and_step_basket(G, cur, next, lp, ld, pstep, false, none, dist_out, node_out);
  }

  // FindNextBoundaryAndStep (:340-470).  `next` is updated from `cur` (the two may
  // be one).  Returns false if a path would exceed kNavMaxLevels.
  static VGB_HD bool step(const NavGeom &G, const NavPath &cur, NavPath &next, const V3<R> &lp,
                          const V3<R> &ld, R pstep, R &step_out) {
    int hit;
    const R step = nearest(G, cur, lp, ld, pstep, hit);
    return advance(G, cur, next, lp, ld, pstep, step, hit, step_out);
  }

  // GetSafety and FindNextBoundaryAndStep: the daughters are searched once for both
  // (each daughter's frame change serves both answers).
  static VGB_HD bool safety_and_step(const NavGeom &G, const NavPath &cur, NavPath &next,
                                     const V3<R> &lp, const V3<R> &ld, R pstep, R &safety_out,
                                     R &step_out) {
    if constexpr (kScreen) {
      safety_out = safety(G, cur, lp);
      return step(G, cur, next, lp, ld, pstep, step_out);
    }
    const NavVol lr = nav_vol(G, cur.top());
    R sf = S::safety_to_out(G, lr, lp);
    R step = S::distance_to_out(G, lr, lp, ld, pstep);
    if (step <= 0.) step = Lim<R>::inf();
    R best = step;
    int hit = -1;
    search<false>(G, lr, lp, ld, true, step, sf, best, hit);
    safety_out = sf;
    return advance(G, cur, next, lp, ld, pstep, best, hit, step_out);
  }

  // the distance to the nearest boundary, and the daughter it belongs to (-1: the
  // mother)
  static VGB_HD R nearest(const NavGeom &G, const NavPath &cur, const V3<R> &lp, const V3<R> &ld,
                          R pstep, int &hit) {
    const NavVol lr = nav_vol(G, cur.top());
    R step = S::distance_to_out(G, lr, lp, ld, pstep);
    if (step <= 0.) step = Lim<R>::inf();
    R best = step;
    int bi = -1;
    if constexpr (kScreen) {
      // the boxes by which the FP64 form's warps leave daughters out, and those of the
      // shapes not argued there; a torus, whose directions move as points, is never left
      // out
      const bool boxes = G.slot_box != nullptr;
      const WidePoint wp = wide_point(lp);
      const WideLine wl = wide_line(lp, ld);
      for (int d = L::lane(); d < lr.dcount; d += L::N) {
        const int32_t k = lr.dfirst + d;
        if (boxes) {
          SlotBox b = {G.slot_box[2 * k], G.slot_box[2 * k + 1]};
          if (b.lo.w != 0.f) b = slot_box_of(G.pl_box + 6 * (int64_t)nav_placed(G, k), true);
          if (!wide_meets(b.lo, b.hi, wp, wl, best)) continue;
        }
        const R dd = S::distance_to_in(G, k, lp, ld, step);
        const bool valid = dd < best && !isinf(dd);
        if (valid) {
          best = dd;
          bi = d;
        }
      }
      nav_min_reduce<L>(best, bi);
    } else {
      R none = 0;
      search<false>(G, lr, lp, ld, false, step, none, best, bi);
    }
    hit = bi;
    return best;
  }

  // the step decisions after the search (:420-470)
  static VGB_HD bool advance(const NavGeom &G, const NavPath &cur, NavPath &next, const V3<R> &lp,
                             const V3<R> &ld, R pstep, R step, int hit, R &step_out) {
    const int32_t first = nav_vol(G, cur.top()).dfirst;
    next = cur;
    if (step == Lim<R>::inf() && pstep > 0.) {
      step_out = 0.;
      next.pop();
      next.boundary = true;
      return true;
    }
    if (step > pstep) {
      step_out = pstep;
      next.boundary = false;
      return true;
    }
    next.boundary = true;
    if (step < 0.) step = 0.;
    step_out = step;
    const R s6 = step + (R)1e-6;
    V3<R> np = {ld.x * s6, ld.y * s6, ld.z * s6};
    np = {np.x + lp.x, np.y + lp.y, np.z + lp.z};
    if (hit != -1) {
      const int32_t nv = nav_placed(G, first + hit);
      if (next.level >= kNavMaxLevels) return false;
      next.push(nv);
      return descend<true>(G, next, nv, nav_generic_point(G.raw[nav_vol(G, nv).raw_xform], np), -1);
    }
    return relocate_from_path(G, next, np);
  }
};

}  // namespace vgb
