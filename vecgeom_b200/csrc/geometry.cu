// geometry.cu -- geometry construction, derived shape parameters and the bulk
// device upload (replaces CudaManager, source/CudaManager.cpp:39-322).
//
// Host code here is compiled with -ffp-contract=off: the derived parameters of
// each shape are computed with the same formulas and rounding as the reference
// constructors, so the device kernels see bit-identical constants.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <limits>
#include <new>

#include "geometry.h"
#include "shapes.cuh"

namespace vgb {

static thread_local char g_err[512] = "";
static thread_local int64_t g_launches = 0;

vgb_status set_error(vgb_status s, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return s;
}

vgb_status cuda_error(cudaError_t e, const char *what) {
  if (e == cudaErrorMemoryAllocation)
    return set_error(VGB_ENOMEM, "%s: %s", what, cudaGetErrorString(e));
  return set_error(VGB_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

void count_launch(int n) { g_launches += n; }

// ---------------------------------------------------------------------------
// Transformation3D (source/Transformation3D.cpp)
// ---------------------------------------------------------------------------

// :138-150 GenerateRotationCode
static int gen_rot_code(const double *r) {
  int code = 0;
  for (int i = 0; i < 9; ++i) code |= (1 << i) * (std::fabs(r[i]) > kTolerance);
  if (code == 0x111 && (r[0] == 1. && r[4] == 1. && r[8] == 1.)) code = 0x200;
  return code;
}

// management/TransformationSpecializations.icc: codes with a specialised
// placed volume; everything else runs the generic rotation.
static int specialised_rot(int code) {
  static const int codes[] = {0x1b1, 0x18e, 0x076, 0x16a, 0x155, 0x0ad, 0x0dc, 0x0e3,
                              0x11b, 0x0a1, 0x10a, 0x046, 0x062, 0x054, 0x111, 0x200};
  for (int c : codes)
    if (c == code) return code;
  return -1;
}

static void set_codes(RawXform &x) {
  // :80-89 SetProperties; source/UnplacedVolume.cpp:23-24
  const bool has_t = std::fabs(x.t[0]) > kTolerance || std::fabs(x.t[1]) > kTolerance ||
                     std::fabs(x.t[2]) > kTolerance;
  x.trans_code = has_t ? -1 : 0;
  x.rot_code = specialised_rot(gen_rot_code(x.r));
}

// The effective device transform of one placement.  generic_only mirrors
// shapes whose placed volumes always take Transform<kGeneric,kGeneric>
// (source/UnplacedPolyhedron.cpp:321-333).
DXform effective_xform(const RawXform &x, bool generic_only) {
  DXform d;
  std::memset(&d, 0, sizeof(d));
  const int tcode = generic_only ? -1 : x.trans_code;
  const int rcode = generic_only ? -1 : x.rot_code;
  if (tcode != 0) {
    d.flags |= kXfHasTrans;
    for (int i = 0; i < 3; ++i) d.t[i] = x.t[i];
  }
  if (rcode != 0x200) {
    d.flags |= kXfHasRot;
    for (int i = 0; i < 9; ++i) {
      const bool keep = (rcode == -1) || ((rcode >> i) & 1);
      d.r[i] = keep ? x.r[i] : 0.;
    }
    if (rcode == 0x16a) d.flags |= kXfQuirk16A;
  } else {
    d.r[0] = d.r[4] = d.r[8] = 1.;
  }
  return d;
}

}  // namespace vgb

using namespace vgb;

vgb_status vgb::add_unplaced(vgb_geometry *g, int type, const void *rec, size_t bytes,
                             int32_t extra, int32_t *id) {
  // 16-byte aligned records in the pool
  while (g->params.size() % 2) g->params.push_back(0.);
  const size_t nd = (bytes + sizeof(double) - 1) / sizeof(double);
  UnplacedRec u;
  u.type = type;
  u.param_off = (int32_t)g->params.size();
  u.param_len = (int32_t)nd;
  u.extra = extra;
  g->params.resize(g->params.size() + nd + (nd % 2), 0.);
  std::memcpy(g->params.data() + u.param_off, rec, bytes);
  g->unplaced.push_back(u);
  g->ctor_form.push_back(kCtorDefault);
  g->ctor_args.emplace_back();
  if (id) *id = (int32_t)g->unplaced.size() - 1;
  return VGB_OK;
}

// Depth of the tree below a logical volume (GeoManager::getMaxDepth counts
// levels from the world, management/GeoManager.h:191).
static int depth_of(const vgb_geometry *g, int32_t logical, int guard) {
  if (guard > 64) return -1;
  int best = 0;
  for (int32_t d : g->logical_daughters[logical]) {
    const int sub = depth_of(g, g->placed[d].logical, guard + 1);
    if (sub < 0) return -1;
    if (sub > best) best = sub;
  }
  return best + 1;
}

template <class T>
static vgb_status upload(const std::vector<T> &h, T **d, int64_t *bytes) {
  const size_t n = h.empty() ? 1 : h.size();
  cudaError_t e = cudaMalloc((void **)d, n * sizeof(T));
  if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: cudaMalloc");
  *bytes += (int64_t)(n * sizeof(T));
  if (!h.empty()) {
    e = cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: cudaMemcpy");
  }
  return VGB_OK;
}

extern "C" {

const char *vgb_last_error(void) { return vgb::g_err; }
const char *vgb_version(void) { return "vgb 0.1 (sm_100a)"; }
int64_t vgb_launch_count(void) { return vgb::g_launches; }
void vgb_launch_count_reset(void) { vgb::g_launches = 0; }

vgb_status vgb_geometry_create(vgb_geometry **g) {
  if (!g) return set_error(VGB_EINVAL, "vgb_geometry_create: out pointer is NULL");
  *g = new (std::nothrow) vgb_geometry();
  if (!*g) return set_error(VGB_ENOMEM, "vgb_geometry_create: out of host memory");
  return VGB_OK;
}

vgb_status vgb_geometry_destroy(vgb_geometry *g) {
  if (!g) return VGB_OK;
  if (g->device >= 0) {
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(g->device);
    cudaFree(g->dev.params);
    cudaFree(g->dev.unplaced);
    cudaFree(g->dev.xforms);
    cudaFree(g->dev.raw);
    cudaFree(g->dev.nav_flags);
    cudaFree(g->dev.pl_box);
    cudaFree(g->dev.ab_box);
    cudaFree(g->dev.ab_slot);
    cudaFree(g->dev.nav_tables);
    cudaFree(g->dev.placed);
    cudaFree(g->dev.logicals);
    cudaFree(g->dev.daughters);
    cudaFree(g->staging);
    for (cudaStream_t st : g->staging_streams)
      if (st) cudaStreamDestroy(st);
    if (g->staging_start) cudaEventDestroy(g->staging_start);
    for (auto &slot : g->staging_ev)
      for (cudaEvent_t ev : slot)
        if (ev) cudaEventDestroy(ev);
    cudaSetDevice(prev);
  }
  delete g;
  return VGB_OK;
}

vgb_status vgb_transformation(vgb_geometry *g, double tx, double ty, double tz, double phi,
                              double theta, double psi, int32_t *id) {
  VGB_CHECK_OPEN(g);
  RawXform x;
  // source/Transformation3D.cpp:93-114 SetRotation(phi, theta, psi), degrees
  const double sinphi = std::sin(kDegToRad * phi), cosphi = std::cos(kDegToRad * phi);
  const double sinthe = std::sin(kDegToRad * theta), costhe = std::cos(kDegToRad * theta);
  const double sinpsi = std::sin(kDegToRad * psi), cospsi = std::cos(kDegToRad * psi);
  x.t[0] = tx;
  x.t[1] = ty;
  x.t[2] = tz;
  x.r[0] = cospsi * cosphi - costhe * sinphi * sinpsi;
  x.r[1] = -sinpsi * cosphi - costhe * sinphi * cospsi;
  x.r[2] = sinthe * sinphi;
  x.r[3] = cospsi * sinphi + costhe * cosphi * sinpsi;
  x.r[4] = -sinpsi * sinphi + costhe * cosphi * cospsi;
  x.r[5] = -sinthe * cosphi;
  x.r[6] = sinpsi * sinthe;
  x.r[7] = cospsi * sinthe;
  x.r[8] = costhe;
  set_codes(x);
  g->raw_xforms.push_back(x);
  if (id) *id = (int32_t)g->raw_xforms.size() - 1;
  return VGB_OK;
}

vgb_status vgb_transformation_matrix(vgb_geometry *g, double tx, double ty, double tz,
                                     const double *r9, int32_t *id) {
  VGB_CHECK_OPEN(g);
  if (!r9) return set_error(VGB_EINVAL, "vgb_transformation_matrix: r9 is NULL");
  RawXform x;
  x.t[0] = tx;
  x.t[1] = ty;
  x.t[2] = tz;
  for (int i = 0; i < 9; ++i) x.r[i] = r9[i];
  set_codes(x);
  g->raw_xforms.push_back(x);
  if (id) *id = (int32_t)g->raw_xforms.size() - 1;
  return VGB_OK;
}

vgb_status vgb_logical_volume(vgb_geometry *g, const char *label, int32_t unplaced,
                              int32_t *id) {
  VGB_CHECK_OPEN(g);
  if (unplaced < 0 || unplaced >= (int32_t)g->unplaced.size())
    return set_error(VGB_EINVAL, "vgb_logical_volume: unknown unplaced id %d", unplaced);
  LogicalRec l;
  l.unplaced = unplaced;
  l.dfirst = 0;
  l.dcount = 0;
  l.wide = l.grid = 0;
  for (int32_t &v : l.pad) v = 0;
  g->logicals.push_back(l);
  g->logical_daughters.emplace_back();
  g->labels.push_back(label ? label : "");
  if (id) *id = (int32_t)g->logicals.size() - 1;
  return VGB_OK;
}

vgb_status vgb_place(vgb_geometry *g, int32_t logical, int32_t transformation,
                     int32_t *placed) {
  VGB_CHECK_OPEN(g);
  if (logical < 0 || logical >= (int32_t)g->logicals.size())
    return set_error(VGB_EINVAL, "vgb_place: unknown logical volume %d", logical);
  if (transformation < 0 || transformation >= (int32_t)g->raw_xforms.size())
    return set_error(VGB_EINVAL, "vgb_place: unknown transformation %d", transformation);
  PlacedRec p;
  p.logical = logical;
  p.unplaced = g->logicals[logical].unplaced;
  p.xform = (int32_t)g->xforms.size();
  p.raw_xform = transformation;
  const int type = g->unplaced[p.unplaced].type;
  g->xforms.push_back(
      effective_xform(g->raw_xforms[transformation], type == VGB_SHAPE_POLYHEDRON));
  g->placed.push_back(p);
  if (placed) *placed = (int32_t)g->placed.size() - 1;
  return VGB_OK;
}

vgb_status vgb_place_daughter(vgb_geometry *g, int32_t mother_logical, int32_t daughter_logical,
                              int32_t transformation, int32_t *placed) {
  VGB_CHECK_OPEN(g);
  if (mother_logical < 0 || mother_logical >= (int32_t)g->logicals.size())
    return set_error(VGB_EINVAL, "vgb_place_daughter: unknown mother %d", mother_logical);
  int32_t id = -1;
  vgb_status s = vgb_place(g, daughter_logical, transformation, &id);
  if (s != VGB_OK) return s;
  g->logical_daughters[mother_logical].push_back(id);
  if (placed) *placed = id;
  return VGB_OK;
}

vgb_status vgb_set_world(vgb_geometry *g, int32_t placed) {
  VGB_CHECK_OPEN(g);
  if (placed < 0 || placed >= (int32_t)g->placed.size())
    return set_error(VGB_EINVAL, "vgb_set_world: unknown placed volume %d", placed);
  g->world = placed;
  return VGB_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// boxes of the daughters, and cells over those of wide volumes (navigation.cuh)
// ---------------------------------------------------------------------------
namespace vgb {
namespace {

// Whether a shape's answers are bounded by its box: Contains, and every finite
// DistanceToIn that can be the nearest, is answered by a point of the shape within
// its tolerance.
//   box   hits are points of a face; a point within the tolerance of a face's
//         plane may answer a hit behind it, so boxes are tested along the whole
//         line;
//   tube, trd, cone, sphere, orb, polycone  hits lie at or ahead of the point, within
//         the z planes and the radii (or on the faces); the formulas take the
//         direction as a unit vector, which the caller checks;
//   polyhedron  the same, or the step limit, which is never nearer than the mother's
//         boundary;
//   subtraction  points of the left component, or on the right one's surface inside
//         the left one.
// The torus moves directions as points, so its hits do not lie on the ray; the other
// shapes are not argued here.
bool bounded_shape(int type, const double *rec) {
  switch (type) {
    case VGB_SHAPE_BOX:
    case VGB_SHAPE_TUBE:
    case VGB_SHAPE_TRD:
    case VGB_SHAPE_CONE:
    case VGB_SHAPE_SPHERE:
    case VGB_SHAPE_ORB:
    case VGB_SHAPE_POLYCONE:
    case VGB_SHAPE_POLYHEDRON:
      return true;
    case VGB_SHAPE_BOOLEAN: {
      const BooleanP &b = *reinterpret_cast<const BooleanP *>(rec);
      return b.op == VGB_BOOL_SUBTRACTION && b.left.type != VGB_SHAPE_BOOLEAN &&
             b.left.type != VGB_SHAPE_POLYHEDRON && bounded_shape(b.left.type, nullptr);
    }
    default:
      return false;
  }
}

// Whether a shape moves directions as points, itself or in a component.
bool holds_torus(int type, const double *rec) {
  if (type != VGB_SHAPE_BOOLEAN) return type == VGB_SHAPE_TORUS;
  const BooleanP &b = *reinterpret_cast<const BooleanP *>(rec);
  return b.left.type == VGB_SHAPE_TORUS || b.right.type == VGB_SHAPE_TORUS;
}

// Whether each placed volume's box may stand for it among its mother's daughters: its
// shape is bounded and its placement a rigid motion, so that the box can be moved to
// the mother's frame.  The FP32+refine form's screen takes the boxes of the other shapes
// too, but for a torus.
void mark_bounded(vgb_geometry *g) {
  std::vector<uint8_t> shape(g->unplaced.size()), screen(g->unplaced.size()),
      rigid(g->raw_xforms.size());
  for (size_t u = 0; u < shape.size(); ++u) {
    const double *rec = g->params.data() + g->unplaced[u].param_off;
    shape[u] = bounded_shape(g->unplaced[u].type, rec);
    screen[u] = !holds_torus(g->unplaced[u].type, rec);
  }
  for (size_t i = 0; i < rigid.size(); ++i) {
    const double *r = g->raw_xforms[i].r;
    bool ok = true;
    for (int a = 0; a < 3; ++a)
      for (int b = a; b < 3; ++b)
        ok &= std::fabs(r[a] * r[b] + r[3 + a] * r[3 + b] + r[6 + a] * r[6 + b] -
                        (a == b ? 1. : 0.)) < 1e-8;
    rigid[i] = ok;
  }
  g->bounded.resize(g->placed.size());
  g->screened.resize(g->placed.size());
  for (size_t pv = 0; pv < g->placed.size(); ++pv) {
    const PlacedRec &p = g->placed[pv];
    bool ok = rigid[p.raw_xform] && !(g->xforms[p.xform].flags & kXfQuirk16A);
    for (int k = 0; ok && k < 6; ++k) ok = std::fabs(g->pl_box[6 * pv + k]) < 1e30f;
    g->bounded[pv] = ok && shape[p.unplaced];
    g->screened[pv] = ok && screen[p.unplaced];
  }
}

struct BoxItem {
  float lo[3], hi[3];
  int32_t d;
};

// The cell grid over a volume's daughters: cells of half the daughters' mean box
// size, at most 64 along an axis.  A point's cell and a box's cells come from the
// same float expression, which is monotone, so a box's range holds the cell of
// every point of the box.
// Small daughters far apart would make most cells empty, and large ones fill every cell,
// so the longest axis is halved until there are no more than kCellsPerDaughter cells and
// as many list entries a daughter: the tables grow with the daughters, by at most the
// size of two of their NavSlots each (the layered detector's layers have 2 to 25 of
// both).  One cell would be the whole list: no grid then (0).
constexpr int64_t kCellsPerDaughter = 32;
int32_t build_grid(vgb_geometry *g, const std::vector<BoxItem> &it) {
  CellGrid c = {};
  double extent[3];
  for (int k = 0; k < 3; ++k) {
    float hi = -3e38f;
    c.org[k] = 3e38f;
    double size = 0.;
    for (const BoxItem &b : it) {
      c.org[k] = std::min(c.org[k], b.lo[k]);
      hi = std::max(hi, b.hi[k]);
      size += (double)b.hi[k] - b.lo[k];
    }
    extent[k] = (double)hi - c.org[k];
    const double cells = std::ceil(extent[k] / (0.5 * size / it.size()));
    c.n[k] = (int32_t)std::min(64., std::max(1., cells));
  }
  // the cells of a box, first and last along each axis
  auto range = [&](const BoxItem &b, int a[3], int z[3]) {
    for (int k = 0; k < 3; ++k) {
      a[k] = cell_of(c, k, b.lo[k]);
      z[k] = std::min(cell_of(c, k, b.hi[k]), c.n[k] - 1);
    }
  };
  const int64_t most = kCellsPerDaughter * (int64_t)it.size();
  int64_t entries;
  for (;;) {
    for (int k = 0; k < 3; ++k)
      c.inv[k] = (float)(c.n[k] / (extent[k] * (1. + 1e-5)));  // the last box ends inside the grid
    entries = 0;
    for (const BoxItem &b : it) {
      int a[3], z[3];
      range(b, a, z);
      entries += (int64_t)(z[0] - a[0] + 1) * (z[1] - a[1] + 1) * (z[2] - a[2] + 1);
    }
    if ((int64_t)c.n[0] * c.n[1] * c.n[2] <= most && entries <= most) break;
    int32_t *n = std::max_element(c.n, c.n + 3);
    *n = (*n + 1) / 2;
  }
  const size_t ncell = (size_t)c.n[0] * c.n[1] * c.n[2];
  // offsets are 32-bit (64-bit ones cost a trace 0.6 %): no grid past their range
  if (ncell == 1 || g->cell_start.size() + ncell >= INT32_MAX ||
      g->cell_items.size() + entries >= INT32_MAX)
    return 0;
  c.first = (int32_t)g->cell_start.size();
  // counted first, then filled in daughter order
  auto each_cell = [&](const BoxItem &b, auto f) {
    int a[3], z[3];
    range(b, a, z);
    for (int iz = a[2]; iz <= z[2]; ++iz)
      for (int iy = a[1]; iy <= z[1]; ++iy)
        for (int ix = a[0]; ix <= z[0]; ++ix) f(((size_t)iz * c.n[1] + iy) * c.n[0] + ix);
  };
  std::vector<int32_t> at(ncell + 1, 0);
  for (const BoxItem &b : it) each_cell(b, [&](size_t k) { ++at[k + 1]; });
  at[0] = (int32_t)g->cell_items.size();
  for (size_t k = 0; k < ncell; ++k) at[k + 1] += at[k];
  g->cell_start.insert(g->cell_start.end(), at.begin(), at.end());
  g->cell_items.resize(at[ncell]);
  for (const BoxItem &b : it) each_cell(b, [&](size_t k) { g->cell_items[at[k]++] = b.d; });
  g->grids.push_back(c);
  return (int32_t)g->grids.size();
}

void build_wide(vgb_geometry *g) {
  g->grids.clear();
  g->cell_start.clear();
  g->cell_items.clear();
  std::vector<BoxItem> it;
  for (LogicalRec &l : g->logicals) {
    l.wide = l.grid = 0;
    if (l.dcount <= kWideDaughters) continue;
    it.resize(l.dcount);
    bool all = true, safety = true;
    for (int d = 0; d < l.dcount; ++d) {
      const int32_t pv = g->daughters[l.dfirst + d];
      const int type = g->unplaced[g->placed[pv].unplaced].type;
      all &= g->bounded[pv] != 0;
      // a box's or a tube's SafetyToIn is at least its largest excess over an axis
      // (or the radius), and so at least the distance to its box over sqrt(3); the
      // other shapes' safeties are not argued to have such a bound
      safety &= g->bounded[pv] && (type == VGB_SHAPE_BOX || type == VGB_SHAPE_TUBE);
      it[d].d = d;
      for (int k = 0; k < 3; ++k) {
        it[d].lo[k] = g->pl_box[6 * (size_t)pv + k];
        it[d].hi[k] = g->pl_box[6 * (size_t)pv + 3 + k];
      }
    }
    l.wide = kWide | (safety ? kWideSafety : 0);
    if (all) l.grid = build_grid(g, it);
  }
}

// The navigator's records, from the tables already on the device.
__global__ void k_nav_records(const PlacedRec *placed, const UnplacedRec *unplaced,
                              const LogicalRec *logicals, const DXform *xforms,
                              const int32_t *daughters, const float *pl_box,
                              const uint8_t *bounded, const uint8_t *screened, int32_t nplaced,
                              int32_t nslots, NavVol *vols,
                              NavSlot *slots, float4 *slot_box) {
  const int32_t stride = gridDim.x * blockDim.x;
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nplaced; k += stride) {
    const PlacedRec p = placed[k];
    const UnplacedRec u = unplaced[p.unplaced];
    const LogicalRec l = logicals[p.logical];
    vols[k] = NavVol{u.type, u.param_off, l.dfirst, l.dcount, l.wide, l.grid, p.raw_xform, p.xform};
  }
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nslots; k += stride) {
    const int32_t pv = daughters[k];
    const PlacedRec p = placed[pv];
    const UnplacedRec u = unplaced[p.unplaced];
    slots[k] = NavSlot{xforms[p.xform], u.type, u.param_off, pv, 0};
    SlotBox b = slot_box_of(pl_box + 6 * (int64_t)pv, bounded[pv] != 0);
    b.lo.w = screened[pv] && !bounded[pv] ? 1.f : 0.f;
    slot_box[2 * k] = b.lo;
    slot_box[2 * k + 1] = b.hi;
  }
}

}  // namespace
}  // namespace vgb

vgb_status vgb::prepare_tables(vgb_geometry *g) {
  // CSR of daughters in insertion order (source/LogicalVolume.cpp:84-102)
  g->daughters.clear();
  for (size_t l = 0; l < g->logicals.size(); ++l) {
    g->logicals[l].dfirst = (int32_t)g->daughters.size();
    g->logicals[l].dcount = (int32_t)g->logical_daughters[l].size();
    for (int32_t d : g->logical_daughters[l]) g->daughters.push_back(d);
  }
  g->max_daughters = 0;
  for (const LogicalRec &l : g->logicals)
    if (l.dcount > g->max_daughters) g->max_daughters = l.dcount;
  if (g->world >= 0) {
    g->max_depth = depth_of(g, g->placed[g->world].logical, 0);
    if (g->max_depth < 0)
      return set_error(VGB_EINVAL, "vgb_geometry_close: volume tree deeper than 64 levels");
  }
  g->nav_raw.resize(g->raw_xforms.size());
  for (size_t i = 0; i < g->raw_xforms.size(); ++i) {
    const RawXform &x = g->raw_xforms[i];
    NavXform &n = g->nav_raw[i];
    std::memset(&n, 0, sizeof(n));
    for (int k = 0; k < 3; ++k) n.t[k] = x.t[k];
    for (int k = 0; k < 9; ++k) n.r[k] = x.r[k];
    const bool has_t = x.trans_code != 0, has_r = x.rot_code != 0x200;
    n.flags = (has_t ? kNavHasTrans : 0u) | (has_r ? kNavHasRot : 0u) |
              ((!has_t && !has_r) ? kNavIdentity : 0u);
  }
  g->type_mask = 0;
  for (const UnplacedRec &u : g->unplaced) g->type_mask |= 1u << u.type;
  // the FP32 screen's boxes, widened so that float rounding of the point, the
  // direction and the slab arithmetic cannot move a ray across them
  g->bbox.assign(6 * g->unplaced.size(), 0.f);
  for (size_t u = 0; u < g->unplaced.size(); ++u) {
    double b[6];
    if (!shape_bbox(g, (int32_t)u, b)) {
      for (int k = 0; k < 3; ++k) {
        g->bbox[6 * u + k] = -3.0e38f;
        g->bbox[6 * u + 3 + k] = 3.0e38f;
      }
      continue;
    }
    double ext = 0.;
    for (int k = 0; k < 6; ++k) ext = std::max(ext, std::fabs(b[k]));
    const double pad = 1e-3 + 1e-5 * ext;
    for (int k = 0; k < 3; ++k) {
      g->bbox[6 * u + k] = std::nextafter((float)(b[k] - pad), -3.0e38f);
      g->bbox[6 * u + 3 + k] = std::nextafter((float)(b[3 + k] + pad), 3.0e38f);
    }
  }
  // each placed volume's box in its mother's frame (corners moved with the full
  // matrix, InverseTransform), for the navigator's float screen
  g->pl_box.assign(6 * g->placed.size(), 0.f);
  for (size_t pv = 0; pv < g->placed.size(); ++pv) {
    float *o = &g->pl_box[6 * pv];
    double b[6];
    if (!shape_bbox(g, g->placed[pv].unplaced, b)) {
      for (int k = 0; k < 3; ++k) {
        o[k] = -3.0e38f;
        o[3 + k] = 3.0e38f;
      }
      continue;
    }
    const RawXform &x = g->raw_xforms[g->placed[pv].raw_xform];
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int c = 0; c < 8; ++c) {
      const double l[3] = {b[(c & 1) ? 3 : 0], b[(c & 2) ? 4 : 1], b[(c & 4) ? 5 : 2]};
      for (int k = 0; k < 3; ++k) {
        const double m = x.t[k] + l[0] * x.r[3 * k] + l[1] * x.r[3 * k + 1] + l[2] * x.r[3 * k + 2];
        lo[k] = std::min(lo[k], m);
        hi[k] = std::max(hi[k], m);
      }
    }
    double ext = 0.;
    for (int k = 0; k < 3; ++k) ext = std::max(ext, std::max(std::fabs(lo[k]), std::fabs(hi[k])));
    const double pad = 1e-3 + 1e-5 * ext;
    for (int k = 0; k < 3; ++k) {
      o[k] = std::nextafter((float)(lo[k] - pad), -3.0e38f);
      o[3 + k] = std::nextafter((float)(hi[k] + pad), 3.0e38f);
    }
  }
  // ABBoxManager::ComputeABBox (source/ABBoxManager.cpp:128-161): the 8 corners
  // of the shape's Extent, moved to the mother's frame with InverseTransform
  // (base/Transformation3D.h:598-632), their min / max (std::min, std::max, in
  // the reference's corner order) widened by 1e-3; InitABBoxes
  // (:185-262) keeps a float copy for the navigator's hit test
  g->abbox_ok = true;
  g->ab_box_d.assign(6 * g->placed.size(), 0.);
  g->ab_box.assign(6 * g->placed.size(), 0.f);
  for (size_t pv = 0; pv < g->placed.size(); ++pv) {
    const UnplacedRec &u = g->unplaced[g->placed[pv].unplaced];
    double lo[3], hi[3];
    if (!reference_extent(u.type, g->params.data() + u.param_off, lo, hi)) {
      // the reference's VPlacedVolume::Extent asserts for this shape
      // (volumes/PlacedVolume.h:260-263); its volumes get no box and the ABBox
      // navigator refuses the geometry
      g->abbox_ok = false;
      for (int k = 0; k < 6; ++k) g->ab_box_d[6 * pv + k] = std::numeric_limits<double>::quiet_NaN();
      continue;
    }
    const RawXform &x = g->raw_xforms[g->placed[pv].raw_xform];
    const double delta[3] = {hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]};
    double mn[3], mx[3];
    for (int k = 0; k < 3; ++k) {
      mn[k] = std::numeric_limits<double>::infinity();
      mx[k] = -std::numeric_limits<double>::infinity();
    }
    for (int cx = 0; cx <= 1; ++cx)
      for (int cy = 0; cy <= 1; ++cy)
        for (int cz = 0; cz <= 1; ++cz) {
          const double c[3] = {lo[0] + cx * delta[0], lo[1] + cy * delta[1], lo[2] + cz * delta[2]};
          for (int k = 0; k < 3; ++k) {
            double m = x.t[k];
            m = m + c[0] * x.r[3 * k];
            m = m + c[1] * x.r[3 * k + 1];
            m = m + c[2] * x.r[3 * k + 2];
            mn[k] = vmin(mn[k], m);
            mx[k] = vmax(mx[k], m);
          }
        }
    for (int k = 0; k < 3; ++k) {
      g->ab_box_d[6 * pv + k] = mn[k] - 1E-3;
      g->ab_box_d[6 * pv + 3 + k] = mx[k] + 1E-3;
    }
    for (int k = 0; k < 6; ++k) g->ab_box[6 * pv + k] = (float)g->ab_box_d[6 * pv + k];
  }
  // the navigator reads the boxes of a volume's daughters in daughter order
  g->ab_slot.assign(2 * g->daughters.size(), float4{0.f, 0.f, 0.f, 0.f});
  for (size_t k = 0; k < g->daughters.size(); ++k) {
    const float *b = &g->ab_box[6 * (size_t)g->daughters[k]];
    g->ab_slot[2 * k] = float4{b[0], b[1], b[2], 0.f};
    g->ab_slot[2 * k + 1] = float4{b[3], b[4], b[5], 0.f};
  }
  mark_bounded(g);
  build_wide(g);
  return VGB_OK;
}

extern "C" {

vgb_status vgb_geometry_close(vgb_geometry *g) {
  VGB_CHECK_OPEN(g);
  vgb_status s0 = prepare_tables(g);
  if (s0 != VGB_OK) return s0;
  // shape records that hold device pointers are fixed up after the pool lands
  cudaError_t e = cudaGetDevice(&g->device);
  if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: cudaGetDevice");
  vgb_status s;
  {
    // allocate the pool, let shape records that reference other parts of the
    // pool store device addresses, then copy it
    const size_t n = g->params.empty() ? 2 : g->params.size();
    e = cudaMalloc((void **)&g->dev.params, n * sizeof(double));
    if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: cudaMalloc");
    g->dev.bytes += (int64_t)(n * sizeof(double));
    if ((s = finalize_shapes(g)) != VGB_OK) return s;
    if (!g->params.empty()) {
      e = cudaMemcpy(g->dev.params, g->params.data(), g->params.size() * sizeof(double),
                     cudaMemcpyHostToDevice);
      if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: cudaMemcpy");
    }
  }
  if ((s = upload(g->unplaced, &g->dev.unplaced, &g->dev.bytes)) != VGB_OK) return s;
  if ((s = upload(g->xforms, &g->dev.xforms, &g->dev.bytes)) != VGB_OK) return s;
  if ((s = upload(g->nav_raw, &g->dev.raw, &g->dev.bytes)) != VGB_OK) return s;
  if ((s = upload(g->placed, &g->dev.placed, &g->dev.bytes)) != VGB_OK) return s;
  if ((s = upload(g->logicals, &g->dev.logicals, &g->dev.bytes)) != VGB_OK) return s;
  if ((s = upload(g->daughters, &g->dev.daughters, &g->dev.bytes)) != VGB_OK) return s;
  {
    const std::vector<uint32_t> zero(1, 0u);
    if ((s = upload(zero, &g->dev.nav_flags, &g->dev.bytes)) != VGB_OK) return s;
  }
  if ((s = upload(g->pl_box, &g->dev.pl_box, &g->dev.bytes)) != VGB_OK) return s;
  if ((s = upload(g->ab_box, &g->dev.ab_box, &g->dev.bytes)) != VGB_OK) return s;
  if ((s = upload(g->ab_slot, &g->dev.ab_slot, &g->dev.bytes)) != VGB_OK) return s;
  {
    // the navigator's tables, one allocation: what the host made in one copy, then
    // the records a kernel makes from the tables above
    std::vector<char> host;
    auto put = [&](const auto &v) {
      const size_t off = host.size(), bytes = v.size() * sizeof(v[0]);
      host.resize((off + bytes + 255) / 256 * 256);
      if (bytes) std::memcpy(host.data() + off, v.data(), bytes);
      return off;
    };
    const size_t o_bounded = put(g->bounded), o_screened = put(g->screened), o_grids = put(g->grids),
                 o_start = put(g->cell_start), o_items = put(g->cell_items);
    size_t bytes = host.size();
    auto room = [&](size_t n) {
      const size_t off = bytes;
      bytes += (n + 255) / 256 * 256;
      return off;
    };
    const size_t np = g->placed.size(), ns = g->daughters.size();
    const size_t o_vols = room(np * sizeof(NavVol)), o_slots = room(ns * sizeof(NavSlot)),
                 o_box = room(2 * ns * sizeof(float4));
    e = cudaMalloc((void **)&g->dev.nav_tables, bytes > 0 ? bytes : 1);
    if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: cudaMalloc");
    g->dev.bytes += (int64_t)bytes;
    char *base = g->dev.nav_tables;
    if (!host.empty()) {
      e = cudaMemcpy(base, host.data(), host.size(), cudaMemcpyHostToDevice);
      if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: cudaMemcpy");
    }
    g->dev.grids = reinterpret_cast<CellGrid *>(base + o_grids);
    g->dev.cell_start = reinterpret_cast<int32_t *>(base + o_start);
    g->dev.cell_items = reinterpret_cast<int32_t *>(base + o_items);
    g->dev.vols = reinterpret_cast<NavVol *>(base + o_vols);
    g->dev.slots = reinterpret_cast<NavSlot *>(base + o_slots);
    g->dev.slot_box = reinterpret_cast<float4 *>(base + o_box);
    if (np > 0) {
      const int grid = (int)std::min<size_t>((std::max(np, ns) + 255) / 256, 148 * 8);
      k_nav_records<<<grid, 256>>>(g->dev.placed, g->dev.unplaced, g->dev.logicals, g->dev.xforms,
                                   g->dev.daughters, g->dev.pl_box,
                                   reinterpret_cast<uint8_t *>(base + o_bounded),
                                   reinterpret_cast<uint8_t *>(base + o_screened), (int32_t)np,
                                   (int32_t)ns, g->dev.vols, g->dev.slots, g->dev.slot_box);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
      if (e != cudaSuccess) return cuda_error(e, "vgb_geometry_close: navigation records");
    }
  }
  g->closed = true;
  return VGB_OK;
}

vgb_status vgb_abbox_compute(const vgb_geometry *g, int32_t placed, double *lower_upper) {
  if (!g || !lower_upper) return set_error(VGB_EINVAL, "vgb_abbox_compute: NULL argument");
  if (placed < 0 || placed >= (int32_t)g->placed.size())
    return set_error(VGB_EINVAL, "vgb_abbox_compute: unknown placed volume %d", placed);
  vgb_geometry *gm = const_cast<vgb_geometry *>(g);
  if (!g->closed) {
    vgb_status s = prepare_tables(gm);
    if (s != VGB_OK) return s;
  }
  const UnplacedRec &u = g->unplaced[g->placed[placed].unplaced];
  double lo[3], hi[3];
  if (!reference_extent(u.type, g->params.data() + u.param_off, lo, hi))
    return set_error(VGB_ENOTSUP, "vgb_abbox_compute: shape type %d has no Extent in the reference",
                     u.type);
  for (int k = 0; k < 6; ++k) lower_upper[k] = g->ab_box_d[6 * (size_t)placed + k];
  return VGB_OK;
}

vgb_status vgb_geometry_max_depth(const vgb_geometry *g, int32_t *depth) {
  VGB_CHECK_G(g);
  if (!depth) return set_error(VGB_EINVAL, "vgb_geometry_max_depth: out pointer is NULL");
  *depth = g->max_depth;
  return VGB_OK;
}

vgb_status vgb_geometry_device_bytes(const vgb_geometry *g, int64_t *bytes) {
  VGB_CHECK_G(g);
  if (!bytes) return set_error(VGB_EINVAL, "vgb_geometry_device_bytes: out pointer is NULL");
  *bytes = g->dev.bytes;
  return VGB_OK;
}

}  // extern "C"

namespace vgb {
vgb_status finalize_shapes(vgb_geometry *g) {
  (void)g;
  return VGB_OK;
}
}  // namespace vgb

