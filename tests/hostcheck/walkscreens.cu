// walkscreens.cu -- test infrastructure: the polycone's and polyhedron's distances with
// and without the tests that pass sections and inner sides over, on the host.
#include <cstring>
#include <vector>

#include "../../vecgeom_b200/csrc/batch.cuh"
#include "../../vecgeom_b200/csrc/geometry.h"

using namespace vgb;

namespace {
// The polycone's reachability test written out for one section, with its divisions.
bool out_of_reach(const PolySec &s, const V3<double> &q, const V3<double> &v) {
  if (!(fabs(v.x * v.x + v.y * v.y + v.z * v.z - 1) < 1e-10)) return false;
  if (!(fabs(q.x) + fabs(q.y) + fabs(q.z) < Lim<double>::inf())) return false;
  const double dz = s.cone.dz, zc = s.shift, mz = 1e-3 + 1e-6 * (fabs(zc) + dz);
  const double zlo = zc - dz - mz, zhi = zc + dz + mz;
  const double rmax = vmax(s.cone.rmax1, s.cone.rmax2), rb = rmax + 1e-3 + 1e-6 * rmax;
  double t0 = 0, t1 = Lim<double>::inf();
  if (v.z != 0) {
    const double ta = (zlo - q.z) / v.z, tb = (zhi - q.z) / v.z;
    t0 = vmax(vmin(ta, tb), 0.);
    t1 = vmax(ta, tb);
    if (t0 > t1) return true;
  } else if (q.z < zlo || q.z > zhi) {
    return true;
  }
  const double a = v.x * v.x + v.y * v.y;
  double tm = a > 0 ? -(q.x * v.x + q.y * v.y) / a : 0.;
  tm = vmin(vmax(tm, t0), t1);
  const double x = q.x + tm * v.x, y = q.y + tm * v.y;
  return x * x + y * y > rb * rb;
}
}  // namespace

// op 2: DistanceToIn, 3: DistanceToOut, local frame; plain 1: nothing is passed over,
// 2: the sections that the test above rejects
extern "C" int ws_distance(const vgb_geometry *g, int32_t placed, int32_t op, int32_t plain,
                           int64_t n, const double *x, const double *y, const double *z,
                           const double *dx, const double *dy, const double *dz, double *out) {
  const UnplacedRec &u = g->unplaced[g->placed[placed].unplaced];
  std::vector<double> rec(g->params.begin() + u.param_off,
                          g->params.begin() + u.param_off + u.param_len);
  for (int64_t i = 0; i < n; ++i) {
    const V3<double> q = {x[i], y[i], z[i]}, v = {dx[i], dy[i], dz[i]};
    if (u.type == VGB_SHAPE_POLYCONE) {
      using O = PolyconeOps<double>;
      const PolyconeP p = bind_params(*reinterpret_cast<const PolyconeP *>(rec.data()), rec.data());
      if (op != 2) return -1;
      O::Walk w;
      double r;
      O::dti_begin(p, q, v, 1e30, w, r);
      if (plain) w.test = false;
      for (;;) {
        if (plain == 2 && out_of_reach(O::sec(p, w.index), q, v)) {
          w.distance = Lim<double>::inf();
          w.index += w.increment;
          if (!w.increment || !(w.index >= 0 && w.index < p.nsec)) break;
        } else if (O::dti_step(p, q, v, 1e30, w)) {
          break;
        }
      }
      out[i] = O::dti_end(p, q, v, 1e30, w);
    } else {
      using O = PolyhedronOps<double>;
      const PolyhedronP p =
          bind_params(*reinterpret_cast<const PolyhedronP *>(rec.data()), rec.data());
      PhSeg *segs = reinterpret_cast<PhSeg *>(rec.data() + p.seg_off);
      for (int k = 0; plain && k < p.nseg; ++k) segs[k].inner_r = 0.f;
      out[i] = op == 2 ? O::distance_to_in(p, q, v, 1e30) : O::distance_to_out(p, q, v, 1e30);
    }
  }
  return 0;
}
