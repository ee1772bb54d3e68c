// widesearch.cu -- test infrastructure: the search of a wide volume's daughters from a
// given point of the world, with the shape calls it makes counted.
#include "navboxes.cuh"

namespace {
constexpr uint32_t kCounted = kNavMaskAll | (1u << 31);
int64_t calls[2];  // SafetyToIn, DistanceToIn
}  // namespace

namespace vgb {
template <> struct NavKernels<kCounted> : NavKernels<kNavMaskAll> {
  using B = NavKernels<kNavMaskAll>;
  static R distance_to_in(const NavGeom &G, int type, int32_t off, const V3<R> &l, const V3<R> &v,
                          R smax) {
    ++calls[1];
    return B::distance_to_in(G, type, off, l, v, smax);
  }
  static R safety_to_in(const NavGeom &G, int type, int32_t off, const V3<R> &l) {
    ++calls[0];
    return B::safety_to_in(G, type, off, l);
  }
};
}  // namespace vgb

// GetSafety (what 0), FindNextBoundaryAndStep (1), both at once (2) or the basket form of
// both (3) of points taken to be in the world volume itself.  next: the id stepped to.
extern "C" int ws_from_world(vgb_geometry *g, int64_t n, const double *x, const double *y,
                             const double *z, const double *dx, const double *dy,
                             const double *dz, int32_t boxes, int32_t what, double pstep,
                             int32_t *next, double *step, double *safety, int64_t *counts) {
  if (prepare_tables(g) != VGB_OK) return -1;
  NavGeom G = {g->params.data(),    g->unplaced.data(), g->placed.data(),
               g->xforms.data(),    g->nav_raw.data(),  g->logicals.data(),
               g->daughters.data(), g->pl_box.data(),   g->ab_box.data(),
               g->ab_slot.data(),   g->world,           g->max_depth};
  std::vector<float4> slot_box;
  for (int32_t pv : g->daughters) {
    const SlotBox b = slot_box_of(&g->pl_box[6 * (size_t)pv], g->bounded[pv] != 0);
    slot_box.push_back(b.lo);
    slot_box.push_back(b.hi);
  }
  if (boxes) {
    G.slot_box = slot_box.data();
    G.grids = g->grids.data();
    G.cell_start = g->cell_start.data();
    G.cell_items = g->cell_items.data();
  }
  using Nav = Navigator<BoxLane, kCounted>;
  calls[0] = calls[1] = 0;
  for (int64_t i = 0; i < n; ++i) {
    const V3<double> p = {x[i], y[i], z[i]}, d = {dx[i], dy[i], dz[i]};
    NavPath cur, nxt;
    cur.level = 0;
    cur.boundary = false;
    for (int32_t &v : cur.v) v = -1;
    cur.push(g->world);
    nxt = cur;
    int32_t node = 0;
    bool ok = true;
    step[i] = safety[i] = 0.;
    if (what == 0) safety[i] = Nav::safety(G, cur, p);
    if (what == 1) ok = Nav::step(G, cur, nxt, p, d, pstep, step[i]);
    if (what == 2) ok = Nav::safety_and_step(G, cur, nxt, p, d, pstep, safety[i], step[i]);
    if (what == 3)
      ok = Nav::safety_and_step_basket(G, cur, nxt, p, d, pstep, true, safety[i], step[i], node);
    next[i] = ok ? 1000 * node + nxt.top() : -99;
  }
  counts[0] = calls[0];
  counts[1] = calls[1];
  return 0;
}
