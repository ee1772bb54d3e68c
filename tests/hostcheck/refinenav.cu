// refinenav.cu -- test infrastructure: a step from the world volume by the FP64 and the
// FP32+refine form of the navigator, with the daughters' boxes, on the host.
#include "navboxes.cuh"

template <bool kScreen>
static void from_world(const NavGeom &G, const V3<double> &p, const V3<double> &d, int32_t &next,
                       double &step, double &safety) {
  using Nav = Navigator<BoxLane, kNavMaskAll, kScreen>;
  NavPath cur, nxt;
  cur.level = 0;
  cur.boundary = false;
  for (int32_t &v : cur.v) v = -1;
  cur.push(G.world);
  next = Nav::safety_and_step(G, cur, nxt, p, d, 1e30, safety, step) ? nxt.top() : -99;
}

extern "C" int rn_from_world(vgb_geometry *g, int64_t n, const double *x, const double *y,
                             const double *z, const double *dx, const double *dy,
                             const double *dz, int32_t screen, int32_t *next, double *step,
                             double *safety) {
  if (prepare_tables(g) != VGB_OK) return -1;
  NavGeom G = {g->params.data(),    g->unplaced.data(), g->placed.data(),
               g->xforms.data(),    g->nav_raw.data(),  g->logicals.data(),
               g->daughters.data(), g->pl_box.data(),   g->ab_box.data(),
               g->ab_slot.data(),   g->world,           g->max_depth};
  std::vector<float4> slot_box;
  for (int32_t pv : g->daughters) {
    SlotBox b = slot_box_of(&g->pl_box[6 * (size_t)pv], g->bounded[pv] != 0);
    b.lo.w = g->screened[pv] && !g->bounded[pv] ? 1.f : 0.f;
    slot_box.push_back(b.lo);
    slot_box.push_back(b.hi);
  }
  if (screen) G.slot_box = slot_box.data();
  for (int64_t i = 0; i < n; ++i) {
    const V3<double> p = {x[i], y[i], z[i]}, d = {dx[i], dy[i], dz[i]};
    if (screen)
      from_world<true>(G, p, d, next[i], step[i], safety[i]);
    else
      from_world<false>(G, p, d, next[i], step[i], safety[i]);
  }
  return 0;
}
