// navboxes.cu -- test infrastructure: the navigator's searches through the daughters'
// boxes and cells (navigation.cuh search, search_wide, cell_list), which the GPU's
// warps use, run on the host with a single lane over a geometry's own tables, so the
// tests can compare them with the plain scan of the daughters (hc_nav_trace).
#include <vector>

#include "../../vecgeom_b200/csrc/geometry.h"
#include "../../vecgeom_b200/csrc/navigation.cuh"

using namespace vgb;

namespace {
struct BoxLane : OneLane {
  static constexpr bool kBoxes = true;
  static int32_t *scratch() {
    static thread_local int32_t buf[64];
    return buf;
  }
};
}  // namespace

// The trace of hc_nav_trace; basket: every step as the basket form takes it (pstep
// infinite), its node index in place of the safety.
extern "C" int nb_trace(vgb_geometry *g, int64_t n, const double *x, const double *y,
                        const double *z, const double *dx, const double *dy, const double *dz,
                        int32_t boxes, int32_t basket, int32_t max_steps, int32_t *next_ids,
                        double *steps, double *safeties, int32_t *nsteps) {
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
  using Nav = Navigator<BoxLane, kNavMaskAll>;
  for (int64_t i = 0; i < n; ++i) {
    V3<double> p = {x[i], y[i], z[i]};
    const V3<double> d = {dx[i], dy[i], dz[i]};
    NavPath cur;
    bool ok = Nav::locate_from_world(G, cur, p);
    int32_t k = 0;
    while (ok && cur.level > 0 && k < max_steps) {
      const DXform m = nav_top_matrix(G, cur);
      const V3<double> lp = xf_point(m, p), ld = xf_dir(m, d);
      double st = 0., sf = 0.;
      int32_t node = 0;
      if (basket) {
        ok = Nav::safety_and_step_basket(G, cur, cur, lp, ld, Lim<double>::inf(), true, sf, st, node);
        if (!(st < Lim<double>::inf())) ok = false;
      } else {
        ok = Nav::safety_and_step(G, cur, cur, lp, ld, 1e30, sf, st);
      }
      if (!ok) break;
      const int64_t r = i * (int64_t)max_steps + k;
      next_ids[r] = basket ? 2 * cur.top() + (node & 1) : cur.top();
      steps[r] = st;
      safeties[r] = sf;
      p = {p.x + d.x * st, p.y + d.y * st, p.z + d.z * st};
      ++k;
    }
    nsteps[i] = ok ? k : -1 - k;
  }
  return 0;
}
