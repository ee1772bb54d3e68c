// cellgrids.cu -- test infrastructure: the sizes of the cell grids that prepare_tables
// makes over the daughters of wide volumes, beside the searches through them.
#include "navboxes.cuh"

// out: daughter slots, grids, entries of the start table, entries of the lists
extern "C" int cg_sizes(vgb_geometry *g, int64_t *out) {
  if (prepare_tables(g) != VGB_OK) return -1;
  out[0] = (int64_t)g->daughters.size();
  out[1] = (int64_t)g->grids.size();
  out[2] = (int64_t)g->cell_start.size();
  out[3] = (int64_t)g->cell_items.size();
  return 0;
}
