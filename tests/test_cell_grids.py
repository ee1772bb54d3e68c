"""The cell grids over the daughters of wide volumes: their tables grow with the
daughters, whatever the daughters' sizes, and searches through them find what the plain
scan of the daughters finds."""
import numpy as np
import pytest

import hostlib
from vecgeom_b200 import workloads as W

MOST = 32  # cells and list entries a daughter (kCellsPerDaughter)


@pytest.fixture(scope="module")
def cg():
    return hostlib.navsearch()


def build(cg, volumes, daughters, layout):
    """A world of `volumes` boxes side by side, each with the given number of daughter
    boxes: `sparse` ones of 2 mm, `shells` that fill their mother from the inside out, or
    `mixed`, as many small ones beside the shells."""
    from vecgeom_b200.geometry import Geometry
    g = Geometry(library=cg)
    b = W.VgbBuilder(g, close=False)
    rng = np.random.default_rng(daughters)
    world_lv = b.logical("world", b.box(600. * volumes, 600., 600.))
    world = b.place(world_lv, b.transform())
    dot = b.logical("dot", b.box(1., 1., 1.))
    for v in range(volumes):
        lv = b.logical(f"v{v}", b.box(500., 500., 500.))
        for k in range(daughters):
            if layout == "shells" or (layout == "mixed" and k % 2):
                h = 499. * (k + 1) / daughters
                b.place_daughter(lv, b.logical(f"s{v}_{k}", b.box(h, h, h)), b.transform())
            else:
                b.place_daughter(lv, dot, b.transform(*rng.uniform(-490., 490., 3)))
        b.place_daughter(world_lv, lv, b.transform(1200. * v - 600. * (volumes - 1), 0., 0.))
    b.set_world(world)
    return g


@pytest.mark.parametrize("layout", ["sparse", "shells", "mixed"])
@pytest.mark.parametrize("volumes,daughters", [(1, 33), (40, 33), (3, 500)])
def test_tables_grow_with_the_daughters(cg, volumes, daughters, layout):
    g = build(cg, volumes, daughters, layout)
    out = np.zeros(4, np.int64)
    assert cg.cg_sizes(g.handle, out.ctypes.data) == 0
    slots, grids, cells, entries = out
    assert grids <= volumes + 1
    assert cells <= MOST * slots + grids
    assert entries <= MOST * slots


@pytest.mark.parametrize("layout", ["sparse", "shells", "mixed"])
@pytest.mark.parametrize("daughters", [33, 64, 300])
def test_search_through_the_cells_equals_the_scan(cg, daughters, layout):
    n, m = 400, 24
    g = build(cg, 2, daughters, layout)
    rng = np.random.default_rng(4)
    p = np.ascontiguousarray(rng.uniform(-1., 1., (3, n)) * np.array([[1150.], [550.], [550.]]))
    d = np.ascontiguousarray(W.isotropic(rng, n))
    got = []
    for boxes in (0, 1):
        ids, ns = np.full(n * m, -7, np.int32), np.zeros(n, np.int32)
        st, sf = np.zeros(n * m), np.zeros(n * m)
        assert cg.nb_trace(g.handle, n, *(a.ctypes.data for a in (*p, *d)), boxes, 0, m,
                           ids.ctypes.data, st.ctypes.data, sf.ctypes.data, ns.ctypes.data) == 0
        got.append([a.tobytes() for a in (ids, ns, st, sf)])
    assert got[0] == got[1]
