"""The polycone's DistanceToIn from very far away, where the reachability test decides by
rounding: on the host, bit for bit, the walk with the test written out with its divisions."""
import numpy as np
import pytest

from test_walk_screens import SHAPES, ws  # noqa: F401 (the fixture)
from vecgeom_b200 import workloads as W


@pytest.mark.parametrize("name", sorted(k for k in SHAPES if k.startswith("polycone")))
def test_far_points_walk_the_same_sections(ws, name):
    from vecgeom_b200.geometry import Geometry
    spec = SHAPES[name]
    n = 120000
    rng = np.random.default_rng(7)
    wl = W.make_workload(spec, n, 9)
    d = np.array(W.isotropic(rng, n))
    d[2, : n // 3] *= 1e-3  # almost across the axis
    d /= np.sqrt((d ** 2).sum(0))
    p = np.ascontiguousarray(np.stack([wl.x, wl.y, wl.z]) - d * 10. ** rng.uniform(8., 30., n))
    d = np.ascontiguousarray(d)
    g = Geometry(library=ws)
    pv = g.LogicalVolume("s", W.build_unplaced(g, spec)).Place(g.Transformation3D())
    got = []
    for plain in (0, 2):
        out = np.zeros(n)
        assert ws.ws_distance(g.handle, pv.id, 2, plain, n, *(a.ctypes.data for a in (*p, *d)),
                              out.ctypes.data) == 0
        got.append(out)
    assert np.isfinite(got[0]).any()
    assert got[0].tobytes() == got[1].tobytes()
