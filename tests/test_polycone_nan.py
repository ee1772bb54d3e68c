"""A point whose z is not a number is in no section of a polycone: Contains and Inside
answer outside without reading a section."""
import numpy as np
import pytest

from test_hostcheck import hc, host_run  # noqa: F401 (the fixture)
from vecgeom_b200 import workloads as W

SPEC = W.polycone_spec(0., 6.283185307179586, [-40., -10., 20., 60.], [0., 0., 5., 5.],
                       [20., 30., 30., 10.])


def points(n=4000):
    rng = np.random.default_rng(1)
    p = rng.uniform(-30., 30., (3, n))
    p[2] = np.nan
    return [np.ascontiguousarray(a) for a in p]


def test_host(hc):
    from vecgeom_b200.geometry import Geometry
    g = Geometry(library=hc)
    # records before the polycone's, as a read before its sections would find them
    for k in range(20):
        g.UnplacedCone(0., 50. + k, 0., 50. + k, 50., 0., 6.283185307179586)
    pv = g.LogicalVolume("p", W.build_unplaced(g, SPEC)).Place(g.Transformation3D())
    assert not host_run(hc, g, pv, 0, points()).any()
    assert (host_run(hc, g, pv, 1, points()) == 2).all()


@pytest.mark.gpu
def test_gpu():
    import torch

    import vecgeom_b200 as V
    g = V.Geometry()
    pv = g.LogicalVolume("p", W.build_unplaced(g, SPEC)).Place(g.Transformation3D())
    g.CloseGeometry()
    p = [torch.from_numpy(a).cuda() for a in points()]
    c = torch.ones(len(p[0]), dtype=torch.uint8, device="cuda")
    i = torch.zeros(len(p[0]), dtype=torch.int32, device="cuda")
    pv.Contains(V.SOA3D(*p), c)
    pv.Inside(V.SOA3D(*p), i)
    assert not c.any() and (i == 2).all()
