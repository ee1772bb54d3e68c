"""The navigator's FP32+refine form gives the FP64 form's results whatever the daughters:
shapes whose answers their boxes do not bound (the torus moves directions as points),
placements that are not rigid motions, hits just behind the point, directions that are
not unit vectors; in calls of both of the GPU's forms."""
import numpy as np
import pytest

import hostlib
from vecgeom_b200 import workloads as W


@pytest.fixture(scope="module")
def rn():
    return hostlib.navsearch()


SPECS = {f"{s.kind}{k}": s for k, s in enumerate(W.zoo_specs() + W.zoo2_specs())}


def build(geometry, names, placement, close):
    """A world box with 24 shapes of the given kinds that may overlap."""
    b = W.VgbBuilder(geometry, close=close)
    rng = np.random.default_rng(3)
    world_lv = b.logical("world", b.box(800., 800., 800.))
    world = b.place(world_lv, b.transform())
    for k in range(24):
        rot = {"plain": (0., 0., 0.), "euler": tuple(rng.uniform(0., 360., 3)),
               "code 0x16A": (0., 30., 90.)}[placement]
        b.place_daughter(world_lv, b.logical(f"d{k}", b.shape(SPECS[names[k % len(names)]])),
                         b.transform(*rng.uniform(-300., 300., 3), *rot))
    b.set_world(world)
    b.close()


def tracks(n, scaled):
    rng = np.random.default_rng(8)
    d = np.array(W.isotropic(rng, n))
    if scaled:
        d *= rng.uniform(0.5, 2., n)
    return np.ascontiguousarray(rng.uniform(-400., 400., (3, n))), np.ascontiguousarray(d)


def host(rn, g, p, d, screen):
    n = p.shape[1]
    nxt, st, sf = np.zeros(n, np.int32), np.zeros(n), np.zeros(n)
    assert rn.rn_from_world(g.handle, n, *(a.ctypes.data for a in (*p, *d)), screen,
                            nxt.ctypes.data, st.ctypes.data, sf.ctypes.data) == 0
    return [a.tobytes() for a in (nxt, st, sf)]


@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("placement", ["plain", "euler", "code 0x16A"])
@pytest.mark.parametrize("name", [*sorted(SPECS), "all"])
def test_host_forms_agree(rn, name, placement, scaled):
    from vecgeom_b200.geometry import Geometry
    if placement == "code 0x16A" and (name == "all" or name.startswith("bool")):
        pytest.skip("the booleans' components want unit directions")
    g = Geometry(library=rn)
    build(g, sorted(SPECS) if name == "all" else [name], placement, False)
    p, d = tracks(4000, scaled)
    assert host(rn, g, p, d, 1) == host(rn, g, p, d, 0)


def test_host_a_hit_behind_the_point(rn):
    from vecgeom_b200.geometry import Geometry
    g = Geometry(library=rn)
    b = W.VgbBuilder(g, close=False)
    lv = b.logical("world", b.box(500., 500., 500.))
    world = b.place(lv, b.transform())
    b.place_daughter(lv, b.logical("a", b.box(10., 10., 10.)), b.transform())
    b.place_daughter(lv, b.logical("b", b.box(5., 5., 5.)), b.transform(10., 14.9, 0.))
    b.set_world(world)
    # its face is 0.5 behind the point along the ray; alone, and beside one the point is in
    p, d = np.array([[10. - 1e-10] * 2, [10.2, 10.6], [0., 9.]]), np.array([[-2e-10, -1e-10], [1., 1.], [0., 0.]])
    assert host(rn, g, p, d, 1) == host(rn, g, p, d, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3001, 41001])
@pytest.mark.parametrize("name", ["torus4", "all"])
def test_gpu_forms_agree(name, n):
    import torch

    import vecgeom_b200 as V
    g = V.Geometry()
    build(g, sorted(SPECS) if name == "all" else [name], "euler", True)
    P, D = (V.SOA3D(*(torch.from_numpy(a[j].copy()).cuda() for j in range(3)))
            for a in tracks(n, False))
    nav = V.SimpleNavigator(g)
    cur, nxt = V.NavStatePool(g, n), V.NavStatePool(g, n)
    nav.LocatePoint(P, cur)
    got = []
    for precision in (0, 1):
        far = torch.full((n,), 1e30, dtype=torch.float64, device="cuda")
        st, sf = torch.zeros_like(far), torch.zeros_like(far)
        nav.FindNextBoundaryAndStep(P, D, cur, nxt, far, st, sf, precision=precision)
        ns = torch.zeros(n, dtype=torch.int32, device="cuda")
        ts = torch.zeros(n, 8, dtype=torch.float64, device="cuda")
        tf = torch.zeros_like(ts)
        nav.Trace(P, D, 1e30, 8, ns, None, ts, tf, precision=precision)
        got.append([nxt.to_numpy().tobytes(), *(t.cpu().numpy().tobytes() for t in (st, sf, ns, ts, tf))])
    assert got[0] == got[1]
