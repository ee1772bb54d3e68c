"""The search of a wide volume's daughters by a warp (navigation.cuh search_wide).
CPU, one lane: only the answers asked for are evaluated.  GPU: the queue of a warp, at
numbers of daughters about multiples of 32, against the host's scan of all of them."""
import numpy as np
import pytest

import hostlib
from vecgeom_b200 import workloads as W


@pytest.fixture(scope="module")
def ws():
    return hostlib.navsearch()


def build(geometry, specs, count, close):
    """A world box with `count` shapes of the given kinds on a 5 x 5 x 5 lattice."""
    b = W.VgbBuilder(geometry, close=close)
    rng = np.random.default_rng(count)
    world_lv = b.logical("world", b.box(800., 800., 800.))
    world = b.place(world_lv, b.transform())
    lvs = [b.logical(f"c{k}", b.shape(s)) for k, s in enumerate(specs)]
    for c, cell in enumerate(rng.permutation(125)[:count]):
        pos = np.array([cell // 25, cell // 5 % 5, cell % 5]) * 280. - 560.
        b.place_daughter(world_lv, lvs[c % len(lvs)],
                         b.transform(*(pos + rng.uniform(-5., 5., 3)), *rng.uniform(0., 360., 3)))
    b.set_world(world)
    b.close()


KINDS = {"boxes": lambda: [W.box_spec(30., 40., 50.), W.tube_spec(10., 60., 70., 0., 4.)],
         "crowd": lambda: W.zoo_specs() + W.zoo2_specs()}


def points(n, seed=1):
    rng = np.random.default_rng(seed)
    return (np.ascontiguousarray(rng.uniform(-790., 790., (3, n))),
            np.ascontiguousarray(W.isotropic(rng, n)))


def from_world(ws, g, p, d, boxes, what, pstep=1e30):
    n = p.shape[1]
    nxt, st, sf, c = np.zeros(n, np.int32), np.zeros(n), np.zeros(n), np.zeros(2, np.int64)
    assert ws.ws_from_world(g.handle, n, *(a.ctypes.data for a in (*p, *d)), boxes, what, pstep,
                            nxt.ctypes.data, st.ctypes.data, sf.ctypes.data, c.ctypes.data) == 0
    return [a.tobytes() for a in (nxt, st, sf)], c


@pytest.mark.parametrize("what", [0, 1, 2, 3])
@pytest.mark.parametrize("count", [33, 125])
@pytest.mark.parametrize("kinds", sorted(KINDS))
def test_only_what_is_asked_for_is_evaluated(ws, kinds, count, what):
    from vecgeom_b200.geometry import Geometry
    g = Geometry(library=ws)
    build(g, KINDS[kinds](), count, False)
    p, d = points(300)
    (want, every), (got, some) = (from_world(ws, g, p, d, boxes, what) for boxes in (0, 1))
    assert got == want
    assert (some <= every).all()
    if what == 0:
        assert some[1] == 0
    if what == 1:
        assert some[0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("count", [33, 63, 64, 65, 97, 125])
@pytest.mark.parametrize("kinds", sorted(KINDS))
def test_gpu_warps_equal_the_hosts_scan(ws, kinds, count):
    import torch

    import vecgeom_b200 as V
    n, m = 700, 16
    p, d = points(n, count)
    host = V.Geometry(library=ws)
    build(host, KINDS[kinds](), count, False)
    ids, ns = np.full(n * m, -7, np.int32), np.zeros(n, np.int32)
    st, sf = np.zeros(n * m), np.zeros(n * m)
    assert ws.nb_trace(host.handle, n, *(a.ctypes.data for a in (*p, *d)), 0, 0, m, ids.ctypes.data,
                       st.ctypes.data, sf.ctypes.data, ns.ctypes.data) == 0
    g = V.Geometry()
    build(g, KINDS[kinds](), count, True)
    P, D = (V.SOA3D(*(torch.from_numpy(a[j]).cuda() for j in range(3))) for a in (p, d))
    t_ns = torch.zeros(n, dtype=torch.int32, device="cuda")
    t_ids = torch.full((n, m), -7, dtype=torch.int32, device="cuda")
    t_st = torch.zeros(n, m, dtype=torch.float64, device="cuda")
    t_sf = torch.zeros_like(t_st)
    V.SimpleNavigator(g).Trace(P, D, 1e30, m, t_ns, t_ids, t_st, t_sf)
    for got, want in ((t_ns, ns), (t_ids, ids), (t_st, st), (t_sf, sf)):
        assert got.cpu().numpy().tobytes() == want.tobytes()
    if kinds == "boxes":  # the ABBox navigator's GetSafety asks for safeties alone
        V.ABBoxNavigator(g).Trace(P, D, 1e30, m, t_ns, t_ids, t_st, t_sf)
        k = ns.clip(0, 1) == 1
        assert np.array_equal(t_sf.cpu().numpy()[k, 0], sf.reshape(n, m)[k, 0])
