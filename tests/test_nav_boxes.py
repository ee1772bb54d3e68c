"""The navigator's searches through the daughters' boxes and cells, and its two forms
on the GPU (a warp or a thread per track).

CPU: the box searches of navigation.cuh, run on the host with one lane, against the
plain scan of every daughter (the same host code without box tables), bit for bit, in
geometries whose volumes hold few daughters, hundreds of boxes, and wide volumes of
mixed kinds (some without a usable box), with unit directions, directions along the
axes, and directions that are not unit vectors.
GPU: a batch large enough to run by threads against the same tracks in batches small
enough to run by warps, bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from vecgeom_b200 import _lib
from vecgeom_b200 import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "vecgeom_b200", "csrc")
OUT = os.path.join(os.path.dirname(HERE), "_build", "hostcheck")


@pytest.fixture(scope="module")
def nb():
    so = os.path.join(OUT, "libvgb_navboxes.so")
    os.makedirs(OUT, exist_ok=True)
    srcs = [os.path.join(HERE, "hostcheck", "navboxes.cu")] + [
        os.path.join(SRC, f) for f in ("geometry.cu", "unplaced.cu", "geometry_io.cu")]
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-shared", "-o", so, *srcs, "-lcudart"], check=True,
                   stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
    L = ctypes.CDLL(so)
    for name, (res, args) in _lib.SIGNATURES.items():
        f = getattr(L, name, None)
        if f is not None:
            f.restype, f.argtypes = res, args
    vp = ctypes.c_void_p
    L.nb_trace.argtypes = ([vp, ctypes.c_int64] + [vp] * 6 + [ctypes.c_int32] * 3 + [vp] * 4)
    return L


def build_crowd(b, specs, seed=3):
    """A world box holding 4 x 4 x 4 shapes of the given kinds (a wide volume), each
    at its own rotation; every fourth one is unrotated, so faces lie along axes."""
    rng = np.random.default_rng(seed)
    world_lv = b.logical("world", b.box(800., 800., 800.))
    world = b.place(world_lv, b.transform())
    lvs = [b.logical(f"c{k}", b.shape(s)) for k, s in enumerate(specs)]
    placed = [world]
    c = 0
    for i in range(4):
        for j in range(4):
            for k in range(4):
                rot = (0., 0., 0.) if c % 4 == 0 else tuple(rng.uniform(0., 360., 3))
                pos = np.array([i, j, k]) * 280. - 420. + rng.uniform(-5., 5., 3)
                placed.append(b.place_daughter(world_lv, lvs[c % len(lvs)],
                                               b.transform(*pos, *rot)))
                c += 1
    b.set_world(world)
    b.close()
    return placed


def build(geometry, name, close):
    b = W.VgbBuilder(geometry, close=close)
    if name == "detector":
        return W.build_detector(b)
    if name == "zoo":
        return W.build_zoo(b, W.zoo_specs())
    if name == "zoo2":
        return W.build_zoo(b, W.zoo2_specs())
    if name == "boxes":
        return build_crowd(b, [W.box_spec(30., 40., 50.), W.tube_spec(10., 60., 70., 0., 4.)])
    return build_crowd(b, W.zoo_specs() + W.zoo2_specs())  # "crowd": mixed, some unbounded


def tracks(name, n, seed, directions):
    rng = np.random.default_rng(seed)
    if name == "detector":
        p = rng.uniform(-1., 1., (3, n)) * np.array([[1100.], [1100.], [1250.]])
        p[:, : n // 4] = 0.
    elif name in ("boxes", "crowd"):
        p = rng.uniform(-700., 700., (3, n))
    else:
        p = np.array(W.zoo_tracks(n, seed)[0])
    d = np.array(W.isotropic(rng, n))
    if directions == "axis":
        d = np.zeros((3, n))
        d[rng.integers(0, 3, n), np.arange(n)] = rng.choice([-1., 1.], n)
    elif directions == "scaled":
        d *= rng.uniform(0.5, 2., n)
    elif directions == "grazing":  # almost along an axis: tiny components
        d = rng.uniform(-1., 1., (3, n)) * 10. ** rng.uniform(-16., -6., (3, n))
        d[rng.integers(0, 3, n), np.arange(n)] = 1.
    return np.ascontiguousarray(p), np.ascontiguousarray(d)


@pytest.mark.parametrize("directions", ["unit", "axis", "grazing", "scaled"])
@pytest.mark.parametrize("basket", [0, 1])
@pytest.mark.parametrize("name", ["detector", "zoo", "zoo2", "boxes", "crowd"])
def test_box_search_equals_the_scan(nb, name, basket, directions):
    from vecgeom_b200.geometry import Geometry
    n, m = 600, 24
    p, d = tracks(name, n, 11, directions)
    g = Geometry(library=nb)
    build(g, name, close=False)
    got = []
    for boxes in (0, 1):
        ids, ns = np.full(n * m, -7, np.int32), np.zeros(n, np.int32)
        st, sf = np.zeros(n * m), np.zeros(n * m)
        assert nb.nb_trace(g.handle, n, *(a.ctypes.data for a in (*p, *d)), boxes, basket, m,
                           ids.ctypes.data, st.ctypes.data, sf.ctypes.data, ns.ctypes.data) == 0
        got.append([a.tobytes() for a in (ids, ns, st, sf)])
    assert got[0] == got[1]


# one track past the sizes from which every call runs by threads
LARGE = 40961


@pytest.mark.gpu
@pytest.mark.parametrize("navigator", ["simple", "basket", "abbox"])
@pytest.mark.parametrize("name", ["detector", "zoo", "boxes", "crowd"])
def test_gpu_threads_equal_warps(name, navigator):
    import torch

    import vecgeom_b200 as V
    if navigator == "abbox" and name == "crowd":
        pytest.skip("a parallelepiped has no aligned box")
    g = V.Geometry()
    build(g, name, close=True)
    n, m = LARGE, 12
    p, d = (torch.from_numpy(a).cuda() for a in tracks(name, n, 5, "unit"))
    nav = V.ABBoxNavigator(g) if navigator == "abbox" else V.SimpleNavigator(g)

    def step(a, b):
        k = b - a
        P, D = (V.SOA3D(*(v[j, a:b].contiguous() for j in range(3))) for v in (p, d))
        cur, nxt = V.NavStatePool(g, k), V.NavStatePool(g, k)
        far = torch.full((k,), 1e30, dtype=torch.float64, device="cuda")
        st, sf = torch.zeros_like(far), torch.zeros_like(far)
        node = torch.zeros(k, dtype=torch.int32, device="cuda")
        nav.LocatePoint(P, cur)
        if navigator == "basket":
            nav.FindNextBoundaryAndStepBasket(P, D, cur, nxt, far, st, sf, node)
        else:
            nav.FindNextBoundaryAndStep(P, D, cur, nxt, far, st, sf)
        return [cur.to_numpy().view(np.uint8).reshape(k, -1), nxt.to_numpy().view(np.uint8).reshape(k, -1),
                st.cpu().numpy(), sf.cpu().numpy(), node.cpu().numpy()]

    def trace(a, b):
        k = b - a
        P, D = (V.SOA3D(*(v[j, a:b].contiguous() for j in range(3))) for v in (p, d))
        ns = torch.zeros(k, dtype=torch.int32, device="cuda")
        ids = torch.full((k, m), -7, dtype=torch.int32, device="cuda")
        st = torch.zeros(k, m, dtype=torch.float64, device="cuda")
        sf = torch.zeros_like(st)
        nav.Trace(P, D, 1e30, m, ns, ids, st, sf)
        return [t.cpu().numpy() for t in (ns, ids, st, sf)]

    for call in (step,) if navigator == "basket" else (step, trace):
        whole = call(0, n)
        cuts = list(range(0, n, 2500)) + [n]
        parts = [call(a, b) for a, b in zip(cuts[:-1], cuts[1:])]
        for k, w in enumerate(whole):
            assert w.tobytes() == np.concatenate([q[k] for q in parts]).tobytes(), (call, k)
    assert nav.error_flags() == 0
