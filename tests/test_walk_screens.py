"""The tests by which the polycone's DistanceToIn passes sections over and the
polyhedron's distances pass inner sides over, against the same walks without them, bit
for bit on the host (from far away, where the cone's roots lose their digits, the
polycone against the test written out with its divisions): shapes with and without an inner radius, phi cuts, pointed inner
surfaces; unit directions, directions along and almost along the axes, directions that
are not unit vectors, and far points."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

from vecgeom_b200 import _lib
from vecgeom_b200 import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "vecgeom_b200", "csrc")
OUT = os.path.join(os.path.dirname(HERE), "_build", "hostcheck")

SHAPES = {
    **{k: v for k, v in W.config3_shapes().items() if k in ("polycone", "polyhedron")},
    "polycone_full": W.polycone_spec(0.4, 2 * math.pi, [-40., -10., 20., 60.], [0., 0., 5., 5.],
                                     [20., 30., 30., 10.]),
    "polycone_one": W.polycone_spec(0., 2., [-5., 5.], [1., 2.], [3., 4.]),
    "polyhedron_varying": W.polyhedron_spec(20., 360., 5, [-50., -10., 0., 30., 60.],
                                            [2., 5., 20., 20., 3.], [30., 40., 45., 45., 20.]),
    "polyhedron_cut": W.polyhedron_spec(0., 200., 6, [-50., -10., 30., 60.], [5., 10., 20., 3.],
                                        [30., 40., 45., 20.]),
    "polyhedron_solid": W.polyhedron_spec(0., 360., 4, [-10., 10.], [0., 0.], [10., 12.]),
}


@pytest.fixture(scope="module")
def ws():
    so = os.path.join(OUT, "libvgb_walkscreens.so")
    os.makedirs(OUT, exist_ok=True)
    srcs = [os.path.join(HERE, "hostcheck", "walkscreens.cu")] + [
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
    vp, i32 = ctypes.c_void_p, ctypes.c_int32
    L.ws_distance.argtypes = [vp, i32, i32, i32, ctypes.c_int64] + [vp] * 7
    return L


@pytest.mark.parametrize("directions", ["unit", "axis", "grazing", "scaled", "far"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_walks_equal_the_plain_walks(ws, name, directions):
    from vecgeom_b200.geometry import Geometry
    spec = SHAPES[name]
    n = 40000
    rng = np.random.default_rng(6)
    wl = W.make_workload(spec, n, 9)
    p = np.stack([wl.x, wl.y, wl.z])
    d = np.stack([wl.dx, wl.dy, wl.dz])
    if directions == "axis":
        d = np.zeros((3, n))
        d[rng.integers(0, 3, n), np.arange(n)] = rng.choice([-1., 1.], n)
    elif directions == "grazing":
        d = rng.uniform(-1., 1., (3, n)) * 10. ** rng.uniform(-16., -3., (3, n))
        d[rng.integers(0, 3, n), np.arange(n)] = 1.
    elif directions == "scaled":
        d = d * rng.uniform(0.5, 2., n)
    elif directions == "far":  # from far away, aimed at the shape
        p = p - d * 10. ** rng.uniform(2., 10., n)
    p, d = np.ascontiguousarray(p), np.ascontiguousarray(d)
    g = Geometry(library=ws)
    pv = g.LogicalVolume("s", W.build_unplaced(g, spec)).Place(g.Transformation3D())
    for op in (2,) if spec.kind == "polycone" else (2, 3):
        got = []
        for plain in (0, 2 if directions == "far" else 1):
            out = np.zeros(n)
            assert ws.ws_distance(g.handle, pv.id, op, plain, n, *(a.ctypes.data for a in (*p, *d)),
                                  out.ctypes.data) == 0
            got.append(out)
        assert got[0].tobytes() == got[1].tobytes(), op
