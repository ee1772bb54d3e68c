"""The short forms of the correctly rounded sin, cos and atan2 (crmath.cuh): the same
doubles as the double-double series wherever they answer, and an error bound that holds
against 250-bit values."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(os.path.dirname(HERE), "_build", "hostcheck")


@pytest.fixture(scope="module")
def cs():
    so = os.path.join(OUT, "libvgb_crshort.so")
    os.makedirs(OUT, exist_ok=True)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-shared", "-o", so, os.path.join(HERE, "hostcheck", "crshort.cu")],
                   check=True, stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
    return ctypes.CDLL(so)


def p(a):
    return ctypes.c_void_p(a.ctypes.data)


def angles(kind, rng, n):
    if kind == "wide":
        return rng.uniform(-4.2, 4.2, n)
    if kind == "tiny":
        return rng.uniform(-1., 1., n) * 10. ** rng.uniform(-300., 0., n)
    # a few ulp around every multiple of pi/128: both ends of every table cell
    x = np.repeat(np.arange(-162, 163) * np.pi / 128, n // 325)
    for _ in range(3):
        x = np.nextafter(x, rng.choice([-10., 10.], len(x)))
    return x


@pytest.mark.parametrize("kind", ["wide", "tiny", "cells"])
def test_short_sincos_equals_the_series(cs, kind):
    x = angles(kind, np.random.default_rng(2), 300000)
    s, c, ss, sc = (np.zeros(len(x)) for _ in range(4))
    fell = np.zeros(1, np.int64)
    cs.cs_sincos(ctypes.c_int64(len(x)), p(x), p(s), p(c), p(ss), p(sc), p(fell))
    assert s.tobytes() == ss.tobytes() and c.tobytes() == sc.tobytes()
    if kind != "cells":  # the short form answers nearly always
        assert fell[0] < 0.01 * len(x)


@pytest.mark.parametrize("kind", ["wide", "tiny", "cells"])
def test_short_sincos_error_bound(cs, kind):
    mp = pytest.importorskip("mpmath")
    x = angles(kind, np.random.default_rng(3), 1300)
    x = np.ascontiguousarray(x[np.abs(x) < 4.0])
    out = np.zeros((len(x), 6))
    cs.cs_short(ctypes.c_int64(len(x)), p(x), p(out))
    with mp.workprec(1300):
        for v, (sh, sl, ch, cl, es, ec) in zip(x, out):
            v = mp.mpf(v)
            assert abs(mp.sin(v) - mp.mpf(sh) - mp.mpf(sl)) <= es
            assert abs(mp.cos(v) - mp.mpf(ch) - mp.mpf(cl)) <= ec


@pytest.mark.parametrize("spread", [0., 8., 200.])
def test_short_atan2_equals_the_series(cs, spread):
    rng = np.random.default_rng(4)
    n = 300000
    y, x = (rng.standard_normal(n) * 10. ** rng.uniform(-spread, spread, n) for _ in range(2))
    edge = np.array([0., -0., 1., -1., 5e-324, -5e-324, 1e308, -1e308, np.inf, -np.inf])
    ey, ex = (a.ravel() for a in np.meshgrid(edge, edge))
    y, x = np.concatenate([y, ey]), np.concatenate([x, ex])
    t, ts = np.zeros(len(y)), np.zeros(len(y))
    cs.cs_atan2(ctypes.c_int64(len(y)), p(y), p(x), p(t), p(ts))
    assert t.tobytes() == ts.tobytes()
