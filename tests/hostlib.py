"""A host library of the navigator's searches (hostcheck/navsearch.cu), built once a run."""
import ctypes
import functools
import os
import subprocess

from vecgeom_b200 import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "vecgeom_b200", "csrc")
OUT = os.path.join(os.path.dirname(HERE), "_build", "hostcheck")


@functools.lru_cache(maxsize=None)
def navsearch():
    so = os.path.join(OUT, "libvgb_navsearch.so")
    os.makedirs(OUT, exist_ok=True)
    srcs = [os.path.join(HERE, "hostcheck", "navsearch.cu")] + [
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
    vp, i32, i64 = ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64
    L.nb_trace.argtypes = [vp, i64] + [vp] * 6 + [i32] * 3 + [vp] * 4
    L.cg_sizes.argtypes = [vp, vp]
    L.rn_from_world.argtypes = [vp, i64] + [vp] * 6 + [i32] + [vp] * 3
    L.ws_from_world.argtypes = [vp, i64] + [vp] * 6 + [i32] * 2 + [ctypes.c_double] + [vp] * 4
    return L
