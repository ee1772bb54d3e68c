"""The native call of PlacedVolume.batch (csrc/pycall.cpp): what it hands to the library,
and that it leaves everything but plain, contiguous, long enough tensors of the right
types to the general path (by returning None without calling)."""
import ctypes

import numpy as np
import pytest
import torch

from vecgeom_b200 import _lib

N = 7
FN = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_int32, ctypes.c_int32,
                      ctypes.c_int64, *[ctypes.c_void_p] * 9, ctypes.c_int32, ctypes.c_int32,
                      ctypes.c_void_p)


def f8(n=N):
    return torch.zeros(n, dtype=torch.float64)


@pytest.fixture
def call():
    if not __import__("os").path.exists(_lib.LIB_PATH.replace("libvgb", "_pycall")):
        pytest.skip("the library is not built here")
    seen = []

    @FN
    def fn(*args):
        seen.append(args)
        return 3
    addr = ctypes.cast(fn, ctypes.c_void_p).value

    def run(pts=None, dirs=None, step=None, out=None, aux=None, stream=None):
        seen.clear()
        pts = pts if pts is not None else [f8() for _ in range(3)]
        dirs = dirs if dirs is not None else [None] * 3
        out = out if out is not None else f8()
        st = _lib.pycall().batch(addr, addr, 0x1234, 5, 2, *pts, *dirs, step, out, aux, 9, 1, stream)
        run.keep = (pts, dirs, step, out, aux)
        return st, (seen[0] if seen else None)
    run.fn = fn
    return run


def test_arguments_arrive(call):
    dirs, step, aux = [f8() for _ in range(3)], f8(N + 2), torch.zeros(N, dtype=torch.int32)
    st, a = call(dirs=dirs, step=step, aux=aux, stream=0x77)
    pts, _, _, out, _ = call.keep
    assert st == 3
    assert a[:4] == (0x1234, 5, 2, N)
    assert list(a[4:13]) == [t.data_ptr() for t in (*pts, *dirs, step, out, aux)]
    assert a[13:] == (9, 1, 0x77)
    st, a = call()
    assert st == 3 and a[7:11] == (None,) * 4 and a[12] is None and a[15] is None


class Sub(torch.Tensor):
    pass


@pytest.mark.parametrize("bad", [
    lambda: f8(2 * N)[::2], lambda: f8(N - 1), lambda: f8(N + 1), lambda: f8().float(),
    lambda: np.zeros(N), lambda: f8().as_subclass(Sub), lambda: [0.] * N, lambda: None,
    lambda: torch.zeros((), dtype=torch.float64)])
@pytest.mark.parametrize("where", ["x", "z", "dx", "dz", "step", "out", "aux"])
def test_anything_else_is_left_to_the_general_path(call, where, bad):
    v = bad()
    pts, dirs = [f8() for _ in range(3)], [f8() for _ in range(3)]
    kw = dict(step=f8(), out=f8(), aux=torch.zeros(N, dtype=torch.int32))
    longer = v is not None and getattr(v, "shape", None) == (N + 1,)
    if where in kw:
        if v is None or where == "out" and isinstance(v, torch.Tensor) and v.dtype == torch.float32:
            return  # an absent step or aux, and any type of output, are plain calls
        if where == "aux" and isinstance(v, torch.Tensor) and v.dim():
            v = v.to(torch.int32) if v.is_contiguous() and not longer and len(v) < N else v
        if longer and where != "aux":
            return  # a longer step or output is a plain call
        kw[where] = v
    else:
        target = pts if where in "xz" else dirs
        if where == "dx" and v is None:
            return  # no directions
        target[0 if where in ("x", "dx") else 2] = v
        if where == "x" and isinstance(v, torch.Tensor) and v.dim() and len(v) == N - 1:
            pass  # the other components are longer than x: left to the general path
    st, a = call(pts=pts, dirs=dirs, **kw)
    assert st is None and a is None


def test_empty_batch_is_left_to_the_general_path(call):
    st, a = call(pts=[f8(0) for _ in range(3)], out=f8(0))
    assert st is None and a is None


@pytest.mark.gpu
def test_gpu_errors_are_the_general_paths(call):
    import vecgeom_b200 as V
    g = V.Geometry()
    pv = g.LogicalVolume("b", g.UnplacedBox(1., 2., 3.)).Place(g.Transformation3D())
    g.CloseGeometry()
    x = [torch.rand(100, dtype=torch.float64, device="cuda") for _ in range(6)]
    P, D = V.SOA3D(*x[:3]), V.SOA3D(*x[3:])
    out = torch.zeros(100, dtype=torch.float64, device="cuda")
    far = torch.full_like(out, 1e30)
    with pytest.raises(ValueError, match="contiguous"):
        pv.DistanceToIn(P, D, torch.zeros(200, dtype=torch.float64, device="cuda")[::2], out)
    with pytest.raises(ValueError, match="shorter"):
        pv.SafetyToIn(P, out[:50])
    with pytest.raises(TypeError):
        pv.DistanceToIn(P, D, far.float(), out)
    with pytest.raises(TypeError):
        pv.Inside(P, out)
    with pytest.raises(V.VgbError):
        pv.DistanceToIn(P, None, far, out)
    with pytest.raises(V.VgbError):
        pv.SafetyToIn(P, out.cpu())
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    pv.DistanceToIn(P, D, far, out, stream=s)
    s.synchronize()
    host = np.zeros(100)
    pv.DistanceToIn(V.SOA3D(*(t.cpu().numpy() for t in x[:3])),
                    V.SOA3D(*(t.cpu().numpy() for t in x[3:])), np.full(100, 1e30), host)
    assert np.array_equal(out.cpu().numpy(), host)
