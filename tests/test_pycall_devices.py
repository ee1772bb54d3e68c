"""One batch call's arrays are on one device: the native call (csrc/pycall.cpp) takes the
entry that skips the driver's pointer queries only where all of them are on a GPU and
leaves a mix of devices to the general path, which refuses it before any launch."""
import ctypes
import os
import types

import numpy as np
import pytest
import torch

from vecgeom_b200 import _lib
from vecgeom_b200.geometry import _check_reachable

N = 7
FN = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_int32, ctypes.c_int32,
                      ctypes.c_int64, *[ctypes.c_void_p] * 9, ctypes.c_int32, ctypes.c_int32,
                      ctypes.c_void_p)


def tensors(device="cpu"):
    t = {k: torch.zeros(N, dtype=torch.float64, device=device)
         for k in ("x", "y", "z", "dx", "dy", "dz", "step", "out")}
    t["aux"] = torch.zeros(N, dtype=torch.int32, device=device)
    return t


def native(t):
    """The native call's status and the entries it called, in order."""
    if not os.path.exists(_lib.LIB_PATH.replace("libvgb", "_pycall")):
        pytest.skip("the library is not built here")
    seen = []
    fns = [FN(lambda *a, k=k: seen.append(k) or 0) for k in ("general", "device")]
    addrs = [ctypes.cast(f, ctypes.c_void_p).value for f in fns]
    st = _lib.pycall().batch(*addrs, 0x1234, 0, 6, t["x"], t["y"], t["z"], t["dx"], t["dy"],
                             t["dz"], t["step"], t["out"], t["aux"], 0, 0, None)
    return st, seen


def test_host_tensors_go_to_the_general_entry():
    assert native(tensors()) == (0, ["general"])


@pytest.mark.parametrize("where", ["x", "y", "z", "dx", "dz", "step", "out", "aux"])
def test_a_mix_of_devices_is_left_to_the_general_path(where):
    t = tensors()
    t[where] = t[where].to("meta")
    assert native(t) == (None, [])


def fake(device, pinned=False):
    return types.SimpleNamespace(device=device, is_cuda=device.startswith("cuda"),
                                 is_pinned=lambda: pinned)


def test_what_the_kernels_can_reach():
    x, out = fake("cuda:0"), fake("cuda:0")
    _check_reachable(x, out, None, fake("cuda:0"), fake("cpu", pinned=True))
    _check_reachable(x, fake("cpu"))  # the library refuses it with its own error
    _check_reachable(np.zeros(N), np.zeros(N), np.zeros(N))
    _check_reachable(fake("cpu"), fake("cpu"), fake("cpu"))
    for bad in (fake("cpu"), fake("cuda:1"), np.zeros(N)):
        with pytest.raises(ValueError, match="one device"):
            _check_reachable(x, out, None, bad)
    with pytest.raises(ValueError, match="one device"):
        _check_reachable(x, fake("cuda:1"))


@pytest.mark.gpu
def test_gpu_mixes_are_refused_and_pinned_arrays_read():
    import vecgeom_b200 as V
    assert native(tensors("cuda")) == (0, ["device"])
    g = V.Geometry()
    pv = g.LogicalVolume("b", g.UnplacedBox(1., 2., 3.)).Place(g.Transformation3D())
    g.CloseGeometry()
    x = [torch.rand(100, dtype=torch.float64, device="cuda") * 8. - 4. for _ in range(6)]
    P, D = V.SOA3D(*x[:3]), V.SOA3D(*x[3:])
    far = torch.full((100,), 1e30, dtype=torch.float64)
    want, out = (torch.zeros(100, dtype=torch.float64, device="cuda") for _ in range(2))
    pv.DistanceToIn(P, D, far.cuda(), want)
    with pytest.raises(ValueError, match="one device"):
        pv.DistanceToIn(P, D, far, out)
    with pytest.raises(ValueError, match="one device"):
        pv.DistanceToIn(P, D, far.numpy(), out)
    with pytest.raises(ValueError, match="one device"):
        pv.SafetyToIn(V.SOA3D(x[0], x[1].cpu(), x[2]), out)
    torch.cuda.synchronize()
    assert not out.any()
    pv.DistanceToIn(P, D, far.pin_memory(), out)
    assert torch.equal(out, want)
