"""Batch calls do not need the native call module (csrc/pycall.cpp): where it is not
built, was built for another torch, or torch is not loaded, they take the general path; so
do calls through a library handle without the entries it uses.  The C library's build
needs no torch."""
import ctypes
import os
import shutil
import subprocess
import sys
import types

import numpy as np
import pytest
import torch

from vecgeom_b200 import _lib
from vecgeom_b200 import geometry as G

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "vecgeom_b200", "csrc")
N = 5


class FakeLib:
    """A library whose vgb_batch notes its calls."""

    def __init__(self):
        self.calls = []

    def vgb_batch(self, *args):
        self.calls.append(args)
        return _lib.OK


def volume(lib):
    g = G.Geometry.__new__(G.Geometry)
    g.L, g.handle, g.closed = lib, ctypes.c_void_p(0x1234), True
    g.__class__ = type("G", (G.Geometry,), {"__del__": lambda self: None})
    return G.PlacedVolume(g, 3, None)


def safety(lib, x=None):
    x = [torch.zeros(N, dtype=torch.float64) for _ in range(3)] if x is None else x
    out = torch.zeros(N, dtype=torch.float64)
    volume(lib).SafetyToIn(G.SOA3D(*x), out)
    assert [c[3] for c in lib.calls] == [N]
    assert lib.calls[0][4:7] == tuple(a.data_ptr() for a in x) and lib.calls[0][11] == out.data_ptr()


def test_a_library_without_the_device_entry(monkeypatch):
    monkeypatch.setattr(_lib, "_pycall", None)
    safety(FakeLib())


@pytest.mark.parametrize("case", ["missing", "broken", "other torch"])
def test_a_module_that_cannot_be_used(monkeypatch, tmp_path, case):
    built = _lib.PYCALL_PATH
    path = tmp_path / "_pycall.so"
    if case == "broken":
        path.write_bytes(b"not a library")
    elif case == "other torch":
        if not os.path.exists(built):
            pytest.skip("the module is not built here")
        shutil.copy(built, path)
        monkeypatch.setattr(torch, "__version__", "0.0.1")
    monkeypatch.setattr(_lib, "_pycall", None)
    monkeypatch.setattr(_lib, "PYCALL_PATH", str(path))
    assert _lib.pycall() is None
    safety(FakeLib())


def test_arrays_of_another_kind_without_torch(monkeypatch):
    a = [np.zeros(N) for _ in range(3)]
    x = [types.SimpleNamespace(shape=(N,), dtype=v.dtype, data_ptr=lambda v=v: v.ctypes.data,
                               is_contiguous=lambda: True) for v in a]
    monkeypatch.setattr(_lib, "_pycall", None)
    monkeypatch.delitem(sys.modules, "torch")
    assert _lib.pycall() is None and _lib._pycall is None
    lib = FakeLib()
    out = np.zeros(N)
    volume(lib).SafetyToIn(G.SOA3D(*x), out)
    assert lib.calls[0][4] == a[0].ctypes.data


def test_the_c_library_builds_without_torch(tmp_path):
    python = tmp_path / "python3"
    python.write_text("#!/bin/sh\nexec %s -S -E \"$@\"\n" % sys.executable)
    python.chmod(0o755)
    r = subprocess.run([str(python), "-c", "import importlib.util as u; print(u.find_spec('torch'))"],
                       capture_output=True, text=True)
    if r.stdout.strip() != "None":
        pytest.skip("torch is on every interpreter's path here")
    for target in ("all", "lib"):
        r = subprocess.run(["make", "-C", SRC, "-n", "-B", target, f"PYTHON={python}"],
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        assert "libvgb.so" in r.stdout and "pycall" not in r.stdout
