"""The device reads the sin and cos table of crmath.cuh in 16-byte words, so its type has
to ask for 16-byte alignment (a table of doubles may be placed on 8)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "vecgeom_b200", "csrc")


def test_sincos_table_is_aligned_for_its_loads(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    r = subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-I", SRC, "-c", "-o",
                        str(tmp_path / "crtable.o"),
                        os.path.join(HERE, "hostcheck", "crtable.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
