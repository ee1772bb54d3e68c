"""Fused calls whose outputs are among their input arrays: the results of the same call
into arrays of their own, for shapes with and without block rows, on device and host
arrays, at the edges of a block and past the grids."""
import numpy as np
import pytest

from vecgeom_b200 import workloads as W

SPECS = {**{k: v for k, v in W.config2_shapes().items()}, **W.config3_shapes(),
         "boolinter": W.zoo2_specs()[-1]}

# op -> the input array it is written over
INTO = [{4: "x"}, {4: "y", 2: "step"}, {2: "x", 3: "dy", 4: "z", 5: "step"}, {3: "dz"}]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 257, 303107])
@pytest.mark.parametrize("name", sorted(SPECS))
def test_outputs_over_inputs(name, n):
    import torch

    import vecgeom_b200 as V
    spec = SPECS[name]
    wl = W.make_workload(spec, min(n, 20000), 3)
    g = V.Geometry()
    pv = g.LogicalVolume("s", W.build_unplaced(g, spec)).Place(g.Transformation3D())
    g.CloseGeometry()
    a = {"x": wl.x, "y": wl.y, "z": wl.z, "dx": wl.dx, "dy": wl.dy, "dz": wl.dz, "step": wl.step}
    a = {k: np.ascontiguousarray(np.resize(v, n)) for k, v in a.items()}
    types = {0: np.uint8, 1: np.int32}

    def run(into, host):
        t = {k: v.copy() if host else torch.from_numpy(v).cuda() for k, v in a.items()}
        outs = {op: np.zeros(n, types.get(op, np.float64)) for op in range(6)}
        if not host:
            outs = {op: torch.from_numpy(o).cuda() for op, o in outs.items()}
        outs.update({op: t[k] for op, k in into.items()})
        pv.fused(0x3f, V.SOA3D(t["x"], t["y"], t["z"]), outs, V.SOA3D(t["dx"], t["dy"], t["dz"]),
                 t["step"])
        return [o.tobytes() if host else o.cpu().numpy().tobytes() for o in outs.values()]

    want = run({}, False)
    for into in INTO:
        for host in (False, True):
            assert run(into, host) == want, (into, host)
