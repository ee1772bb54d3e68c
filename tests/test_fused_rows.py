"""The fused call of the expensive shapes (one launch, a block row per group of ops)
against one call per op, bit for bit on the GPU, at the edges of a warp, a block and the
grids, for every op group alone and together, and every flag."""
import math

import numpy as np
import pytest

from vecgeom_b200 import workloads as W

SPECS = {"cone": W.config2_shapes()["cone"], "sphere": W.config2_shapes()["sphere"],
         **W.config3_shapes(), "torus_cut": W.torus_spec(2., 5., 50., 0.3, 4.),
         "boolinter": W.zoo2_specs()[-1],
         "polycone_one": W.polycone_spec(0., 2., [-5., 5.], [1., 2.], [3., 4.]),
         "polyhedron_cut": W.polyhedron_spec(0., 200., 6, [-50., -10., 30., 60.],
                                             [5., 10., 20., 3.], [30., 40., 45., 20.])}


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 257, 4099, 303107])
@pytest.mark.parametrize("name", sorted(SPECS))
def test_rows_equal_single_ops(name, n):
    import torch

    import vecgeom_b200 as V
    spec = SPECS[name]
    m = min(n, 20000)
    wl = W.make_workload(spec, m, 3)
    place = (3., -2., 1., 30., 40., 50.)
    R = W.euler_rotation(*place[3:])
    rep = -(-n // m)
    p = R @ np.stack([wl.x, wl.y, wl.z]) + np.array(place[:3])[:, None]
    d = R @ np.stack([wl.dx, wl.dy, wl.dz])
    p, d = (np.tile(a, rep)[:, :n] for a in (p, d))
    g = V.Geometry()
    pv = g.LogicalVolume("s", W.build_unplaced(g, spec)).Place(g.Transformation3D(*place))
    g.CloseGeometry()
    P, D = (V.SOA3D(*(torch.from_numpy(np.ascontiguousarray(a[j])).cuda() for j in range(3)))
            for a in (p, d))
    step = torch.full((n,), 1e30, dtype=torch.float64, device="cuda")
    kinds = {0: torch.uint8, 1: torch.int32}

    def buf(op):
        return torch.full((n,), 7, dtype=kinds.get(op, torch.float64), device="cuda")
    want = {op: buf(op) for op in range(6)}
    for op in range(6):
        dist = op in (2, 3)
        pv.batch(op, P, want[op], D if dist else None, step if dist else None)
    inside = want[0] != 0
    inf = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    for ops in (0x3f, 0x04, 0x08, 0x33, 0x0c, 0x28, 0x15):
        for dto, local in ((False, False), (True, False), (False, True)):
            outs = {op: buf(op) for op in range(6) if (ops >> op) & 1}
            pv.fused(ops, P, outs, D, step, dto_inside_only=dto, local_inside_only=local)
            for op, got in outs.items():
                w = want[op]
                if (op == 3 and (dto or local)) or (op == 5 and local):
                    w = torch.where(inside, w, inf)
                assert torch.equal(got.view(torch.uint8), w.contiguous().view(torch.uint8)), (ops, op)
