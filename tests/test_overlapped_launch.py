"""Batch kernels launched back to back overlap their set-up with the kernel before them:
chains in which each call reads what the one before it wrote, and writes what it read,
give what the same calls give with a synchronisation after each, eagerly and replayed
from a captured graph, with other kernels and fills between them."""
import math

import numpy as np
import pytest

from vecgeom_b200 import workloads as W


@pytest.mark.gpu
@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n", [1, 1000, 70001, 400003])
def test_chains_of_dependent_calls(n, captured):
    import torch

    import vecgeom_b200 as V
    specs = [W.box_spec(10., 20., 30.), W.config2_shapes()["tube"], W.config3_shapes()["polycone"]]
    g = V.Geometry()
    pvs = [g.LogicalVolume("s", W.build_unplaced(g, s)).Place(g.Transformation3D(1., 2., 3.))
           for s in specs]
    g.CloseGeometry()
    rng = np.random.default_rng(8)
    p = torch.from_numpy(rng.uniform(-60., 60., (3, n))).cuda()
    d = torch.from_numpy(np.array(W.isotropic(rng, n))).cuda()
    D = V.SOA3D(*(d[j].contiguous() for j in range(3)))
    x0 = [p[j].contiguous() for j in range(3)]
    x = [t.clone() for t in x0]
    P = V.SOA3D(*x)
    a, b, c = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3))
    node = torch.zeros(n, dtype=torch.int32, device="cuda")
    outs = {2: torch.zeros_like(a), 4: torch.zeros_like(a), 0: torch.zeros(n, dtype=torch.uint8, device="cuda")}

    def chain(wait):
        for t, t0 in zip(x, x0):
            t.copy_(t0)
        s = torch.cuda.current_stream()
        a.fill_(math.inf)
        node.zero_()
        for k in range(12):
            pv = pvs[k % 3]
            pv.SafetyToIn(P, b, stream=s)
            wait()
            pv.SafetyToInMinimize(P, a, stream=s)          # reads and writes a
            wait()
            pv.DistanceToIn(P, D, a, c, stream=s)          # step limit: the call before
            wait()
            pv.DistanceToInMinimize(P, D, k, b, node, stream=s)
            wait()
            pv.fused((1 << 2) | (1 << 4) | 1, P, outs, D, b, stream=s)
            wait()
            x[k % 3].add_(torch.clamp(outs[4], -1., 1.))   # another library's kernel
            wait()
        return [t.clone() for t in (*x, a, b, c, node, *outs.values())]

    want = chain(torch.cuda.synchronize)
    torch.cuda.synchronize()
    if captured:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = chain(lambda: None)
        for _ in range(3):
            graph.replay()
    else:
        for _ in range(3):
            got = chain(lambda: None)
    torch.cuda.synchronize()
    for w, q in zip(want, got):
        assert torch.equal(w.view(torch.uint8), q.view(torch.uint8))
