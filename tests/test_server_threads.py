"""The navigation server's launches with a thread per track, which servers of many slots
take: the results of every request equal, bit for bit, those of the same tracks served in
small parts by a server whose launches give each track a warp.  Requests of uneven sizes
(padded chunks) arrive and finish at different iterations, so launches change between the
two forms, and tracks outside the world are finished from the start."""
import numpy as np
import pytest

from test_server import assert_same, serve
from vecgeom_b200 import workloads as W

MAX_STEPS = 48


def requests(name, sizes):
    out = []
    for k, n in enumerate(sizes):
        if name == "zoo":
            pts, dirs = W.zoo_tracks(n, 900 + k)
        else:
            pts, dirs = W.isotropic_tracks(n, 900 + k)
            if k % 2:
                rng = np.random.default_rng(k)
                pts = [rng.uniform(-1000., 1000., n) for _ in range(3)]
        pts = [np.array(a) for a in pts]
        pts[0][::11] = 1e6  # outside the world
        out.append((pts, dirs))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name,precision,big", [("detector", 0, 20000), ("detector", 1, 20000),
                                                ("zoo", 0, 40500)])
def test_many_slots_equal_few(name, precision, big):
    import vecgeom_b200 as V
    g = V.Geometry()
    b = W.VgbBuilder(g)
    if name == "zoo":
        W.build_zoo(b, W.zoo_specs())
    else:
        W.build_detector(b)
    # the slots of the first launch are past the lines of 20,480 and 40,960
    reqs = requests(name, [big, 300, 17, 600, 2500, 1, 5000, 777])
    many = serve(V.NavServer(g, max_tracks=big + 6000, steps_per_launch=5, max_steps=MAX_STEPS,
                             precision=precision),
                 reqs, arrivals=[0, 0, 0, 0, 1, 2, 4, 12])
    few = V.NavServer(g, max_tracks=2048, steps_per_launch=7, max_steps=MAX_STEPS)
    for k, (pts, dirs) in enumerate(reqs):
        n = len(pts[0])
        cuts = list(range(0, n, 2000)) + [n]
        parts = [([a[i:j] for a in pts], [a[i:j] for a in dirs]) for i, j in zip(cuts, cuts[1:])]
        res = serve(few, parts, arrivals=[0] * len(parts))
        want = {key: np.concatenate([res[i][key] for i in range(len(parts))])
                for key in ("nsteps", "hash", "x", "y", "z")}
        assert_same(many[k], want, f"request {k}")
        assert (want["nsteps"][::11] == 0).all()
        assert n == 1 or want["nsteps"].max() > 5
