"""Cases that time the library through its Python API: the work a user has it do.

Shape batches (the VPlacedVolume SOA3D calls, one call per op or the fused form,
device or pinned host buffers), mixed baskets, and navigation (LocatePoint,
FindNextBoundaryAndStep, whole traces, the server) in the layered detector and in
the mixed-shape geometry.  Shapes and geometries are those of
vecgeom_b200.workloads; points are a third inside the shape, a third outside it in
1.5 times its box and a third within 1e-6 mm of its surface, directions isotropic.
All points are drawn on the GPU from the seed alone.
"""
import ctypes
import math

import numpy as np
import torch

import vecgeom_b200 as V
from vecgeom_b200 import workloads as W
from vecgeom_b200 import _lib as L

# op name -> (op code of the C ABI, output dtype, takes directions, local frame)
OPS = {
    "contains": (L.OP_CONTAINS, torch.uint8, False, False),
    "inside": (L.OP_INSIDE, torch.int32, False, False),
    "safety_to_in": (L.OP_SAFETY_TO_IN, torch.float64, False, False),
    "safety_to_out": (L.OP_SAFETY_TO_OUT, torch.float64, False, True),
    "distance_to_in": (L.OP_DISTANCE_TO_IN, torch.float64, True, False),
    "distance_to_out": (L.OP_DISTANCE_TO_OUT, torch.float64, True, True),
}
TCS = "tube+cone+sphere"
HEAVY = "torus+polycone+polyhedron+boolsub"
OTHERS = "trd+orb+parallelepiped+paraboloid+trapezoid+boolunion+boolinter"
KINDS = ["box"] + TCS.split("+") + HEAVY.split("+") + OTHERS.split("+")
STEP_MAX = 1e30


def listed():
    return [
        # one volume asks for the distances of a handful of tracks: call overhead
        {"name": "box_dti_100", "path": "batch", "shapes": "box", "ops": "distance_to_in",
         "n": 100, "placed": False, "jitter": 0},
        # a basket of particles against three rotated volumes, every op: an ordinary call
        {"name": "tube_cone_sphere_16k", "path": "batch", "shapes": TCS, "ops": "all",
         "n": 16411, "placed": True, "jitter": 0},
        # the benchmark's main workload: 2^22 points per shape, every op
        {"name": "tube_cone_sphere_4m", "path": "batch", "shapes": TCS, "ops": "all",
         "n": 1 << 22, "placed": False, "jitter": 0},
        # the benchmark's compute-heavy shapes
        {"name": "heavy_4m", "path": "batch", "shapes": HEAVY, "ops": "all", "n": 1 << 22,
         "placed": False, "jitter": 0},
        # the remaining shapes, rotated, an odd size
        {"name": "other_shapes_500k", "path": "batch", "shapes": OTHERS, "ops": "all",
         "n": 500009, "placed": True, "jitter": 0},
        # everything about a point in one call (local ops where the point is inside)
        {"name": "fused_seven_500k", "path": "fused", "shapes": TCS + "+" + HEAVY, "n": 500009,
         "placed": True, "jitter": 0},
        # the same call on a client's pinned host arrays: the benchmark's end-to-end form
        {"name": "hosted_fused_512k", "path": "hosted", "shapes": TCS, "n": 1 << 19,
         "placed": False, "jitter": 0},
        # many volumes with their own small batches in one launch
        {"name": "baskets_1024", "path": "baskets", "baskets": 1024, "median": 1024, "jitter": 4},
        # one navigation step of a transport loop in a geometry of every shape
        {"name": "step_zoo_50k", "path": "step", "geometry": "zoo", "navigator": "simple",
         "n": 50021},
        # whole tracks through the layered detector, both navigators
        {"name": "trace_detector_64k", "path": "trace", "geometry": "detector",
         "navigator": "simple", "n": 1 << 16, "max_steps": 64},
        {"name": "trace_abbox_32k", "path": "trace", "geometry": "detector",
         "navigator": "abbox", "n": 1 << 15, "max_steps": 64},
        # requests of a few to some thousand tracks through the navigation server
        {"name": "served_48", "path": "served", "geometry": "detector", "requests": 48,
         "largest": 4096, "max_steps": 64, "steps_per_launch": 8},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["batch", "batch", "batch", "fused", "hosted", "baskets", "step", "trace",
                       "served"])
    if path in ("batch", "fused", "hosted"):
        group = rng.choice([TCS, HEAVY, OTHERS, "one", "one"])
        if group == "one":
            group = rng.choice(KINDS)
        case = {"path": path, "shapes": group, "placed": rng.random() < 0.5,
                "jitter": rng.randrange(1, 1000)}
        if path == "batch":
            case["ops"] = rng.choice(["all", "all", rng.choice(list(OPS))])
            case["n"] = _log_uniform(rng, 1, 1 << 22)
        else:
            case["n"] = _log_uniform(rng, 1, 1 << (20 if path == "fused" else 19))
        return case
    if path == "baskets":
        return {"path": path, "baskets": _log_uniform(rng, 8, 1024),
                "median": _log_uniform(rng, 64, 1024), "jitter": rng.randrange(1, 1000)}
    case = {"path": path, "geometry": rng.choice(["detector", "zoo"])}
    if path == "step":
        case.update(navigator=rng.choice(["simple", "abbox", "basket"]),
                    n=_log_uniform(rng, 1, 1 << 17))
    elif path == "trace":
        case.update(navigator=rng.choice(["simple", "abbox"]), n=_log_uniform(rng, 1, 1 << 16),
                    max_steps=rng.randrange(8, 65))
    else:
        case.update(requests=_log_uniform(rng, 1, 64), largest=_log_uniform(rng, 16, 4096),
                    max_steps=rng.randrange(16, 65), steps_per_launch=rng.choice([4, 8, 16]))
    return case


# ---------------------------------------------------------------------------
# shapes and their points
# ---------------------------------------------------------------------------
def _specs(case):
    base = {**W.basket_base_specs(), "trd": W.trd_spec(20., 10., 25., 15., 30.)}
    base.update({s.kind: s for s in W.zoo2_specs() if s.kind != "trapezoidcorners"})
    rng = np.random.default_rng(case["jitter"])
    out = {}
    for kind in case["shapes"].split("+"):
        s = base[kind]
        out[kind] = W.jitter_spec(s, rng) if case["jitter"] and kind in W.BASKET_KINDS else s
    return out


def _place(case, k):
    """Placement (tx, ty, tz, Euler angles) of a batch case's k-th shape."""
    if not case["placed"]:
        return W.IDENTITY_PLACE
    return (3. - k, -2. + k, 1. + 2. * k, 30. + 11. * k, 40. + 7. * k, 50. + 5. * k)


def _phi_in(x, y, sphi, dphi):
    return torch.remainder(torch.atan2(y, x) - sphi, 2 * math.pi) <= dphi + 1e-15


def _stack_in(p, z, radial):
    """Sections of a polycone or polyhedron: rmin <= radial <= rmax at height z."""
    ok = torch.zeros_like(z, dtype=torch.bool)
    for k in range(len(p["z"]) - 1):
        z0, z1 = p["z"][k], p["z"][k + 1]
        t = (z - z0) / (z1 - z0)
        lo = p["rmin"][k] + (p["rmin"][k + 1] - p["rmin"][k]) * t
        hi = p["rmax"][k] + (p["rmax"][k + 1] - p["rmax"][k]) * t
        ok |= (z >= z0) & (z <= z1) & (radial >= lo) & (radial <= hi)
    return ok


def _local(place, x, y, z):
    rot = W.euler_rotation(*place[3:])
    a = (x - place[0], y - place[1], z - place[2])
    return tuple(a[0] * rot[0, j] + a[1] * rot[1, j] + a[2] * rot[2, j] for j in range(3))


def _contains(kind, p, x, y, z):
    """Containment without tolerances, used to draw points; the parameters are
    numbers or one value per point."""
    if kind == "box":
        return (x.abs() <= p["dx"]) & (y.abs() <= p["dy"]) & (z.abs() <= p["dz"])
    if kind in ("tube", "cone"):
        r = torch.sqrt(x * x + y * y)
        if kind == "tube":
            lo, hi = p["rmin"], p["rmax"]
        else:
            t = (z + p["dz"]) / (2 * p["dz"])
            lo = p["rmin1"] + (p["rmin2"] - p["rmin1"]) * t
            hi = p["rmax1"] + (p["rmax2"] - p["rmax1"]) * t
        return (z.abs() <= p["dz"]) & (r >= lo) & (r <= hi) & _phi_in(x, y, p["sphi"], p["dphi"])
    if kind in ("sphere", "orb"):
        r = torch.sqrt(x * x + y * y + z * z)
        if kind == "orb":
            return r <= p["r"]
        th = torch.atan2(torch.sqrt(x * x + y * y), z)
        return ((r >= p["rmin"]) & (r <= p["rmax"]) & (th >= p["stheta"])
                & (th <= p["stheta"] + p["dtheta"]) & _phi_in(x, y, p["sphi"], p["dphi"]))
    if kind == "torus":
        rho = torch.sqrt(x * x + y * y) - p["rtor"]
        d = torch.sqrt(rho * rho + z * z)
        return (d >= p["rmin"]) & (d <= p["rmax"]) & _phi_in(x, y, p["sphi"], p["dphi"])
    if kind == "polycone":
        return _stack_in(p, z, torch.sqrt(x * x + y * y)) & _phi_in(x, y, p["sphi"], p["dphi"])
    if kind == "polyhedron":
        sw = 2 * math.pi / p["sides"]
        rel = torch.remainder(torch.atan2(y, x), 2 * math.pi)
        mid = (torch.clamp(torch.floor(rel / sw), max=p["sides"] - 1) + 0.5) * sw
        return _stack_in(p, z, x * torch.cos(mid) + y * torch.sin(mid))
    if kind == "trd":
        t = (z + p["dz"]) / (2 * p["dz"])
        return ((z.abs() <= p["dz"]) & (x.abs() <= p["dx1"] + (p["dx2"] - p["dx1"]) * t)
                & (y.abs() <= p["dy1"] + (p["dy2"] - p["dy1"]) * t))
    if kind == "parallelepiped":
        ta, tt = math.tan(math.radians(p["alpha"])), math.tan(math.radians(p["theta"]))
        ly = y - tt * math.sin(math.radians(p["phi"])) * z
        lx = x - (tt * math.cos(math.radians(p["phi"])) * z + ta * ly)
        return (lx.abs() <= p["x"]) & (ly.abs() <= p["y"]) & (z.abs() <= p["z"])
    if kind == "paraboloid":
        a = 2. * p["dz"] / (p["rhi"] ** 2 - p["rlo"] ** 2)
        b = -p["dz"] * (p["rlo"] ** 2 + p["rhi"] ** 2) / (p["rhi"] ** 2 - p["rlo"] ** 2)
        return (z.abs() <= p["dz"]) & (z >= a * (x * x + y * y) + b)
    if kind == "trapezoid":
        c = W.trapezoid_corners(*p.values())
        ok = z.abs() <= p["dz"]
        for i1, i2, i3, i4 in ((0, 1, 5, 4), (2, 6, 7, 3), (0, 4, 6, 2), (1, 3, 7, 5)):
            m = np.cross(c[i3] - c[i1], c[i4] - c[i2])
            ok &= m[0] * x + m[1] * y + m[2] * z <= m.dot(c[i1])
        return ok
    # booleans of a box and a full tube
    lx, ly, lz = _local(p.get("left_place", W.IDENTITY_PLACE), x, y, z)
    rx, ry, rz = _local(p.get("right_place", W.IDENTITY_PLACE), x, y, z)
    h = p["box_half"]
    box = (lx.abs() <= h[0]) & (ly.abs() <= h[1]) & (lz.abs() <= h[2])
    tube = (rx * rx + ry * ry <= p["tube_rmax"] ** 2) & (rz.abs() <= p["tube_dz"])
    return {"boolsub": box & ~tube, "boolunion": box | tube, "boolinter": box & tube}[kind]


def _take(v, idx):
    """Per-point values of a parameter (or of a list of them) at some points."""
    if isinstance(v, torch.Tensor):
        return v[idx]
    if isinstance(v, (list, tuple)) and v and isinstance(v[0], torch.Tensor):
        return [a[idx] for a in v]
    return v


def _reject(kind, p, half, center, want, scale, n, gen):
    """n points uniform in the scaled box with Contains == want."""
    out = torch.empty(3, n, dtype=torch.float64, device="cuda")
    todo = torch.arange(n, device="cuda")
    while todo.numel():
        u = torch.rand(3, todo.numel(), dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        q = torch.stack([_take(center[j], todo) + u[j] * _take(half[j], todo) * scale
                         for j in range(3)])
        out[:, todo] = q
        ok = _contains(kind, {k: _take(v, todo) for k, v in p.items()}, q[0], q[1], q[2]) == want
        todo = todo[~ok]
    return out


def _points(kind, p, half, center, n, gen):
    """The mixed points of a shape, and which of them are inside."""
    n1, n2 = n // 3, n // 3
    role = torch.full((n,), 2, device="cuda")
    role[:n1] = 0
    role[n1:n1 + n2] = 1
    role = role[torch.randperm(n, device="cuda", generator=gen)]

    def some(idx):
        return ({k: _take(v, idx) for k, v in p.items()}, [_take(h, idx) for h in half],
                [_take(c, idx) for c in center])
    pts = torch.empty(3, n, dtype=torch.float64, device="cuda")
    for r, want, scale in ((0, True, 1.0), (1, False, 1.5)):
        idx = torch.nonzero(role == r).flatten()
        pts[:, idx] = _reject(kind, *some(idx), want, scale, idx.numel(), gen)
    idx = torch.nonzero(role == 2).flatten()
    if idx.numel():
        q, h, c = some(idx)
        lo = _reject(kind, q, h, c, True, 1.0, idx.numel(), gen)
        hi = _reject(kind, q, h, c, False, 1.5, idx.numel(), gen)
        d = (hi - lo) / (hi - lo).norm(dim=0)
        for _ in range(56):
            mid = 0.5 * (lo + hi)
            ok = _contains(kind, q, mid[0], mid[1], mid[2])
            lo, hi = torch.where(ok, mid, lo), torch.where(ok, hi, mid)
        off = torch.rand(idx.numel(), dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        pts[:, idx] = 0.5 * (lo + hi) + d * (off * 1e-6)
    return pts, _contains(kind, p, pts[0], pts[1], pts[2])


def _directions(n, gen):
    v = torch.randn(3, n, dtype=torch.float64, device="cuda", generator=gen)
    return v / v.norm(dim=0)


def _soa(a):
    return V.SOA3D(*(a[j].contiguous() for j in range(3)))


def _mother(place, a, move):
    """Local points (or directions: move=False) in the frame the shape is placed in."""
    if tuple(place) == W.IDENTITY_PLACE:
        return a
    rot = torch.from_numpy(W.euler_rotation(*place[3:])).cuda()
    out = rot @ a
    if move:
        out = out + torch.tensor(place[:3], dtype=torch.float64, device="cuda")[:, None]
    return out


def _shape_states(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = V.Geometry()
    shapes = []
    for k, (kind, spec) in enumerate(_specs(case).items()):
        place = _place(case, k)
        lv = g.LogicalVolume(kind, W.build_unplaced(g, spec))
        pv = lv.Place(g.Transformation3D(*place))
        pts, ins = _points(kind, spec.params, spec.half, spec.center, case["n"], gen)
        shapes.append((kind, spec, place, pv, pts, ins, _directions(case["n"], gen)))
    g.CloseGeometry()
    return g, shapes


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def _names(case):
    return list(OPS) if case.get("ops", "all") == "all" else case["ops"].split("+")


def _local_points(ins):
    """The points of the local ops: inside the shape, half as many as there are
    points (about half of the mixed points are inside; the first come again where
    they are fewer)."""
    idx = torch.nonzero(ins).flatten()
    if not idx.numel():
        idx = torch.arange(1, device="cuda")
    return idx[torch.arange(max(1, len(ins) // 2), device="cuda") % idx.numel()]


def _prepare_batch(case, seed):
    g, shapes = _shape_states(case, seed)
    calls = []
    for kind, spec, place, pv, pts, ins, dirs in shapes:
        mother = (_soa(_mother(place, pts, True)), _soa(_mother(place, dirs, False)))
        idx = _local_points(ins)
        local = (_soa(pts[:, idx]), _soa(dirs[:, idx]))
        for name in _names(case):
            op, dtype, dist, loc = OPS[name]
            p, d = local if loc else mother
            step = torch.full((len(p),), STEP_MAX, dtype=torch.float64, device="cuda")
            out = torch.zeros(len(p), dtype=dtype, device="cuda")
            calls.append((kind, name, pv, p, d if dist else None, step if dist else None, out))
    return {"geometry": g, "calls": calls}


def _prepare_fused(case, seed, hosted):
    g, shapes = _shape_states(case, seed)
    calls = []

    def mine(t):
        return t.cpu().pin_memory() if hosted else t.contiguous()
    for kind, spec, place, pv, pts, ins, dirs in shapes:
        m, d = _mother(place, pts, True), _mother(place, dirs, False)
        p = V.SOA3D(*(mine(m[j]) for j in range(3)))
        v = V.SOA3D(*(mine(d[j]) for j in range(3)))
        step = mine(torch.full((len(p),), STEP_MAX, dtype=torch.float64, device="cuda"))
        outs = {op: mine(torch.zeros(len(p), dtype=dtype, device="cuda"))
                for op, dtype, _, _ in OPS.values()}
        calls.append((kind, pv, p, v, step, outs))
    return {"geometry": g, "calls": calls}


def _prepare_baskets(case, seed):
    """Jittered instances of the eight basket shapes at their own placements; the
    points of all baskets of one kind are drawn together."""
    rng = np.random.default_rng(case["jitter"])
    nb = case["baskets"]
    sizes = np.clip(np.round(rng.lognormal(math.log(case["median"]), 1.0, nb)), 16, 8192)
    sizes = sizes.astype(np.int64)
    kinds = rng.integers(0, len(W.BASKET_KINDS), nb)
    base = W.basket_base_specs()
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    g = V.Geometry()
    specs, places, baskets = [], [], []
    for b in range(nb):
        spec = W.jitter_spec(base[W.BASKET_KINDS[kinds[b]]], rng)
        place = (*rng.uniform(-100., 100., 3), *rng.uniform(0., 360., 3))
        lv = g.LogicalVolume("basket", W.build_unplaced(g, spec))
        baskets.append((lv.Place(g.Transformation3D(*place)), offsets[b], sizes[b]))
        specs.append(spec)
        places.append(place)
    g.CloseGeometry()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    total = int(offsets[-1])
    pts = torch.empty(3, total, dtype=torch.float64, device="cuda")
    dirs = torch.empty(3, total, dtype=torch.float64, device="cuda")
    for k, kind in enumerate(W.BASKET_KINDS):
        mine = np.flatnonzero(kinds == k)
        if not len(mine):
            continue
        counts = torch.from_numpy(sizes[mine]).cuda()
        where = torch.from_numpy(np.concatenate(
            [np.arange(offsets[b], offsets[b + 1]) for b in mine])).cuda()

        def each(values):
            t = torch.tensor(np.array(values, np.float64), device="cuda")
            return t.repeat_interleave(counts, dim=0)
        p = {}
        for name, v in specs[mine[0]].params.items():
            vals = each([specs[b].params[name] for b in mine])
            p[name] = vals if vals.dim() == 1 else [c.contiguous() for c in vals.T]
        if kind == "polyhedron":
            p["sides"] = specs[mine[0]].params["sides"]
        half = [each([specs[b].half[j] for b in mine]) for j in range(3)]
        center = [each([specs[b].center[j] for b in mine]) for j in range(3)]
        q, _ = _points(kind, p, half, center, where.numel(), gen)
        v = _directions(where.numel(), gen)
        rot = each([W.euler_rotation(*places[b][3:]) for b in mine])
        t = each([places[b][:3] for b in mine])
        pts[:, where] = torch.einsum("nij,jn->in", rot, q) + t.T
        dirs[:, where] = torch.einsum("nij,jn->in", rot, v)
    ops = (1 << L.OP_DISTANCE_TO_IN) | (1 << L.OP_SAFETY_TO_IN)
    outs = {op: torch.zeros(total, dtype=torch.float64, device="cuda")
            for op in (L.OP_DISTANCE_TO_IN, L.OP_SAFETY_TO_IN)}
    return {"geometry": g, "plan": V.BasketPlan(g, baskets, ops), "points": _soa(pts),
            "dirs": _soa(dirs), "outs": outs,
            "step": torch.full((total,), STEP_MAX, dtype=torch.float64, device="cuda")}


def _geometry(case):
    g = V.Geometry()
    if case["geometry"] == "detector":
        W.build_detector(W.VgbBuilder(g))
    else:
        W.build_zoo(W.VgbBuilder(g), W.zoo_specs())
    return g


def _track_points(case, n, gen, whole):
    """Starting points: whole tracks leave the detector's origin, a step of a
    transport loop starts anywhere in the detector; in the zoo a third start near
    a shape."""
    u = torch.rand(3, n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    if case["geometry"] == "detector":
        if whole:
            return torch.zeros_like(u)
        return u * torch.tensor([1100., 1100., 1250.], dtype=torch.float64, device="cuda")[:, None]
    cell = torch.randint(0, 3, (3, n), device="cuda", generator=gen).double() * 600. - 600.
    near = torch.rand(n, device="cuda", generator=gen) < 1. / 3.
    return torch.where(near, cell + u * 30., u * 900.)


class _PoolBytes:
    """A NavStatePool's device memory, as an array of its states' bytes (a tensor
    made of it holds this object, and with it the pool)."""

    def __init__(self, pool):
        self.pool = pool
        dev = ctypes.c_void_p()
        L.check(pool.geometry.L.vgb_navpool_info(pool.handle, ctypes.byref(dev), None, None))
        self.__cuda_array_interface__ = {"shape": (pool.n, pool.stride), "typestr": "|u1",
                                         "data": (dev.value, False), "version": 3}


def _prepare_step(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = _geometry(case)
    n = case["n"]
    nav = V.ABBoxNavigator(g) if case["navigator"] == "abbox" else V.SimpleNavigator(g)
    cur, nxt = V.NavStatePool(g, n), V.NavStatePool(g, n)

    def buf(dtype=torch.float64, fill=0):
        return torch.full((n,), fill, dtype=dtype, device="cuda")
    return {"geometry": g, "nav": nav, "basket": case["navigator"] == "basket",
            "points": _soa(_track_points(case, n, gen, False)), "dirs": _soa(_directions(n, gen)),
            "cur": cur, "next": nxt, "pstep": buf(fill=STEP_MAX), "step": buf(), "safety": buf(),
            "node": buf(torch.int32),
            "next_bytes": torch.as_tensor(_PoolBytes(nxt), device="cuda")}


def _prepare_trace(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = _geometry(case)
    n, m = case["n"], case["max_steps"]
    nav = V.ABBoxNavigator(g) if case["navigator"] == "abbox" else V.SimpleNavigator(g)
    return {"geometry": g, "nav": nav, "max_steps": m,
            "points": _soa(_track_points(case, n, gen, True)), "dirs": _soa(_directions(n, gen)),
            "nsteps": torch.zeros(n, dtype=torch.int32, device="cuda"),
            "next_ids": torch.zeros(n, m, dtype=torch.int32, device="cuda"),
            "steps": torch.zeros(n, m, dtype=torch.float64, device="cuda"),
            "safeties": torch.zeros(n, m, dtype=torch.float64, device="cuda")}


def _prepare_served(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = _geometry(case)
    # the requests' sizes, spread over their logarithm, are the case's own
    rng = np.random.default_rng(case["requests"])
    sizes = np.round(np.exp(rng.uniform(0., math.log(case["largest"]), case["requests"])))
    reqs = []
    for n in sizes.astype(int):
        p = _track_points(case, int(n), gen, True).cpu().numpy()
        d = _directions(int(n), gen).cpu().numpy()
        reqs.append(([np.ascontiguousarray(a) for a in p], [np.ascontiguousarray(a) for a in d]))
    server = V.NavServer(g, max_tracks=1 << 15, steps_per_launch=case["steps_per_launch"],
                         max_steps=case["max_steps"])
    return {"geometry": g, "server": server, "requests": reqs}


def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        state = _prepare_batch(case, seed)
    elif path in ("fused", "hosted"):
        state = _prepare_fused(case, seed, path == "hosted")
    else:
        state = {"baskets": _prepare_baskets, "step": _prepare_step, "trace": _prepare_trace,
                 "served": _prepare_served}[path](case, seed)
    state["path"] = path
    return state


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
ALL_OPS = sum(1 << op for op, _, _, _ in OPS.values())


def _run_batch(s):
    out = {}
    for kind, name, pv, p, d, step, o in s["calls"]:
        if name == "contains":
            pv.Contains(p, o)
        elif name == "inside":
            pv.Inside(p, o)
        elif name == "safety_to_in":
            pv.SafetyToIn(p, o)
        elif name == "safety_to_out":
            pv.SafetyToOut(p, o)
        elif name == "distance_to_in":
            pv.DistanceToIn(p, d, step, o)
        else:
            pv.DistanceToOut(p, d, step, o)
        out.setdefault(kind, {})[name] = o
    return out


def _run_fused(s):
    out = {}
    for kind, pv, p, v, step, outs in s["calls"]:
        pv.fused(ALL_OPS, p, outs, v, step, local_inside_only=True)
        out[kind] = {name: outs[op] for name, (op, _, _, _) in OPS.items()}
    return out


def _run_baskets(s):
    s["plan"].run(s["points"], s["dirs"], s["step"], s["outs"])
    return {"distance_to_in": s["outs"][L.OP_DISTANCE_TO_IN],
            "safety_to_in": s["outs"][L.OP_SAFETY_TO_IN]}


def _run_step(s):
    nav = s["nav"]
    nav.LocatePoint(s["points"], s["cur"])
    if s["basket"]:
        nav.FindNextBoundaryAndStepBasket(s["points"], s["dirs"], s["cur"], s["next"], s["pstep"],
                                          s["step"], s["safety"], s["node"])
    else:
        nav.FindNextBoundaryAndStep(s["points"], s["dirs"], s["cur"], s["next"], s["pstep"],
                                    s["step"], s["safety"])
    return {"step": s["step"], "safety": s["safety"], "node": s["node"], "next": s["next_bytes"]}


def _run_trace(s):
    s["nav"].Trace(s["points"], s["dirs"], STEP_MAX, s["max_steps"], s["nsteps"], s["next_ids"],
                   s["steps"], s["safeties"])
    return {k: s[k] for k in ("nsteps", "next_ids", "steps", "safeties")}


def _run_served(s):
    server = s["server"]
    ids = [server.submit(p, d) for p, d in s["requests"]]
    left = len(ids)
    while left:
        done, _, _ = server.step()
        left -= len(done)
    results = [server.result(i) for i in ids]
    out = {k: np.concatenate([r[k] for r in results]) for k in ("nsteps", "x", "y", "z", "hash")}
    out["hash"] = out["hash"].view(np.int64)
    return out


def run(state):
    return {"batch": _run_batch, "fused": _run_fused, "hosted": _run_fused,
            "baskets": _run_baskets, "step": _run_step, "trace": _run_trace,
            "served": _run_served}[state["path"]](state)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# Arithmetic of a point, op by op (additions, products, divisions, roots), as
# counted for the benchmark's shapes; 60 stands for the others.
FLOPS = {"box": 25, "tube": 60, "cone": 110, "sphere": 120, "torus": 350, "polycone": 250,
         "polyhedron": 300}


def work(case):
    path = case["path"]
    if path in ("batch", "fused", "hosted"):
        kinds = case["shapes"].split("+")
        n, nbytes, flops = case["n"], 0., 0.
        for kind in kinds:
            if path == "batch":
                for name in _names(case):
                    _, dtype, dist, loc = OPS[name]
                    m = n // 2 if loc else n
                    nbytes += m * (56 if dist else 24) + m * torch.empty(0, dtype=dtype).element_size()
                    flops += m * FLOPS.get(kind, 60) * (1. if dist else 0.2)
            else:
                nbytes += n * (56 + 1 + 4 + 4 * 8)
                flops += n * FLOPS.get(kind, 60) * 2.
        return {"bytes": nbytes, "flops": flops}
    if path == "baskets":
        n = case["baskets"] * case["median"] * math.exp(0.5)
        return {"bytes": n * (56 + 16), "flops": n * 200.}
    if path == "step":
        # points in, states out and in again, step and safety out; a few shapes a track
        return {"bytes": case["n"] * (48 + 8 + 3 * 56 + 16.), "flops": case["n"] * 2000.}
    if path == "trace":
        records = case["n"] * case["max_steps"]
        return {"bytes": case["n"] * 52. + records * 20., "flops": records * 1000.}
    n = case["requests"] * case["largest"] / math.log(case["largest"])
    return {"bytes": n * (48 + 36.), "flops": n * case["max_steps"] * 1000.}


# ---------------------------------------------------------------------------
# exact: 64-bit values in plain torch
# ---------------------------------------------------------------------------
# Safeties of the shapes whose safety is a closed formula of the point, and the
# box's and orb's distances.  The other distances depend on the library's
# tolerances for the third of the points that lie within 1e-6 mm of a surface, so
# no formula without those rules gives them.
def _exact_safety(kind, p, q, to_in):
    x, y, z = q
    r = torch.sqrt(x * x + y * y)
    if kind == "box":
        s = torch.stack([x.abs() - p["dx"], y.abs() - p["dy"], z.abs() - p["dz"]]).amax(0)
        return s if to_in else -s
    if kind == "torus" and p["rmin"] == 0 and p["dphi"] >= 2 * math.pi:
        s = torch.sqrt((r - p["rtor"]) ** 2 + z * z) - p["rmax"]
        return s if to_in else -s
    if kind == "orb":
        s = torch.sqrt(x * x + y * y + z * z) - p["r"]
        return (s if to_in else -s).clamp(min=0.)
    return None


def _exact_distance(kind, p, q, v, to_in):
    if kind != "box":
        return None
    h = [p["dx"], p["dy"], p["dz"]]
    inf = torch.full_like(q[0], math.inf)
    if not to_in:
        t = [(torch.copysign(torch.full_like(inf, h[j]), v[j]) - q[j]) / v[j] for j in range(3)]
        return torch.minimum(torch.minimum(t[0], t[1]), t[2])
    s = [q[j].abs() - h[j] for j in range(3)]
    out = inf.clone()
    for j in (2, 1, 0):
        a, b = [k for k in range(3) if k != j]
        t = s[j] / v[j].abs()
        hit = ((s[j] >= -0.5e-9) & (q[j] * v[j] < 0) & ((q[a] + t * v[a]).abs() <= h[a])
               & ((q[b] + t * v[b]).abs() <= h[b]))
        out = torch.where(hit, t, out)
    return torch.where((s[0] < 0) & (s[1] < 0) & (s[2] < 0), torch.full_like(inf, -1.), out)


def exact(case, seed):
    if case["path"] not in ("batch", "fused", "hosted"):
        return None
    _, shapes = _shape_states(case, seed)
    fused = case["path"] != "batch"
    out = {}
    for kind, spec, place, _, pts, ins, dirs in shapes:
        out[kind] = {}
        idx = _local_points(ins)
        for name in _names(case):
            out[kind][name] = None
            _, dtype, dist, loc = OPS[name]
            if dtype != torch.float64 or (fused and loc):
                continue
            q, v = (pts[:, idx], dirs[:, idx]) if loc else (pts, dirs)
            if dist:
                out[kind][name] = _exact_distance(kind, spec.params, q, v, not loc)
            else:
                out[kind][name] = _exact_safety(kind, spec.params, q, not loc)
    return out if any(v is not None for ops in out.values() for v in ops.values()) else None
