"""The box tests of a wide volume's search (navigation.cuh wide_meets, wide_near) where the
bound they compare with is special, against the scan of all daughters on the host."""
import numpy as np
import pytest

from test_wide_search import from_world, ws  # noqa: F401 (the fixture)
from vecgeom_b200 import workloads as W


def world(ws, half, daughters, filler):
    """A world box holding the given (half lengths, position) boxes, then 40 small ones."""
    from vecgeom_b200.geometry import Geometry
    g = Geometry(library=ws)
    b = W.VgbBuilder(g, close=False)
    lv = b.logical("world", b.box(half, half, half))
    placed = b.place(lv, b.transform())
    for k, (h, pos) in enumerate(daughters):
        b.place_daughter(lv, b.logical(f"d{k}", b.box(*h)), b.transform(*pos))
    dot = b.logical("dot", b.box(*filler[0]))
    for k in range(40):
        b.place_daughter(lv, dot, b.transform(filler[1], filler[1], filler[1] * (k - 20) / 20))
    b.set_world(placed)
    return g


@pytest.mark.parametrize("what", [1, 2, 3])
def test_an_inside_answer_beats_a_hit_behind_the_point(ws, what):
    """The first box answers with its face just behind the point, -0.5 away along the ray;
    the second, which the point is in, with -1, though its own face is 0.3 behind."""
    g = world(ws, 500., [((10., 10., 10.), (0., 0., 0.)), ((5., 5., 5.), (10., 14.9, 0.))],
              ((1., 1., 1.), 400.))
    p = np.array([[10. - 1e-10], [10.2], [0.]])
    d = np.array([[-2e-10], [1.], [0.]])
    want, got = (from_world(ws, g, p, d, boxes, what)[0] for boxes in (0, 1))
    assert got == want


@pytest.mark.parametrize("what", [0, 2])
@pytest.mark.parametrize("unit", [1., 1e6, 1e16, 1e20])
def test_safeties_at_any_scale(ws, what, unit):
    g = world(ws, 1000. * unit, [((50. * unit,) * 3, (500. * unit, 10. * unit, 0.))],
              ((10. * unit,) * 3, 700. * unit))
    rng = np.random.default_rng(2)
    p = np.ascontiguousarray(rng.uniform(-300., 300., (3, 200)) * unit)
    d = np.ascontiguousarray(W.isotropic(rng, 200))
    want, got = (from_world(ws, g, p, d, boxes, what)[0] for boxes in (0, 1))
    assert got == want
