"""Edits of a 2D body and the block kernel's rules: brushes without a rebuild of the flags resolve the rules of
their own box, a stroke resolves them once. Bit for bit against the oracle in the exact build, with brushes across
the grid's edges (the box's cells have links over a periodic side, also where only one side is periodic)."""
import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Solver
from cells_b200.rng import perturbed_rest2
from oracle.oracle import OracleSolver2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("modes", [(2, 2, 2, 2), (0, 0, 0, 0), (0, 1, 0, 2), (1, 0, 2, 0)])
@pytest.mark.parametrize("size", [(60, 40), (11, 9)])
def test_brush_without_rebuild(precision, modes, size):
    W, H = size
    cfg = dict(zip(("left", "right", "bottom", "top"), modes), tau=0.56, uIn=0.05, forceEvery=0)
    s = Solver.create(width=W, height=H, precision=precision, exactArithmetic=True, **cfg)
    o = OracleSolver2D(width=W, height=H, precision=precision, **cfg)
    spots = [(W / 2, H / 2), (0.4, H / 3), (W - 1.2, H / 2), (W / 3, 0.3), (W / 2, H - 1.1), (0, 0), (W - 1, H - 1)]
    for x in (s, o):
        sdf = g.empty_sdf(W, H)
        for cx, cy in spots:
            g.add_circle(sdf, W, H, cx, cy, 1.4)
        x.setSdf(sdf)
        x.initField(perturbed_rest2(W, H, 1e-3))
        x.encodeSteps(3)
        for cx, cy in spots:  # the fractions of their links move, the flags stay
            x.brush(cx + 0.1, cy - 0.1, 1.6, False, False)
            x.encodeSteps(4)
    a, b = s.readPopulations(), np.ascontiguousarray(o.populations())
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    s.destroy()


def test_stroke_resolves_the_rules_once():
    W, H, n = 200, 120, 20
    s = Solver.create(width=W, height=H, exactArithmetic=True, left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05)
    o = OracleSolver2D(width=W, height=H, left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05)
    xy = [(60 + 2.0 * k, 60 + 0.7 * k) for k in range(n)]
    for x in (s, o):
        x.initField(perturbed_rest2(W, H, 1e-3))
        x.encodeSteps(7)
    before = s.launchCount()
    s.brushStroke(xy, 3.0, False)
    assert s.launchCount() - before <= n + 4  # each point's SDF; macro, counter, flags and rules
    for k, (cx, cy) in enumerate(xy):
        o.brush(cx, cy, 3.0, False, k + 1 == n)
    for x in (s, o):
        x.encodeSteps(9)
    a, b = s.readPopulations(), np.ascontiguousarray(o.populations())
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    s.destroy()
