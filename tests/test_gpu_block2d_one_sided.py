"""Axes that are periodic on one side only: the margin behind that side holds cells whose own far side is a wall
or open, next to the real first or last column. Bit for bit against the oracle in the exact build, with and
without the list of links, with bodies at the seam: fluid in the first column and solid in the second at more than
half the link (the rule that reads the cell's own population), solids beside slip rows, and a body in each corner."""
import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Solver
from cells_b200.rng import perturbed_rest2
from oracle.oracle import OracleSolver2D

pytestmark = pytest.mark.gpu

# left, right, bottom, top; 0 periodic, x: 1 wall 2 open, y: 1 wall 2 slip 3 moving
X_MODES = [(0, 1, 1, 1), (0, 2, 2, 2), (1, 0, 2, 2), (2, 0, 1, 1), (0, 1, 0, 0)]
Y_MODES = [(2, 2, 0, 1), (2, 2, 0, 2), (1, 1, 0, 3), (2, 2, 1, 0), (2, 2, 2, 0), (1, 1, 3, 0), (0, 0, 2, 0), (0, 0, 0, 2)]
BOTH = [(0, 1, 0, 2), (1, 0, 2, 0), (0, 2, 2, 0), (2, 0, 0, 3)]


# FP32: one tile, two tiles a row, 64x32 regions, 64x48 without a list; FP64: 32x24, 32x32 without a list
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("size", [(15, 9), (40, 33), (300, 200), (905, 605)])
@pytest.mark.parametrize("modes", X_MODES + Y_MODES + BOTH)
def test_one_sided(precision, size, modes):
    W, H = size
    left, right, bottom, top = modes
    cfg = dict(left=left, right=right, bottom=bottom, top=top, tau=0.56, uIn=0.05, uLid=0.03, forceEvery=2, smagorinsky=0.1)
    sdf = g.empty_sdf(W, H)
    # a cell between fluid columns 0 | 2 and rows 0 | 2, and solids in the first and last columns and rows themselves
    for x, y, r in [(2.0, H / 2, 1.3), (W - 3.0, H / 2 + 1, 1.3), (W / 2, 2.0, 1.3), (W / 2 - 2, H - 3.0, 1.3),
                    (0.2, H / 4, 1.2), (W - 1.3, 3 * H / 4, 1.2), (W / 4, 0.3, 1.2), (3 * W / 4, H - 1.2, 1.2), (0, 0, 0.7),
                    (W - 1, H - 1, 0.7)]:
        g.add_circle(sdf, W, H, x, y, r)
    s = Solver.create(width=W, height=H, precision=precision, exactArithmetic=True, **cfg)
    o = OracleSolver2D(width=W, height=H, precision=precision, **cfg)
    for x in (s, o):
        x.setSdf(sdf)
        x.initField(perturbed_rest2(W, H, 1e-3))
        for n in (7, 4, 2):
            x.encodeSteps(n)
    a, b = s.readPopulations(), np.ascontiguousarray(o.populations())
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    fa, fb = s.readForces(), o.readForces()
    assert [v["step"] for v in fa] == [v["step"] for v in fb]
    for v, w in zip(fa, fb):  # an f64 sum of at most 1,600 link terms below 1 in another order
        assert abs(v["fx"] - w["fx"]) <= 1e-10 and abs(v["fy"] - w["fy"]) <= 1e-10
    s.destroy()
