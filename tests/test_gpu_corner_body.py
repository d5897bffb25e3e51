"""A body that touches the row y = z = 0: the row's inlet cell, the first cell of every buffer, is then in the body
list, and none of its sources may be looked up (they lie before the buffers' first element). The flags of the larger
grids are an allocation of their own. Bit for bit against the oracle in the exact build."""
import numpy as np
import pytest

from cells_b200 import Solver3D, geometry as g
from cells_b200.rng import perturbed_rest3
from oracle.oracle import OracleSolver3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16", "fp64"])
@pytest.mark.parametrize("size,steps", [((3, 1, 1), 5), ((5, 2, 2), 5), ((33, 7, 6), 6), ((64, 12, 11), 6), ((140, 64, 62), 3),
                                        ((141, 64, 62), 3)])
def test_body_on_the_first_row(precision, size, steps):
    W, H, D = size
    cfg = dict(tau=0.56, uIn=0.05, spongeFraction=0.15, absorb=0.02, forceEvery=1)
    s = Solver3D.create(W, H, D, precision=precision, exactArithmetic=True, **cfg)
    o = OracleSolver3D(W, H, D, precision, **cfg)
    sdf = g.empty_sdf3(W, H, D)
    g.add_sphere(sdf, W, H, D, 1.4, 0.2, 0.1, 1.3)
    for x in (s, o):
        x.setSdf(sdf)
        x.initField(perturbed_rest3(W, H, D, 1e-4, ux=0.05))
        x.encodeSteps(steps)
    a, b = s.readPopulations(), np.ascontiguousarray(o.populations())
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    assert len(s.readForces()) == steps
    s.destroy()
