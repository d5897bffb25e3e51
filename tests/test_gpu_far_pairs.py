"""FP32 at odd widths: cells x and x + 32 of a row in one thread (fast build) against the exact build's one cell
per thread, at the widths where the second cell is missing, the outlet changes sides or a tile holds one column."""
import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Solver3D
from cells_b200.rng import perturbed_rest3

pytestmark = pytest.mark.gpu

STEPS = 12
# one step leaves at most 40 roundings of the largest population, which relaxation does not amplify in 12 steps
TOL = STEPS * 40 * 6e-8


def run(W, H, D, exact, smag, body, **kw):
    s = Solver3D.create(W, H, D, tau=0.56, uIn=0.05, spongeFraction=0.2, absorb=0.05, forceEvery=1, smagorinsky=smag,
                        exactArithmetic=exact, **kw)
    sdf = g.empty_sdf3(W, H, D)
    for x, y, z, r in body:
        g.add_sphere(sdf, W, H, D, x, y, z, r)
    s.setSdf(sdf)
    s.initField(perturbed_rest3(W, H, D, 1e-3, ux=0.05))
    s.encodeSteps(STEPS)
    out = s.readPopulations(), s.readForcesArray()
    assert s.readStatus() == 0
    s.destroy()
    return out


@pytest.mark.parametrize("W", [3, 31, 33, 63, 65, 95, 97, 129])
@pytest.mark.parametrize("H,D", [(7, 6), (2, 5), (5, 2), (3, 3), (1, 1)])
@pytest.mark.parametrize("smag", [0.0, 0.1])
def test_matches_one_cell_per_thread(W, H, D, smag):
    body = [(W / 3, H / 2, D / 2, 1.3)] if min(W, H, D) >= 6 else []
    a, b = (run(W, H, D, exact, smag, body)[0] for exact in (False, True))
    assert np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b))


# bodies that hold the first or the second cell of a thread, a tile's edge, the inlet and the outlet column
@pytest.mark.parametrize("x", [0, 4, 31, 32, 36, 63, 64, 95, 96])
@pytest.mark.parametrize("workgroup", [0, 32, 64, 256])
def test_bodies_at_tile_edges(x, workgroup):
    a, fa = run(97, 11, 10, False, 0.1, [(x, 5, 5, 2.6)], workgroupSize=workgroup)
    b, fb = run(97, 11, 10, True, 0.1, [(x, 5, 5, 2.6)])
    assert np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b))
    # a sample adds up at most 400 links of two populations each
    assert fa.shape == fb.shape and np.max(np.abs(fa - fb)) <= 400 * 2 * TOL * np.max(np.abs(b))
