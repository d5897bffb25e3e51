"""Force samples of runs of steps, whose body blocks' partials are added up once per run (a step graph, or
steps launched one by one), against steps taken one at a time, each of which reduces its own force."""
import numpy as np
import pytest

from cells_b200 import Solver3D, geometry as g
from cells_b200.rng import perturbed_rest3

pytestmark = pytest.mark.gpu


def solver(W, H, D, precision, every, body):
    s = Solver3D.create(W, H, D, precision=precision, tau=0.56, uIn=0.05, spongeFraction=0.2, absorb=0.02,
                        forceEvery=every)
    if body:
        sdf = g.empty_sdf3(W, H, D)
        g.add_sphere(sdf, W, H, D, *body)
        s.setSdf(sdf)
    s.initField(perturbed_rest3(W, H, D, 1e-3, ux=0.05))
    return s


@pytest.mark.parametrize("precision", ["fp32", "fp16", "fp64"])
@pytest.mark.parametrize("every", [1, 3, 17])
@pytest.mark.parametrize("body", [None, (8, 6, 5, 0.6), (9, 6, 5, 4.2)])  # none; one block's cells; many blocks
def test_runs_match_single_steps(precision, every, body):
    W, H, D = 26, 12, 10
    a, b = (solver(W, H, D, precision, every, body) for _ in range(2))
    for n in (2, 131, 256, 1, 40):  # a short run, a graph and a rest, graphs only, a single step, a rest
        a.encodeSteps(n)
        for _ in range(n):
            b.encodeSteps(1)
    fa, fb = a.readForcesArray(), b.readForcesArray()
    assert fa.shape == fb.shape and len(fa) == 430 // every
    assert np.array_equal(fa, fb)  # the same partials in the same order
    assert np.array_equal(a.readPopulations().view(np.uint8), b.readPopulations().view(np.uint8))
    assert a.readStatus() == 0
    a.destroy()
    b.destroy()
