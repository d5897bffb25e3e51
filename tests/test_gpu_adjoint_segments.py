"""A recorded run that fits one segment (steps <= checkpointEvery): its states are recomputed on the sweep's own
stream, right before the first adjoint step, so only that step's launch orders the two. Against the same run
in short segments: the states are the same bits and every sum has a fixed order, so the results are equal."""
import numpy as np
import pytest

from cells_b200 import Solver3D, geometry as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("W,H,D", [(96, 48, 40), (97, 40, 33), (34, 9, 7)])
@pytest.mark.parametrize("steps", [2, 7, 12])
def test_one_segment_equals_short_segments(precision, W, H, D, steps):
    sdf = g.empty_sdf3(W, H, D)
    g.add_sphere(sdf, W, H, D, W / 3, H / 2, D / 2, H / 5)
    out = []
    for every in (steps, steps + 9, 1):
        s = Solver3D.create(W, H, D, precision=precision, tau=0.6, uIn=0.05, spongeFraction=0.3, absorb=0.02, forceEvery=0)
        s.setSdf(sdf)
        s.initField()
        s.encodeSteps(5)
        first = s.step
        j = s.adjointForward(steps, first + 1, first + steps, checkpointEvery=every, component=0)
        # the second sweep finds the states of the first in its buffers, the first one what was there before
        out += [(j, s.adjointBackward(wantAdjoint=True)) for _ in range(2)]
        s.destroy()
    for j, o in out[1:]:
        assert j == out[0][0] and o["du"] == out[0][1]["du"]
        for k in ("adjoint", "dsdf"):
            assert np.array_equal(o[k].view(np.uint8), out[0][1][k].view(np.uint8))


# More slices of blocks than one launch holds: the adjoint step of a thin, deep grid goes out in two launches.
@pytest.mark.parametrize("precision,size", [("fp64", (32, 3, 22000)), ("fp32", (64, 2, 20000))])
def test_more_slices_than_a_launch_holds(precision, size):
    W, H, D = size
    out = []
    for every in (3, 1):
        s = Solver3D.create(W, H, D, precision=precision, tau=0.6, uIn=0.05, forceEvery=0)
        sdf = g.empty_sdf3(W, H, D)
        g.add_sphere(sdf, W, H, D, W / 3, 0.6, D - 40, 2.2)
        s.setSdf(sdf)
        s.initField()
        s.encodeSteps(2)
        first = s.step
        s.adjointForward(3, first + 1, first + 3, checkpointEvery=every, component=0)
        out.append(s.adjointBackward(wantAdjoint=True))
        s.destroy()
    for k in ("adjoint", "dsdf"):
        assert np.any(out[0][k]) and np.array_equal(out[0][k].view(np.uint8), out[1][k].view(np.uint8))
    assert out[0]["du"] == out[1]["du"]
