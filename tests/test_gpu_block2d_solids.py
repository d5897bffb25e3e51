"""Cells that become solid between steps beside a slip wall. No step writes a solid cell, so it keeps the
populations that each of the two buffers held at that moment; a slip row mirrors populations of its own row, a
solid's too, and so must see the two buffers in turn, in one launch of several steps as step by step. Bit for
bit in the exact build, with and without the list of links."""
import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Batch2D, Solver
from cells_b200.rng import perturbed_rest2
from oracle.oracle import OracleSolver2D

pytestmark = pytest.mark.gpu

# FP32: 32x24 regions, 64x32 regions, 64x48 without a list. FP64: 32x24, 32x32 with 5 steps without a list (both sizes)
SMALL, MIDDLE, LARGE = (60, 40), (300, 200), (905, 605)


def solvers(W, H, precision, left=2):
    cfg = dict(left=left, right=left, bottom=2, top=2, tau=0.56, uIn=0.05, absorb=0.02,
               spongeFraction=0.2 if left == 2 else 0, bodyForce=(0, 0) if left == 2 else (1e-5, 2e-6))
    return [Solver.create(width=W, height=H, precision=precision, exactArithmetic=True, **cfg),
            OracleSolver2D(width=W, height=H, precision=precision, **cfg)]


def equal(s, o):
    a, b = s.readPopulations(), np.ascontiguousarray(o.populations())
    return np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("size", [SMALL, MIDDLE, LARGE])
@pytest.mark.parametrize("wall", ["bottom", "top"])
@pytest.mark.parametrize("before", [3, 4])
@pytest.mark.parametrize("how", ["brush", "setSdf"])
def test_body_onto_a_slip_wall(precision, size, wall, before, how):
    W, H = size
    y = 1 if wall == "bottom" else H - 2
    s, o = solvers(W, H, precision)
    moved = g.empty_sdf(W, H)
    g.add_circle(moved, W, H, W / 2, y, 3.4)
    for x in (s, o):
        sdf = g.empty_sdf(W, H)
        g.add_circle(sdf, W, H, W / 4, H / 2, 2.8)
        x.setSdf(sdf)
        x.initField(perturbed_rest2(W, H, 1e-3))
        x.encodeSteps(before)
        if how == "brush":
            x.brush(W / 2, y, 3.4, False, True)
        else:
            x.setSdf(moved)
        for n in (7, 2, 1):
            x.encodeSteps(n)
    assert equal(s, o)
    s.destroy()


# the row's end is periodic: a solid in the last column stands in a margin of the first tile
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("left", [0, 2])
def test_split_runs_agree(precision, left):
    W, H = SMALL
    out = []
    for counts in ((7, 8), (1,) * 15):
        s, o = solvers(W, H, precision, left)
        for x in (s, o):
            x.initField(perturbed_rest2(W, H, 1e-3))
            x.encodeSteps(5)
            x.brush(W - 2, 1, 2.6, False, True)
            for n in counts:
                x.encodeSteps(n)
        assert equal(s, o)
        out.append(s.readPopulations())
        s.destroy()
    assert np.array_equal(out[0], out[1])


# several rebuilds between two runs: cells covered by the second, uncovered (refilled) and covered again
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("before", [(7,), (3, 1), (5, 2)])
def test_rebuilds_between_runs(precision, before):
    W, H = SMALL
    s, o = solvers(W, H, precision)
    for x in (s, o):
        x.initField(perturbed_rest2(W, H, 1e-3))
        for n in before:
            x.encodeSteps(n)
        x.brush(20, 1, 2.6, False, True)
        x.brush(40, 0, 2.6, False, True)
        x.brush(20, 1, 3.6, True, True)
        x.brush(21, 0, 2.6, False, True)
        x.encodeSteps(3)
        x.brush(30, H - 1, 2.6, False, True)
        x.encodeSteps(5)
    assert equal(s, o)
    s.destroy()


# the autotuner's trials step the flow and restore it: a body drawn after them finds both buffers as they were
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("before", [4, 7])
def test_body_after_autotune(precision, before):
    W, H = SMALL
    cfg = dict(left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05)
    b = Batch2D([dict(cfg, width=W, height=H, precision=precision, exactArithmetic=True)])
    o = OracleSolver2D(width=W, height=H, precision=precision, **cfg)
    t, m = b.tunnels[0], perturbed_rest2(W, H, 1e-3)
    t.initField(m)
    o.initField(m)
    b.step(before)
    o.encodeSteps(before)
    b.autotune(11)
    for x in (t, o):
        x.brush(30, 1, 3.2, False, True)
    b.step(5)
    o.encodeSteps(5)
    assert equal(t, o)
    b.destroy()
