"""Several D2Q9 steps per launch (tiles with margins in shared memory) against the CPU oracle, bit for bit in
the exact build, at tile edges, remainders, periodic seams, every region shape and mixed step counts."""
import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Batch2D, Solver
from cells_b200.rng import perturbed_rest2
from oracle.oracle import OracleSolver2D

pytestmark = pytest.mark.gpu

CHANNEL, PERIODIC, CAVITY, SLIP = (2, 2, 2, 2), (0, 0, 0, 0), (1, 1, 1, 3), (2, 2, 0, 0)
# a force sample is an f64 sum of at most 1,600 link terms below 1 in another order: 1600 eps sum|t| < 1e-10 as a
# bound; the terms are near 0.2 and cancel
FORCE_TOL = 1e-10


def case(modes, every=1, smag=0.0):
    left, right, bottom, top = modes
    return dict(left=left, right=right, bottom=bottom, top=top, tau=0.56, uIn=0.05, uLid=0.03, absorb=0.02,
                spongeFraction=0.2 if left == 2 else 0, forceEvery=every, smagorinsky=smag,
                bodyForce=(1e-5, 2e-6) if left == 0 else (0, 0))


def body(W, H, seam):
    sdf = g.empty_sdf(W, H)
    if min(W, H) >= 7:
        g.add_circle(sdf, W, H, W / 4, H / 2, max(1.3, min(W, H) / 9))
        if seam:  # across the periodic x seam
            g.add_circle(sdf, W, H, W - 1, H / 3, 2.2)
    return sdf


def compare(W, H, cfg, precision, counts, edit=None):
    s = Solver.create(width=W, height=H, precision=precision, exactArithmetic=True, **cfg)
    o = OracleSolver2D(width=W, height=H, precision=precision, **cfg)
    for x in (s, o):
        x.setSdf(body(W, H, cfg["left"] == 0))
        x.initField(perturbed_rest2(W, H, 1e-3))
        for n in counts:
            x.encodeSteps(n)
        if edit:
            edit(x)
            for n in counts:
                x.encodeSteps(n)
    a, b = s.readPopulations(), np.ascontiguousarray(o.populations())
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    fa, fb = s.readForces(), o.readForces()
    assert [v["step"] for v in fa] == [v["step"] for v in fb]
    for v, w in zip(fa, fb):
        assert abs(v["fx"] - w["fx"]) <= FORCE_TOL and abs(v["fy"] - w["fy"]) <= FORCE_TOL
    s.destroy()


# 18 x 10 cells per tile of a small tunnel: exact, one over, one short, one row, one cell
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("size", [(36, 28), (37, 29), (35, 41), (50, 1), (3, 3), (64, 7)])
@pytest.mark.parametrize("modes", [CHANNEL, PERIODIC, CAVITY, SLIP])
def test_tile_edges(precision, size, modes):
    compare(*size, case(modes, every=3, smag=0.1), precision, (2, 7, 1, 130, 4))


# the smallest grids take 32x24 regions; larger ones 32x32, 64x32, 64x48 with and without a list of links (FP64 32x32
# with 7 steps and a list, with 5 and with 3 steps without)
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("size", [(400, 100), (300, 200), (500, 300), (905, 605)])
@pytest.mark.parametrize("modes", [CHANNEL, PERIODIC])
def test_region_shapes(precision, size, modes):
    compare(*size, case(modes, smag=0.1), precision, (7, 6))


@pytest.mark.parametrize("rebuild", [False, True])
def test_brush(rebuild):
    def edit(x):
        x.brush(20, 12, 2.4, False, rebuild)

    compare(60, 40, case(CHANNEL), "fp32", (9, 2), edit)


def test_more_body_cells_than_coefficient_slots():
    W, H = 120, 90
    sdf = g.empty_sdf(W, H)
    for y in range(4, H - 4, 5):
        for x in range(4, W - 4, 5):
            g.add_circle(sdf, W, H, x + 0.3, y + 0.1, 1.2)
    cfg = case(CHANNEL, every=2)
    s = Solver.create(width=W, height=H, exactArithmetic=True, **cfg)
    o = OracleSolver2D(width=W, height=H, **cfg)
    for x in (s, o):
        x.setSdf(sdf)
        x.initField(perturbed_rest2(W, H, 1e-3))
        x.encodeSteps(40)
    assert np.array_equal(s.readPopulations().view(np.uint8), np.ascontiguousarray(o.populations()).view(np.uint8))
    s.destroy()


# The fast builds of the two kernels round differently: each step leaves at most 18 roundings of the largest
# population, which relaxation does not amplify.
@pytest.mark.parametrize("precision,eps", [("fp32", 6e-8), ("fp64", 1.1e-16)])
@pytest.mark.parametrize("modes", [CHANNEL, PERIODIC])
def test_fast_build_and_batches_match_single_steps(precision, eps, modes):
    sizes, n = [(40, 33), (131, 64), (18, 14)], 131
    batch = Batch2D([dict(case(modes, every=2, smag=0.1), width=W, height=H, precision=precision) for W, H in sizes])
    for t, (W, H) in zip(batch.tunnels, sizes):
        t.setSdf(body(W, H, modes is PERIODIC))
        t.initField(perturbed_rest2(W, H, 1e-3))
    batch.step(n)
    for t, (W, H) in zip(batch.tunnels, sizes):
        one = Solver.create(width=W, height=H, precision=precision, workgroupSize=128, **case(modes, every=2, smag=0.1))
        one.setSdf(body(W, H, modes is PERIODIC))
        one.initField(perturbed_rest2(W, H, 1e-3))
        one.encodeSteps(n)
        a, b = t.readPopulations(), one.readPopulations()
        assert np.max(np.abs(a - b)) <= 2 * n * 18 * eps * np.max(np.abs(b))
        assert len(t.readForces()) == len(one.readForces()) == n // 2
        one.destroy()
    batch.destroy()


# a periodic side bounds the steps per launch; below 3 cells steps go one by one, as they do for a fixed block size
@pytest.mark.parametrize("size", [(40, 2), (40, 4), (5, 30)])
def test_new_modes_choose_again(size):
    out = []
    for workgroup in (0, 128):
        s = Solver.create(width=size[0], height=size[1], exactArithmetic=True, workgroupSize=workgroup, **case(CHANNEL, 2))
        s.initField(perturbed_rest2(*size, 1e-3))
        s.encodeSteps(9)
        s.update(left=0, right=0, bottom=0, top=0, uIn=0.0)
        s.encodeSteps(9)
        s.update(left=2, right=2, bottom=2, top=2, uIn=0.05)
        s.encodeSteps(11)
        out.append(s.readPopulations())
        s.destroy()
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(out[0], out[1])
