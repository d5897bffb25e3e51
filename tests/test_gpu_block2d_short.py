"""Short 2D runs without force samples on grids of many tiles: steps that no launch of three or more takes go through
the one-step kernel. Bit for bit against the oracle in the exact build, for every remainder, with a body drawn onto
a slip wall after each run (solid cells keep what both buffers held, whichever kernel took the last steps)."""
import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Batch2D, Solver
from cells_b200.rng import perturbed_rest2
from oracle.oracle import OracleSolver2D

pytestmark = pytest.mark.gpu


# FP32: 64x48 with a list, without one; FP64: 32x32 without a list, with 5 and with 3 steps
@pytest.mark.parametrize("precision,size,K", [("fp32", (500, 300), 5), ("fp32", (905, 605), 5), ("fp64", (300, 200), 5),
                                              ("fp64", (905, 605), 3)])
def test_remainders(precision, size, K):
    W, H = size
    cfg = dict(left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05, forceEvery=0)
    s = Solver.create(width=W, height=H, precision=precision, exactArithmetic=True, **cfg)
    o = OracleSolver2D(width=W, height=H, precision=precision, **cfg)
    for x in (s, o):
        sdf = g.empty_sdf(W, H)
        g.add_circle(sdf, W, H, W / 4, H / 2, H / 9)
        x.setSdf(sdf)
        x.initField(perturbed_rest2(W, H, 1e-3))
    for k, n in enumerate((2, 4, 6, 7, 9, 1, 12, 3)):
        before = s.launchCount()
        s.encodeSteps(n)
        few = precision == "fp32" and W > 500 and n < K  # one by one
        assert s.launchCount() - before == (n if few else n // K + (0, 1, 2, 1, 2)[n % K])
        o.encodeSteps(n)
        for x in (s, o):
            x.brush(40 + 40 * k, H - 1 if k % 2 else 0, 3.3, False, True)
    s.encodeSteps(5)
    o.encodeSteps(5)
    a, b = s.readPopulations(), np.ascontiguousarray(o.populations())
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    s.destroy()


# How a caller groups its steps: in the fast build, single steps and runs round differently. Each step leaves at most 18
# roundings of the largest population, which relaxation does not amplify. A fixed workgroup size takes one kernel.
@pytest.mark.parametrize("workgroup", [0, 128])
@pytest.mark.parametrize("precision,eps", [("fp32", 6e-8), ("fp64", 1.1e-16)])
@pytest.mark.parametrize("size", [(64, 48), (400, 100), (905, 605)])
def test_grouping_of_steps(workgroup, precision, eps, size):
    W, H = size
    out, n = [], 60
    for counts in ((n,), (1,) * n, (7, 1, 2, 1, 1, 13, 5, 30)):
        s = Solver.create(width=W, height=H, precision=precision, workgroupSize=workgroup, left=2, right=2, bottom=2,
                          top=2, tau=0.56, uIn=0.05, smagorinsky=0.1)
        sdf = g.empty_sdf(W, H)
        g.add_circle(sdf, W, H, W / 4, H / 2, H / 9)
        s.setSdf(sdf)
        s.initField(perturbed_rest2(W, H, 1e-3))
        for k in counts:
            s.encodeSteps(k)
        assert [v["step"] for v in s.readForces()] == list(range(1, n + 1))
        out.append(s.readPopulations())
        s.destroy()
    for a in out[1:]:
        if workgroup:
            assert np.array_equal(a, out[0])
        assert np.max(np.abs(a - out[0])) <= 2 * n * 18 * eps * np.max(np.abs(out[0]))


# Two sampled steps of a large batch of small tunnels: one by one, as a single tunnel of as many cells does not
@pytest.mark.parametrize("sizes,one_by_one", [([(500, 200)] * 24, True), ([(2400, 1000)], False)])
def test_two_sampled_steps(sizes, one_by_one):
    cfg = dict(left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05, exactArithmetic=True)
    b = Batch2D([dict(cfg, width=W, height=H) for W, H in sizes])
    W, H = sizes[0]
    sdf = g.empty_sdf(W, H)
    g.add_circle(sdf, W, H, W / 4, H / 2, H / 9)
    m = perturbed_rest2(W, H, 1e-3)
    for t in b.tunnels:
        t.setSdf(sdf)
        t.initField(m)
    before = b.launchCount()
    b.step(2)
    assert b.launchCount() - before == (2 if one_by_one else 3)  # and the force sums
    b.step(7)
    b.step(2)
    o = OracleSolver2D(width=W, height=H, **{k: v for k, v in cfg.items() if k != "exactArithmetic"})
    o.setSdf(sdf)
    o.initField(m)
    o.encodeSteps(11)
    f = np.ascontiguousarray(o.populations())
    for t in {0: b.tunnels[0], len(sizes) - 1: b.tunnels[-1]}.values():
        assert np.array_equal(t.readPopulations().view(np.uint8), f.view(np.uint8))
        assert [v["step"] for v in t.readForces()] == list(range(1, 12))
    b.destroy()


# a longer run goes through one kernel whatever its remainder: the same bits as its steps in launches of one
@pytest.mark.parametrize("size", [(500, 300), (905, 605)])
def test_longer_runs_take_one_kernel(size):
    W, H = size
    out = []
    for counts in ((16, 17), (15, 13, 5)):
        s = Solver.create(width=W, height=H, left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05, forceEvery=0)
        s.initField(perturbed_rest2(W, H, 1e-3))
        for n in counts:
            s.encodeSteps(n)
        out.append(s.readPopulations())
        s.destroy()
    assert np.array_equal(out[0], out[1])
