"""Short 3D runs with force samples: the force is summed in the step, or by one kernel after the run where that is
faster. The sums have one order, so runs of n steps and n runs of one step give the same bits; and a run without a
body, or on a grid whose steps do not wait for the sum, launches nothing but its steps."""
import numpy as np
import pytest

from cells_b200 import Solver3D, geometry as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16", "fp64"])
@pytest.mark.parametrize("W,H,D", [(48, 24, 24), (90, 40, 38), (160, 64, 62)])
@pytest.mark.parametrize("every", [1, 3])
def test_grouping(precision, W, H, D, every):
    sdf = g.empty_sdf3(W, H, D)
    g.add_sphere(sdf, W, H, D, W / 4, H / 2, D / 2, H / 7)
    out = []
    for counts in ((1,) * 62, (2, 3, 4, 53), (60, 2)):
        s = Solver3D.create(W, H, D, precision=precision, tau=0.56, uIn=0.05, forceEvery=every)
        s.setSdf(sdf)
        s.initField()
        for n in counts:
            s.encodeSteps(n)
        out.append((s.readPopulations(), s.readForces()))
        s.destroy()
    for f, forces in out[1:]:
        assert np.array_equal(f.view(np.uint8), out[0][0].view(np.uint8))
        assert forces == out[0][1] and len(forces) == 62 // every


@pytest.mark.parametrize("size,body,launches", [((48, 24, 24), True, {2: 3, 3: 4, 8: 9}), ((48, 24, 24), False, {2: 2, 8: 8, 60: 60}),
                                                ((128, 64, 64), True, {2: 2, 3: 4}),
                                                ((160, 64, 62), True, {2: 2, 8: 8, 47: 47, 48: 49})])
def test_launches(size, body, launches):
    W, H, D = size
    s = Solver3D.create(W, H, D, precision="fp32", tau=0.56, uIn=0.05, forceEvery=1)
    if body:
        sdf = g.empty_sdf3(W, H, D)
        g.add_sphere(sdf, W, H, D, W / 4, H / 2, D / 2, H / 7)
        s.setSdf(sdf)
    s.initField()
    for n, want in launches.items():
        before = s.launchCount()
        s.encodeSteps(n)
        assert s.launchCount() - before == want
    assert [v["step"] for v in s.readForces()] == list(range(1, sum(launches) + 1))
    s.destroy()


# a cylinder across the grid: many body blocks, for whose count the steps of a larger grid or of FP16 wait after all
@pytest.mark.parametrize("precision,size,launches", [("fp16", (64, 32, 32), {3: 3, 4: 5}), ("fp32", (160, 80, 80), {11: 11, 12: 13})])
def test_launches_with_a_large_body(precision, size, launches):
    W, H, D = size
    x, y = np.meshgrid(np.arange(W), np.arange(H))
    sdf = np.tile((np.hypot(x - W / 4, y - H / 2 - 0.3) - 0.12 * H).astype(np.float32).reshape(-1), D)
    out = []
    for alone in (False, True):
        s = Solver3D.create(W, H, D, precision=precision, tau=0.56, uIn=0.05, forceEvery=1)
        s.setSdf(sdf)
        s.initField()
        for n, want in launches.items():
            before = s.launchCount()
            for _ in range(n if alone else 1):
                s.encodeSteps(1 if alone else n)
            assert s.launchCount() - before == (n if alone else want)
        out.append((s.readPopulations(), s.readForces()))
        s.destroy()
    assert np.array_equal(out[0][0].view(np.uint8), out[1][0].view(np.uint8)) and out[0][1] == out[1][1]
