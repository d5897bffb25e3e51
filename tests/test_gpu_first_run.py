"""The first run of a handle that samples forces allocates nothing: what it needs comes with the handle (2D) or with
the body (3D). The free memory of the device shows an allocation of some MB; the kernels are loaded by a run of
another handle before."""
import pytest

import cells_b200.geometry as g
from cells_b200 import Batch2D, Solver, Solver3D

pytestmark = pytest.mark.gpu


def free():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [2, 28])
def test_2d(precision, n):
    W, H = 3000, 1000  # force partials of a run: 3 MB (FP32) and more
    cfg = dict(width=W, height=H, precision=precision, left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05)
    sdf = g.empty_sdf(W, H)
    g.add_circle(sdf, W, H, W / 4, H / 2, 40)
    for measured in (False, True):
        s = Solver.create(**cfg)
        s.setSdf(sdf)
        s.initField()
        s.synchronize()
        before = free()
        s.encodeSteps(n)
        s.synchronize()
        if measured:
            assert free() == before
        assert len(s.readForces()) == n
        s.destroy()


def test_2d_batch():
    for measured in (False, True):
        b = Batch2D([dict(width=900, height=300, left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05) for _ in range(16)])
        b.synchronize()
        before = free()
        b.step(10)
        b.synchronize()
        if measured:
            assert free() == before
        b.destroy()


@pytest.mark.parametrize("precision", ["fp32", "fp16", "fp64"])
def test_3d(precision):
    W, H, D = 160, 96, 96  # about 60,000 body cells: 7 MB of force partials
    sdf = g.empty_sdf3(W, H, D)
    g.add_sphere(sdf, W, H, D, 60, 48, 48, 40)
    for measured in (False, True):
        s = Solver3D.create(W, H, D, precision=precision, tau=0.6, uIn=0.05, forceEvery=1)
        s.setSdf(sdf)
        s.initField()
        s.synchronize()
        before = free()
        s.encodeSteps(8)
        s.synchronize()
        if measured:
            assert free() == before
        assert len(s.readForces()) == 8
        s.destroy()
