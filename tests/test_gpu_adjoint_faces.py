"""The FP32 adjoint step against the FP64 one (the transposed step that the dot-product and
finite-difference tests pin) where its work split changes: x-pairs with face rows on the packed path,
odd widths on the one-cell path, partial tiles, bodies that touch slip faces (their rows leave the
packed path), and a segment of odd length with a terminal adjoint."""
import numpy as np
import pytest

from cells_b200 import Solver3D, geometry as g

pytestmark = pytest.mark.gpu


def run(precision, W, H, D, center, r, steps, K, terminal):
    sdf = g.empty_sdf3(W, H, D)
    g.add_sphere(sdf, W, H, D, *center, r)
    s = Solver3D.create(W, H, D, precision=precision, tau=0.6, uIn=0.05, spongeFraction=0.3, absorb=0.02, forceEvery=0)
    s.setSdf(sdf)
    s.initField()
    s.encodeSteps(8)
    first = s.step
    j = s.adjointForward(steps, first + steps // 2, first + steps, checkpointEvery=K, component=0)
    t = terminal.astype(np.float32 if precision == "fp32" else np.float64) if terminal is not None else None
    out = s.adjointBackward(terminal=t, wantAdjoint=True)
    solid = (s.readFlags() >> 19) & 1
    s.destroy()
    return j, out, solid


@pytest.mark.parametrize("terminal", [False, True])
@pytest.mark.parametrize("W,H,D,center,r", [
    (64, 6, 6, (20, 3, 3), 1.6),       # one whole tile per row, one tile of rows and planes
    (66, 7, 11, (30, 3, 5), 2.2),      # a second tile of one pair; rows and planes past the last tile
    (62, 12, 9, (20, 0.5, 4), 2.7),    # a body through the y = 0 face
    (70, 9, 12, (31, 4, 11.2), 2.9),   # a body through the z = D-1 face
    (33, 8, 10, (12, 7.5, 9.5), 3.1),  # odd width, a body in the corner of two faces
    (4, 3, 3, (9, 9, 9), 0.5),         # the thinnest grid with an interior; no body
])
def test_fp32_matches_fp64(W, H, D, center, r, terminal):
    steps, K = 9, 4
    t = np.random.default_rng(5).standard_normal(19 * W * H * D) if terminal else None
    j32, o32, solid = run("fp32", W, H, D, center, r, steps, K, t)
    j64, o64, _ = run("fp64", W, H, D, center, r, steps, K, t)
    fluid = np.tile(solid == 0, 19)
    # f32 rounding: about ten roundings of 6e-8 per step and value over 17 steps, in the norm
    tol = 2e-5
    a, b = o32["adjoint"].astype(np.float64)[fluid], o64["adjoint"][fluid]
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
    assert np.linalg.norm(o32["dsdf"] - o64["dsdf"]) <= tol * np.linalg.norm(o64["dsdf"])
    # sums over signed terms: against the sum of the magnitudes that enter
    assert abs(o32["du"] - o64["du"]) <= tol * (abs(o64["du"]) + np.sum(np.abs(b)))
    assert abs(j32 - j64) <= tol * max(abs(j64), 1e-3)
