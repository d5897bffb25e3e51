"""A batch whose tunnels each respect their largest allowed buffer keeps several steps per launch: the limit is
one buffer's, so no table may exceed it, and the tables of all tunnels together may. Populations are bit for bit
those of an unlimited batch."""
import numpy as np
import pytest

import cells_b200.geometry as g
from cells_b200 import Batch2D
from cells_b200.rng import perturbed_rest2

pytestmark = pytest.mark.gpu

SIZES = [(300, 80), (400, 100), (37, 29), (64, 64)]


def run(limit, every):
    # limit: bytes per buffer beyond the largest population buffer; None: unlimited
    most = max(36 * W * H for W, H in SIZES)
    b = Batch2D([dict(left=2, right=2, bottom=2, top=2, tau=0.56, uIn=0.05, width=W, height=H, forceEvery=every,
                      exactArithmetic=True, maxBufferBytes=0 if limit is None else most + limit) for W, H in SIZES * 6])
    for t, (W, H) in zip(b.tunnels, SIZES * 6):
        sdf = g.empty_sdf(W, H)
        for k in range(6):  # enough body cells to fill the coefficient slots of the smallest tunnel
            g.add_circle(sdf, W, H, 5 + 5 * k, H / 2 + (-1) ** k * H / 5, 1.6)
        t.setSdf(sdf)
        t.initField(perturbed_rest2(W, H, 1e-3))
    before = b.launchCount()
    b.step(28)
    launches = b.launchCount() - before
    out = [t.readPopulations() for t in b.tunnels], [t.readForces() for t in b.tunnels]
    b.destroy()
    return launches, out


@pytest.mark.parametrize("every", [0, 2])
@pytest.mark.parametrize("limit", [0, 1 << 20])
def test_limited_batch_takes_several_steps_per_launch(limit, every):
    many, free = run(None, every)
    few, held = run(limit, every)
    assert many <= 14 and few <= 14  # 28 steps, at least 3 of them per launch, and the force sums
    for a, b in zip(free[0], held[0]):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    for a, b in zip(free[1], held[1]):
        assert a == b
