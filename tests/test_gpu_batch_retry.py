"""A batch that goes on after a frame that blew up: what the solve left behind (a step that need not be finite) has no part in
the frames that follow the restore, whose line search starts from the energy at no step at all."""
import numpy as np
import pytest

from drape_b200 import batch as BT
from drape_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuning", [None, (0, 512)], ids=["resident", "slot_parallel"])
def test_frames_after_a_blow_up_equal_a_new_batchs(gpu, tuning):
    sizes = (600, 9000, 2500)
    a, b = BT.BatchSolver(0), BT.BatchSolver(0)
    for s in (a, b):
        for k, n in enumerate(sizes):
            s.add(S.tube_variant(70 + k, n, field_n=32))
        s.build()
        if tuning:
            s.set_tuning(*tuning)
        s.step(1.0 / 60.0, 1, 2)
        s.save()
    b.step(1.0 / 60.0, 1, 2)
    for dt in (1e6, 1e12, 1e18, 1e25):
        a.step(dt, 1, 2)
        a.restore()
        a.reset_counters()
        b.reset_counters()
        b.restore()
        for s in (a, b):
            s.step(1.0 / 60.0, 1, 2)
        for k in range(len(sizes)):
            assert np.array_equal(a.positions(k), b.positions(k))
            ca, cb = a.counters(k), b.counters(k)
            assert ca.line_search_halvings == cb.line_search_halvings and ca.cg_iterations == cb.cg_iterations
        a.restore()
    a.close()
    b.close()
