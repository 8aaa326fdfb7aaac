"""Bounded waits that run out in the middle of a solve: with a limit of a nanosecond any exchange may give up, in some
blocks and not in others. The step either succeeds or fails with the device error, and the solver goes on as if nothing had
been: from the same state it then takes the same step as one whose waits never ran out."""
import numpy as np
import pytest

from drape_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [12, 40, 59, 70], ids=["cluster_small", "cluster", "cluster_largest", "grid"])
def test_solver_survives_waits_that_run_out(gpu, side):
    scene = S.sheet_on_sphere(n=side, height=0.16, cg_tolerance=1e-6, max_cg=200)
    a, b = gpu.CudaSolver(0), gpu.CudaSolver(0)
    for s in (a, b):
        s.build(scene)
        s.step(1.0 / 60.0, 1, 2)
    start = b.snapshot()
    b.step(1.0 / 60.0, 1, 2)
    ref = b.positions()
    for _ in range(20):
        a.set_barrier_limit(1)
        try:
            a.step(1.0 / 60.0, 1, 2)
        except RuntimeError as e:
            assert "timed out" in str(e), e
        a.set_barrier_limit(0)
        a.restore(start)
        a.step(1.0 / 60.0, 1, 2)
        assert np.array_equal(a.positions(), ref)
        a.restore(start)
    a.close()
    b.close()
