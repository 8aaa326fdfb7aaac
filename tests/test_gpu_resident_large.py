"""Several rows a thread: with pinned rows and columns in every block, beyond 213k particles (where the 1024-thread kernel
takes over), and with the PCG capped at one and at three iterations (the line to the 1024-thread kernel), against that
kernel, whose row products and recurrences the resident-row kernels repeat: bit-identical positions, the same counts."""
import numpy as np
import pytest

from drape_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _pinned_sheet(n):
    scene = S.sheet_on_sphere(n=n, height=0.16, cg_tolerance=1e-2, max_cg=50)
    x = scene.garments[0].initial_positions
    scene.pins += [(v, tuple(x[v])) for v in range(0, n * n, 61)]
    scene.pins += [(v, tuple(x[v])) for v in range(5000, 5700)]  # whole slices of 32 rows
    return scene


CASES = {
    "pinned_90k": (lambda: _pinned_sheet(300), 512),
    "pinned_160k": (lambda: _pinned_sheet(400), 512),
    "beyond_213k": (lambda: S.sheet_on_sphere(n=465, height=0.16, cg_tolerance=1e-2, max_cg=50), 1024),
    "one_iteration": (lambda: S.sheet_on_sphere(n=300, height=0.16, cg_tolerance=1e-6, max_cg=1), 1024),
    "three_iterations": (lambda: S.sheet_on_sphere(n=300, height=0.16, cg_tolerance=1e-6, max_cg=3), 512),
}


@pytest.mark.parametrize("name", list(CASES))
def test_large_scenes_match_the_1024_thread_kernel(gpu, name):
    make, threads = CASES[name]
    out = []
    for variant in (0, 3):
        s = gpu.CudaSolver(0)
        s.set_pcg_variant(variant)
        s.build(make())
        assert s.solve_threads() == (threads if variant == 0 else 1024)
        for _ in range(2):
            s.step(1.0 / 60.0, 1, 2)
        out.append((s.positions(), s.cg_history()))
        s.close()
    (xa, ha), (xb, hb) = out
    assert np.isfinite(xa).all() and np.array_equal(ha, hb), (ha, hb)
    assert np.array_equal(xa, xb), np.abs(xa - xb).max()


@pytest.mark.parametrize("cap, resident", [(3, False), (6, True)])
def test_batch_of_capped_solves(gpu, cap, resident):
    from drape_b200 import batch as BT
    from drape_b200.scene import Settings
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    out = []
    for tuning in ((0, 256), (0, 512)):
        b = BT.BatchSolver(0)
        for k in range(4):
            b.add(S.tube_variant(40 + k, 30000, field_n=16, settings=Settings(cg_tolerance=1e-6, max_cg_iterations=cap)))
        b.build()
        t = b.set_tuning(*tuning)
        assert t["blocks"] == (sms * (1024 // tuning[1]) if tuning[1] == 512 or not resident else sms)
        b.step(1.0 / 60.0, 1, 2)
        out.append([b.positions(k) for k in range(4)])
        b.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y), np.abs(x - y).max()
