"""The batch's resident-row plan over frames in which no garment advances (phase changes, statistics, saved states), and what
the tuning reports of it: with the default variant one block per SM, whatever frame ran last."""
import numpy as np
import pytest

from drape_b200 import batch as BT
from drape_b200 import scenes as S

pytestmark = pytest.mark.gpu

SIZES = (600, 9000, 2500)


def _run(tuning):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    b = BT.BatchSolver(0)
    for k, n in enumerate(SIZES):
        b.add(S.tube_variant(80 + k, n, field_n=32))
    b.build()
    out = []
    for f in range(6):
        if f == 0:
            for k in range(len(SIZES)):
                b.set_phase(k, 0)
        if f == 3:
            b.set_phase(1, 1)
        b.stats(0)
        t = b.set_tuning(*tuning)  # sets what is set
        assert t["blocks"] == (sms if tuning == (0, 256) else sms * (1024 // tuning[1]))
        assert (t["row_lanes"], t["block_threads"]) == tuning
        b.step(1.0 / 60.0, 1, 2)
        out += [b.positions(k) for k in range(len(SIZES))]
    b.close()
    return out


def test_plan_over_frames_without_substeps(gpu):
    for a, b in zip(_run((0, 256)), _run((0, 512))):
        assert np.array_equal(a, b), np.abs(a - b).max()


def test_autotune_reports_the_launch_of_the_variant_it_chose(gpu):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    b = BT.BatchSolver(0)
    for k, n in enumerate(SIZES):
        b.add(S.tube_variant(80 + k, n, field_n=32))
    b.build()
    t = b.autotune(1)
    resident = (t["row_lanes"], t["block_threads"]) == (0, 256)
    assert t["blocks"] == (sms if resident else sms * (1024 // t["block_threads"]))
    b.close()


@pytest.mark.parametrize("garments, side, resident", [(297, 10, False), (296, 10, True), (297, 11, True)])
def test_many_tiny_garments_run_on_the_variants_own_blocks(gpu, garments, side, resident):
    """From three launches' worth of garments on, garments of at most 104 particles stay with the slot-parallel kernel. One
    frame within 1e-5 m of the same garments in two batches on 512-thread blocks, which has fewer blocks than garments
    here; the same PCG counts."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sms == 148

    def run(which, tuning):
        b = BT.BatchSolver(0)
        for k in which:
            b.add(S.sheet_on_sphere(n=side, height=0.16 + 0.001 * (k % 7), cg_tolerance=1e-2, max_cg=50))
        b.build()
        blocks = b.set_tuning(*tuning)["blocks"]
        b.step(1.0 / 60.0, 1, 2)
        x = [b.positions(k) for k in range(len(which))]
        its = [b.counters(k).cg_iterations for k in range(len(which))]
        b.close()
        return x, its, blocks

    x, its, blocks = run(range(garments), (0, 256))
    assert blocks == (sms if resident else 4 * sms)
    half = garments // 2
    xa, ia, _ = run(range(half), (0, 512))
    xb, ib, _ = run(range(half, garments), (0, 512))
    assert its == ia + ib
    assert max(np.abs(a.astype(np.float64) - b).max() for a, b in zip(x, xa + xb)) < 1e-5
