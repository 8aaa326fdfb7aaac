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
