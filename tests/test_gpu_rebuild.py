"""A solver that is built again between drapes, whose frames replay captured graphs: with the same mesh and other pins the
device view and every address can stay the same while the cluster kernel's layout changes (16 blocks see more unpinned rows
together than before, 148 blocks do not). The drape equals a new solver's."""
import numpy as np
import pytest

from drape_b200 import scenes as S
from drape_b200.scene import drape_drape_options

pytestmark = pytest.mark.gpu


def _sheet(lo, hi):
    """A 40 x 40 sheet of which particles lo to hi are free."""
    scene = S.sheet_on_sphere(n=40, cg_tolerance=1e-2, max_cg=50)
    x = scene.garments[0].initial_positions
    scene.pins += [(v, tuple(x[v])) for v in range(1600) if not lo <= v < hi]
    return scene


def _drape(solver, scene):
    solver.build(scene)
    o = drape_drape_options(substeps=1, iterations=2, frame_dt=1.0 / 60.0, max_assembly_seconds=0.05, seam_gap_done=0.001,
                            settle_rms_speed=1e-4, settle_hold_frames=3, max_sim_seconds=0.3, snapshot_every=30,
                            max_retries=3, energy_rise_frames=60, frames_per_wait=10)
    res = solver.drape_to_rest([scene.garments[0].id], o)
    return solver.positions(), int(res.frames_run)


def test_drape_after_a_rebuild_equals_a_new_solvers(gpu):
    scenes = [_sheet(745, 850), _sheet(700, 805), S.sheet_on_sphere(n=12, height=0.16, cg_tolerance=1e-2, max_cg=50),
              _sheet(745, 850), _sheet(0, 1600)]
    a = gpu.CudaSolver(0)
    for scene in scenes:
        xa, fa = _drape(a, scene)
        b = gpu.CudaSolver(0)
        xb, fb = _drape(b, scene)
        b.close()
        assert fa == fb
        assert np.array_equal(xa, xb), np.abs(xa - xb).max()
    a.close()
