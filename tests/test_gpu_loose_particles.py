"""Particles without neighbours (in no triangle and no seam), placed so that they fill the last warp of every solve block:
their rows are a diagonal block alone, kept in registers, so these warps have no slots in shared memory. The resident-row
kernels against the 1024-thread ones, with the initial network and without."""
import numpy as np
import pytest

from drape_b200 import learned
from drape_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _sheet_with_loose_particles():
    """148 x 64 sheet particles in rows of 128, four loose ones after every 64: on 148 SMs, 68 rows a block."""
    nx, ny = 128, 74
    g = S.piece_garment("sheet", 0.6, 0.4, nx, ny, S.jersey_fabric())
    n = g.vertex_count
    new = np.arange(n) + 4 * (np.arange(n) // 64)
    total = n + 4 * (n // 64)

    def spread(a, fill):
        out = np.broadcast_to(np.asarray(fill, a.dtype), (total, *a.shape[1:])).copy()
        out[new] = a
        return out

    loose = np.setdiff1d(np.arange(total), new)
    x = spread(np.stack([g.rest[:, 0], np.full(n, 0.5), g.rest[:, 1]], axis=1), 0.0)
    x[loose] = np.stack([np.linspace(-1, 1, len(loose)), np.ones(len(loose)), np.zeros(len(loose))], axis=1)
    scene = S.Scene([S.Garment(g.id, spread(g.rest, 0.0), spread(g.vertex_piece, 0),
                               spread(g.vertex_area, g.vertex_area.mean()), new[g.triangles].astype(np.uint32),
                               g.triangle_piece, g.piece_grain, g.piece_fabric, g.seam_pairs, x,
                               spread(g.boundary, False))])
    scene.pins.append((0, tuple(x[0])))
    return scene


@pytest.mark.parametrize("network", [False, True])
def test_rows_of_a_diagonal_block_alone(gpu, network):
    runs = []
    for variant in (0, 3):
        s = gpu.CudaSolver(0)
        s.set_pcg_variant(variant)
        if network:
            s.set_precond(learned.LearnedPreconditioner(0))
        s.build(_sheet_with_loose_particles())
        assert s.solve_threads() == (512 if variant == 0 else 1024)
        s.step(1.0 / 60.0, 1, 1)
        c = s.counters()
        assert c.precond_fallbacks == 0 and c.learned_solves == int(network)
        runs.append((s.positions().astype(np.float64), s.cg_history()))
        s.close()
    (xa, ha), (xb, hb) = runs
    assert np.array_equal(ha, hb), (ha, hb)
    # Without the network the two kernels repeat the same products; with it they sum in different orders.
    assert np.abs(xa - xb).max() <= (1e-5 if network else 0.0)
