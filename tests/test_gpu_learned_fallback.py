"""The block-Jacobi solve that follows a learned one which broke down, where the blocks' halos differ most: half of the
particles numbered along the sheet (small halos), half at random (halos of a thousand particles and more). Blocks with
small halos end the learned solve first, and must not publish the next solve's z while others still wait for this one's.
Bit-identical to a solver without the network, frame for frame, and no wait runs out."""
import numpy as np
import pytest

from drape_b200 import learned
from drape_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _half_shuffled(n, seed):
    sc = S.sheet_on_sphere(n=n, height=0.16, cg_tolerance=1e-2, max_cg=50)
    g = sc.garments[0]
    perm = np.arange(g.vertex_count)
    np.random.default_rng(seed).shuffle(perm[g.vertex_count // 2:])
    inv = np.argsort(perm).astype(np.uint32)
    sc.garments[0] = S.Garment(g.id, g.rest[perm], g.vertex_piece[perm], g.vertex_area[perm],
                               inv[g.triangles.astype(np.int64)], g.triangle_piece, g.piece_grain, g.piece_fabric,
                               g.seam_pairs, g.initial_positions[perm], g.boundary[perm])
    return sc


@pytest.mark.parametrize("side", [61, 140])
def test_fallback_with_unequal_halos(gpu, side):
    params = learned.init_params(0)
    k = learned.param_count() - 16 - 16 * 192  # W_o
    params[k:k + 16 * 192] = np.nan
    scene = _half_shuffled(side, 5)
    a, b = gpu.CudaSolver(0), gpu.CudaSolver(0)
    b.set_precond(learned.LearnedPreconditioner(0, params))
    for s in (a, b):
        s.build(scene)
        assert s.solve_threads() == 512
    for _ in range(30):
        a.step(1 / 60, 1, 2)
        b.step(1 / 60, 1, 2)
        assert np.array_equal(a.positions(), b.positions())
    c = b.counters()
    assert c.precond_fallbacks == c.learned_solves == c.newton_iterations > 0
    a.close()
    b.close()
