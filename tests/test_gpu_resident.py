"""The resident-row solve kernel at the edges of its layout: fewer particles than blocks, blocks with no rows, ragged
warps and rows, pinned rows and columns, halos that span most of the garment, and scenes near its size limit. Its oracle
is the 1024-thread reference-order kernel (variant 3), whose row products and recurrences it repeats in the same order:
bit-identical positions and the same PCG counts."""
import numpy as np
import pytest

from drape_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _hanging(n):
    g = S.piece_garment("sheet", 0.5, 0.5, n, n, S.jersey_fabric())
    g.initial_positions = np.stack([g.rest[:, 0], 0.5 + g.rest[:, 1], np.zeros(g.vertex_count)], axis=1)
    scene = S.Scene([g])
    for v in list(range(0, n * n, max(1, n // 3))):  # pins in every block, corners and interior
        scene.pins.append((v, tuple(g.initial_positions[v])))
    return scene


def _shuffled(n, seed):
    """A sheet whose vertices are numbered at random: every block's halo holds most of the garment."""
    sc = S.sheet_on_sphere(n=n, height=0.16, cg_tolerance=1e-2, max_cg=50)
    g = sc.garments[0]
    perm = np.random.default_rng(seed).permutation(g.vertex_count)
    inv = np.argsort(perm).astype(np.uint32)
    sc.garments[0] = S.Garment(g.id, g.rest[perm], g.vertex_piece[perm], g.vertex_area[perm],
                               inv[g.triangles.astype(np.int64)], g.triangle_piece, g.piece_grain, g.piece_fabric,
                               g.seam_pairs, g.initial_positions[perm], g.boundary[perm])
    return sc


CASES = {
    "sheet_4x4": lambda: S.sheet_on_sphere(n=4, height=0.16, cg_tolerance=1e-2, max_cg=50),
    "sheet_12x12": lambda: S.sheet_on_sphere(n=12, height=0.16, cg_tolerance=1e-2, max_cg=50),
    "sheet_13x13": lambda: S.sheet_on_sphere(n=13, height=0.16, cg_tolerance=1e-2, max_cg=50),
    "sheet_70x70": lambda: S.sheet_on_sphere(n=70, height=0.16, cg_tolerance=1e-6, max_cg=200),
    "pinned_37x37": lambda: _hanging(37),
    # One cluster up to 3,500 particles (59 x 59), the whole grid from there on.
    "cluster_59x59": lambda: S.sheet_on_sphere(n=59, height=0.16, cg_tolerance=1e-2, max_cg=50),
    "cluster_shuffled_50x50": lambda: _shuffled(50, 4),
    "grid_60x60": lambda: S.sheet_on_sphere(n=60, height=0.16, cg_tolerance=1e-2, max_cg=50),
    "shuffled_60x60": lambda: _shuffled(60, 3),
    "tube_66k": lambda: S.seamed_tube(161, 205, field_n=64, field_cell=0.012),
    # Several rows a thread, the matrix partly in the L2: the smallest and largest of two rows, and three rows.
    "tube_72k": lambda: S.seamed_tube(169, 213, field_n=64, field_cell=0.012),
    "tube_141k": lambda: S.seamed_tube(236, 299, field_n=64, field_cell=0.012),
    "tube_150k": lambda: S.seamed_tube(243, 309, field_n=64, field_cell=0.012),
}


def _run(gpu, scene, variant, frames=3):
    s = gpu.CudaSolver(0)
    s.set_pcg_variant(variant)
    s.build(scene)
    threads = s.solve_threads()
    for _ in range(frames):
        s.step(1.0 / 60.0, 1, 2)
    out = s.positions(), s.velocities(), s.cg_history(), threads
    s.close()
    return out


@pytest.mark.parametrize("name", list(CASES))
def test_resident_rows_match_the_1024_thread_kernel(gpu, name):
    x3, v3, h3, t3 = _run(gpu, CASES[name](), 3)
    x0, v0, h0, t0 = _run(gpu, CASES[name](), 0)
    assert (t3, t0) == (1024, 512)
    assert np.isfinite(x0).all()
    assert np.array_equal(h0, h3), (h0, h3)
    assert np.array_equal(x0, x3) and np.array_equal(v0, v3), np.abs(x0 - x3).max()


@pytest.mark.parametrize("name", ["sheet_13x13", "pinned_37x37", "shuffled_60x60", "tube_60k"])
def test_resident_learned_pcg_with_a_zero_output_layer_is_block_jacobi(gpu, name):
    """With the initial network (zero output layer) the factor is exactly block-Jacobi's Cholesky factor, so the learned
    resident kernel (the factor on chip for the small scenes, in the L2 for the 60k tube) follows the block-Jacobi one:
    the same PCG counts in the first frame and positions that differ by the roundings of L L^T r against M^-1 r."""
    from drape_b200 import learned
    make = CASES.get(name, lambda: S.seamed_tube(154, 195, field_n=64, field_cell=0.012))
    xj, _, hj, _ = _run(gpu, make(), 0, frames=1)
    s = gpu.CudaSolver(0)
    s.set_precond(learned.LearnedPreconditioner(0))
    s.build(make())
    assert s.solve_threads() == 512
    s.step(1.0 / 60.0, 1, 2)
    x, h, c = s.positions(), s.cg_history(), s.counters()
    s.close()
    assert c.learned_solves == c.newton_iterations == 2 and c.precond_fallbacks == 0
    assert np.abs(np.asarray(h) - np.asarray(hj)).max() <= 1, (h, hj)
    assert np.abs(x.astype(np.float64) - xj).max() < 1e-4


@pytest.mark.parametrize("side", [3, 128, 129])
def test_reads_in_chunks_equal_the_snapshot(gpu, side):
    """Positions and velocities are read through a 16,384-particle staging buffer: below, at and past one chunk they
    equal the snapshot's, which copies the padded vectors."""
    s = gpu.CudaSolver(0)
    s.build(S.sheet_on_sphere(n=side, height=0.16, cg_tolerance=1e-2, max_cg=50))
    s.step(1.0 / 60.0, 1, 2)
    snap = s.snapshot()
    assert np.array_equal(s.positions(), snap["positions"]) and np.array_equal(s.velocities(), snap["velocities"])
    s.close()


def _batch(gpu, sizes, tuning=None, frames=2):
    from drape_b200 import batch
    b = batch.BatchSolver(0)
    for k, n in enumerate(sizes):
        b.add(S.tube_variant(40 + k, n, field_n=32))
    b.build()
    if tuning:
        b.set_tuning(*tuning)
    for _ in range(frames):
        b.step(1.0 / 60.0, 1, 2)
    out = [b.positions(k) for k in range(len(sizes))], [b.counters(k).cg_iterations for k in range(len(sizes))]
    b.close()
    return out


@pytest.mark.parametrize("sizes", [(64,), (300, 5000), (900, 700, 2100, 500), (30000,) * 6 + (2000,), (40000,) * 6],
                         ids=["tiny", "two", "four", "one_wave_182k", "two_waves_240k"])
def test_resident_batch_matches_the_slot_parallel_kernel(gpu, sizes):
    """The batch's resident-row solve (the default variant) against the slot-parallel kernel on 512-thread blocks, whose
    row sums it repeats in the same order: bit-identical positions and the same PCG counts, with one to three rows a
    thread and one or two launches."""
    xa, ca = _batch(gpu, sizes)
    xb, cb = _batch(gpu, sizes, (0, 512))
    assert ca == cb
    for a, b in zip(xa, xb):
        assert np.isfinite(a).all() and np.array_equal(a, b), np.abs(a - b).max()


def test_resident_batch_after_the_partition_changes(gpu):
    """Garments that end their drape leave the frame and the others' groups, halos and mailboxes move: the drape's end
    state equals the slot-parallel kernel's."""
    from drape_b200 import batch
    from drape_b200.scene import drape_drape_options
    out = []
    for tuning in (None, (0, 512)):
        b = batch.BatchSolver(0)
        for k, n in enumerate((600, 3000, 1200)):
            b.add(S.tube_variant(60 + k, n, field_n=32))
        b.build()
        if tuning:
            b.set_tuning(*tuning)
        o = drape_drape_options(substeps=1, iterations=2, frame_dt=1.0 / 60.0, max_assembly_seconds=0.05,
                                seam_gap_done=0.001, settle_rms_speed=0.5, settle_hold_frames=3, max_sim_seconds=0.4,
                                snapshot_every=30, max_retries=3, energy_rise_frames=60, frames_per_wait=10)
        res, _ = b.drape_to_rest(o)
        out.append(([b.positions(k) for k in range(3)], [int(r.frames_run) for r in res]))
        b.close()
    (xa, fa), (xb, fb) = out
    assert fa == fb and len(set(fa)) > 1, fa
    for a, b in zip(xa, xb):
        assert np.array_equal(a, b), np.abs(a - b).max()


def _system(n, degree, seed, local):
    """A seeded SPD block-CSR system: a diagonal block and about `degree` symmetric neighbours a row, near the diagonal
    (`local`) or anywhere; some rows pinned, some with an active contact."""
    rng = np.random.default_rng(seed)
    m = n * degree // 2
    a = rng.integers(0, n, m)
    b = (a + rng.integers(1, max(2, degree), m)) % n if local else rng.integers(0, n, m)
    pairs = np.unique(np.sort(np.stack([a, b], 1)[a != b], 1), axis=0)
    d = rng.standard_normal((len(pairs), 3))
    block = (d[:, :, None] * d[:, None, :] + 0.1 * np.eye(3)).astype(np.float32)
    diag = np.tile(0.5 * np.eye(3, dtype=np.float32), (n, 1, 1))
    for k in (0, 1):
        np.add.at(diag, pairs[:, k], block)
    row = np.concatenate([np.arange(n), pairs[:, 0], pairs[:, 1]])
    col = np.concatenate([np.arange(n), pairs[:, 1], pairs[:, 0]])
    blocks = np.concatenate([diag, -block, -block])
    order = np.lexsort((col, row))
    start = np.zeros(n + 1, np.uint32)
    start[1:] = np.cumsum(np.bincount(row, minlength=n))
    normals = rng.standard_normal((n, 3)).astype(np.float32)
    normals /= np.linalg.norm(normals, axis=1, keepdims=True)
    pinned = (rng.random(n) < 0.05).astype(np.uint8)
    grad = (rng.standard_normal((n, 3)) * (1 - pinned)[:, None]).astype(np.float32)
    return dict(row_start=start, col_index=col[order].astype(np.uint32), blocks=blocks[order].reshape(-1, 9),
                pinned=pinned, active=(rng.random(n) < 0.2).astype(np.uint8), normals=normals, grad=grad)


@pytest.mark.parametrize("n, degree, local", [(1, 0, True), (7, 4, True), (148, 12, True), (149, 12, True),
                                              (8190, 14, True), (8192, 12, False), (3000, 40, False)])
def test_noalloc_pcg_over_resident_rows(gpu, n, degree, local):
    """The allocation-free PCG against the allocating entry point (the 1024-thread kernel) where its blocks' rows and
    halos fit the resident-row form and where they do not (scattered couplings: the 1024-thread form), twice in a row in
    either order of the two forms: the same iteration count and iterates."""
    import torch
    from test_zz_no_alloc import _noalloc
    small = _system(200, 8, 1, True)
    for k in range(2):
        sysd = dict(_system(n, degree, 10 + n, local), max_it=60, tol=1e-5)
        ref = gpu.pcg(sysd["row_start"], sysd["col_index"], sysd["blocks"], sysd["pinned"], sysd["active"],
                      sysd["normals"], sysd["grad"], 60, 1e-5)
        step, resid, its = _noalloc(gpu, sysd)
        assert its == ref[2]
        assert np.linalg.norm(step - ref[0]) <= 1e-6 * np.linalg.norm(ref[0])
        assert np.linalg.norm(resid - ref[1]) <= 1e-6 * max(np.linalg.norm(ref[1]), 1e-6)
        _noalloc(gpu, dict(small, max_it=20, tol=1e-3))
    torch.cuda.synchronize()


def test_solve_kernels_of_different_grids_take_turns(gpu):
    """One solver, three frames each with the cluster kernel, the 1024-thread kernel and the learned kernel in turn: the
    barrier counter starts anew for each, and the block-Jacobi frames equal a solver's that never changed."""
    from drape_b200 import learned
    net = learned.LearnedPreconditioner(0)
    scene = CASES["cluster_59x59"]()
    a, b = gpu.CudaSolver(0), gpu.CudaSolver(0)
    for s in (a, b):
        s.build(scene)
    for k in range(3):
        start = b.snapshot()
        a.set_pcg_variant(3 if k == 1 else 0)
        a.step(1.0 / 60.0, 1, 2)
        b.step(1.0 / 60.0, 1, 2)
        assert np.array_equal(a.positions(), b.positions())
        a.set_precond(net)
        a.step(1.0 / 60.0, 1, 2)
        a.set_precond(None)
        a.restore(b.snapshot())
        assert np.isfinite(start["positions"]).all()
    a.close()
    b.close()
