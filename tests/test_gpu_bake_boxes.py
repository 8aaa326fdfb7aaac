"""The bake's per-component boxes, shared sample boxes, distance bounds and bit-word sweeps where they can go wrong, bit for
bit against the oracle's serial restatement: boxes cut off by the grid, few large and askew triangles, slivers, a body far
from the origin, bands wider and far narrower than the triangles, components without any sample near them, a pocket that
the flood must not reach and a maze that takes it many turns, rows of one, two and three words."""
import numpy as np
import pytest

from drape_b200 import bake as BK
from drape_b200 import meshes as M

pytestmark = pytest.mark.gpu


def _rotation(seed):
    q, _ = np.linalg.qr(np.random.default_rng(seed).standard_normal((3, 3)))
    return q * np.sign(np.linalg.det(q))


def _joined(parts):
    """One mesh of several closed surfaces."""
    v, t, at = [], [], 0
    for p in parts:
        v.append(p.vertices)
        t.append(p.triangles + at)
        at += len(p.vertices)
    return M.TriangleMesh(np.concatenate(v), np.concatenate(t).astype(np.uint32))


def _maze():
    """A shell of walls with one opening and baffles that leave a gap at alternating ends."""
    w = [M.box((0, -0.1, 0), (0.2, 0.004, 0.06)), M.box((0, 0.1, 0), (0.2, 0.004, 0.06)),
         M.box((0, 0, -0.06), (0.2, 0.1, 0.004)), M.box((0, 0, 0.06), (0.2, 0.1, 0.004)),
         M.box((-0.2, 0, 0), (0.004, 0.1, 0.06)), M.box((0.2, 0.03, 0), (0.004, 0.07, 0.06))]
    for k in range(7):
        w.append(M.box((0.15 - 0.05 * k, 0.03 if k % 2 else -0.03, 0), (0.004, 0.07, 0.06)))
    return [_joined(w)]


def _hollow():
    inner = M.icosphere((0, 0, 0), 0.06, 3)
    return [_joined([M.icosphere((0, 0, 0), 0.1, 3), M.TriangleMesh(inner.vertices, inner.triangles[:, ::-1].copy())])]


CASES = {
    "boxes_cut_by_the_grid": (lambda: M.test_body(), (0.011, 0.0, 0.03)),
    "large_triangles": (lambda: [M.box((0.1, 0, 0), (0.3, 0.02, 0.2))], (0.006, 0.05, 0.02)),
    "askew_triangles": (lambda: [M.box((0, 0, 0.1), (0.3, 0.05, 0.2), _rotation(1)),
                                 M.box((0.1, 0, 0), (0.02, 0.25, 0.01), _rotation(2))], (0.007, 0.03, 0.02)),
    "slivers": (lambda: [M.box((0, 0, 0), (0.3, 0.0001, 0.001), _rotation(3))], (0.004, 0.03, 0.02)),
    "far_from_origin": (lambda: [M.icosphere((4000.0, -2500.0, 900.0), 0.1, 3)], (0.006, 0.03, 0.02)),
    "wide_band": (lambda: [M.icosphere((0, 0, 0), 0.02, 2), M.box((0.1, 0, 0), (0.02, 0.02, 0.02))], (0.01, 0.2, 0.15)),
    "between_samples": (lambda: [M.icosphere((0, 0, 0), 0.08, 2), M.icosphere((0.1234, 0.0312, 0.0101), 0.0004, 1),
                                 M.icosphere((-0.1117, 0.0021, 0.0303), 0.0003, 1)], (0.01, 0.02, 0.0005)),
    "hollow": (_hollow, (0.004, 0.03, 0.01)),
    "maze": (_maze, (0.004, 0.02, 0.006)),
    "overlapping": (lambda: M.capsule_union_body(), (0.009, 0.05, 0.02)),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_field_is_bit_exact(gpu, oracle_mod, case):
    make, (cell, padding, band) = CASES[case]
    comps = make()
    ref = oracle_mod.bake(comps, cell, padding, band)
    got = BK.bake_field(comps, BK.options(cell, padding, band))
    assert tuple(got.dims) == tuple(ref.dims)
    assert np.array_equal(got.values, ref.values), int(np.sum(got.values != ref.values))
