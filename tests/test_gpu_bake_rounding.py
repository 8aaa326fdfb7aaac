"""The bake where the rounded closest point lies out of its triangle's bounding box, so that the box's distance exceeds the
computed one: a box at 1 m whose vertices differ in their last bits. Bit for bit against the oracle's serial restatement;
each seed has samples above a face (7, 4, 2 and 1 of them) whose nearest triangle the box alone would reject."""
import numpy as np
import pytest

from drape_b200 import bake as BK
from drape_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [5, 26, 29, 51])
def test_field_where_rounding_leaves_the_bounding_box(gpu, oracle_mod, seed):
    box = M.box((0, 0, 0), (1.0, 0.05, 0.2))
    v = box.vertices.copy()
    v[:, 0] = np.sign(v[:, 0]) * (1 + np.random.default_rng(seed).integers(-4, 5, len(v)) * 2.0**-53)
    comps = [M.TriangleMesh(v, box.triangles)]
    ref = oracle_mod.bake(comps, 0.02, 0.03, 0.03)
    got = BK.bake_field(comps, BK.options(0.02, 0.03, 0.03))
    assert np.array_equal(got.values, ref.values), int(np.sum(got.values != ref.values))
