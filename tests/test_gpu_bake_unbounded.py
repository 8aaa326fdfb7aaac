"""The bake with a band whose square overflows (infinite, or 1e200): every sample is within it, and the field is the signed
distance to each component, bit for bit the oracle's."""
import numpy as np
import pytest

from drape_b200 import bake as BK
from drape_b200 import meshes as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("band", [1e3, 1e200, float("inf")])
def test_field_without_a_far_side(gpu, oracle_mod, band):
    comps = [M.icosphere((0, 0, 0), 0.08, 2), M.box((0.1, 0.05, 0), (0.03, 0.1, 0.02))]
    ref = oracle_mod.bake(comps, 0.013, 0.05, band)
    got = BK.bake_field(comps, BK.options(0.013, 0.05, band))
    assert np.isfinite(ref.values).all() and (ref.values < 0).any() and (ref.values > 0).any()
    assert np.array_equal(got.values, ref.values), int(np.sum(got.values != ref.values))
