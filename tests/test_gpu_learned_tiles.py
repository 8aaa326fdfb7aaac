"""The backward tile kernels (transposed operands in place, two CTAs an SM) where their tiling can go wrong: a system of
one partial tile, and one with more tiles than CTAs, so that each CTA accumulates several. Against the CPU oracle with the
bars of tests/test_gpu_learned.py (gradients to 3e-2 relative in norm, per-group cosine above 0.99)."""
import mpnn
import numpy as np
import pytest

from drape_b200 import learned
from test_gpu_learned import _groups_close, _random_params, _sample
from test_mpnn_oracle import graph_of, sheet_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [3, 60])
def test_gradient_matches_oracle_at_the_edges_of_the_tiling(gpu, oracle_mod, nx):
    sysm = sheet_system(oracle_mod, nx=nx)
    flat = _random_params(2)
    n = len(sysm["diag_slot"])
    probe = np.random.default_rng(5).standard_normal((n, 3)).astype(np.float32)
    net = learned.LearnedPreconditioner(0, flat)
    sid = _sample(net, sysm, residuals=[probe])
    loss, grad = net.loss_grad(sid, 0)
    ref, gref = mpnn.kaporin_and_grad(graph_of(sysm), flat.astype(np.float64), probe, emulate=True)
    assert abs(loss - ref) <= 1e-3 * max(1.0, abs(ref))
    _groups_close(grad, gref)
