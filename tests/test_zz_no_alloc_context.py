"""The allocation-free PCG in a context that was created again: after a cudaDeviceReset, which the header allows between calls
outside a capture, it solves as before. In a process of its own, since the reset ends the other tests' context too."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r'''
import ctypes as C
import numpy as np
from cuda.bindings import runtime as rt
from drape_b200 import cuda as G


def ok(r):
    assert int(r[0]) == 0, r
    return r[1] if len(r) > 1 else None


def device(a):
    a = np.ascontiguousarray(a)
    p = ok(rt.cudaMalloc(a.nbytes))
    ok(rt.cudaMemcpy(p, a.ctypes.data, a.nbytes, rt.cudaMemcpyKind.cudaMemcpyHostToDevice))
    return p


def solve(n=300):
    rows = [[j for j in (i - 1, i, i + 1) if 0 <= j < n] for i in range(n)]
    start = np.cumsum([0] + [len(r) for r in rows])
    col = np.concatenate(rows)
    slots, padded = len(col), (len(col) + 31) // 32 * 32
    planes = np.zeros((9, padded), np.float32)
    planes[::4, :slots] = np.where(col == np.repeat(np.arange(n), np.diff(start)), 4.0, -1.0)
    grad = np.zeros((n, 4), np.float32)
    grad[:, :3] = np.random.default_rng(1).standard_normal((n, 3))
    step, its = np.zeros((n, 4), np.float32), np.zeros(1, np.int32)
    d = [device(a) for a in (start.astype(np.uint32), col.astype(np.uint32), planes, np.zeros(n, np.uint8), grad, step,
                             step, its)]
    code = L.drape_cuda_pcg_noalloc(n, slots, d[0], d[1], d[2], padded, d[3], None, None, d[4], 50, 1e-4, d[5], d[6],
                                    d[7], None)
    assert code == 0, L.drape_cuda_last_error(None)
    ok(rt.cudaDeviceSynchronize())
    for a, p in ((step, d[5]), (its, d[7])):
        ok(rt.cudaMemcpy(a.ctypes.data, p, a.nbytes, rt.cudaMemcpyKind.cudaMemcpyDeviceToHost))
    assert its[0] > 0 and np.isfinite(step).all() and np.abs(step).max() > 0
    return step, int(its[0])


L = G.load()
ok(rt.cudaSetDevice(0))
before = solve()
ok(rt.cudaDeviceReset())
ok(rt.cudaSetDevice(0))
for _ in range(2):
    after = solve()
    assert after[1] == before[1] and np.array_equal(after[0], before[0])
print("same")
'''


def test_noalloc_pcg_after_a_device_reset(gpu):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "drape-2_b200"))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
