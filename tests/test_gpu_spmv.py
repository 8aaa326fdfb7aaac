"""The standalone block-CSR product at the edges of its two kernels: the four-slots-a-thread one (16-byte aligned planes, one
or two full waves of blocks) and the general one. Rows without slots, rows longer than a chunk, row ranges that start at every
remainder of four, pinned rows and columns. The oracle is the same sum in FP64; a row of K slots adds 3 K products in FP32,
so its error is at most (3 K + 1) * 2^-24 times the sum of the products' magnitudes (first order, with a factor 1.01 for
the rest)."""
import ctypes as C

import numpy as np
import pytest

from drape_b200 import cuda as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SMS_ROWS = 148 * 4 * 128  # rows of one wave of full blocks on 148 SMs


def _system(n, seed, longest):
    rng = np.random.default_rng(seed)
    count = rng.integers(0, 9, n)
    if longest:
        count[rng.integers(0, n, 3)] = longest
    start = np.concatenate([[0], np.cumsum(count)]).astype(np.uint32)
    slots = int(start[-1])
    return dict(n=n, start=start, slots=slots, col=rng.integers(0, n, slots).astype(np.uint32),
                a=rng.standard_normal((9, slots)).astype(np.float32), pin=(rng.random(n) < 0.1).astype(np.uint8),
                x=rng.standard_normal((n, 4)).astype(np.float32))


def _product(s, pad, shift):
    """The device product with the planes padded to a multiple of four plus `pad` slots and the columns' array `shift`
    words off its 16-byte boundary."""
    stride = (s["slots"] + 3) // 4 * 4 + pad
    planes = np.zeros((9, max(stride, 4)), np.float32)
    planes[:, :s["slots"]] = s["a"]
    cols = np.zeros(s["slots"] + 4, np.uint32)
    cols[shift:shift + s["slots"]] = s["col"]
    d = {k: torch.from_numpy(np.ascontiguousarray(v).view(np.uint8).reshape(-1)).cuda()
         for k, v in dict(start=s["start"], col=cols, a=planes, pin=s["pin"], x=s["x"]).items()}
    y = torch.full((s["n"], 4), 7.0, device="cuda")
    code = D.load().drape_cuda_spmv_device(s["n"], d["start"].data_ptr(), d["col"].data_ptr() + 4 * shift,
                                           d["a"].data_ptr(), planes.shape[1], d["pin"].data_ptr(), d["x"].data_ptr(),
                                           y.data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert code == 0
    torch.cuda.synchronize()
    return y.cpu().numpy()[:, :3]


@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 0), (0, 1)], ids=["aligned", "odd_stride", "odd_columns"])
@pytest.mark.parametrize("n,longest", [(1, 0), (1, 5), (3, 0), (31, 1100), (33, 0), (127, 2051), (129, 0), (9473, 40),
                                       (18945, 0), (37889, 1023), (SMS_ROWS, 0), (SMS_ROWS + 1, 0),
                                       (SMS_ROWS * 3 // 2, 0), (SMS_ROWS * 3 // 2 + 1, 0),
                                       (2 * SMS_ROWS, 0), (2 * SMS_ROWS + 1, 0)])
def test_product_matches_fp64(gpu, n, longest, pad, shift):
    s = _system(n, n + longest, longest)
    y = _product(s, pad, shift)
    row = np.repeat(np.arange(n), np.diff(s["start"].astype(np.int64)))
    live = (s["pin"][row] == 0) & (s["pin"][s["col"]] == 0)
    a = s["a"].T.reshape(-1, 3, 3).astype(np.float64) * live[:, None, None]
    terms = a * s["x"][s["col"], None, :3].astype(np.float64)
    ref, size = np.zeros((n, 3)), np.zeros((n, 3))
    np.add.at(ref, row, terms.sum(2))
    np.add.at(size, row, np.abs(terms).sum(2))
    k = np.diff(s["start"].astype(np.int64))[:, None]
    assert (np.abs(y - ref) <= 1.01 * (3 * k + 1) * 2.0 ** -24 * size).all()
