"""The block-CSR product on both sides of the lines between its two kernels: 256 slots, and one whole block of the narrow
kernel more than its wave. The bound and the oracle are test_gpu_spmv's."""
import pytest
from test_gpu_spmv import SMS_ROWS, test_product_matches_fp64 as product_matches_fp64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,longest", [(3, 242), (3, 247), (40, 100), (60, 40), (70, 0), (SMS_ROWS * 3 // 2 + 127, 0),
                                       (SMS_ROWS * 3 // 2 + 128, 0)])
def test_product_at_the_lines(gpu, n, longest):
    product_matches_fp64(gpu, n, longest, 0, 0)
