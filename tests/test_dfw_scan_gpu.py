"""Delta-rule scan kernels at the edges of the line sizes (elements per lane, lanes per line), of the lines of a CTA and
of the groups of steps, against the oracle."""
import pytest
import torch

from helpers import dfw_inputs, to_dev
from test_dfw_gpu import check_against_oracle, run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,D,M", [(1, 1, 1, 1), (3, 33, 16, 17), (2, 32, 15, 33), (2, 65, 17, 49), (1, 31, 64, 65),
                                     (2, 40, 81, 80), (1, 70, 104, 105), (3, 9, 129, 128), (1, 5, 256, 257), (1, 3, 512, 512)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.float64])
def test_line_sizes(cuda, B, T, D, M, dtype):
    ins = to_dev(dfw_inputs(B, T, D, M, "softmax", 1.0, 300 + T + D), dtype, cuda)
    check_against_oracle(ins, run_cabi(*ins), dtype)
