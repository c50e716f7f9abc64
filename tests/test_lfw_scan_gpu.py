"""Decay-rule scan kernels at the edges of the line sizes (elements per lane, lanes per line), of the lines of a CTA, of
the steps whose sums are formed together and of the checkpoint interval, against the oracle."""
import pytest
import torch

from helpers import lfw_inputs, to_dev
from test_lfw_gpu import check_against_oracle, run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,D,K", [(1, 1, 1, 1), (3, 33, 16, 17), (2, 32, 15, 33), (2, 65, 17, 49), (1, 71, 64, 65),
                                     (2, 40, 81, 80), (1, 70, 104, 105), (3, 9, 129, 128), (1, 5, 257, 256), (1, 3, 512, 512),
                                     (60, 12, 100, 30)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.float64])
def test_line_sizes(cuda, B, T, D, K, dtype):
    ins = to_dev(lfw_inputs(B, T, D, K, "sigmoid", 1.0, 400 + T + D), dtype, cuda)
    check_against_oracle(ins, run_cabi(*ins), dtype)
