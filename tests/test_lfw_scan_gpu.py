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


# longer and shorter lines in one launch: equal, half and in between, either way round, at 32, 16 and 8 lanes per line
@pytest.mark.parametrize("B,T,D,K", [(1, 20, 64, 33), (1, 20, 96, 48), (1, 20, 48, 96), (1, 20, 96, 60), (1, 20, 128, 97), (2, 5, 20, 32),
                                     (20, 9, 48, 40), (20, 9, 48, 24), (30, 9, 24, 48), (20, 9, 90, 64), (12, 9, 64, 128),
                                     (130, 6, 32, 31), (120, 5, 64, 32), (120, 5, 32, 64), (70, 5, 80, 65), (80, 5, 40, 80),
                                     (70, 5, 80, 50), (60, 5, 52, 104), (60, 5, 104, 60), (40, 4, 128, 105), (50, 4, 128, 7)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_line_pairs(cuda, B, T, D, K, dtype):
    ins = to_dev(lfw_inputs(B, T, D, K, "sigmoid", 1.0, 500 + T + D), dtype, cuda)
    check_against_oracle(ins, run_cabi(*ins), dtype)


@pytest.mark.parametrize("D,K", [(96, 48), (64, 64)])
def test_backward_sees_what_the_kernels_before_it_wrote(cuda, D, K):
    """Inputs overwritten by the kernel just ahead in the stream give what they give after a synchronisation."""
    from t2fw_b200 import cabi

    sets = [to_dev(lfw_inputs(16, 129, D, K, "sigmoid", 1.0, 600 + i), torch.float32, cuda) for i in range(4)]
    buf = [t.clone() for t in sets[0]]

    def grads(i, sync):
        for b, t in zip(buf, sets[i]):
            b.copy_(t)
        x, f, q, k, fk, s, go, gs = buf
        _, ckpt = cabi.lfw_forward(x, f, q, k, fk, s)
        for b, t in zip(buf, sets[i]):
            b.copy_(t)
        if sync:
            torch.cuda.synchronize()
        return cabi.lfw_backward(go, gs, x, f, q, k, fk, s, ckpt)

    got = [grads(i % 4, False) for i in range(12)]
    want = [grads(i, True) for i in range(4)]
    for i, g in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(g, want[i % 4]))
