"""Step-by-step kernel for short sequences (csrc/steps.cu): slab and row-count edges of its CTAs, group edges
of its step ring, all key sizes, both rules, and bit equality of a ring of decode steps with single steps."""
import pytest
import torch

from helpers import OUT_TOL, dfw_inputs, lfw_inputs, max_rel_err, to_dev
from oracle import fw_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,D,K", [(1, 2, 64, 64), (3, 7, 8, 32), (2, 8, 24, 64), (40, 9, 72, 128), (300, 17, 64, 64),
                                     (75, 33, 128, 128), (2, 64, 200, 32), (150, 64, 64, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_short_forward_matches_oracle(cuda, B, T, D, K, dtype):
    from t2fw_b200 import cabi

    x, f, q, k, fk, s, _, _ = to_dev(lfw_inputs(B, T, D, K, "sigmoid", 0.5, B + T), dtype, cuda)
    out, ckpt = cabi.lfw_forward(x, f, q, k, fk, s)
    r_out, r_fin = fw_oracle.lfw_forward(x, f, q, k, fk, s)
    assert max_rel_err(out, r_out) <= OUT_TOL[dtype] and max_rel_err(ckpt[:, -1], r_fin) <= OUT_TOL[dtype]
    qd, kd, v, sd, _, _ = to_dev(dfw_inputs(B, T, D, K, "scaled", 0.5, B + T), dtype, cuda)
    out, fin, _ = cabi.dfw_forward(qd, kd, v, sd)
    r_out, r_fin, _ = fw_oracle.dfw_forward(qd, kd, v, sd)
    assert max_rel_err(out, r_out) <= OUT_TOL[dtype] and max_rel_err(fin, r_fin) <= OUT_TOL[dtype]


@pytest.mark.parametrize("B,n,D,K", [(1, 2, 64, 64), (500, 10, 64, 64), (3, 16, 24, 32), (9, 8, 72, 128)])
def test_ring_equals_single_steps(cuda, B, n, D, K):
    from t2fw_b200.decode import LFWDecodeLoop, lfw_decode_step

    x, f, q, k, fk, s, _, _ = to_dev(lfw_inputs(B, n, D, K, "sigmoid", 0.5, 7 * B + n), torch.float16, cuda)
    ring = [t.transpose(0, 1).unsqueeze(2).contiguous() for t in (x, f, q, k, fk)]
    loop = LFWDecodeLoop(s, ring=n)
    for slot, t in zip((loop.x, loop.f, loop.query, loop.key, loop.f_key), ring):
        slot.copy_(t)
    a, b, o = s.clone(), torch.empty_like(s), torch.empty_like(ring[0][0])
    for _ in range(2):
        got = loop.run_ring()
        for i in range(n):
            lfw_decode_step(*(t[i] for t in ring), a, b, o)
            a, b = b, a
            assert torch.equal(got[i], o)
        assert torch.equal(loop.state, a)


@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 9, 3), (40, 63, 12)])
def test_short_fused_layer_equals_plain_operator(cuda, B, T, H):
    from t2fw_b200.functional_fused import LFWFusedFunction, unfused_reference

    g = torch.Generator().manual_seed(B + T)
    qkvg = torch.randn(B, T, 4 * H * 64, generator=g).half().to(cuda)
    state = torch.randn(B * H, 64, 64, generator=g).half().to(cuda)
    for a, b in zip(LFWFusedFunction.apply(qkvg, state, H), unfused_reference(qkvg, state, H)):
        assert max_rel_err(a, b) <= 1e-3      # torch's sigmoid may round a gate the other way


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gates_are_the_chunk_kernels_gates(cuda, dtype):
    """The fused layer's gate of every finite pre-activation, from a call of one step and from one of a whole chunk (what
    the backward of either uses): a state of ones and nothing else leaves the gate as the next state."""
    from t2fw_b200.functional_fused import LFWFusedFunction

    pre = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(dtype)
    pre = torch.where(torch.isfinite(pre), pre, torch.zeros_like(pre)).reshape(1024, 1, 64).to(cuda)
    state = torch.zeros(1024, 64, 64, dtype=dtype, device=cuda)
    state[:, 0] = 1
    got = []
    for T in (1, 64):
        qkvg = torch.zeros(1024, T, 256, dtype=dtype, device=cuda)
        qkvg[:, :, 192:] = 30      # gate 1
        qkvg[:, :1, 192:] = pre
        got.append(LFWFusedFunction.apply(qkvg, state, 1)[1][:, 0])
    torch.cuda.synchronize()
    assert (got[0] >= 0.125).all() and (got[0] <= 1).all() and torch.equal(got[0], got[1])
