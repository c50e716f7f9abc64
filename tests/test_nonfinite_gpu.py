"""A NaN or an infinity that goes into a call comes out of it: wherever the recurrence, evaluated step by step, is not a finite
number, the kernels' result is none either (never a finite number in its place), and other rows of the batch do not change.
A chunk's products contract over its 64 steps, so the chunked kernels may show it in other steps of the same chunk too."""
import numpy as np
import pytest
import torch

from helpers import dfw_inputs, lfw_inputs, to_dev
from oracle import fw_oracle

pytestmark = pytest.mark.gpu

LFW = ("x", "f", "q", "k", "f_key", "state", "grad_out", "grad_state")
DFW = ("q", "k", "v", "state", "grad_out", "grad_state")


def _spoiled(ins, names, what, value, step):
    """The inputs with one element of row 1 replaced: of a step, or of a state."""
    t = ins[names.index(what)]
    t[1, 20 if "state" in what else step, 5] = value
    return ins


def _compare(got, clean, ref):
    for i, (g, c, r) in enumerate(zip(got, clean, ref)):
        g, c = g.double().cpu().numpy(), c.double().cpu().numpy()
        bad = ~np.isfinite(np.asarray(r, dtype=np.float64))
        assert not np.isfinite(g[bad]).any(), ("result", i, int(np.isfinite(g[bad]).sum()), int(bad.sum()))
        for row in (0, 2):
            assert np.array_equal(g[row], c[row]), ("result", i, "row", row)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("step", [0, 63, 64, 199])
@pytest.mark.parametrize("what", LFW)
@pytest.mark.parametrize("D,K,dtype", [(64, 64, torch.float16), (64, 64, torch.bfloat16), (128, 128, torch.float16),
                                       (128, 64, torch.bfloat16), (64, 128, torch.float16), (192, 128, torch.float16),
                                       (24, 40, torch.float32)])
def test_decay_rule(cuda, D, K, dtype, what, step, value):
    from t2fw_b200 import cabi

    def run(ins):
        out, ckpt = cabi.lfw_forward(*ins[:6])
        grads = cabi.lfw_backward(ins[6], ins[7], *ins[:6], ckpt)
        torch.cuda.synchronize()
        return (out, ckpt[:, -1], *grads)

    ins = to_dev(lfw_inputs(3, 200, D, K, "sigmoid", 0.5, 61), dtype, cuda)
    clean = run(ins)
    ins = _spoiled(ins, LFW, what, value, step)
    with np.errstate(all="ignore"):
        ref = (*fw_oracle.lfw_forward(*ins[:6]), *fw_oracle.lfw_backward(ins[6], ins[7], *ins[:6]))
    _compare(run(ins), clean, ref)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("step", [0, 63, 64, 199])
@pytest.mark.parametrize("what", DFW)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_delta_rule(cuda, dtype, what, step, value):
    from t2fw_b200 import cabi

    def run(ins):
        out, fin, delta = cabi.dfw_forward(*ins[:4])
        grads = cabi.dfw_backward(ins[4], ins[5], ins[0], ins[1], delta, fin)
        torch.cuda.synchronize()
        return (out, fin, *grads)

    ins = to_dev(dfw_inputs(3, 200, 64, 64, "scaled", 0.3, 62), dtype, cuda)
    clean = run(ins)
    ins = _spoiled(ins, DFW, what, value, step)
    with np.errstate(all="ignore"):
        out, fin, _ = fw_oracle.dfw_forward(*ins[:4])
        ref = (out, fin, *fw_oracle.dfw_backward(ins[4], ins[5], *ins[:4]))
    _compare(run(ins), clean, ref)


@pytest.mark.parametrize("step", [0, 63, 64, 199])
@pytest.mark.parametrize("part", ["query", "key", "value", "gate", "state", "grad_out", "grad_state"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_fused_layer(cuda, dtype, part, step):
    """Against the plain operator on folded, activated tensors, step by step in double precision."""
    from t2fw_b200.functional_fused import GATE_FLOOR, LFWFusedFunction

    B, T, H = 3, 200, 2
    C = H * 64
    g = torch.Generator().manual_seed(63)
    ins = [torch.randn(s, generator=g).to(dtype).to(cuda) for s in ((B, T, 4 * C), (B * H, 64, 64), (B, T, C), (B * H, 64, 64))]

    def run(ins):
        leaves = [ins[0].clone().requires_grad_(True), ins[1].clone().requires_grad_(True)]
        out, nxt = LFWFusedFunction.apply(*leaves, H)
        d_qkvg, d_state = torch.autograd.grad([out, nxt], leaves, ins[2:])
        torch.cuda.synchronize()
        return [out.detach(), nxt.detach().reshape(B, -1), d_qkvg, d_state.reshape(B, -1)]

    clean = run(ins)
    col = {"query": 0, "key": C, "value": 2 * C, "gate": 3 * C}
    if part in col:
        ins[0][1, step, col[part] + 5] = float("nan")
    elif part == "grad_out":
        ins[2][1, step, 5] = float("nan")
    else:
        ins[1 if part == "state" else 3][H, 20, 5] = float("nan")

    def fold(t):
        return t.view(B, T, H, 64).permute(0, 2, 1, 3).reshape(B * H, T, 64).double().cpu()

    def unfold(a):
        return np.asarray(a).reshape(B, H, T, 64).transpose(0, 2, 1, 3).reshape(B, T, C)

    q, k, v, a = (fold(t.contiguous()) for t in ins[0].split(C, dim=-1))
    gate = torch.sigmoid(a).clamp_min(GATE_FLOOR)      # (NaN stays NaN)
    args = (v, torch.ones_like(v), q / 8, k, gate, ins[1].double().cpu())
    with np.errstate(all="ignore"):
        out, fin = fw_oracle.lfw_forward(*args)
        dx, _, dq, dk, dfk, ds = fw_oracle.lfw_backward(fold(ins[2]), ins[3].double().cpu(), *args)
    # the gate's derivative is 0 below the floor, NaN where the pre-activation is
    der = np.where(np.isnan(a.numpy()), np.nan, np.where(torch.sigmoid(a).numpy() > GATE_FLOOR, 1.0, 0.0))
    dfk = np.where(der == 0.0, 0.0, np.asarray(dfk) * der)
    ref = [unfold(out), np.asarray(fin).reshape(B, -1), np.concatenate([unfold(t) for t in (dq, dk, dx, dfk)], -1),
           np.asarray(ds).reshape(B, -1)]
    _compare(run(ins), clean, ref)
