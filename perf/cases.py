"""Performance cases of the fast-weight recurrences, through the public entry points.

A case names an entry point (`op`), whether only the forward pass or forward + backward runs (`pass`), sizes, storage
type, and the distribution of its gates (decay rule) or keys (delta rule):

  op      lfw    LFWFunction.apply: decay rule on [B, T, D] / [B, T, K] tensors
          dfw    DFWFunction.apply: delta rule
          fused  LFWFusedFunction.apply: decay-rule attention core on a projection output [B, T, 4*H*64]
          step   lfw_decode_step: one recurrent step into caller-owned buffers
          loop   LFWDecodeLoop.run_ring: `ring` chained steps, replayed as one CUDA graph
  pass    fwd    inference (no_grad)
          train  forward, then gradients of every input through autograd
  gates   raw_f1   forget gate 1, f_key ~ N(0,1): the benchmark configuration
          sigmoid  sigmoid(N(0,1)) on both sides
          open     sigmoid(4 + N(0,1)) on both sides: gates near 1, as a trained or freshly initialised layer has them
  keys    scaled   q, k ~ N(0,1) / sqrt(M)
          softmax  softmax over the features times a sigmoid write strength
"""
import math

import torch

from t2fw_b200.decode import LFWDecodeLoop, lfw_decode_step
from t2fw_b200.functional_dfw import DFWFunction
from t2fw_b200.functional_fused import LFWFusedFunction
from t2fw_b200.functional_lfw import LFWFunction

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


def _lfw(name, kind, B, T, D, K, dtype, gates):
    return {"name": name, "op": "lfw", "pass": kind, "B": B, "T": T, "D": D, "K": K, "dtype": dtype, "gates": gates}


def _dfw(name, kind, B, T, D, K, dtype, keys):
    return {"name": name, "op": "dfw", "pass": kind, "B": B, "T": T, "D": D, "K": K, "dtype": dtype, "keys": keys}


def listed():
    return [
        # one recurrent token of a small batch through the autograd wrapper (latency of a single small call)
        _lfw("lfw_token_b32", "fwd", 32, 1, 64, 64, "fp16", "open"),
        _dfw("dfw_token_b32", "fwd", 32, 1, 64, 64, "fp16", "softmax"),
        # serving: one decode step of 256 sequences x 16 heads; 1/8 of that in a graph-replayed loop
        {"name": "decode_step_b4096", "op": "step", "pass": "fwd", "B": 4096, "T": 1, "D": 64, "K": 64, "ring": 1,
         "dtype": "fp16", "gates": "sigmoid"},
        {"name": "decode_loop_b512", "op": "loop", "pass": "fwd", "B": 512, "T": 1, "D": 64, "K": 64, "ring": 8,
         "dtype": "bf16", "gates": "open"},
        # prefill of one prompt of ragged length over the 12 heads of a small model, and of a batch of prompts
        _lfw("lfw_prefill_b12", "fwd", 12, 777, 64, 64, "bf16", "open"),
        _dfw("dfw_prefill_b48", "fwd", 48, 1333, 64, 64, "bf16", "softmax"),
        # training: batch 8 x 12 heads at sequence 1024 (the benchmark shape) for both rules and the fused layer
        _lfw("lfw_train_b96", "train", 96, 1024, 64, 64, "fp16", "raw_f1"),
        _dfw("dfw_train_b96", "train", 96, 1024, 64, 64, "fp16", "scaled"),
        {"name": "fused_train_b8h12", "op": "fused", "pass": "train", "B": 8, "H": 12, "T": 1024, "D": 64, "K": 64,
         "dtype": "bf16", "gates": "open"},
        # fine-tuning on short sequences, both gates: many launches for little work
        _lfw("lfw_train_short", "train", 24, 160, 64, 64, "fp16", "sigmoid"),
        # full precision at a state shape that is no multiple of the tile
        _lfw("lfw_train_fp32", "train", 16, 129, 96, 48, "fp32", "sigmoid"),
        # long sequences with 128-wide heads
        _lfw("lfw_train_long", "train", 16, 16384, 128, 128, "fp16", "sigmoid"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["token", "decode", "lfw", "lfw", "lfw", "dfw", "dfw", "fused", "any"])
    dt16 = rng.choice(["fp16", "fp16", "bf16"])
    gates = rng.choice(["raw_f1", "sigmoid", "open"])
    keys = rng.choice(["scaled", "softmax"])
    step = rng.choice(["train", "train", "fwd"])
    if kind == "token":
        op, B = rng.choice(["lfw", "lfw", "dfw"]), _log(rng, 1, 2048)
        c = _lfw("", "fwd", B, 1, 64, 64, dt16, gates) if op == "lfw" else _dfw("", "fwd", B, 1, 64, 64, dt16, keys)
    elif kind == "decode":
        op = rng.choice(["step", "loop"])
        c = {"op": op, "pass": "fwd", "B": _log(rng, 8, 8192), "T": 1, "D": 64, "K": 64,
             "ring": rng.choice([2, 4, 8, 16]) if op == "loop" else 1, "dtype": dt16, "gates": gates}
    elif kind == "lfw":
        D, K = rng.choice([(64, 64), (64, 64), (64, 64), (128, 128), (128, 64)])
        T = _log(rng, 2, 16384)
        c = _lfw("", step, _log(rng, 1, max(1, min(384, 196608 // T))), T, D, K, dt16, gates)
    elif kind == "dfw":
        T = _log(rng, 2, 4096)
        c = _dfw("", step, _log(rng, 1, max(1, min(384, 131072 // T))), T, 64, 64, dt16, keys)
    elif kind == "fused":
        H, T = rng.choice([6, 8, 12, 16]), _log(rng, 16, 4096)
        c = {"op": "fused", "pass": step, "B": _log(rng, 1, max(1, min(32, 131072 // (T * H)))), "H": H, "T": T, "D": 64,
             "K": 64, "dtype": dt16, "gates": rng.choice(["sigmoid", "open"])}
    else:      # every other state shape, and full precision
        D = _log(rng, 12, 100)
        K = rng.choice([D, (D + 1) // 2])
        dt = rng.choice(["fp32", "fp32", "fp16"])
        B, T = _log(rng, 1, 48), _log(rng, 4, 300)
        c = _lfw("", step, B, T, D, K, dt, rng.choice(["sigmoid", "open"])) if rng.random() < 0.6 else \
            _dfw("", step, B, T, D, K, dt, "softmax")
    c.pop("name", None)
    return c


def _gate(rnd, shape, kind):
    return torch.sigmoid(rnd(*shape) + (4.0 if kind == "open" else 0.0))


def prepare(case, seed):
    dev, dtype = torch.device("cuda"), DTYPES[case["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device=dev)

    op, B, T, D, K = case["op"], case["B"], case["T"], case["D"], case["K"]
    train = case["pass"] == "train"
    if op == "fused":
        H = case["H"]
        qkvg = rnd(B, T, 4 * H * 64)
        if case["gates"] == "open":
            qkvg[..., 3 * H * 64:] += 4.0
        ins = [qkvg, 0.1 * rnd(B * H, 64, 64)]
        up = [rnd(B, T, H * 64), rnd(B * H, 64, 64)]
    elif op == "dfw":
        if case["keys"] == "softmax":
            q = torch.softmax(rnd(B, T, K), -1)
            k = torch.softmax(rnd(B, T, K), -1) * torch.sigmoid(rnd(B, T, 1))
        else:
            q, k = rnd(B, T, K) / math.sqrt(K), rnd(B, T, K) / math.sqrt(K)
        ins = [q, k, rnd(B, T, D), 0.1 * rnd(B, D, K)]
        up = [rnd(B, T, D), rnd(B, D, K)]
    else:
        n = case.get("ring", 1)
        bt = (n, B, 1) if op in ("step", "loop") else (B, T)
        x, q, k = rnd(*bt, D), rnd(*bt, K) / math.sqrt(K), rnd(*bt, K) / math.sqrt(K)
        raw = case["gates"] == "raw_f1"
        f = torch.ones(*bt, D, device=dev) if raw else _gate(rnd, (*bt, D), case["gates"])
        fk = rnd(*bt, K) if raw else _gate(rnd, (*bt, K), case["gates"])
        s = 0.1 * rnd(B, D, K)
        if op == "loop":
            loop = LFWDecodeLoop(s.to(dtype), ring=n)
            for slot, t in ((loop.x, x), (loop.f, f), (loop.query, q), (loop.key, k), (loop.f_key, fk)):
                slot.copy_(t)
            loop.run_ring()      # a serving loop captures its graph once, at start-up
            return {"case": case, "loop": loop}
        ins = [x, f, q, k, fk, s]
        if op == "step":
            ins = [t[0] if t.dim() == 4 else t for t in ins]
        up = [rnd(B, T, D), rnd(B, D, K)]
    st = {"case": case, "in": [t.to(dtype).contiguous().requires_grad_(train) for t in ins]}
    if train:
        st["up"] = [t.to(dtype) for t in up]
    if op == "step":
        st["out"] = torch.empty(B, 1, D, dtype=dtype, device=dev)
        st["next"] = torch.empty(B, D, K, dtype=dtype, device=dev)
    return st


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "loop":
        return state["loop"].run_ring(), state["loop"].state
    if op == "step":
        return lfw_decode_step(*state["in"], state["next"], state["out"])
    fn = {"lfw": LFWFunction, "dfw": DFWFunction, "fused": LFWFusedFunction}[op]
    args = state["in"] + ([case["H"]] if op == "fused" else [])
    if case["pass"] == "fwd":
        with torch.no_grad():
            return fn.apply(*args)
    out, nxt = fn.apply(*args)
    return (out.detach(), nxt.detach(), *torch.autograd.grad([out, nxt], state["in"], state["up"]))


def work(case):
    """Inputs once, outputs once; operations of the step-by-step definition of the recurrence."""
    e = 4 if case["dtype"] == "fp32" else 2
    op, B, T, D, K = case["op"], case["B"], case["T"], case["D"], case["K"]
    train = case["pass"] == "train"
    if op == "fused":
        B, seq = B * case["H"], 4 * 64
    elif op == "dfw":
        seq = D + 2 * K
    else:
        seq = 2 * D + 3 * K
    n = B * T * case.get("ring", 1)
    elems = n * (seq + D) + 2 * B * D * K                    # sequence inputs, outputs, state in and out
    if train:
        elems += n * (D + seq) + 2 * B * D * K               # both upstream gradients, gradients of all inputs
    per = (6, 21) if op != "dfw" else (6, 18)                # multiplies and adds per step and state element
    return {"bytes": e * elems, "flops": per[train] * n * D * K}


def tolerance(case):
    # storage rounding of the results plus the contractions' operand rounding (10 mantissa bits for 16-bit storage);
    # fp32: sums of up to a few hundred terms in another order, divided by gates in the gate gradients
    return {"rel": {"fp16": 5e-3, "bf16": 1e-2, "fp32": 2e-5}[case["dtype"]]}
