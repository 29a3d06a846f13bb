"""The work a user of this package has it do, as timed cases: what is called, with which sizes, and how closely two
implementations of it must agree.

Six kinds of call, all through the package's public entry points:
  step      `causal_attention` and its gradients through autograd, on dense [B, H, T, D] tensors (fp32 or bf16)
  packed    `causal_attention_packed` and its gradient, on a fused [B, T, 3*H*D] projection output (bf16)
  fwd       `attention_forward` alone: scoring or prefill, no gradients (bf16 or fp32)
  linear    a `Linear` projection, forward and backward (bf16)
  sublayer  projection -> packed attention -> projection, forward and backward: the attention half of a transformer block
  host      `HostAttention.run`: operands and results in pinned host memory, copies pipelined under the kernels
"""
from __future__ import annotations

import math

import torch

from inferno_b200 import attention as A
from inferno_b200.host_pipeline import HostAttention
from inferno_b200.linear import Linear

_DT = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # the smallest training call: the shape of the CPU unit example; launches and host work are all there is
        dict(name="tiny_step_f32", kind="step", B=4, H=4, T=128, D=64, dtype="f32", std=1.0, do_std=1.0),
        # one layer of a GPT-2-small-shaped model trained in fp32
        dict(name="gpt2_step_f32", kind="step", B=8, H=12, T=1024, D=64, dtype="f32", std=1.0, do_std=0.1),
        # a batch of mid-length sequences whose length divides no tile
        dict(name="ragged_step_bf16", kind="step", B=3, H=5, T=777, D=128, dtype="bf16", std=1.0, do_std=0.1),
        # long-context training: few heads, long walks
        dict(name="long_step_bf16", kind="step", B=2, H=16, T=8192, D=128, dtype="bf16", std=0.5, do_std=0.1),
        # the largest: a whole batch of 4k sequences on one GPU, the benchmark's default workload
        dict(name="box_step_bf16", kind="step", B=64, H=16, T=4096, D=128, dtype="bf16", std=1.0, do_std=0.1),
        # one layer of a 12-layer GPT trained in bf16, operands read in place inside the projection output
        dict(name="gpt_packed_step", kind="packed", B=16, H=12, T=1024, D=64, std=1.0, do_std=0.1),
        # scoring one short prompt with a small model: latency
        dict(name="short_fwd_bf16", kind="fwd", B=1, H=12, T=200, D=64, dtype="bf16", std=1.0),
        # prefill of one long prompt
        dict(name="prefill_fwd_bf16", kind="fwd", B=1, H=16, T=4096, D=128, dtype="bf16", std=1.0),
        # the fused QKV projection of the same GPT at its training batch
        dict(name="qkv_linear_step", kind="linear", M=16384, K=768, N=2304),
        # an output projection at a small ragged batch
        dict(name="small_linear_step", kind="linear", M=1000, K=768, N=768),
        # the attention half of one GPT block, everything on this package
        dict(name="gpt_sublayer_step", kind="sublayer", B=16, H=12, T=1024, D=64),
        # heads whose operands live in host memory, in eight chunks
        dict(name="host_step_bf16", kind="host", heads=32, chunk=4, T=4096, D=128, std=1.0, do_std=0.1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, n):
    """Half of the sizes are left odd or ragged, the others are rounded to the multiples that models use."""
    if n < 64 or rng.random() < 0.5:
        return n
    return max(64, n // 64 * 64)


def _mult8(n):
    return max(8, (n + 4) // 8 * 8)


_MOST = None


def _cost(case):
    w = work(case)
    return max(w["flops"] / 1.0e15, w["bytes"] / 4.0e12)


def draw(rng):
    global _MOST
    if _MOST is None:
        _MOST = max(_cost(c) for c in listed() if c["kind"] != "host")
    while True:
        kind = rng.choices(["step", "packed", "fwd", "linear", "sublayer", "host"], weights=[6, 2, 3, 2, 2, 1])[0]
        if kind in ("step", "fwd"):
            dtype = rng.choice(["bf16", "bf16", "f32"])
            D = 64 if dtype == "f32" else rng.choice([64, 128])
            T = _odd(rng, _log_int(rng, 32, 8192 if dtype == "bf16" else 4096))
            H = rng.choice([1, 2, 4, 5, 8, 12, 16])
            B = _log_int(rng, 1, 64 if kind == "step" else 8)
            case = dict(kind=kind, B=B, H=H, T=T, D=D, dtype=dtype, std=rng.choice([0.5, 1.0]))
            if kind == "step":
                case["do_std"] = rng.choice([0.1, 1.0])
            size = B * H * T * D
            if size > (1 << 29 if dtype == "bf16" else 1 << 26):
                continue
        elif kind == "packed":
            D = rng.choice([64, 128])
            case = dict(kind=kind, B=_log_int(rng, 1, 32), H=rng.choice([4, 8, 12, 16]), T=_odd(rng, _log_int(rng, 64, 4096)), D=D,
                        std=1.0, do_std=0.1)
            if case["B"] * case["H"] * case["T"] * D > 1 << 27:
                continue
        elif kind == "linear":
            case = dict(kind=kind, M=_mult8(_log_int(rng, 64, 32768)), K=_mult8(_log_int(rng, 64, 4096)), N=_mult8(_log_int(rng, 64, 4096)))
        elif kind == "sublayer":
            # the projections take a number of tokens that is a multiple of 8
            case = dict(kind=kind, B=_log_int(rng, 1, 16), H=rng.choice([4, 8, 12]), T=_mult8(_log_int(rng, 64, 2048)), D=64)
        else:
            chunk = rng.choice([2, 4, 8])
            case = dict(kind=kind, heads=chunk * rng.randint(3, 8), chunk=chunk, T=_odd(rng, _log_int(rng, 256, 4096)), D=rng.choice([64, 128]),
                        std=1.0, do_std=0.1)
            if case["heads"] * case["T"] * case["D"] > 32 * 4096 * 128:
                continue
        if _cost(case) <= _MOST:
            return case


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, shape, std, dtype):
    # drawn in slices of the leading axis: the fp32 draws behind a large bf16 tensor then need little memory
    out = torch.empty(shape, dtype=dtype, device="cuda")
    rows = max(1, (1 << 26) // max(1, out[0].numel()))
    for i in range(0, shape[0], rows):
        part = out[i:i + rows]
        part.copy_(torch.randn(part.shape, device="cuda", generator=g).mul_(std))
    return out


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind in ("step", "fwd"):
        shape, dt = (case["B"], case["H"], case["T"], case["D"]), _DT[case["dtype"]]
        q, k, v = (_normal(g, shape, case["std"], dt) for _ in range(3))
        if kind == "fwd":
            return kind, q, k, v
        do = _normal(g, shape, case["do_std"], dt)
        return kind, q.requires_grad_(), k.requires_grad_(), v.requires_grad_(), do
    if kind == "packed":
        B, T, C = case["B"], case["T"], case["H"] * case["D"]
        qkv = _normal(g, (B, T, 3 * C), case["std"], torch.bfloat16)
        return kind, qkv.requires_grad_(), case["H"], _normal(g, (B, T, C), case["do_std"], torch.bfloat16)
    if kind == "linear":
        lin = _linear(g, case["K"], case["N"])
        x = _normal(g, (case["M"], case["K"]), 1.0, torch.bfloat16)
        return kind, lin, x.requires_grad_(), _normal(g, (case["M"], case["N"]), 0.1, torch.bfloat16)
    if kind == "sublayer":
        B, T, C = case["B"], case["T"], case["H"] * case["D"]
        wqkv, wout = _linear(g, C, 3 * C), _linear(g, C, C)
        x = _normal(g, (B, T, C), 1.0, torch.bfloat16)
        return kind, wqkv, wout, case["H"], x.requires_grad_(), _normal(g, (B, T, C), 0.1, torch.bfloat16)
    heads, T, D = case["heads"], case["T"], case["D"]
    pin = lambda t: torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)
    ins = [pin(_normal(g, (heads, 1, T, D), std, torch.bfloat16)) for std in (case["std"],) * 3 + (case["do_std"],)]
    outs = [torch.empty((heads, 1, T, D), dtype=torch.bfloat16, pin_memory=True) for _ in range(4)]
    return kind, HostAttention(case["chunk"], T, D, torch.bfloat16, "cuda", nbuf=3), ins, outs


def _linear(g, K, N):
    """A projection as a bf16 model holds it, with weights at the scale a trained one has."""
    lin = Linear(K, N).cuda().to(torch.bfloat16)
    with torch.no_grad():
        lin.weight.copy_(torch.randn(K, N, device="cuda", generator=g).mul_(K ** -0.5))
        lin.bias.copy_(torch.randn(N, device="cuda", generator=g).mul_(0.02))
    return lin


def run(state):
    kind = state[0]
    if kind == "step":
        _, q, k, v, do = state
        y = A.causal_attention(q, k, v)
        return (y,) + torch.autograd.grad(y, (q, k, v), do)
    if kind == "fwd":
        _, q, k, v = state
        return A.attention_forward(q, k, v)
    if kind == "packed":
        _, qkv, H, dy = state
        y = A.causal_attention_packed(qkv, H)
        return (y,) + torch.autograd.grad(y, (qkv,), dy)
    if kind == "linear":
        _, lin, x, dy = state
        y = lin(x)
        return (y,) + torch.autograd.grad(y, (x, lin.weight, lin.bias), dy)
    if kind == "sublayer":
        _, wqkv, wout, H, x, dy = state
        y = wout(A.causal_attention_packed(wqkv(x), H))
        return (y,) + torch.autograd.grad(y, (x, wqkv.weight, wqkv.bias, wout.weight, wout.bias), dy)
    _, pipe, ins, outs = state
    pipe.run(*ins, *outs)
    return tuple(outs)


def _attention_work(BH, T, D, elt, backward):
    """Causal pairs only; q, k, v (and dO) read once, o and lse (and dq, dk, dv) written once."""
    pairs = T * (T + 1) / 2.0
    tensor = BH * T * D * elt
    return dict(bytes=(8 if backward else 4) * tensor + (0 if backward else 4.0 * BH * T), flops=(14.0 if backward else 4.0) * BH * pairs * D)


def _linear_work(M, K, N):
    return dict(bytes=2.0 * (2 * M * K + 2 * K * N + 2 * M * N + 2 * N), flops=6.0 * M * K * N)


def work(case):
    kind = case["kind"]
    if kind in ("step", "fwd"):
        return _attention_work(case["B"] * case["H"], case["T"], case["D"], 4 if case["dtype"] == "f32" else 2, kind == "step")
    if kind == "packed":
        return _attention_work(case["B"] * case["H"], case["T"], case["D"], 2, True)
    if kind == "linear":
        return _linear_work(case["M"], case["K"], case["N"])
    if kind == "sublayer":
        M, C = case["B"] * case["T"], case["H"] * case["D"]
        attn = _attention_work(case["B"] * case["H"], case["T"], case["D"], 2, True)
        # x, dy read; y, dx written; both weights and biases read and their gradients written
        return dict(bytes=2.0 * (4 * M * C + 2 * 4 * C * C + 2 * 4 * C), flops=attn["flops"] + 6.0 * M * C * 4 * C)
    return _attention_work(case["heads"], case["T"], case["D"], 2, True)


def tolerance(case):
    if case.get("dtype") == "f32":
        # products of fp32 operands carried as bf16 pairs: 2^-16 each, fp32 sums
        return dict(rel=5e-5)
    return dict(rel=1e-2)
