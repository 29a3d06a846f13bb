"""Host-side mirror of the reference's ``Linear`` for the two projections around attention.

``Linear::forward`` in the reference is ``matmul(x, W) + b`` with the weight stored ``[in, out]``
(src/inferno/modules/linear.cpp:19-106); its backward is MMBackward + the bias' sum_to_shape
(src/inferno/gradfn/mmbackward.cpp:36-98).  Here both directions run on the tcgen05 GEMM of
``csrc/linear_gemm.cuh`` through the C ABI (bf16 tensors, a bias of either type, fp32 accumulation).
"""
from __future__ import annotations

import torch

from . import _capi


def linear_forward(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """y = x @ w + bias with x [..., K], w [K, N] (the reference's [in, out] storage), bias [N]."""
    return _capi.host().linear_forward(x, w, bias)


def linear_backward(x, w, dy, need_dx=True, need_dw=True, need_db=True):
    """(dx, dw, db) of ``linear_forward``; db is fp32; what is not needed comes back as None.

    A dW whose tiles alone would not fill the GPU evenly is cut along the tokens and its parts are added up in fp32 in the order in
    which they finish: its bits can differ from run to run in the last place.  dx, db and y repeat bit for bit."""
    return _capi.host().linear_backward(x, w, dy, need_dx, need_dw, need_db)


class LinearFunction:
    """The differentiable projection (backward node in csrc/host_ops.cpp), under the name it had as an autograd function."""

    @staticmethod
    def apply(x, w, bias):
        return _capi.host().linear(x, w, bias)


class Linear(torch.nn.Module):
    """``x @ W + b`` with W stored [in, out] like the reference's Linear; bf16 weight, fp32-accumulated GEMM."""

    def __init__(self, in_features: int, out_features: int, bias: bool = True):
        super().__init__()
        self.weight = torch.nn.Parameter(torch.empty(in_features, out_features))
        self.bias = torch.nn.Parameter(torch.zeros(out_features)) if bias else None
        torch.nn.init.normal_(self.weight, 0.0, 0.02)

    def forward(self, x):
        return _capi.host().linear(x, self.weight, self.bias)


def _time_shape(M: int, K: int, N: int, iters: int = 20):
    """Forward and backward of one projection on synthetic bf16 data, timed with CUDA events."""
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(K, N, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16)
    b = torch.randn(N, device="cuda", generator=g)
    dy = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)

    def timed(fn):
        for _ in range(3):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(iters):
            fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / iters

    fwd = timed(lambda: linear_forward(x, w, b))
    bwd = timed(lambda: linear_backward(x, w, dy))
    flop = 2.0 * M * K * N
    return dict(M=M, K=K, N=N, fwd_ms=fwd, fwd_tflops=flop / fwd / 1e9, bwd_ms=bwd, bwd_tflops=2 * flop / bwd / 1e9)


if __name__ == "__main__":
    import argparse
    import json

    ap = argparse.ArgumentParser(description="time y = x W + b and its backward (dX, dW, db) on one GPU")
    ap.add_argument("M", type=int, nargs="?", default=16384)
    ap.add_argument("K", type=int, nargs="?", default=768)
    ap.add_argument("N", type=int, nargs="?", default=2304)
    ap.add_argument("--iters", type=int, default=20)
    a = ap.parse_args()
    print(json.dumps(_time_shape(a.M, a.K, a.N, a.iters)))
