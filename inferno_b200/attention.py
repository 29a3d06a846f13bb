"""Host-side mirror of the reference's operator idiom for the fused attention op.

In the reference an op is a free function ``Inferno::op(const Tensor&...) -> Tensor`` that
checks devices and shapes, allocates the output, switches on the device type, calls the
CUDA launcher with raw pointers, and attaches a backward node when gradients are enabled
(src/inferno/core/ops.cpp:204-270; nodes: src/inferno/gradfn/node.h:23-45).  The fused op
stands where InfernoApp/main.cpp:737-754 composes matmul / scale / mask / Softmax / matmul:

    y = causal_attention(q, k, v, scale)         # q, k, v: dense [B, H, T, D] on a CUDA device

Here the tensor type is ``torch.Tensor`` (device memory, streams) and the launcher is the C ABI
of ``include/inferno_b200_attn.h``; the checks, allocations and autograd nodes between the two are
native (``csrc/host_ops.cpp``).  There is no CPU arm: a CPU tensor is rejected, exactly as the
library itself refuses to run without an sm_100 device.
"""
from __future__ import annotations

import torch

from . import _capi

class _Workspace:
    """The caller-owned scratch of the C ABI, one buffer per (device, stream), grown on demand; the native host path keeps it."""

    @property
    def _bufs(self) -> dict:
        return _capi.host().workspaces()


_workspace = _Workspace()


def empty_bthd(B: int, H: int, T: int, D: int, dtype, device) -> torch.Tensor:
    """A [B, H, T, D] view over [B, T, H, D] memory: what the attention output must look like for
    ``y.transpose(1, 2).reshape(B, T, C)`` to be free (InfernoApp/main.cpp:758-761 pays a copy for it)."""
    return torch.empty((B, T, H, D), dtype=dtype, device=device).transpose(1, 2)


def _raise(rc: int, where: str):
    if rc != _capi.OK:
        raise _capi.Ib200Error(rc, where)


def attention_forward(q, k, v, scale: float | None = None, causal: bool = True, math_mode: int = _capi.MATH_SPLIT_BF16,
                      out=None, lse=None, total_heads: int | None = None):
    """Launch the forward kernel.  Returns (o [B,H,T,D], lse [B,H,T] fp32).  Asynchronous on the current stream.

    ``total_heads``: the heads of the whole problem when this call computes a part of them (a shard, a chunk).  The order in which
    a row's keys are summed depends on how many heads there are; given the whole number, a head gets the bits that one call on
    all heads would give it.

    q, k, v (and ``out``) may be arbitrary [B,H,T,D] views with a contiguous last axis -- e.g. slices of a packed
    [B,T,3,H,D] projection, or an output laid out [B,T,H,D] -- and are then read and written in place."""
    return _capi.host().attention_forward(q, k, v, scale, causal, math_mode, out, lse, total_heads)


def attention_backward(q, k, v, o, dO, lse, scale: float | None = None, causal: bool = True,
                       math_mode: int = _capi.MATH_SPLIT_BF16, dq=None, dk=None, dv=None):
    """Launch the backward kernels.  Returns (dq, dk, dv).  Asynchronous on the current stream.
    Operands and outputs may be strided views as in ``attention_forward``."""
    return _capi.host().attention_backward(q, k, v, o, dO, lse, scale, causal, math_mode, dq, dk, dv)


def check_device_status(device=None) -> None:
    """Synchronise the current stream and raise if a kernel reported an expired wait.  The status word is sticky:
    one check after any number of forward / backward calls on this stream sees the first failure among them."""
    import ctypes
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    key = (device.index, torch.cuda.current_stream(device).cuda_stream)
    buf = _workspace._bufs.get(key)
    if buf is None:
        return
    code = ctypes.c_int(0)
    with torch.cuda.device(device):
        rc = _capi.lib().ib200_attn_check(buf.data_ptr(), torch.cuda.current_stream().cuda_stream, ctypes.byref(code))
    if rc != _capi.OK:
        raise _capi.Ib200Error(rc, f"ib200_attn_check (device code {code.value})")


def set_timing_events(fwd_start=None, fwd_stop=None, bwd_start=None, bwd_stop=None) -> None:
    """Have later calls on this thread record these ``torch.cuda.Event``s (timing enabled, created on the
    current device) right around the forward / backward main kernels.  No arguments switches it off."""
    handles = []
    for ev in (fwd_start, fwd_stop, bwd_start, bwd_stop):
        if ev is None:
            handles.append(None)
        else:
            if not ev.cuda_event:          # torch creates the event lazily, on first record
                ev.record()
            handles.append(ev.cuda_event)
    _raise(_capi.lib().ib200_attn_set_timing_events(*handles), "ib200_attn_set_timing_events")


def queue_timing_events(forward=(), backward=()) -> None:
    """Have the next attention calls of this process record these (start, stop) pairs of ``torch.cuda.Event``s right around
    their main kernels: one pair per call, in call order, whichever thread makes the call (autograd runs backward nodes on
    a worker thread of its own, which ``set_timing_events`` does not reach).  No arguments drops what is left."""
    def handles(pairs):
        for e in (e for pair in pairs for e in pair):
            if not e.cuda_event:           # torch creates the event lazily, on first record
                e.record()
        return [(a.cuda_event, b.cuda_event) for a, b in pairs]
    _capi.host().queue_timing_events(handles(list(forward)), handles(list(backward)))


class AttentionBackward:
    """The differentiable op with every option, under the name it had as an autograd function.  Its backward node (csrc/host_ops.cpp) saves q, k, v, out and lse, produces
    dq, dk, dv, and plays the role a ``class AttentionBackward : public Node`` would in the reference
    (src/inferno/gradfn/node.h:23-45: ``backward()``, ``release()``, ``get_inputs()``).
    With ``bthd_out`` the output is laid out [B,T,H,D] in memory (returned as a [B,H,T,D] view).  When q, k, v are
    slices of one packed [B,T,3,H,D] buffer the gradients are written into one packed buffer of the same layout.
    """

    @staticmethod
    def apply(q, k, v, scale, causal, math_mode, bthd_out):
        return _capi.host().causal_attention(q, k, v, scale, causal, math_mode, bthd_out, None)


def causal_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float | None = None,
                     math_mode: int = _capi.MATH_SPLIT_BF16, bthd_out: bool = False, total_heads: int | None = None) -> torch.Tensor:
    """``softmax(mask(q k^T * scale)) v`` with a causal mask; differentiable.  q, k, v: [B,H,T,D] tensors or views.
    ``total_heads`` as in ``attention_forward``."""
    return _capi.host().causal_attention(q, k, v, scale, True, math_mode, bthd_out, total_heads)


def causal_attention_packed(qkv: torch.Tensor, num_heads: int, scale: float | None = None,
                            math_mode: int = _capi.MATH_SPLIT_BF16, total_heads: int | None = None) -> torch.Tensor:
    """Attention straight on the fused projection output: ``qkv`` is [B, T, 3*C] (= [B,T,3,H,D]); returns [B, T, C].
    Replaces slice / contiguous / reshape / transpose / contiguous before the kernels and transpose / contiguous /
    reshape after them (InfernoApp/main.cpp:716-737, 758-761) with stride arithmetic: no copy kernel runs, and the
    gradient is written into one [B, T, 3*C] buffer by the kernels themselves.  ``total_heads`` (batch times heads of the
    whole problem) as in ``attention_forward``."""
    return _capi.host().causal_attention_packed(qkv, num_heads, scale, math_mode, total_heads)
