"""Calls captured into CUDA graphs: the first call of a process or thread, and what later calls do to a captured one's scratch."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_FIRST_CALL = r"""
import sys, torch
from inferno_b200 import attention as A
from inferno_b200.linear import Linear
bf16 = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
q, k, v, do = (bf16(2, 4, 256, 64) for _ in range(4))
qkv, dz = bf16(2, 200, 384), bf16(2, 200, 128)
lin, x, dy = Linear(768, 768).cuda().to(torch.bfloat16), bf16(1000, 768), bf16(1000, 768)
for t in (q, k, v, qkv, x):
    t.requires_grad_()
def forward():
    return A.attention_forward(q.detach(), k.detach(), v.detach())
def step():
    y = A.causal_attention(q, k, v)
    return (y,) + torch.autograd.grad(y, (q, k, v), do)
def packed():
    y = A.causal_attention_packed(qkv, 2)
    return (y,) + torch.autograd.grad(y, qkv, dz)
def linear():
    y = lin(x)
    return (y,) + torch.autograd.grad(y, (x, lin.weight, lin.bias), dy)
if sys.argv[1] == "step":
    forward()                  # this thread has made a call, autograd's worker has not
    torch.cuda.synchronize()
fn = dict(forward=forward, step=step, packed=packed, linear=linear)[sys.argv[1]]
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    captured = fn()
g.replay()
eager = fn()
torch.cuda.synchronize()
for a, b in zip(captured, eager):
    assert float((a.float() - b.float()).norm()) <= 1e-3 * float(b.float().norm())
print("captured and replayed")
"""


@pytest.mark.parametrize("what", ["forward", "step", "packed", "linear"])
def test_the_first_call_of_a_process_or_thread_can_be_captured(what):
    res = subprocess.run([sys.executable, "-c", _FIRST_CALL, what], env=dict(os.environ, PYTHONPATH=ROOT), cwd=ROOT, capture_output=True, text=True,
                         timeout=120)
    assert res.returncode == 0 and "captured and replayed" in res.stdout, res.stdout[-500:] + res.stderr[-2000:]


@pytest.mark.parametrize("captured", ["linear", "attention"])
def test_a_captured_call_keeps_its_scratch_when_a_projection_needs_more(captured):
    """Replaying a graph after a larger eager projection on the capture stream writes to the graph's own memory, not to what has since been
    handed to somebody else."""
    from inferno_b200 import attention as A
    from inferno_b200.linear import Linear
    bf16 = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        lin, x, dy = Linear(512, 512).cuda().to(torch.bfloat16), bf16(2048, 512).requires_grad_(), bf16(2048, 512)
        big, xb, dyb = Linear(4096, 4096).cuda().to(torch.bfloat16), bf16(4096, 4096).requires_grad_(), bf16(4096, 4096)
        q = torch.randn(1, 4, 512, 64, device="cuda")
        step = (lambda: torch.autograd.grad(lin(x), (x, lin.weight, lin.bias), dy)) if captured == "linear" else (lambda: A.attention_forward(q, q, q))
        want = [t.clone() for t in step()]
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            out = step()
        torch.autograd.grad(big(xb), (xb, big.weight, big.bias), dyb)
        # whatever that gave back to the allocator is handed out again
        junk = [torch.full((n,), 7, device="cuda", dtype=torch.uint8) for n in (1 << 16, 1 << 18, 1 << 20, 1 << 21, 1 << 22, 1 << 23) for _ in range(4)]
        g.replay()
        s.synchronize()
        assert all(bool((j == 7).all()) for j in junk)
        for a, b in zip(out, want):
            assert float((a.float() - b.float()).norm()) <= 1e-3 * float(b.float().norm())
