"""The projection GEMM (bf16 tcgen05, fp32 accumulate, bias epilogue) against a float32 PyTorch matmul.
Tolerance: normwise relative error 1e-2 (bf16 output rounding is 2^-9 per element)."""
import pytest
import torch

from inferno_b200 import _capi
from inferno_b200 import linear as L

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


@pytest.mark.parametrize("M,K,N", [(128, 64, 256), (256, 768, 2304), (1000, 768, 768), (136, 72, 264), (4096, 3072, 768),
                                   (8192, 256, 256),     # weight gradient: 2 output tiles, split-K over 8 slabs
                                   (128, 8192, 256)])    # forward: 1 output tile, split-K with the bias going in once
def test_forward_and_backward_match_float32_reference(M, K, N):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(K, N, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    b = torch.randn(N, device="cuda", generator=g)
    dy = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    y = L.linear_forward(x, w, b)
    dx, dw, db = L.linear_backward(x, w, dy)
    torch.cuda.synchronize()
    xf, wf, dyf = x.float(), w.float(), dy.float()
    assert rel(y, xf @ wf + b) < 1e-2
    assert rel(dx, dyf @ wf.t()) < 1e-2
    assert rel(dw, xf.t() @ dyf) < 1e-2
    assert rel(db, dyf.sum(0)) < 1e-4


def test_generic_entry_point_all_operand_majors():
    M, N, K = 256, 512, 192
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(K, N, device="cuda").to(torch.bfloat16)
    want = a.float() @ b.float()
    lib = _capi.lib()
    s = torch.cuda.current_stream().cuda_stream
    for a_t in (0, 1):
        for b_t in (0, 1):
            aa = a.t().contiguous() if a_t else a
            bb = b.t().contiguous() if b_t else b
            c = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
            rc = lib.ib200_gemm_bf16(aa.data_ptr(), bb.data_ptr(), c.data_ptr(), None, M, N, K, a_t, b_t, s)
            assert rc == _capi.OK
            torch.cuda.synchronize()
            assert rel(c, want) < 1e-2, (a_t, b_t)
    assert lib.ib200_gemm_bf16(a.data_ptr(), b.data_ptr(), c.data_ptr(), None, M, N, 100, 0, 0, s) == _capi.ERR_UNSUPPORTED
    assert lib.ib200_gemm_bf16(None, b.data_ptr(), c.data_ptr(), None, M, N, K, 0, 0, s) == _capi.ERR_INVALID_ARGUMENT


def test_linear_module_autograd():
    torch.manual_seed(1)
    lin = L.Linear(256, 384).cuda().to(torch.bfloat16)
    x = torch.randn(4, 96, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = lin(x)
    y.backward(torch.ones_like(y))
    ref = x.detach().float() @ lin.weight.detach().float() + lin.bias.detach().float()
    assert rel(y.detach(), ref) < 1e-2
    assert rel(lin.bias.grad, torch.full((384,), 4 * 96.0, device="cuda")) < 1e-2
    assert x.grad is not None and lin.weight.grad is not None


@pytest.mark.parametrize("M,K,N", [(8, 8, 8),              # less than one k-step, one corner of a tile
                                   (256, 64, 256),         # exactly one tile of a CTA pair
                                   (264, 72, 520),         # one step past it in every direction
                                   (136, 4104, 264),       # forward cut along K, ragged last slice
                                   (4104, 136, 264),       # weight gradient cut along K, ragged last slice
                                   (1000, 768, 768), (20000, 256, 512),
                                   (9480, 1032, 2056)])    # more tiles than CTA pairs in dX, dW's slices even out the load
def test_tile_edges_and_split_products(M, K, N):
    """Every output has one bf16 rounding on top of fp32 sums: at most 2^-9 of each value, so 2^-9 of the norm; the
    summation error (2^-24 sqrt(K) at K <= 20000) is far below the factor of 1.5 left for it."""
    g = torch.Generator(device="cuda").manual_seed(3 * M + K + N)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
    lin = L.Linear(K, N).cuda().to(torch.bfloat16)
    with torch.no_grad():
        lin.bias.copy_(torch.randn(N, device="cuda", generator=g))
    dy = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    y = lin(x)
    dx, dw, db = torch.autograd.grad(y, (x, lin.weight, lin.bias), dy)
    _, _, db32 = L.linear_backward(x.detach(), lin.weight.detach(), dy, need_dx=False)
    _, dw1, _ = L.linear_backward(x.detach(), lin.weight.detach(), dy, need_dx=False, need_db=False)
    torch.cuda.synchronize()
    xd, wd, dyd = x.detach().double(), lin.weight.detach().double(), dy.double()
    tol = 1.5 * 2.0 ** -9
    assert rel(y.double(), xd @ wd + lin.bias.detach().double()) < tol
    assert rel(dx.double(), dyd @ wd.t()) < tol
    assert rel(dw.double(), xd.t() @ dyd) < tol and rel(dw1.double(), xd.t() @ dyd) < tol
    assert db.dtype == torch.bfloat16 and rel(db.double(), dyd.sum(0)) < tol
    assert rel(db32.double(), dyd.sum(0)) < 1e-5


@pytest.mark.parametrize("offset", [1, 3, 4, 8])      # 2, 6, 8 and 16 bytes past an aligned address
def test_bias_may_be_a_slice(offset):
    x, w = (torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((64, 64), (64, 264)))
    buf = torch.randn(300, device="cuda").to(torch.bfloat16)
    b = buf[offset:offset + 264]
    y = L.linear_forward(x, w, b)
    assert torch.equal(y, L.linear_forward(x, w, b.clone())) and rel(y, x.float() @ w.float() + b.float()) < 1e-2


@pytest.mark.parametrize("M,K,N", [(16384, 768, 2304), (8192, 512, 768), (1000, 768, 768)])
def test_weight_gradient_without_a_workspace_has_few_roundings(M, K, N):
    """ib200_linear_bwd adds its parts in bf16.  With tiles of 256 x 256 that leave 74 CTA pairs half idle these have two to eight parts; where
    two suffice (the first shape: 27 tiles) the result is the same from run to run."""
    g = torch.Generator(device="cuda").manual_seed(5)
    x, w, dy = (torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16) for s in ((M, K), (K, N), (M, N)))
    s = torch.cuda.current_stream().cuda_stream
    runs = []
    for _ in range(6):
        dx, dw, db = torch.empty_like(x), torch.empty_like(w), torch.empty(N, device="cuda")
        assert _capi.lib().ib200_linear_bwd(x.data_ptr(), w.data_ptr(), dy.data_ptr(), dx.data_ptr(), dw.data_ptr(), db.data_ptr(), M, K, N, s) == _capi.OK
        runs.append(dw)
    ref = x.double().t() @ dy.double()
    parts = min(8, 74 // (-(-K // 256) * -(-N // 256)), M // 64 // 8)
    # each part and each sum is rounded to 8 bits: relative error of at most 2^-9 of a running sum, whose norm grows as the square root
    tol = 2.0 ** -9 * (1 + sum(((i + 1) / parts) ** 0.5 for i in range(parts)))
    assert rel(runs[0].double(), ref) < tol
    if parts == 2:
        assert all(torch.equal(r, runs[0]) for r in runs)
