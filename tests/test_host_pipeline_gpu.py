"""The pinned-host pipeline (inferno_b200.host_pipeline.HostAttention): operands in host memory, chunked over heads on
three streams with two staging sets.  Its results must equal, bit for bit, those of the same kernels run on resident
tensors, for every head of every chunk, also when the last chunk is short and when the pipeline object is reused."""
import pytest
import torch

from inferno_b200 import attention as A
from inferno_b200.host_pipeline import HostAttention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,hc,T,D", [(10, 3, 256, 128), (7, 2, 200, 64), (4, 8, 128, 128)])
def test_pipeline_matches_resident_path(heads, hc, T, D):
    g = torch.Generator().manual_seed(heads * 1000 + T)
    hin = [torch.randn((heads, 1, T, D), generator=g).to(torch.bfloat16).pin_memory() for _ in range(4)]
    hout = [torch.empty((heads, 1, T, D), dtype=torch.bfloat16).pin_memory() for _ in range(4)]
    pipe = HostAttention(hc, T, D, torch.bfloat16, "cuda")
    for _ in range(3):                                   # reuse: staging sets and events of the previous run
        for t in hout:
            t.fill_(float("nan"))
        pipe.run(*hin, *hout)
        torch.cuda.synchronize()
        q, k, v, do = (t.cuda() for t in hin)
        o, lse = A.attention_forward(q, k, v)
        dq, dk, dv = A.attention_backward(q, k, v, o, do, lse)
        torch.cuda.synchronize()
        # dQ goes through fp32 atomics whose order is not fixed, so it is compared to a tolerance; the rest bitwise
        assert torch.equal(hout[0], o.cpu())
        assert torch.equal(hout[2], dk.cpu()) and torch.equal(hout[3], dv.cpu())
        assert float((hout[1].float() - dq.cpu().float()).abs().max()) <= 1e-2 * float(dq.float().abs().max())


def test_chunk_of_a_large_problem_is_walked_like_the_whole():
    """One head alone would be walked in single query tiles, 600 heads in pairs: as a chunk, one head must give the bits of the 600."""
    from inferno_b200 import _capi
    one = [torch.randn((1, 1, 700, 64), device="cuda").to(torch.bfloat16) for _ in range(3)]
    o, lse = _capi.host().attention_forward(*one, None, True, _capi.MATH_SPLIT_BF16, None, None, 600)
    o2, lse2 = A.attention_forward(*(t.expand(600, 1, 700, 64).contiguous() for t in one))
    torch.cuda.synchronize()
    assert torch.equal(o[0], o2[599]) and torch.equal(lse[0], lse2[599])
    with pytest.raises(_capi.Ib200Error):
        _capi.host().attention_forward(*(t.expand(3, 1, 700, 64).contiguous() for t in one), None, True, _capi.MATH_SPLIT_BF16, None, None, 2)
