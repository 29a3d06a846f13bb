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


# Configurations whose shards, cut by their own number of heads, would be walked in single query tiles where the whole is walked in pairs.
@pytest.mark.parametrize("B,H,T,D,dt,ranks", [(2, 16, 8192, 128, torch.bfloat16, 8), (8, 12, 1024, 64, torch.float32, 8), (16, 12, 1024, 64, torch.bfloat16, 8)])
def test_shards_get_the_bits_of_the_whole(B, H, T, D, dt, ranks):
    from inferno_b200 import _capi
    from inferno_b200.shard import shard_range
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = [_capi.lib().ib200_attn_fwd_item_rows(n, T, 1, sms) for n in (B * H, B * H // ranks)]
    assert rows == [256, 128]
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn(B * H, 1, T, D, device="cuda", generator=g).to(dt) for _ in range(4))
    o, lse = A.attention_forward(q, k, v)
    _, dk, dv = A.attention_backward(q, k, v, o, do, lse)
    for r in range(ranks):
        s = slice(shard_range(B * H, r, ranks).start, shard_range(B * H, r, ranks).stop)
        o1, lse1 = A.attention_forward(q[s], k[s], v[s], total_heads=B * H)
        _, dk1, dv1 = A.attention_backward(q[s], k[s], v[s], o1, do[s], lse1)
        assert all(torch.equal(a, b[s]) for a, b in ((o1, o), (lse1, lse), (dk1, dk), (dv1, dv)))
    assert torch.equal(A.causal_attention(q[s], k[s], v[s], total_heads=B * H), o[s])


def test_packed_op_and_host_pipeline_take_the_number_of_heads_of_the_whole():
    B, H, T, D, heads = 1, 4, 700, 64, 600
    g = torch.Generator(device="cuda").manual_seed(4)
    qkv = torch.randn(B, T, 3 * H * D, device="cuda", generator=g).to(torch.bfloat16)
    many = A.causal_attention_packed(qkv.expand(150, T, 3 * H * D).contiguous(), H)
    assert torch.equal(A.causal_attention_packed(qkv, H, total_heads=heads)[0], many[149])
    q, k, v = (qkv.view(B, T, 3, H, D)[:, :, i].transpose(1, 2).reshape(B * H, 1, T, D) for i in range(3))
    hin = [t.cpu().pin_memory() for t in (q, k, v, q)]
    hout = [torch.empty_like(hin[0]).pin_memory() for _ in range(4)]
    HostAttention(2, T, D, torch.bfloat16, "cuda").run(*hin, *hout, total_heads=heads)
    assert torch.equal(hout[0].view(H, T, D).transpose(0, 1).reshape(T, H * D), many[149].cpu())
    for bad in (0, -1, 2 ** 40):
        with pytest.raises(ValueError, match="total_heads"):
            A.causal_attention_packed(qkv, H, total_heads=bad)
    for call in (lambda: A.causal_attention_packed(qkv, H, total_heads=3), lambda: A.attention_forward(q, k, v, total_heads=3)):
        with pytest.raises(Exception, match="invalid argument"):      # fewer heads than the call itself has
            call()
