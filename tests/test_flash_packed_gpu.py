"""Attention on packed QKV (rotary, forward, gradients in place) and the backward's edges: ragged tiles, unseen key tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(qkv, cos, sin, g, p, causal, interleaved, dout):
    """64-bit attention of the packed activation and its gradient."""
    x = qkv.double().requires_grad_(True)
    s, b, _ = x.shape
    v5 = x.view(s, b, g, p + 2, 128)

    def rot(t):
        if cos is None:
            return t
        r = cos.shape[-1]
        a, rest = t[..., :r], t[..., r:]
        half = torch.stack((-a[..., 1::2], a[..., 0::2]), -1).reshape(a.shape) if interleaved else \
            torch.cat((-a[..., r // 2:], a[..., :r // 2]), -1)
        return torch.cat((a * cos.double().view(s, 1, 1, 1, r) + half * sin.double().view(s, 1, 1, 1, r), rest), -1)
    q, k, v = rot(v5[:, :, :, :p]), rot(v5[:, :, :, p:p + 1]), v5[:, :, :, p + 1:]
    sc = torch.einsum("sbgpd,tbgqd->bgpst", q, k) * 128 ** -0.5
    if causal:
        sc = sc.masked_fill(torch.ones(s, s, dtype=torch.bool, device=x.device).triu(1), float("-inf"))
    out = torch.einsum("bgpst,tbgqd->sbgpd", sc.softmax(-1), v).reshape(s, b, g * p, 128)
    out.backward(dout.double())
    return out.detach(), x.grad


@pytest.mark.parametrize("s,b,g,p", [(1, 1, 1, 1), (127, 2, 2, 3), (128, 1, 3, 1), (300, 1, 2, 4), (640, 2, 1, 2), (1025, 1, 4, 1)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("rope", [None, "half", "interleaved"])
def test_packed_attention(s, b, g, p, causal, rope):
    """bf16 operands, probabilities and score gradients, fp32 sums: 1e-2 of the norm, as between any two bf16 attentions."""
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops.flash_sm100_impl import flash_attention_packed
    torch.manual_seed(s + g)
    base = torch.randn(s, b, g * (p + 2) * 128, device="cuda", dtype=torch.bfloat16)
    ang = torch.rand(s, 128, device="cuda") * 6
    if rope == "half":
        ang[:, 64:] = ang[:, :64]
    elif rope:
        ang[:, 1::2] = ang[:, 0::2]
    cos, sin = (ang.cos(), ang.sin()) if rope else (None, None)
    dout = torch.randn(s, b, g * p, 128, device="cuda", dtype=torch.bfloat16)
    leaf = base.clone().requires_grad_(True)
    out = flash_attention_packed(leaf * 1.0, cos, sin, g, p, rope == "interleaved", causal, 128 ** -0.5)
    out.backward(dout)
    torch.cuda.synchronize()
    G.check_status()
    ro, rg = _oracle(base, cos, sin, g, p, causal, rope == "interleaved", dout)
    assert ((out.double() - ro).norm() / ro.norm()).item() < 1e-2
    assert ((leaf.grad.double() - rg).norm() / rg.norm().clamp_min(1e-3)).item() < 1e-2
    v_grad = leaf.grad.view(s, b, g, p + 2, 128)[:, :, :, p + 1].double()
    assert ((v_grad - rg.view(s, b, g, p + 2, 128)[:, :, :, p + 1]).norm() / rg.norm()).item() < 1e-2


@pytest.mark.parametrize("sq,sk,nq,nkv", [(128, 384, 2, 2), (100, 700, 4, 1), (256, 520, 300, 300)])
def test_key_tiles_that_no_query_sees_get_zero_gradients(sq, sk, nq, nkv):
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops.attention import attention_ref, attn_bwd_ref
    from mindspeed_b200.ops.flash_sm100_impl import flash_bwd, flash_fwd
    torch.manual_seed(sq)
    q, k, v, do = (torch.randn(n, 1, h, 128, device="cuda", dtype=torch.bfloat16) for n, h in ((sq, nq), (sk, nkv), (sk, nkv), (sq, nq)))
    o, lse = flash_fwd(q, k, v, True, 128 ** -0.5, q_offset=0)
    junk = [torch.full_like(t, float("nan")) for t in (q, k, v)]
    dq, dk, dv = flash_bwd(do, q, k, v, o, lse, True, 128 ** -0.5, q_offset=0, out=junk)
    torch.cuda.synchronize()
    G.check_status()
    assert dk[sq:].abs().max().item() == 0 and dv[sq:].abs().max().item() == 0
    for a, r in zip((dq, dk, dv), attn_bwd_ref(do, q, k, v, o, lse, True, 128 ** -0.5)):
        assert ((a.float() - r.float()).norm() / r.float().norm()).item() < 1e-2
