"""Self attention as a module: the packed route against the one through the core attention module."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,groups", [(4, 4), (4, 2), (4, 1)])
@pytest.mark.parametrize("rope", [None, "half", "interleaved"])
@pytest.mark.parametrize("hooks", [False, True])
def test_packed_and_unpacked_agree(heads, groups, rope, hooks, monkeypatch):
    """The same kernels on the same numbers, so outputs are equal; of the gradients dQ is a sum of fp32 atomics that is rounded to bf16
    once (2^-8 relative for one element in another order's place, far less over a norm) and passes through one bf16 product."""
    from mindspeed_b200.config import TransformerConfig
    from mindspeed_b200.models.attention import SelfAttention
    from mindspeed_b200.ops import flash_sm100_impl as F
    from mindspeed_b200.ops import gemm as G
    torch.manual_seed(heads + groups)
    cfg = TransformerConfig(num_layers=1, hidden_size=heads * 128, num_attention_heads=heads, num_query_groups=groups, optimization_level=2,
                            params_dtype=torch.bfloat16, attention_dropout=0.0, rotary_interleaved=rope == "interleaved")
    m = SelfAttention(cfg).cuda().bfloat16()
    calls, own = [], F.flash_attention_packed
    monkeypatch.setattr(F, "flash_attention_packed", lambda *a: (calls.append(1), own(*a))[1])
    x = torch.randn(300, 2, heads * 128, device="cuda", dtype=torch.bfloat16)
    ang = torch.rand(300, 128, device="cuda") * 6
    if rope == "half":
        ang[:, 64:] = ang[:, :64]
    elif rope:
        ang[:, 1::2] = ang[:, 0::2]
    rpe = (ang.cos(), ang.sin()) if rope else None
    dout = torch.randn_like(x)

    def run():
        m.zero_grad(set_to_none=True)
        leaf = x.clone().requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t) if hooks else contextlib.nullcontext():
            out = m(leaf, rotary_pos_emb=rpe)[0]
            out.backward(dout)
        return [out, leaf.grad] + [p.grad for p in m.parameters() if p.grad is not None]
    got = run()
    assert calls
    handle = m.core_attention.register_forward_hook(lambda *a: None)
    calls.clear()
    want = run()
    handle.remove()
    torch.cuda.synchronize()
    G.check_status()
    assert not calls and torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 2e-3
