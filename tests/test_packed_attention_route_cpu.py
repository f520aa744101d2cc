"""When self attention runs on the packed QKV activation, and when it goes through the core attention module as before.  Availability of
the kernels is let through; what is tested is the choice."""
import pytest
import torch


@pytest.fixture
def layer(monkeypatch):
    from mindspeed_b200.config import TransformerConfig
    from mindspeed_b200.models.attention import SelfAttention
    from mindspeed_b200.ops import flash_sm100_impl as F
    cfg = TransformerConfig(num_layers=1, hidden_size=256, num_attention_heads=2, use_cpu_initialization=True, optimization_level=2,
                            attention_dropout=0.0)
    m = SelfAttention(cfg)
    m.packed_calls = []

    def packed(qkv, cos, sin, groups, qpg, interleaved, causal, scale):
        m.packed_calls.append(1)
        return torch.zeros(*qkv.shape[:2], groups * qpg, 128)
    monkeypatch.setattr(F, "packed_supports", lambda *a: True)
    monkeypatch.setattr(F, "flash_attention_packed", packed)
    return m


def _run(m):
    m.packed_calls.clear()
    m(torch.randn(8, 1, 256))
    return bool(m.packed_calls)


def test_plain_self_attention_is_packed(layer):
    assert _run(layer)


@pytest.mark.parametrize("kind", ["register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook",
                                  "register_full_backward_pre_hook"])
@pytest.mark.parametrize("everywhere", [False, True])
def test_hooked_core_attention_is_called(layer, kind, everywhere):
    seen = []
    hook = lambda mod, *a: seen.append(type(mod).__name__)
    if everywhere:
        handle = getattr(torch.nn.modules.module, kind.replace("register_", "register_module_"))(hook)
    else:
        handle = getattr(layer.core_attention, kind)(hook)
    try:
        assert not _run(layer)
        if "forward" in kind:
            assert "CoreAttention" in seen
    finally:
        handle.remove()
    assert _run(layer)


@pytest.mark.parametrize("what", ["instance", "class", "flash_attention", "subclass"])
def test_replaced_core_attention_is_called(layer, monkeypatch, what):
    from mindspeed_b200.models import attention as A
    seen = []

    def forward(*args, **kw):
        seen.append(1)
        q = next(a for a in args if torch.is_tensor(a))
        return q.reshape(*q.shape[:2], -1)
    if what == "instance":
        layer.core_attention.forward = forward
    elif what == "class":
        monkeypatch.setattr(A.CoreAttention, "forward", forward)
    elif what == "flash_attention":
        monkeypatch.setattr(A.attn_ops, "flash_attention", lambda q, *a, **k: (seen.append(1), q)[1])
    else:
        layer.core_attention.__class__ = type("Mine", (A.CoreAttention,), {"forward": forward})
    assert not _run(layer) and seen
