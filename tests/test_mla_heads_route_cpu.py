"""Which operands the latent-attention head kernel takes: it reads by the shapes of the queries, so all others have to fit them."""
import pytest
import torch


class _OnGpu(torch.Tensor):
    is_cuda = True


def _operands(s=3, b=2, n=4, nope=8, rope=16, vd=8):
    on = lambda *shape: torch.zeros(*shape).as_subclass(_OnGpu)
    return dict(q=on(s, b, n, nope + rope), kv=on(s, b, n, nope + vd), k_pe=on(s, b, rope), cos=on(s, rope), sin=on(s, rope))


@pytest.mark.parametrize("name,shape", [("kv", (3, 2, 2, 16)), ("kv", (2, 2, 4, 16)), ("k_pe", (3, 1, 16)), ("k_pe", (2, 2, 16)), ("k_pe", (3, 2, 1, 16)),
                                        ("q", (3, 2, 4, 32)), ("sin", (1, 16)), ("cos", (2, 16)), ("cos", (3, 1, 1, 16)), (None, None)])
def test_operands_that_do_not_fit_take_the_torch_form(monkeypatch, name, shape):
    from mindspeed_b200.ops import mla_heads as H
    monkeypatch.setattr(H.loader, "use_kernels", lambda t: t.is_cuda)
    ops = _operands()
    if name is not None:
        ops[name] = torch.zeros(shape).as_subclass(_OnGpu)
    assert H.supports(*(ops[k] for k in ("q", "kv", "k_pe", "cos", "sin")), 8) is (name is None)
    if name is None:
        ops["sin"] = torch.zeros(3, 16)
        assert not H.supports(*(ops[k] for k in ("q", "kv", "k_pe", "cos", "sin")), 8)
