"""Logits of a batch are those of its samples, sample-major."""
import pytest
import torch


def test_logits_of_a_batch():
    from mindspeed_b200.config import TransformerConfig
    from mindspeed_b200.models.gpt_model import GPTModel
    torch.manual_seed(0)
    cfg = TransformerConfig(num_layers=1, hidden_size=32, num_attention_heads=2, use_cpu_initialization=True)
    model = GPTModel(cfg, vocab_size=64, max_sequence_length=16)
    tokens = torch.randint(0, 64, (3, 16))
    pos = torch.arange(16).expand(3, -1)
    with torch.no_grad():
        both = model(tokens, pos, None)
        each = torch.cat([model(tokens[i:i + 1], pos[i:i + 1], None) for i in range(3)])
    assert both.shape == (3, 16, 64) and both.is_contiguous()
    torch.testing.assert_close(both, each, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("how", ["hook", "pre_hook", "global", "class"])
def test_who_watches_the_output_layer_sees_sequence_major(how, monkeypatch):
    """[s, b, h] in, whatever the batch size, as with labels."""
    from mindspeed_b200.config import TransformerConfig
    from mindspeed_b200.models.gpt_model import GPTModel
    from mindspeed_b200.parallel.layers import ColumnParallelLinear
    torch.manual_seed(0)
    cfg = TransformerConfig(num_layers=1, hidden_size=32, num_attention_heads=2, use_cpu_initialization=True)
    model = GPTModel(cfg, vocab_size=64, max_sequence_length=16)
    tokens, pos = torch.randint(0, 64, (3, 16)), torch.arange(16).expand(3, -1)
    with torch.no_grad():
        want = model(tokens, pos, None)
        shapes = []

        def see(mod, args, *_):
            if mod is model.output_layer:
                shapes.append(tuple(args[0].shape))
        if how == "hook":
            handle = model.output_layer.register_forward_hook(see)
        elif how == "pre_hook":
            handle = model.output_layer.register_forward_pre_hook(see)
        elif how == "global":
            handle = torch.nn.modules.module.register_module_forward_hook(see)
        else:
            own = ColumnParallelLinear.forward
            monkeypatch.setattr(ColumnParallelLinear, "forward", lambda self, x, *a, **k: (see(self, (x,)), own(self, x, *a, **k))[1])
            handle = None
        got = model(tokens, pos, None)
        if handle is not None:
            handle.remove()
    assert shapes == [(16, 3, 32)]
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5)
