"""Logits of a batch are those of its samples, sample-major."""
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
