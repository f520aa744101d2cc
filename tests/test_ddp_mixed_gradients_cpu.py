"""Parameters whose gradient comes from a fused op (straight into main_grad) and from autograd in the same backward."""
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from dist_utils import run_distributed


def _tied(rank, world, fusion, overlap, penalty):
    import torch.distributed as dist
    from mindspeed_b200.config import TransformerConfig
    from mindspeed_b200.models.gpt_model import GPTModel
    from mindspeed_b200.ops import permute
    from mindspeed_b200.parallel import layers, parallel_state as ps
    from mindspeed_b200.parallel.distributed.ddp import DistributedDataParallel, DistributedDataParallelConfig
    if not dist.is_initialized():
        dist.init_process_group("gloo", rank=rank, world_size=world)
    ps.initialize_model_parallel()
    torch.manual_seed(0)
    cfg = TransformerConfig(num_layers=1, hidden_size=32, num_attention_heads=2, use_cpu_initialization=True, hidden_dropout=0.0,
                            attention_dropout=0.0, gradient_accumulation_fusion=fusion, optimization_level=2)
    if penalty and fusion:                      # let the lookup's device test through; the kernel stands in as index_add_
        layers.VocabParallelEmbedding._fused = lambda self, ids: torch.is_grad_enabled()
        permute.add_rows_ = lambda out, idx, src: out.index_add_(0, idx, src.float())
    model = GPTModel(cfg, vocab_size=64, max_sequence_length=16, share_embeddings_and_output_weights=not penalty)
    ddp = DistributedDataParallel(cfg, DistributedDataParallelConfig(grad_reduce_in_fp32=True, overlap_grad_reduce=overlap), model)
    ddp.zero_grad_buffer()
    w = model.embedding.word_embeddings.weight
    gen = torch.Generator().manual_seed(rank)
    for step in range(2):
        ids = torch.randint(0, 64, (2, 16), generator=gen)
        loss = ddp(ids, torch.arange(16).expand(2, -1), None, labels=ids.roll(-1, 1)).mean()
        if penalty:
            loss = loss + w.square().sum()
        if step == 0:
            with ddp.no_sync():
                loss.backward()
        else:
            loss.backward()
    ddp.finish_grad_sync()
    return w.main_grad.clone()


@pytest.mark.parametrize("overlap", [False, True])
def test_shared_table_gets_both_gradients(overlap):
    """The output layer's share goes into main_grad by itself, the lookup's comes from autograd, after the wrapper may already have heard
    of the first.  fp32 on both sides, sums in another order."""
    want = run_distributed(_tied, 2, False, False, False)
    got = run_distributed(_tied, 2, True, overlap, False)
    for a, b in zip(got, want):
        torch.testing.assert_close(torch.as_tensor(a), torch.as_tensor(b), rtol=1e-4, atol=1e-6)


def test_penalty_beside_a_fused_lookup():
    want = run_distributed(_tied, 1, False, False, True)
    got = run_distributed(_tied, 1, True, False, True)
    torch.testing.assert_close(torch.as_tensor(got[0]), torch.as_tensor(want[0]), rtol=1e-4, atol=1e-6)
