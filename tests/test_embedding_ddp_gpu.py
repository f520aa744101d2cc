"""Fused embedding gradient under the data-parallel wrapper, accumulated over micro-batches, against the dense one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r'''
import os, socket
with socket.socket() as s:
    s.bind(("127.0.0.1", 0))
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(s.getsockname()[1]), RANK="0", WORLD_SIZE="1", LOCAL_RANK="0")
import torch
torch.distributed.init_process_group("gloo", rank=0, world_size=1)
from mindspeed_b200.config import TransformerConfig
from mindspeed_b200.models.gpt_model import GPTModel
from mindspeed_b200.ops import permute
from mindspeed_b200.parallel import parallel_state as ps
from mindspeed_b200.parallel.distributed.ddp import DistributedDataParallel, DistributedDataParallelConfig
ps.initialize_model_parallel()
torch.manual_seed(0)
cfg = TransformerConfig(num_layers=1, hidden_size=256, num_attention_heads=2, hidden_dropout=0.0, attention_dropout=0.0, optimization_level=2,
                        gradient_accumulation_fusion=True, params_dtype=torch.bfloat16, bf16=True)
model = GPTModel(cfg, vocab_size=512, max_sequence_length=64).cuda()
ddp = DistributedDataParallel(cfg, DistributedDataParallelConfig(grad_reduce_in_fp32=True, overlap_grad_reduce=True), model)
table, calls, own = model.embedding.word_embeddings, [], permute.add_rows_
permute.add_rows_ = lambda *a: (calls.append(1), own(*a))[1]
batches = [torch.randint(0, 40, (2, 64), device="cuda") for _ in range(3)]          # few distinct ids: every row repeats
pos = torch.arange(64, device="cuda").expand(2, -1)
def step():
    ddp.zero_grad_buffer()
    for i, ids in enumerate(batches):
        loss = ddp(ids, pos, None, labels=ids.roll(-1, 1)).mean()
        if i + 1 < len(batches):
            with ddp.no_sync():
                loss.backward()
        else:
            loss.backward()
    ddp.finish_grad_sync()
    torch.cuda.synchronize()
    assert table.weight.grad is None
    return table.weight.main_grad.clone()
fused = step()
assert len(calls) == 3 and table.weight.lookups_in_flight == 0
table.fuse_grad = False
dense = step()
assert len(calls) == 3
print("ERR", ((fused - dense).norm() / dense.norm()).item())
'''


def test_three_micro_batches():
    """The dense gradient of a micro-batch is rounded to bf16 before it is added (2^-9 relative, a value); the fused one is not."""
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert float(r.stdout.split("ERR")[1].split()[0]) < 2.0 ** -8
