"""Whole training steps under the options that open a saved-tensors context around the step."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r'''
import os, sys, json
os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT="29579", RANK="0", WORLD_SIZE="1")
import torch
import pretrain_gpt as pg
from mindspeed_b200.training import initialize_megatron, setup_model_and_optimizer, train_step
al = ["--num-layers","2","--hidden-size","256","--num-attention-heads","2","--group-query-attention","--num-query-groups","1",
 "--ffn-hidden-size","512","--seq-length","256","--max-position-embeddings","256","--micro-batch-size","2","--global-batch-size","4",
 "--vocab-size","2048","--make-vocab-size-divisible-by","1","--bf16","--lr","1e-3","--lr-decay-style","constant","--hidden-dropout","0",
 "--attention-dropout","0","--swiglu","--normalization","RMSNorm","--position-embedding-type","rope","--disable-bias-linear",
 "--untie-embeddings-and-output-weights","--use-flash-attn","--use-distributed-optimizer","--train-iters","5","--optimization-level","2"]
al += sys.argv[1:]
args = initialize_megatron(args_list=al)
model, opt, sched = setup_model_and_optimizer(pg.model_provider)
it = pg.train_valid_test_datasets_provider(args)
table = model[0].module.embedding.word_embeddings.weight
out = []
for _ in range(5):
    ld, _, norm, _ = train_step(pg.forward_step, it, model, opt, sched)
    out.append([float(ld["lm loss"]), float(norm)])
assert table.grad is None and table.lookups_in_flight == 0
print("STEPS", json.dumps(out))
'''


def _steps(*flags):
    r = subprocess.run([sys.executable, "-c", CODE, *flags], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return json.loads([l for l in r.stdout.splitlines() if l.startswith("STEPS")][0][len("STEPS "):])


@pytest.fixture(scope="module")
def plain():
    return _steps()


@pytest.mark.parametrize("flags", [["--smart-swap"], ["--adaptive-recompute-device-swap"], ["--adaptive-recompute-device-size", "1"]])
def test_losses_are_those_of_a_plain_step(plain, flags):
    """The same data, seed and arithmetic; what differs are the orders of fp32 sums (dQ, weight gradients), carried through bf16 and
    five steps of Adam: 1 % of the loss, 5 % of the gradient norm."""
    for (a, na), (b, nb) in zip(plain, _steps(*flags)):
        assert abs(a - b) < 0.01 * a and abs(na - nb) < 0.05 * na
