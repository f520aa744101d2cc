"""Fused embedding gradient where saved tensors pass through hooks (host swap, checkpointing).  The lookup's device test is let through
and the kernel stands in as ``index_add_``: what is tested is the autograd function."""
import contextlib

import pytest
import torch
from torch.utils.checkpoint import checkpoint


@pytest.fixture
def table(monkeypatch):
    from mindspeed_b200.ops import permute
    from mindspeed_b200.parallel import layers

    class Config:
        deterministic_mode = perform_initialization = False
        use_cpu_initialization = gradient_accumulation_fusion = True
        optimization_level, params_dtype = 1, torch.float32
    monkeypatch.setattr(layers.VocabParallelEmbedding, "_fused", lambda self, ids: torch.is_grad_enabled())
    monkeypatch.setattr(permute, "add_rows_", lambda out, idx, src: out.index_add_(0, idx, src.float()))
    m = layers.VocabParallelEmbedding(20, 6, init_method=None, config=Config())
    torch.nn.init.normal_(m.weight)
    m.weight.main_grad = torch.zeros(20, 6)
    m.told = []
    m.weight._main_grad_ready_cb = m.told.append
    return m


def _identity():
    return torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t)


@pytest.mark.parametrize("how", ["plain", "identity", "save_on_cpu", "checkpoint", "reentrant", "identity + checkpoint"])
def test_gradient_reaches_the_accumulator(table, how):
    torch.manual_seed(0)
    ids = torch.randint(0, 20, (4, 9))
    scale = torch.ones((), requires_grad=True)               # reentrant checkpointing differentiates inputs only
    with contextlib.ExitStack() as stack:
        if "identity" in how:
            stack.enter_context(_identity())
        if how == "save_on_cpu":
            stack.enter_context(torch.autograd.graph.save_on_cpu())
        run = lambda x, s: table(x) * s
        out = checkpoint(run, ids, scale, use_reentrant=how == "reentrant") if "checkpoint" in how or how == "reentrant" else run(ids, scale)
        g = torch.randn_like(out)
        out.backward(g)
    want = torch.zeros(20, 6).index_add_(0, ids.flatten(), g.flatten(0, 1))
    torch.testing.assert_close(table.weight.main_grad, want)
    assert table.weight.grad is None and len(table.told) == 1 and table.weight.lookups_in_flight == 0


def test_weight_may_change_between_the_passes(table):
    """The gradient of a lookup does not depend on the weight's values, so neither does the check of their version."""
    out = table(torch.tensor([1, 1, 3]))
    with torch.no_grad():
        table.weight.mul_(2.0)
    out.sum().backward()
    assert table.weight.main_grad[:, 0].tolist()[:4] == [0, 2, 0, 1]


def test_a_graph_that_is_dropped_closes_its_lookups(table):
    kept = table(torch.tensor([2, 3]))
    table(torch.tensor([4]))                                   # never differentiated
    kept.sum().backward()
    assert len(table.told) == 1 and table.weight.lookups_in_flight == 0


def test_ids_of_other_ranks_add_nothing(table, monkeypatch):
    """A vocabulary split: rows 20 .. 39 of 60 are here. Every other id is left out of the sum instead of adding zeros to row 0."""
    from mindspeed_b200.ops import permute
    from mindspeed_b200.parallel import mappings as M
    table.world, table.vocab_start_index, table.vocab_end_index = 3, 20, 40
    monkeypatch.setattr(M, "reduce_from_tensor_model_parallel_region", lambda x, group=None: x)
    seen = []
    monkeypatch.setattr(permute, "add_rows_", lambda out, idx, src: (seen.append(idx), out.index_add_(0, idx[idx >= 0], src[idx >= 0]))[1])
    ids = torch.tensor([[0, 19, 20, 39], [40, 59, 25, 25]])
    out = table(ids)
    here = torch.tensor([[0, 0, 1, 1], [0, 0, 1, 1]], dtype=torch.bool)
    assert torch.equal(out[here], table.weight.detach()[ids[here] - 20]) and not out[~here].any()
    out.backward(torch.ones_like(out))
    assert seen[0].tolist() == [-1, -1, 0, 19, -1, -1, 5, 5]
    assert table.weight.main_grad[:, 0].tolist() == [1.0 if r in (0, 19) else 2.0 if r == 5 else 0.0 for r in range(20)]
