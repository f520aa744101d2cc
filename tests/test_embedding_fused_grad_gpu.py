"""Embedding gradient added straight into main_grad: values, repeated lookups, and when the dense way is kept."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Config:
    deterministic_mode = use_cpu_initialization = perform_initialization = False
    gradient_accumulation_fusion, optimization_level, params_dtype = True, 1, torch.bfloat16


def _table(rows, cols):
    from mindspeed_b200.parallel.layers import VocabParallelEmbedding
    m = VocabParallelEmbedding(rows, cols, init_method=None, config=_Config())
    torch.nn.init.normal_(m.weight)
    m.weight.main_grad = torch.zeros(rows, cols, device="cuda")
    m.told = []
    m.weight._main_grad_ready_cb = m.told.append
    return m


def test_gradient_rows_are_added_once_and_the_wrapper_is_told_last():
    torch.manual_seed(0)
    m = _table(50, 72)
    ids = torch.randint(0, 50, (3, 40), device="cuda")
    a, b = m(ids), m(ids[:1])
    ga, gb = torch.randn_like(a), torch.randn_like(b)
    a.backward(ga)
    assert not m.told                               # the second lookup is outstanding
    b.backward(gb)
    assert len(m.told) == 1 and m.weight.grad is None and m.weight.grad_added_to_main_grad
    want = torch.zeros(50, 72, device="cuda").index_add(0, ids.flatten(), ga.float().flatten(0, 1)).index_add(0, ids[0], gb.float()[0])
    torch.testing.assert_close(m.weight.main_grad, want, rtol=1e-5, atol=1e-5)


def test_shared_tables_and_missing_accumulators_keep_the_dense_gradient():
    m = _table(10, 16)
    m.weight.shared_embedding = True
    m(torch.tensor([[1, 1, 3]], device="cuda")).sum().backward()
    assert m.weight.grad[1, 0].item() == 2 and not m.told
    m = _table(10, 16)
    del m.weight.main_grad
    m(torch.tensor([[1, 1, 3]], device="cuda")).sum().backward()
    assert m.weight.grad[3, 0].item() == 1


def test_hooked_weights_keep_the_dense_gradient():
    ids = torch.tensor([[1, 1, 3]], device="cuda")
    for register in ("register_hook", "register_post_accumulate_grad_hook"):
        m, seen = _table(10, 16), []
        handle = getattr(m.weight, register)(lambda t: seen.append(tuple(t.shape)))
        m(ids).sum().backward()
        assert seen == [(10, 16)] and m.weight.grad[1, 0].item() == 2 and not m.told
        handle.remove()
        m.weight.grad = None
        m(ids).sum().backward()
        assert len(seen) == 1 and m.weight.grad is None and m.weight.main_grad[1, 0].item() == 2


def test_the_wrappers_own_hook_does_not_count():
    def hook(p):
        assert p.grad is None                         # the node runs, but autograd has no gradient for this weight
    hook.fills_main_grad = True
    m = _table(10, 16)
    m.weight.register_post_accumulate_grad_hook(hook)
    m(torch.tensor([[1, 1, 3]], device="cuda")).sum().backward()
    assert m.weight.grad is None and m.weight.main_grad[3, 0].item() == 1 and len(m.told) == 1
