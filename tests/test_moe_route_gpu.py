"""Routing tables on the device against masked selections, and their gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (3, 5, 2), (1024, 8, 2), (1025, 64, 6), (5000, 33, 8), (31, 300, 4)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("skew", [False, True])
def test_tables(T, E, k, dtype, skew):
    from mindspeed_b200.ops.permute import route_tables
    torch.manual_seed(T + E)
    scores = torch.rand(T, E, device="cuda")
    if skew:                                   # some experts take every token, others none
        scores += torch.arange(E, device="cuda") * 10.0
    idx = scores.topk(k, 1)[1]
    rmap = torch.zeros(T, E, dtype=torch.bool, device="cuda").scatter(1, idx, True)
    probs = (torch.rand(T, E, device="cuda") * rmap).to(dtype).requires_grad_(True)
    tok, p, counts = route_tables(probs, rmap, T * k)
    rt = rmap.t()
    assert torch.equal(counts, rt.sum(1))
    assert torch.equal(tok, torch.arange(T, device="cuda").expand(E, -1).masked_select(rt))
    ref = probs.detach().clone().requires_grad_(True)
    want = ref.t().contiguous().masked_select(rt.contiguous())
    assert torch.equal(p, want)
    g = torch.randn_like(p)
    p.backward(g)
    want.backward(g)
    assert torch.equal(probs.grad, ref.grad)
