"""Weight gradient of the grouped GEMM where experts end inside a 64-row block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[0, 1, 63, 64, 65, 0], [64, 128, 192], [5], [1, 1, 1, 1], [300, 0, 257, 31]])
@pytest.mark.parametrize("K,N", [(256, 512), (264, 136)])
def test_wgrad_adds_every_row_once(counts, K, N):
    """fp32 accumulation of bf16 products: 1e-5 of the largest value covers the order of at most 300 terms."""
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops.grouped_gemm import _offsets, grouped_wgrad_acc
    torch.manual_seed(len(counts) + K)
    rows = sum(counts)
    x = torch.randn(rows + 40, K, device="cuda").bfloat16()          # rows behind the last expert belong to nobody
    dy = torch.randn(rows + 40, N, device="cuda").bfloat16()
    x[rows:] = float("nan")
    dy[rows:] = float("inf")
    acc = torch.randn(len(counts), K, N, device="cuda")
    want, s = acc.clone(), 0
    for e, n in enumerate(counts):
        want[e] += (x[s:s + n].double().t() @ dy[s:s + n].double()).float()
        s += n
    grouped_wgrad_acc(x, dy, _offsets(counts, x.device), acc)
    torch.cuda.synchronize()
    G.check_status()
    assert ((acc - want).abs().max() / want.abs().max()).item() < 1e-5
