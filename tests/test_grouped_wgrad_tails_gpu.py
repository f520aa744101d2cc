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


@pytest.mark.parametrize("epilogue", [0, 1])
def test_wgrad_stores(epilogue):
    """The storing forms (bf16, fp32): every expert with rows is written, the others keep what they hold."""
    import ctypes

    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops import loader
    from mindspeed_b200.ops.grouped_gemm import TAIL, _offsets
    torch.manual_seed(epilogue)
    counts, K, N = [70, 0, 1, 64], 264, 136
    rows = sum(counts)
    x, dy = (torch.randn(rows, c, device="cuda").bfloat16() for c in (K, N))
    offs = _offsets(counts, x.device)
    dw = torch.full((len(counts), K, N), 7.0, device="cuda", dtype=(torch.bfloat16, torch.float32)[epilogue])
    xt, dyt = (torch.empty(len(counts) * TAIL, c, device="cuda", dtype=torch.bfloat16) for c in (K, N))
    loader.check(loader.require_lib().msb_grouped_gemm_wgrad(
        loader.p(x), loader.p(dy), loader.p(dw), loader.p(offs), loader.p(xt), loader.p(dyt), len(counts), rows, K, N, epilogue,
        loader.p(G.status_word(x.device)), ctypes.c_void_p(loader.stream_ptr())), "grouped_gemm_wgrad")
    torch.cuda.synchronize()
    G.check_status()
    s = 0
    for e, n in enumerate(counts):
        want = (x[s:s + n].double().t() @ dy[s:s + n].double()) if n else torch.full((K, N), 7.0, device="cuda", dtype=torch.float64)
        s += n
        assert ((dw[e].double() - want).abs().max() / want.abs().max()).item() < (2.0 ** -8 if epilogue == 0 else 1e-5)
