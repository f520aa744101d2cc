"""Edges of the vectorised reduction, row-scale gradient and row scatter-add kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4099, 1 << 20, (1 << 24) + 5])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_l2norm_lengths_and_alignment(n, offset, dtype):
    """Sums of squares (all positive) in fp32 over fewer than 2^10 terms a thread: relative error below 2^10 * 2^-24."""
    from mindspeed_b200.ops import adam as A
    torch.manual_seed(n)
    g = torch.randn(n + offset, device="cuda").to(dtype)[offset:]
    ref = g.double().square().sum().item()
    assert abs(A.l2norm_sq(g).item() - ref) <= 6.2e-5 * ref


@pytest.mark.parametrize("rows,F", [(1, 8), (3, 264), (5000, 64), (37, 14336)])
def test_swiglu_row_scale_gradient(rows, F):
    """bf16 inputs, fp32 sums of F products: the oracle is the same expression in 64 bits; outputs round to bf16."""
    from mindspeed_b200.ops.activation import swiglu
    torch.manual_seed(F)
    x = torch.randn(rows, 2 * F, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    sc = torch.rand(rows, device="cuda", requires_grad=True)
    dy = torch.randn(rows, F, device="cuda", dtype=torch.bfloat16)
    swiglu(x, sc).backward(dy)
    xd, sd = x.detach().double().requires_grad_(True), sc.detach().double().requires_grad_(True)
    a, b = xd.chunk(2, -1)
    (torch.nn.functional.silu(a) * b * sd[:, None]).backward(dy.double())
    assert ((sc.grad - sd.grad).norm() / sd.grad.norm()).item() < 1e-5
    assert ((x.grad - xd.grad).norm() / xd.grad.norm()).item() < 4e-3


@pytest.mark.parametrize("n,rows,cols", [(1, 1, 8), (7, 3, 24), (300, 40, 1000), (6 * 128, 128, 4096), (500, 2, 2048), (64, 1, 133), (65, 1, 136)])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scatter_add_rows(n, rows, cols, weighted, dtype):
    """Repeated and missing targets, more than one list of 64, columns that no vector divides; fp32 sums, one rounding."""
    from mindspeed_b200.ops.permute import scatter_add_rows
    torch.manual_seed(n + cols)
    src = torch.randn(n, cols, device="cuda").to(dtype)
    idx = torch.randint(0, max(1, rows - 1), (n,), device="cuda")
    w = torch.rand(n, device="cuda") if weighted else None
    want = torch.zeros(rows, cols, device="cuda", dtype=torch.float64)
    want.index_add_(0, idx, src.double() * (1.0 if w is None else w.double()[:, None]))
    got = scatter_add_rows(src, idx, rows, w)
    assert got.dtype == dtype
    tol = 4e-3 if dtype == torch.bfloat16 else 3e-5
    assert ((got.double() - want).abs() <= tol * want.abs() + 3e-5 * want.abs().max()).all()


@pytest.mark.parametrize("n,rows,cols", [(1, 1, 8), (300, 7, 264), (5000, 4096, 1536), (64, 3, 133)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_add_rows_into_fp32_table(n, rows, cols, dtype):
    """fp32 sums of at most n terms in any order: n * 2^-24 of the sum of magnitudes."""
    from mindspeed_b200.ops.permute import add_rows_
    torch.manual_seed(n)
    src = torch.randn(n, cols, device="cuda").to(dtype)
    idx = torch.randint(0, rows, (n,), device="cuda")
    out = torch.randn(rows, cols, device="cuda")
    want = out.double().index_add(0, idx, src.double())
    size = out.double().abs().index_add(0, idx, src.double().abs())
    add_rows_(out, idx, src)
    assert ((out.double() - want).abs() <= (n + 1) * 2.0 ** -24 * size).all()


def test_add_rows_leaves_out_negative_rows():
    """Neither read (a NaN there would show) nor added."""
    from mindspeed_b200.ops.permute import add_rows_
    src = torch.full((40, 16), float("nan"), device="cuda")
    idx = torch.full((40,), -1, device="cuda")
    idx[5], idx[9] = 2, 0
    src[5], src[9] = 1.0, 2.0
    out = torch.zeros(3, 16, device="cuda")
    add_rows_(out, idx, src)
    assert out[:, 0].tolist() == [2.0, 0.0, 1.0] and not out.isnan().any()


@pytest.mark.parametrize("n,rows,cols", [(9, 1, 8), (17, 2, 24), (4096, 1, 4096), (5000, 3, 133), (24576, 64, 264), (3000, 1000, 2048)])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_scatter_add_rows_with_many_repeats(n, rows, cols, weighted, dtype):
    """More than eight source rows on an output row: eight in order, the others by atomics in any order.  fp32 sums of m terms in any order
    are within m * 2^-23 of the sum of magnitudes, one rounding to the result's type follows."""
    from mindspeed_b200.ops.permute import scatter_add_rows
    torch.manual_seed(n + cols)
    src = torch.randn(n, cols, device="cuda").to(dtype)
    idx = torch.where(torch.rand(n, device="cuda") < 0.3, 0, torch.randint(0, rows, (n,), device="cuda"))
    w = torch.rand(n, device="cuda") if weighted else None
    terms = src.double() * (1.0 if w is None else w.double()[:, None])
    zero = torch.zeros(rows, cols, device="cuda", dtype=torch.float64)
    want, size = zero.index_add(0, idx, terms), zero.index_add(0, idx, terms.abs())
    m = torch.bincount(idx, minlength=rows)[:, None]
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}[dtype]
    for _ in range(2):                                # the second call meets used scratch
        got = scatter_add_rows(src, idx, rows, w)
        assert got.dtype == dtype
        assert ((got.double() - want).abs() <= (m + 1) * 2.0 ** -23 * size + eps * want.abs() + 1e-7).all()


def test_scatter_add_onto_one_row_is_not_serial():
    """16384 rows on one output row and the same rows spread over 4096 (four each) move the same bytes.  The atomics of the former queue at
    one row's addresses (at most five times the time); one thread that walks a list of them took a hundred times as long."""
    from mindspeed_b200.ops.permute import scatter_add_rows
    src = torch.randn(16384, 4096, device="cuda", dtype=torch.bfloat16)

    def best(idx):
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            scatter_add_rows(src, idx, 4096)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[1:])
    spread = best(torch.arange(16384, device="cuda") % 4096)
    assert best(torch.zeros(16384, dtype=torch.long, device="cuda")) < 20 * spread
