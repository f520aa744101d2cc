"""fp8 quantiser (csrc/kernels/quant_fp8.cu) bit for bit against ops/quant.py, and the CTA-pair block-scaled GEMM."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert a.shape == b.shape
    assert torch.equal(a.flatten().view(torch.uint8), b.flatten().view(torch.uint8))


@pytest.mark.parametrize("M,K", [(1, 128), (127, 256), (128, 128), (129, 384), (1000, 1024), (4096, 512)])
@pytest.mark.parametrize("src", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.float8_e5m2])
def test_activation_forms_are_those_of_the_reference(M, K, src, dtype):
    from mindspeed_b200.ops import gemm_fp8 as F
    from mindspeed_b200.ops.quant import quant_1x128
    torch.manual_seed(M + K)
    x = (torch.randn(M, K, device="cuda") * torch.logspace(-6, 3, M, device="cuda")[:, None]).to(src)
    x[:, :64] = 0
    x[M // 2, :] = 0                                     # a block of zeros: the smallest scale
    q, s, qt, st = F.quant_activation(x, dtype, rows=True, cols=True)
    rq, rs = quant_1x128(x, dtype=dtype)
    xt = torch.nn.functional.pad(x, (0, 0, 0, (-M) % 128)).t().contiguous()
    rqt, rst = quant_1x128(xt, dtype=dtype)
    for a, b in ((q, rq), (s, rs), (qt, rqt), (st, rst)):
        _same(a, b)
    only = F.quant_activation(x, dtype, rows=False, cols=True)
    assert only[0] is None
    _same(only[2], rqt)
    _same(F.quant_activation(x, dtype)[0], rq)


@pytest.mark.parametrize("N,K", [(128, 128), (256, 384), (1536, 512)])
def test_weight_form_and_special_values(N, K):
    from mindspeed_b200.ops import gemm_fp8 as F
    from mindspeed_b200.ops.quant import quant_128x128, quant_1x128
    torch.manual_seed(N)
    w = (torch.randn(N, K, device="cuda") * 0.02).bfloat16()
    q, s, qt, st = F.quant_weight(w)
    rq, rs = quant_128x128(w)
    rqt, rst = quant_128x128(w.t().contiguous())
    for a, b in ((q, rq), (s, rs), (qt, rqt), (st, rst)):
        _same(a, b)
    w[3, 5], w[100, 7] = float("inf"), float("nan")       # scales of their blocks become inf / NaN, as in the reference
    _, s, _, _ = F.quant_weight(w)
    assert torch.equal(torch.nan_to_num(s, nan=-1.0), torch.nan_to_num(quant_128x128(w)[1], nan=-1.0))
    _, s, _, st = F.quant_activation(w, rows=True, cols=True)
    assert torch.equal(torch.nan_to_num(s, nan=-1.0), torch.nan_to_num(quant_1x128(w)[1], nan=-1.0))
    assert torch.equal(torch.nan_to_num(st, nan=-1.0), torch.nan_to_num(quant_1x128(w.t().contiguous())[1], nan=-1.0))


@pytest.mark.parametrize("M,N,K", [(2048, 2304, 128), (2500, 1920, 640), (1537, 2944, 256), (256, 9600, 384), (1, 128, 128), (300, 384, 1152)])
@pytest.mark.parametrize("rowwise", [False, True])
@pytest.mark.parametrize("out", ["bf16", "f32", "acc"])
def test_pair_kernel_matches_reference(M, N, K, rowwise, out):
    """Tiles cut by M and by N (N = 128 mod 256), one k-block, more k-blocks than pipeline stages.  Same operands and the same
    order of k-blocks as the reference: 1e-3 of the largest value for the tensor core's sums inside a k-block (the bound of the
    single-CTA kernel's test), bf16 adds its rounding (2^-8)."""
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops import gemm_fp8 as F
    from mindspeed_b200.ops.quant import quant_128x128, quant_1x128
    torch.manual_seed(M + N)
    xq, xs = quant_1x128(torch.randn(M, K, device="cuda") * torch.rand(M, 1, device="cuda"), dtype=torch.float8_e5m2)
    w = torch.randn(N, K, device="cuda") * torch.rand(N, 1, device="cuda")
    wq, ws = quant_1x128(w) if rowwise else quant_128x128(w)
    ref = F._ref(xq, xs, wq, ws, rowwise, torch.float32)
    if out == "acc":
        acc = torch.randn(M, N, device="cuda")
        ref = ref + acc
        y = F.fp8_gemm(xq, xs, wq, ws, w_rowwise=rowwise, out=acc, accumulate=True)
    else:
        y = F.fp8_gemm(xq, xs, wq, ws, w_rowwise=rowwise, out_dtype=torch.bfloat16 if out == "bf16" else torch.float32)
    torch.cuda.synchronize()
    G.check_status()
    tol = 4e-3 if out == "bf16" else 1e-3
    assert ((y.float() - ref).abs().max() / ref.abs().max()).item() < tol


@pytest.mark.parametrize("M,N,K", [(300, 201, 640), (1, 130, 128), (129, 1, 1152), (2304, 2049, 256)])
@pytest.mark.parametrize("out", ["bf16", "f32", "acc"])
def test_rows_that_tma_cannot_store_take_the_single_cta_kernel(M, N, K, out):
    """Row-wise scales and N % 4 != 0: neither the output's rows nor the scales start on 16-byte boundaries.  Bounds as above."""
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops import gemm_fp8 as F
    from mindspeed_b200.ops.quant import quant_1x128
    torch.manual_seed(M + N)
    xq, xs = quant_1x128(torch.randn(M, K, device="cuda") * torch.rand(M, 1, device="cuda"), dtype=torch.float8_e5m2)
    wq, ws = quant_1x128(torch.randn(N, K, device="cuda") * torch.rand(N, 1, device="cuda"))
    ref = F._ref(xq, xs, wq, ws, True, torch.float32)
    guard = torch.full((M * N + 64,), 7.0, device="cuda", dtype=torch.bfloat16 if out == "bf16" else torch.float32)
    y = guard[:M * N].view(M, N)
    if out == "acc":
        y.copy_(torch.randn(M, N, device="cuda"))
        ref = ref + y
    F.fp8_gemm(xq, xs, wq, ws, w_rowwise=True, out=y, accumulate=out == "acc")
    torch.cuda.synchronize()
    G.check_status()
    tol = 4e-3 if out == "bf16" else 1e-3
    assert ((y.float() - ref).abs().max() / ref.abs().max()).item() < tol
    assert (guard[M * N:] == 7.0).all()


@pytest.mark.parametrize("rowwise", [False, True])
def test_output_columns_of_a_wider_matrix(rowwise):
    """Rows of an fp32 output that start 4 bytes past a 16-byte boundary, in a matrix large enough for the pair kernel."""
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops import gemm_fp8 as F
    from mindspeed_b200.ops.quant import quant_128x128, quant_1x128
    torch.manual_seed(5)
    xq, xs = quant_1x128(torch.randn(2048, 256, device="cuda"))
    w = torch.randn(2304, 256, device="cuda")
    wq, ws = quant_1x128(w) if rowwise else quant_128x128(w)
    wide = torch.full((2048, 2304 + 5), 7.0, device="cuda")
    F.fp8_gemm(xq, xs, wq, ws, w_rowwise=rowwise, out=wide[:, 1:2305])
    torch.cuda.synchronize()
    G.check_status()
    ref = F._ref(xq, xs, wq, ws, rowwise, torch.float32)
    assert ((wide[:, 1:2305] - ref).abs().max() / ref.abs().max()).item() < 1e-3
    assert (wide[:, 0] == 7.0).all() and (wide[:, 2305:] == 7.0).all()


@pytest.mark.parametrize("src", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.float8_e5m2])
def test_subnormal_values_are_not_flushed(src, dtype):
    """Blocks whose largest value lies between 1e-42 and 1e-26: their subnormal values reach fp8 under the smallest scales (1e-30 / fmax
    and a little above), bit for bit as in PyTorch, which keeps subnormals."""
    from mindspeed_b200.ops import gemm_fp8 as F
    from mindspeed_b200.ops.quant import quant_128x128, quant_1x128
    torch.manual_seed(0)
    size = torch.logspace(-42, -26, 256, device="cuda", dtype=torch.float64)
    x = (torch.randn(256, 256, device="cuda", dtype=torch.float64) * size[:, None])
    x[::2, ::3] = torch.randn(128, 86, device="cuda", dtype=torch.float64) * 5e-39
    x = x.to(src)
    tiny = (x != 0) & (x.abs().double() < 2.0 ** -126)
    q, s, qt, st = F.quant_activation(x, dtype, rows=True, cols=True)
    rq, rs = quant_1x128(x, dtype=dtype)
    rqt, rst = quant_1x128(x.t().contiguous(), dtype=dtype)
    for a, b in ((q, rq), (s, rs), (qt, rqt), (st, rst)):
        _same(a, b)
    if dtype == torch.float8_e5m2:
        assert (q.float()[tiny] != 0).any()
    else:
        for a, b in zip(F.quant_weight(x), quant_128x128(x) + quant_128x128(x.t().contiguous())):
            _same(a, b)
