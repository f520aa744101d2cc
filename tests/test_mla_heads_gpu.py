"""Head kernels of multi-head latent attention against their PyTorch form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,b,n,nope,rope,vd", [(1, 1, 1, 8, 16, 8), (5, 2, 3, 128, 64, 128), (33, 1, 16, 64, 32, 96), (7, 3, 32, 128, 64, 128)])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("strided", [False, True])
def test_heads_and_gradients(s, b, n, nope, rope, vd, interleaved, dtype, strided):
    """k_pe as a slice of a wider projection; gradients as the attention returns them (head-major memory).  The oracle runs in 64
    bits: one rounding of each output."""
    from mindspeed_b200.ops.mla_heads import _MlaHeads, mla_heads_ref
    torch.manual_seed(s * n)
    q = torch.randn(s, b, n, nope + rope, device="cuda", dtype=dtype, requires_grad=True)
    kv = torch.randn(s, b, n, nope + vd, device="cuda", dtype=dtype, requires_grad=True)
    low = torch.randn(s, b, 48 + rope, device="cuda", dtype=dtype, requires_grad=True)
    ang = torch.rand(s, rope, device="cuda") * 6
    cos, sin = ang.cos(), ang.sin()
    out = _MlaHeads.apply(q, kv, low[..., 48:], cos, sin, nope, interleaved)
    ref_in = [t.detach().double().requires_grad_(True) for t in (q, kv, low)]

    def rotate(x):
        c, sn = (a.double().view(s, 1, 1, rope) for a in (cos, sin))
        if interleaved:
            half = torch.stack((-x[..., 1::2], x[..., 0::2]), -1).reshape(x.shape)
        else:
            half = torch.cat((-x[..., rope // 2:], x[..., :rope // 2]), -1)
        return x * c + half * sn
    rq, rkv, rlow = ref_in
    ref = (torch.cat((rq[..., :nope], rotate(rq[..., nope:])), -1),
           torch.cat((rkv[..., :nope], rotate(rlow[..., 48:].view(s, b, 1, rope)).expand(s, b, n, rope)), -1), rkv[..., nope:])
    tol = 4e-3 if dtype == torch.bfloat16 else 1e-6
    near = lambda a, r: ((a.double() - r).norm() <= tol * r.norm() + 1e-12).item()
    for a, r in zip(out, ref):
        assert near(a, r)
    grads = []
    for a in out:
        g = torch.randn(b, n, s, a.shape[-1], device="cuda", dtype=dtype).permute(2, 0, 1, 3) if strided else torch.randn_like(a)
        grads.append(g)
    torch.autograd.backward(out, grads)
    torch.autograd.backward(ref, [g.double() for g in grads])
    for t, r in zip((q, kv, low), ref_in):
        assert near(t.grad, r.grad)
    if dtype == torch.float32:
        for a, r in zip(out, mla_heads_ref(q, kv, low[..., 48:], cos, sin, nope, interleaved)):
            torch.testing.assert_close(a, r, rtol=1e-5, atol=1e-5)
