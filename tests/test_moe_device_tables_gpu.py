"""MoE layer on one GPU: routing tables made on the device against the way through host counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(grouped, capacity=None, seed=0):
    from mindspeed_b200.config import TransformerConfig
    from mindspeed_b200.parallel.moe import MoELayer
    torch.manual_seed(seed)
    cfg = TransformerConfig(num_layers=1, hidden_size=256, num_attention_heads=2, num_moe_experts=8, moe_router_topk=2, moe_ffn_hidden_size=384,
                            ffn_hidden_size=384, moe_grouped_gemm=grouped, moe_token_dispatcher_type="alltoall", optimization_level=2,
                            gated_linear_unit=True, activation_func=torch.nn.functional.silu, add_bias_linear=False,
                            moe_expert_capacity_factor=capacity, params_dtype=torch.bfloat16, bf16=True)
    return MoELayer(cfg).cuda().train()


def _run(m, x, dout, on_map):
    handle = m.router.register_forward_hook(lambda mod, args, out: on_map(out[1]))
    try:
        m.zero_grad(set_to_none=True)
        leaf = x.clone().requires_grad_(True)
        out = m(leaf)[0]
        out.backward(dout)
        return [out.detach(), leaf.grad] + [p.grad for p in m.parameters() if p.grad is not None]
    finally:
        handle.remove()


def _drop(rmap):
    rmap[5] = False
    rmap[7, :3] = False


def _unmark(rmap):
    if hasattr(rmap, "rows_per_token"):
        del rmap.rows_per_token


@pytest.mark.parametrize("grouped", [True, False])
@pytest.mark.parametrize("edit", [None, _drop])
@pytest.mark.parametrize("frozen", [False, True])
def test_layer_with_and_without_the_note(grouped, edit, frozen):
    """The same rows in the same order reach the same kernels; gradients of the weights are fp32 sums whose order may differ."""
    from mindspeed_b200.ops import gemm as G
    m = _layer(grouped)
    m.router.weight.requires_grad_(not frozen)
    x = torch.randn(70, 2, 256, device="cuda", dtype=torch.bfloat16)
    dout = torch.randn_like(x)
    edit = edit or (lambda rmap: None)
    got = _run(m, x, dout, lambda rmap: edit(rmap))
    want = _run(m, x, dout, lambda rmap: (edit(rmap), _unmark(rmap))[0])
    torch.cuda.synchronize()
    G.check_status()
    assert len(got) == len(want) and torch.equal(got[0], want[0])
    for a, b in zip(got, want):
        assert ((a.float() - b.float()).norm() <= 1e-5 * b.float().norm()).item()


def test_capacity_limited_maps_carry_no_note():
    m = _layer(True, capacity=1.0)
    x = torch.randn(64, 1, 256, device="cuda", dtype=torch.bfloat16)
    seen = []
    _run(m, x, torch.randn_like(x), lambda rmap: seen.append(hasattr(rmap, "rows_per_token")))
    assert seen == [False]


@pytest.mark.parametrize("more", [True, False])
def test_wrong_row_count_is_an_error_and_stays_in_bounds(more):
    """Writes through ``.data`` are not counted as versions: rows and counts are cut at what was allocated, and the status word tells."""
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops.permute import route_tables
    rmap = torch.zeros(40, 8, dtype=torch.bool, device="cuda").scatter(1, torch.arange(80, device="cuda").view(40, 2) % 8, True)
    if more:
        rmap[::2] = True
    else:
        rmap[3:] = False
    G.check_status()
    idx, prob, counts = route_tables(torch.rand(40, 8, device="cuda"), rmap, 80)
    assert counts.sum().item() == min(80, int(rmap.sum())) and (counts >= 0).all() and ((idx >= 0) & (idx < 40)).all() and prob.numel() == 80
    with pytest.raises(RuntimeError, match="routing map"):
        G.check_status()
    G.check_status()
