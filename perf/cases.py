"""Performance cases of the single-GPU training path.

Each case is one pass of something a training script calls: a whole optimizer step (``training.train_step``), a forward pass
that returns logits, or one forward + backward of a building block that such a step is made of (attention, a linear layer in
bf16 or block-scaled fp8, a mixture-of-experts layer, a multi-head-latent-attention block).  The widths are those of
``mindspeed_b200/models/presets.py``, of the smoke test and of ``mindspeed_b200/benchmarks``; depth, experts and batch are cut
so that a state is a few GB.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) model / weights / inputs on the GPU, made from the seed
  run(state)          one pass; returns what the pass computes
  work(case)          bytes and operations the pass cannot do without
  tolerance(case)     how far another correct implementation of the same precision may be off
  exact(case, seed)   what run returns, in 64 bits and plain torch
"""
import os
import socket

import torch

D = 128          # head size of every dense-attention preset
QK_NOPE, QK_ROPE, V_DIM, Q_LORA, KV_LORA = 128, 64, 128, 1536, 512      # latent attention of the DeepSeek preset


def listed():
    return [
        # a debug-sized model (the smoke test's): what a step costs when every kernel is small and launches dominate
        dict(name="train-tiny", kind="train", layers=2, hidden=512, heads=4, kv=2, ffn=1536, seq=512, mbs=1, gbs=2, vocab=4096),
        # a small model on a length that is no power of two, batched, MHA, GPT-2's vocabulary padded to 128
        dict(name="train-ragged", kind="train", layers=4, hidden=1536, heads=12, kv=12, ffn=4096, seq=1000, mbs=3, gbs=3, vocab=50304),
        # two layers of the Llama-3-8B shape at its training length: the headline configuration's layer, two micro-batches
        dict(name="train-llama", kind="train", layers=2, hidden=4096, heads=32, kv=8, ffn=14336, seq=8192, mbs=1, gbs=2, vocab=32000),
        # scoring a batch: forward only, logits out
        dict(name="logits", kind="logits", layers=2, hidden=4096, heads=32, kv=8, ffn=14336, seq=2048, mbs=2, vocab=32000),
        # attention of the Llama-3-8B layer, forward and backward
        dict(name="attn-8k", kind="attention", sq=8192, sk=8192, b=1, heads=32, kv=8, causal=True),
        # the shortest sequences trained on (also one tensor-parallel rank's heads): few tiles, latency counts
        dict(name="attn-short", kind="attention", sq=512, sk=512, b=2, heads=4, kv=1, causal=True),
        # full (encoder-style) attention over a length that ends inside a tile
        dict(name="attn-ragged", kind="attention", sq=1500, sk=1500, b=4, heads=12, kv=12, causal=False),
        # one tensor-parallel (8) rank's share of the QKV projection: forward, both gradients, weight gradient added in fp32
        dict(name="linear-qkv-tp8", kind="linear", tokens=8192, inp=4096, out=768),
        # FC1 of the Llama-3-8B layer (gate and up projection) under the block-scaled fp8 recipe, half a sequence
        dict(name="fp8-fc1", kind="fp8", tokens=4096, inp=4096, out=28672),
        # the Mixtral layer: few wide experts, top 2, softmax router with balancing loss
        dict(name="moe-mixtral", kind="moe", seq=4096, b=1, hidden=4096, experts=8, topk=2, ffn=14336, shared=0, score="softmax"),
        # the DeepSeek-V3-style layer: many narrow experts, top 6, sigmoid router, shared expert
        dict(name="moe-deepseek", kind="moe", seq=4096, b=1, hidden=4096, experts=64, topk=6, ffn=1536, shared=1536, score="sigmoid"),
        # its attention block: low-rank queries and keys, 192-wide query / key heads, 128-wide value heads
        dict(name="mla-deepseek", kind="mla", seq=4096, b=1, hidden=4096, heads=32),
    ]


def _log_size(rng, lo, hi, step=1):
    v = lo * (hi / lo) ** rng.random()
    return max(lo, int(v) // step * step)


def draw(rng):
    """One more case: sizes log-uniform over the ranges of the listed cases, ragged lengths among them, never more
    arithmetic than the largest listed case."""
    limit = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["train", "train", "logits", "attention", "attention", "attention", "linear", "fp8", "moe", "mla"])
        step = rng.choice([1, 8, 64])
        if kind in ("train", "logits"):
            heads = rng.choice([4, 8, 12, 16, 24, 32])
            hidden = heads * D
            c = dict(kind=kind, layers=rng.randint(1, 4), hidden=hidden, heads=heads, kv=rng.choice([h for h in (1, 2, 4, 8, heads) if heads % h == 0]),
                     ffn=_log_size(rng, 2 * hidden, 4 * hidden, 64), seq=_log_size(rng, 256, 8192, step), mbs=rng.randint(1, 3),
                     vocab=_log_size(rng, 2048, 65536, 128))
            if kind == "train":
                c["gbs"] = c["mbs"] * rng.randint(1, 2)
            most = c["mbs"] * c["seq"] * c["vocab"] <= 8192 * 65536       # the logits of one micro-batch
        elif kind == "attention":
            kv, causal = rng.choice([1, 2, 4, 8, 16]), rng.random() < 0.75
            sq = _log_size(rng, 256, 16384, step)
            sk = sq if rng.random() < 0.8 else sq + _log_size(rng, 64, sq, step)      # later queries of a longer context
            c = dict(kind=kind, sq=sq, sk=sk, b=rng.randint(1, 4), heads=kv * rng.choice([1, 2, 4]), kv=kv, causal=causal)
            most = work(c)["flops"] <= 8e12
        elif kind == "linear":
            c = dict(kind=kind, tokens=_log_size(rng, 256, 16384, step), inp=_log_size(rng, 512, 14336, 64), out=_log_size(rng, 512, 28672, 64))
            most = True
        elif kind == "fp8":
            c = dict(kind=kind, tokens=_log_size(rng, 256, 8192, step), inp=_log_size(rng, 512, 14336, 128), out=_log_size(rng, 512, 28672, 128))
            most = c["tokens"] * (c["inp"] + c["out"]) <= 8192 * 32768
        elif kind == "moe":
            many = rng.random() < 0.5
            c = dict(kind=kind, seq=_log_size(rng, 256, 8192, step), b=rng.randint(1, 2), hidden=rng.choice([1024, 2048, 4096]),
                     experts=rng.choice([32, 64] if many else [4, 8]), topk=rng.randint(4, 8) if many else rng.randint(1, 2),
                     ffn=_log_size(rng, 512, 1536, 64) if many else _log_size(rng, 2048, 14336, 64),
                     shared=rng.choice([0, 1024]) if many else 0, score="sigmoid" if many else "softmax")
            most = c["seq"] * c["b"] * c["topk"] * (c["hidden"] + 3 * c["ffn"]) <= 4096 * 2 * 49152
        else:
            c = dict(kind=kind, seq=_log_size(rng, 256, 4096, step), b=rng.randint(1, 2), hidden=rng.choice([2048, 4096]), heads=rng.choice([16, 32]))
            most = True
        if most and work(c)["flops"] <= limit:
            return c


# ---- flags of the models -----------------------------------------------------------------------------------------------
def _flags(c, seed):
    hidden, seq = c.get("hidden", 512), c.get("seq", 512)
    a = ["--num-layers", str(c.get("layers", 1)), "--hidden-size", str(hidden), "--num-attention-heads", str(c.get("heads", max(1, hidden // D))),
         "--ffn-hidden-size", str(c.get("ffn", 4 * hidden)), "--seq-length", str(seq), "--max-position-embeddings", str(seq),
         "--micro-batch-size", str(c.get("mbs", 1)), "--global-batch-size", str(c.get("gbs", c.get("mbs", 1))), "--vocab-size", str(c.get("vocab", 4096)),
         "--make-vocab-size-divisible-by", "1", "--init-method-std", "0.02", "--hidden-dropout", "0", "--attention-dropout", "0", "--bf16",
         "--lr", "1e-4", "--lr-decay-style", "constant", "--weight-decay", "0.1", "--clip-grad", "1.0", "--adam-beta2", "0.95",
         "--untie-embeddings-and-output-weights", "--disable-bias-linear", "--normalization", "RMSNorm", "--norm-epsilon", "1e-5", "--swiglu",
         "--position-embedding-type", "rope", "--use-flash-attn", "--use-distributed-optimizer", "--train-iters", "1000000",
         "--optimization-level", "2", "--seed", str(seed)]
    if c.get("kv", c.get("heads")) != c.get("heads"):
        a += ["--group-query-attention", "--num-query-groups", str(c["kv"])]
    if c["kind"] == "moe":
        a += ["--num-experts", str(c["experts"]), "--moe-router-topk", str(c["topk"]), "--moe-ffn-hidden-size", str(c["ffn"]), "--moe-grouped-gemm",
              "--moe-token-dispatcher-type", "alltoall", "--moe-router-score-function", c["score"]]
        if c["score"] == "sigmoid":
            a += ["--moe-router-enable-expert-bias", "--moe-router-load-balancing-type", "seq_aux_loss", "--moe-aux-loss-coeff", "0.0001"]
        else:
            a += ["--moe-router-load-balancing-type", "aux_loss", "--moe-aux-loss-coeff", "0.01"]
        if c["shared"]:
            a += ["--moe-shared-expert-intermediate-size", str(c["shared"])]
    if c["kind"] == "mla":
        a += ["--multi-latent-attention", "--q-lora-rank", str(Q_LORA), "--kv-lora-rank", str(KV_LORA), "--qk-nope-head-dim", str(QK_NOPE),
              "--qk-rope-head-dim", str(QK_ROPE), "--v-head-dim", str(V_DIM)]
    if c["kind"] == "fp8":
        a += ["--fp8-format", "e4m3", "--fp8-recipe", "blockwise"]
    return a


def _initialize(c, seed):
    """What a script does first: parse the flags, set up the (one-rank) process group and the model-parallel state."""
    if not torch.distributed.is_initialized():
        with socket.socket() as s:
            s.bind(("127.0.0.1", 0))
            port = s.getsockname()[1]
        os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port), RANK="0", WORLD_SIZE="1", LOCAL_RANK="0")
    from mindspeed_b200.training import initialize_megatron
    return initialize_megatron(args_list=_flags(c, seed))


def _grad_buffers(module):
    """fp32 gradient accumulators, as the data-parallel wrapper attaches them."""
    for p in module.parameters():
        p.main_grad = torch.zeros(p.shape, dtype=torch.float32, device=p.device)


# ---- one state / one pass per kind --------------------------------------------------------------------------------------
def prepare(case, seed):
    c = dict(case)
    args = _initialize(c, seed)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, std=1.0):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.bfloat16).mul_(std)

    st = {"case": c, "args": args}
    if c["kind"] in ("train", "logits"):
        import pretrain_gpt
        tokens = torch.randint(0, c["vocab"], (c.get("gbs", c["mbs"]), c["seq"] + 1), generator=torch.Generator().manual_seed(seed))
        if c["kind"] == "logits":
            from mindspeed_b200.training import get_model
            st["model"] = get_model(pretrain_gpt.model_provider, wrap_with_ddp=False)[0].eval()
            st["tokens"] = tokens[:, :-1].contiguous().cuda()
            st["positions"] = torch.arange(c["seq"], device="cuda").unsqueeze(0).expand(c["mbs"], -1).contiguous()
        else:
            from mindspeed_b200.training import setup_model_and_optimizer
            st["model"], st["optimizer"], st["scheduler"] = setup_model_and_optimizer(pretrain_gpt.model_provider)
            st["forward_step"] = pretrain_gpt.forward_step
            pos = torch.arange(c["seq"]).unsqueeze(0).expand(c["mbs"], -1)
            st["batches"] = [{k: v.contiguous().pin_memory() for k, v in dict(
                tokens=tokens[i:i + c["mbs"], :-1], labels=tokens[i:i + c["mbs"], 1:], loss_mask=torch.ones(c["mbs"], c["seq"]),
                position_ids=pos).items()} for i in range(0, c["gbs"], c["mbs"])]
    elif c["kind"] == "attention":
        st["q"] = randn(c["sq"], c["b"], c["heads"], D).requires_grad_(True)
        st["k"] = randn(c["sk"], c["b"], c["kv"], D).requires_grad_(True)
        st["v"] = randn(c["sk"], c["b"], c["kv"], D).requires_grad_(True)
        st["dout"] = randn(c["sq"], c["b"], c["heads"], D)
    else:
        from mindspeed_b200.training import core_transformer_config_from_args
        config = core_transformer_config_from_args(args)
        if c["kind"] in ("linear", "fp8"):
            from mindspeed_b200.parallel.layers import linear_classes
            st["module"] = linear_classes(config)[0](c["inp"], c["out"], config=config, init_method=config.init_method, bias=False)
            st["x"], st["dout"] = randn(c["tokens"], 1, c["inp"]), randn(c["tokens"], 1, c["out"])
        elif c["kind"] == "moe":
            from mindspeed_b200.parallel.moe.moe_layer import MoELayer
            st["module"] = MoELayer(config)
            st["x"], st["dout"] = randn(c["seq"], c["b"], c["hidden"]), randn(c["seq"], c["b"], c["hidden"], std=0.1)
        else:
            from mindspeed_b200.models.attention import MLASelfAttention
            from mindspeed_b200.models.rotary import RotaryEmbedding
            st["module"] = MLASelfAttention(config)
            st["rotary"] = RotaryEmbedding(QK_ROPE).cuda().get_cos_sin(c["seq"], torch.device("cuda"))
            st["x"], st["dout"] = randn(c["seq"], c["b"], c["hidden"]), randn(c["seq"], c["b"], c["hidden"], std=0.1)
        st["module"].cuda().train()
        st["x"].requires_grad_(True)
        if c["kind"] in ("linear", "moe"):
            _grad_buffers(st["module"])
    return st


def _step_gradients(module, out, x, dout):
    """Backward of a block; weight gradients end up in ``main_grad`` where the block accumulates there, else in ``grad``."""
    for p in module.parameters():
        p.grad = None
    x.grad = None
    out.backward(dout)
    grads = {}
    for name, p in module.named_parameters():
        grads[name] = p.main_grad if p.grad is None else p.grad
    return {"out": out.detach(), "dx": x.grad, "grads": grads}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "train":
        from mindspeed_b200.training import train_step
        from mindspeed_b200.training.global_vars import set_args
        set_args(state["args"])
        model = state["model"]
        loss, _, grad_norm, _ = train_step(state["forward_step"], iter([dict(b) for b in state["batches"]]), model, state["optimizer"], state["scheduler"])
        params = [p for m in model for p in m.parameters()]
        return {"loss": loss["lm loss"], "grad_norm": grad_norm, "weights": [p.detach() for p in params], "grads": [p.main_grad for p in params]}
    if kind == "logits":
        with torch.no_grad():
            return state["model"](state["tokens"], state["positions"], None)
    if kind == "attention":
        from mindspeed_b200.ops.attention import flash_attention
        q, k, v = state["q"], state["k"], state["v"]
        out = flash_attention(q, k, v, causal=c["causal"])
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["dout"])
        return {"out": out.detach(), "dq": dq, "dk": dk, "dv": dv}
    module, x = state["module"], state["x"]
    if kind == "linear":
        return _step_gradients(module, module(x)[0], x, state["dout"])
    if kind == "fp8":
        from mindspeed_b200.models.te_compat import BlockwiseScaling, clear_fp8_weight_cache, fp8_autocast
        clear_fp8_weight_cache()             # the optimizer has moved the weights since the last pass
        with fp8_autocast(True, BlockwiseScaling(fp8_format="e4m3")):
            out = module(x)[0]
        return _step_gradients(module, out, x, state["dout"])
    if kind == "moe":
        return _step_gradients(module, module(x)[0], x, state["dout"])
    return _step_gradients(module, module(x, rotary_pos_emb=state["rotary"])[0], x, state["dout"])


# ---- work and tolerance -------------------------------------------------------------------------------------------------
def _pairs(sq, sk, causal):
    """Visible (query, key) pairs of one head."""
    if not causal:
        return sq * sk
    return sq * (sk - sq) + sq * (sq + 1) // 2


def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind in ("train", "logits"):
        per_layer = c["hidden"] * (c["heads"] + 2 * c["kv"]) * D + c["heads"] * D * c["hidden"] + 3 * c["hidden"] * c["ffn"]
        matmul = c["layers"] * per_layer + c["vocab"] * c["hidden"]
        total = matmul + c["vocab"] * c["hidden"]
        samples = c.get("gbs", c["mbs"])
        fwd = samples * (2 * matmul * c["seq"] + c["layers"] * 4 * D * c["heads"] * _pairs(c["seq"], c["seq"], True))
        if kind == "logits":
            return {"bytes": 2 * matmul + samples * c["seq"] * (2 * c["vocab"] + 2 * c["hidden"]), "flops": fwd}
        # forward + backward; bf16 weight, fp32 gradient written, fp32 master and two moments read and written
        return {"bytes": total * (2 + 2 + 4 + 24), "flops": 3 * fwd}
    if kind == "attention":
        pairs = c["b"] * c["heads"] * _pairs(c["sq"], c["sk"], c["causal"])
        q, kv = c["sq"] * c["b"] * c["heads"] * D, c["sk"] * c["b"] * c["kv"] * D
        return {"bytes": 2 * (4 * q + 4 * kv), "flops": 14 * D * pairs}      # 2 products forward, 5 backward
    if kind in ("linear", "fp8"):
        w = c["inp"] * c["out"]
        io = 2 * 2 * c["tokens"] * (c["inp"] + c["out"])                     # x, dout in; y, dx out
        return {"bytes": io + w * (2 + (8 if kind == "linear" else 2)), "flops": 6 * c["tokens"] * w}
    t = c["seq"] * c["b"]
    if kind == "moe":
        w = 3 * c["hidden"] * c["ffn"]
        rows = 3 * c["hidden"] * c["shared"]
        return {"bytes": 10 * (c["experts"] * w + rows) + 8 * t * c["hidden"],
                "flops": 6 * t * (c["topk"] * w + rows + c["hidden"] * c["experts"])}
    qk = QK_NOPE + QK_ROPE
    w = c["hidden"] * (Q_LORA + KV_LORA + QK_ROPE) + Q_LORA * c["heads"] * qk + KV_LORA * c["heads"] * (QK_NOPE + V_DIM) + c["heads"] * V_DIM * c["hidden"]
    pairs = c["b"] * c["heads"] * _pairs(c["seq"], c["seq"], True)
    return {"bytes": 4 * w + 8 * t * c["hidden"], "flops": 6 * t * w + pairs * (2 * (qk + V_DIM) + 2 * (3 * qk + 2 * V_DIM))}


#: About four times what the path differs by from the same computation with other products and sums: fp32 attention instead of
#: the tiled bf16 one (whole steps, logits, attention, latent attention), library matrix products (linear, experts).  Seen there:
#: gradients of a step 1.6e-2 / 0.58, logits 1.1e-2 / 0.06, attention 3.3e-3 / 0.13, linear and experts 1.7e-3 / 4e-3 (one bf16
#: rounding), latent attention 4.8e-3 / 0.14.
_TOLERANCE = {"train": (0.03, 0.99), "logits": (0.03, 0.25), "attention": (0.013, 0.5), "linear": (0.007, 0.016), "fp8": (0.007, 0.03),
              "moe": (0.01, 0.1), "mla": (0.02, 0.56)}


def tolerance(case):
    rel, most = _TOLERANCE[case["kind"]]
    return {"rel": rel, "max": most}


# ---- the same passes in 64 bits, in plain torch ---------------------------------------------------------------------------
def _rms_norm(x, weight, eps=1e-5):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight


def _rotate(x, dim):
    """Rotary embedding of the last axis of [s, b, heads, dim], halves rotated."""
    inv = 1.0 / (10000.0 ** (torch.arange(0, dim, 2, dtype=torch.float32, device=x.device) / dim))
    angle = torch.outer(torch.arange(x.shape[0], dtype=torch.float32, device=x.device), inv).double()
    cos, sin = (torch.cat((f, f), -1)[:, None, None, :] for f in (angle.cos(), angle.sin()))
    a, b = x.chunk(2, -1)
    return x * cos + torch.cat((-b, a), -1) * sin


def _one_head(q, k, v, causal):
    s = q @ k.t() / q.shape[1] ** 0.5
    if causal:
        s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1 + k.shape[0] - q.shape[0]), float("-inf"))
    return s.softmax(-1) @ v


def _attention(q, k, v, causal):
    """[s, b, heads, d], a head at a time and its scores formed again in backward."""
    from torch.utils.checkpoint import checkpoint
    rep = q.shape[2] // k.shape[2]
    out = [torch.stack([checkpoint(_one_head, q[:, i, h], k[:, i, h // rep], v[:, i, h // rep], causal, use_reentrant=False)
                        for h in range(q.shape[2])], 1) for i in range(q.shape[1])]
    return torch.stack(out, 1)


def _swiglu(x):
    a, b = x.chunk(2, -1)
    return torch.nn.functional.silu(a) * b


def _logits(c, w, tokens):
    """tokens [b, s] -> [b, s, vocab]; w: the model's weights by name."""
    x = w["embedding.word_embeddings.weight"][tokens.t()]
    heads, kv = c["heads"], c["kv"]
    for i in range(c["layers"]):
        p = "decoder.layers.%d." % i
        h = _rms_norm(x, w[p + "input_layernorm.weight"]) @ w[p + "self_attention.linear_qkv.weight"].t()
        h = h.view(*h.shape[:2], kv, heads // kv + 2, D)
        q, k, v = h[..., :-2, :].reshape(*h.shape[:2], heads, D), h[..., -2, :], h[..., -1, :]
        x = x + _attention(_rotate(q, D), _rotate(k, D), v, True).flatten(2) @ w[p + "self_attention.linear_proj.weight"].t()
        h = _rms_norm(x, w[p + "pre_mlp_layernorm.weight"]) @ w[p + "mlp.linear_fc1.weight"].t()
        x = x + _swiglu(h) @ w[p + "mlp.linear_fc2.weight"].t()
    return (_rms_norm(x, w["decoder.final_layernorm.weight"]) @ w["output_layer.weight"].t()).transpose(0, 1)


def _experts(c, w, x):
    flat = x.reshape(-1, x.shape[-1])
    n, e = flat.shape[0], c["experts"]
    logits = flat @ w["router.weight"].t()
    if c["score"] == "softmax":
        top, idx = logits.topk(c["topk"], 1)
        top, scores = top.softmax(-1), logits.softmax(-1)
    else:
        top, idx = logits.sigmoid().topk(c["topk"], 1)
        scores = logits.sigmoid()
        top, scores = top / top.sum(-1, keepdim=True), scores / scores.sum(-1, keepdim=True)
    chosen = torch.zeros_like(logits).scatter(1, idx, 1.0)
    if c["score"] == "softmax":
        balance = (scores.sum(0) * chosen.sum(0)).sum() * (e * 0.01 / (n * n * c["topk"]))
    else:
        per = (scores.view(c["seq"], c["b"], e).sum(0) * chosen.view(c["seq"], c["b"], e).sum(0)).sum()
        balance = per * (e * 0.0001 / (c["seq"] ** 2 * c["topk"] * c["b"]))
    out = torch.zeros_like(flat)
    for i in range(e):
        row, slot = (idx == i).nonzero(as_tuple=True)
        out = out.index_add(0, row, _swiglu(flat[row] @ w["experts.weight1"][i]) @ w["experts.weight2"][i] * top[row, slot, None])
    if c["shared"]:
        out = out + _swiglu(flat @ w["shared_experts.linear_fc1.weight"].t()) @ w["shared_experts.linear_fc2.weight"].t()
    return out.view_as(x), balance


def _latent_attention(c, w, x):
    n, qk = c["heads"], QK_NOPE + QK_ROPE
    q = _rms_norm(x @ w["linear_q_down_proj.weight"].t(), w["q_layernorm.weight"]) @ w["linear_q_up_proj.weight"].t()
    q = q.view(*x.shape[:2], n, qk)
    low, k_pe = (x @ w["linear_kv_down_proj.weight"].t()).split([KV_LORA, QK_ROPE], -1)
    kv = (_rms_norm(low, w["kv_layernorm.weight"]) @ w["linear_kv_up_proj.weight"].t()).view(*x.shape[:2], n, QK_NOPE + V_DIM)
    k_pe = _rotate(k_pe[:, :, None], QK_ROPE).expand(-1, -1, n, -1)
    q = torch.cat((q[..., :QK_NOPE], _rotate(q[..., QK_NOPE:], QK_ROPE)), -1)
    k = torch.cat((kv[..., :QK_NOPE], k_pe), -1)
    return _attention(q, k, kv[..., QK_NOPE:], True).flatten(2) @ w["linear_proj.weight"].t()


def exact(case, seed):
    """What ``run`` returns on the state of ``prepare(case, seed)``, in 64 bits.  The fp8 layer is given without its rounding of
    the operands; the weights after an optimizer step have no such value (their first update is little more than the sign of a
    gradient)."""
    c = dict(case)
    st = prepare(case, seed)
    kind = c["kind"]
    if kind == "attention":
        q, k, v = (st[n].detach().double().requires_grad_(True) for n in "qkv")
        out = _attention(q, k, v, c["causal"])
        return dict(zip(("out", "dq", "dk", "dv"), (out.detach(),) + torch.autograd.grad(out, (q, k, v), st["dout"].double())))
    if kind in ("train", "logits"):
        model = st["model"] if kind == "logits" else st["model"][0]
        while hasattr(model, "module"):
            model = model.module
        names = [n for n, _ in model.named_parameters()]
        w = {n: p.detach().double().requires_grad_(kind == "train") for n, p in model.named_parameters()}
        if kind == "logits":
            with torch.no_grad():
                return _logits(c, w, st["tokens"])
        loss = 0.0
        for b in st["batches"]:
            part = torch.nn.functional.cross_entropy(_logits(c, w, b["tokens"].cuda()).flatten(0, 1), b["labels"].cuda().flatten()) / len(st["batches"])
            part.backward()
            loss += float(part.detach())
        grads = [w[n].grad for n in names]
        norm = float(torch.stack([g.square().sum() for g in grads]).sum().sqrt())
        return {"loss": loss, "grad_norm": norm, "weights": [None] * len(names), "grads": grads}        # clipped inside the update
    w = {n: p.detach().double().requires_grad_(True) for n, p in st["module"].named_parameters()}
    x, dout = st["x"].detach().double().requires_grad_(True), st["dout"].double()
    if kind == "moe":
        out, balance = _experts(c, w, x)
        balance.backward(retain_graph=True)
    else:
        out = _latent_attention(c, w, x) if kind == "mla" else x @ w["weight"].t()
    out.backward(dout)
    return {"out": out.detach(), "dx": x.grad, "grads": {n: p.grad for n, p in w.items()}}
