"""What a user of the framework has it do, as timed cases.

The work is pre-training: micro-batches through ``DualPipeV.step`` (forward and backward of every layer of a model
family, gradients left in the flat fp32 accumulators), the forward-only use of the same step (greedy decoding, scoring
of packed documents), the operators that users call by themselves (attention, expert blocks), and the optimizer step.
Widths are those of the model configurations under ``examples/pretrain_lm``; the depth is cut to two layers (one of each
kind where a family has two) and the vocabulary with it, so that the head keeps about the share it has at full depth.
Routing is the throughput recipes' round-robin replay (``TrainingCfg.benchmark``) in the model cases; the expert-block
cases route by their own logits, so their groups are as ragged as in training.

``draw`` gives other sizes of the same kinds of work: sequence lengths 64 to 4096 in the models, 64 to 16384 in the
attention, 16 to 8192 tokens in the expert blocks, odd ones among them.
"""

import math
from types import SimpleNamespace

import torch

# ------------------------------------------------------------------------------------------------
# sizes
# ------------------------------------------------------------------------------------------------
MODELS = {
    # the smoke configuration: four narrow layers, where launches and the host count
    "small": dict(model_type="qwen3_moe", hidden_size=512, num_attention_heads=8, num_key_value_heads=2, head_dim=128,
                  rms_norm_eps=1e-6, num_experts=16, num_experts_per_tok=4, moe_intermediate_size=256,
                  norm_topk_prob=True, vocab_size=4096, num_hidden_layers=4, rope_theta=1e6, attention_bias=False),
    "qwen3": dict(model_type="qwen3_moe", hidden_size=2048, num_attention_heads=32, num_key_value_heads=4, head_dim=128,
                  rms_norm_eps=1e-6, num_experts=128, num_experts_per_tok=8, moe_intermediate_size=768,
                  norm_topk_prob=True, vocab_size=9496, num_hidden_layers=2, rope_theta=1e6, attention_bias=False),
    # multi-head latent attention; a dense layer, then an expert layer with shared experts
    "deepseek": dict(model_type="deepseek_v2", hidden_size=2048, num_attention_heads=16, qk_rope_head_dim=64,
                     qk_nope_head_dim=128, kv_lora_rank=512, v_head_dim=128, q_lora_rank=None, rms_norm_eps=1e-6,
                     n_routed_experts=64, num_experts_per_tok=6, moe_intermediate_size=1408, n_shared_experts=2,
                     first_k_dense_replace=1, intermediate_size=10944, routed_scaling_factor=1.0, topk_method="greedy",
                     n_group=1, topk_group=1, vocab_size=8192, num_hidden_layers=2, rope_theta=10000.0,
                     rope_scaling=None),
    # a gated-delta-rule layer, then a gated attention layer with head dim 256
    "qwen35": dict(model_type="qwen3_5_moe_text", hidden_size=2048, num_attention_heads=16, num_key_value_heads=2,
                   head_dim=256, attn_output_gate=True, layer_types=["linear_attention", "full_attention"],
                   linear_conv_kernel_dim=4, linear_key_head_dim=128, linear_value_head_dim=128,
                   linear_num_key_heads=16, linear_num_value_heads=32, num_experts=256, num_experts_per_tok=8,
                   moe_intermediate_size=512, shared_expert_intermediate_size=512,
                   rope_parameters=dict(rope_type="default", rope_theta=1e7, partial_rotary_factor=0.25),
                   rms_norm_eps=1e-6, attention_bias=False, vocab_size=15520, num_hidden_layers=2),
}
DEPTH = {"small": 4, "qwen3": 48, "deepseek": 27, "qwen35": 40}  # for the depth-scaled initialisation

# heads, key-value heads, head dim, window, sinks
ATTENTION = {"qwen3": (32, 4, 128, 0, False), "gpt-oss": (64, 8, 64, 0, True), "gpt-oss-window": (64, 8, 64, 127, True)}
# experts, picked, hidden, intermediate, biased clamped activation
EXPERTS = {"qwen3": (128, 8, 2048, 768, False), "gpt-oss": (32, 4, 2880, 2880, True), "deepseek": (64, 6, 2048, 1408, False)}


def listed():
    return [
        # one optimizer step's micro-batches of a debugging run: launches and host time
        dict(name="train_small", kind="train", model="small", seq=512, rows=2),
        # the flagship: two micro-batches of one 4096-token sequence
        dict(name="train_qwen3", kind="train", model="qwen3", seq=4096, rows=2),
        # the recipe lengths of the other families
        dict(name="train_deepseek", kind="train", model="deepseek", seq=2048, rows=2),
        dict(name="train_qwen35", kind="train", model="qwen35", seq=3072, rows=2),
        # one token of the greedy decoder: the whole padded 64-token sequence, forward only
        dict(name="decode_qwen3", kind="forward", model="qwen3", seq=64, rows=2, docs=1),
        # logits of packed documents of uneven lengths
        dict(name="score_packed_qwen3", kind="forward", model="qwen3", seq=3001, rows=2, docs=7),
        # expert blocks, forward and backward, routed by their logits
        dict(name="experts_gpt_oss", kind="experts", shape="gpt-oss", tokens=2048, fp8=False),
        dict(name="experts_fp8", kind="experts", shape="qwen3", tokens=3001, fp8=True),
        # attention, forward and backward: a long sequence, packed documents, sinks
        dict(name="attention_long", kind="attention", shape="qwen3", seq=16384, docs=1),
        dict(name="attention_packed", kind="attention", shape="qwen3", seq=4093, docs=9),
        dict(name="attention_sinks", kind="attention", shape="gpt-oss", seq=2048, docs=1),
        # Muon on a layer's matrices, AdamW on the rest
        dict(name="optimizer", kind="optimizer", experts=64, hidden=2048, intermediate=768, vocab=9496),
    ]


def _size(rng, low, high):
    """Spread over the logarithm; odd, a multiple of 4, of 64 and unrestricted in turn."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    step = rng.choice([1, 4, 64, 1])
    return max(low, min(high, n // step * step))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "forward", "experts", "attention", "attention", "optimizer"])
    if kind == "train":
        model = rng.choice(["small", "qwen3", "deepseek", "qwen35"])
        return dict(kind=kind, model=model, seq=_size(rng, 64, 4096 if model in ("small", "qwen3") else 3072), rows=2)
    if kind == "forward":
        seq = _size(rng, 64, 4096)
        return dict(kind=kind, model=rng.choice(["qwen3", "deepseek"]), seq=seq, rows=2, docs=rng.randint(1, 1 + seq // 64))
    if kind == "experts":
        return dict(kind=kind, shape=rng.choice(sorted(EXPERTS)), tokens=_size(rng, 16, 8192), fp8=rng.random() < 0.4)
    if kind == "attention":
        shape = rng.choice(sorted(ATTENTION))
        seq = _size(rng, 64, 16384 if shape == "qwen3" else 8192)
        if seq > 4096:  # long sequences are trained in round lengths
            seq = seq // 64 * 64
        return dict(kind=kind, shape=shape, seq=seq, docs=rng.choice([1, 1, rng.randint(1, 1 + seq // 64)]))
    return dict(kind=kind, experts=rng.randint(4, 64), hidden=rng.choice([1024, 2048, 2880]),
                intermediate=rng.choice([512, 768, 1408]), vocab=rng.randint(1000, 20000) // 8 * 8)


# ------------------------------------------------------------------------------------------------
# inputs (made from the seed alone)
# ------------------------------------------------------------------------------------------------
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + salt * 7919 + 17) % (1 << 62))


def _normal(seed, salt, shape, std, mean=0.0, dtype=torch.bfloat16):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=_gen(seed, salt))


def _doc_starts(seed, seq, docs):
    """Uneven document boundaries: ``docs`` documents of at least one token."""
    cuts = torch.randperm(seq - 1, generator=torch.Generator().manual_seed(seed))[: docs - 1] + 1
    return [0] + sorted(int(c) for c in cuts) + [seq]


def _shapes(model):
    """{parameter name: (shape, standard deviation, mean)} of a model family."""
    c = MODELS[model]
    H, V, L = c["hidden_size"], c["vocab_size"], c["num_hidden_layers"]
    s, so = 0.02, 0.02 / math.sqrt(2 * DEPTH[model])
    out = {"embed_tokens.weight": ((V, H), s, 0.0)}
    norm_mean = 0.0 if model == "qwen35" else 1.0

    def mlp(p, inter):
        out[p + "gate_proj.weight"], out[p + "up_proj.weight"] = ((inter, H), s, 0.0), ((inter, H), s, 0.0)
        out[p + "down_proj.weight"] = ((H, inter), so, 0.0)

    def experts(p, E, inter):
        out[p + "gate.weight"] = ((E, H), s, 0.0)
        if model == "qwen35":
            out[p + "experts.gate_up_proj.weight"] = ((E, 2 * inter, H), s, 0.0)
        else:
            out[p + "experts.gate_proj.weight"] = ((E, inter, H), s, 0.0)
            out[p + "experts.up_proj.weight"] = ((E, inter, H), s, 0.0)
        out[p + "experts.down_proj.weight"] = ((E, H, inter), so, 0.0)

    for i in range(L):
        p = "layers.%d." % i
        for n in ("input_layernorm", "post_attention_layernorm"):
            out[p + n + ".weight"] = ((H,), 0.1, norm_mean)
        a = p + "self_attn."
        if model in ("small", "qwen3") or (model == "qwen35" and c["layer_types"][i] == "full_attention"):
            D, Hq, Hk = c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"]
            out[a + "q_proj.weight"] = ((Hq * D * (2 if model == "qwen35" else 1), H), s, 0.0)
            out[a + "k_proj.weight"] = ((Hk * D, H), s, 0.0)
            out[a + "v_proj.weight"] = ((Hk * D, H), s, 0.0)
            out[a + "o_proj.weight"] = ((H, Hq * D), so, 0.0)
            out[a + "q_norm.weight"], out[a + "k_norm.weight"] = ((D,), 0.1, norm_mean), ((D,), 0.1, norm_mean)
        elif model == "deepseek":
            nh, dn, dr, dv, r = (c[k] for k in ("num_attention_heads", "qk_nope_head_dim", "qk_rope_head_dim", "v_head_dim", "kv_lora_rank"))
            out[a + "q_proj.weight"] = ((nh * (dn + dr), H), s, 0.0)
            out[a + "kv_a_proj_with_mqa.weight"] = ((r + dr, H), s, 0.0)
            out[a + "kv_a_layernorm.weight"] = ((r,), 0.1, 1.0)
            out[a + "kv_b_proj.weight"] = ((nh * (dn + dv), r), s, 0.0)
            out[a + "o_proj.weight"] = ((H, nh * dv), so, 0.0)
        else:
            a = p + "linear_attn."
            nk, nv, dk, dv = (c["linear_" + k] for k in ("num_key_heads", "num_value_heads", "key_head_dim", "value_head_dim"))
            out[a + "conv1d.weight"] = ((2 * nk * dk + nv * dv, 1, c["linear_conv_kernel_dim"]), 0.3, 0.0)
            out[a + "dt_bias"], out[a + "A_log"] = ((nv,), 0.5, 0.0), ((nv,), 0.7, 0.5)
            out[a + "norm.weight"] = ((dv,), 0.1, 1.0)
            out[a + "in_proj_qkv.weight"] = ((2 * nk * dk + nv * dv, H), s, 0.0)
            out[a + "in_proj_z.weight"] = ((nv * dv, H), s, 0.0)
            out[a + "in_proj_b.weight"], out[a + "in_proj_a.weight"] = ((nv, H), s, 0.0), ((nv, H), s, 0.0)
            out[a + "out_proj.weight"] = ((H, nv * dv), s, 0.0)
        m = p + "mlp."
        if model == "deepseek" and i < c["first_k_dense_replace"]:
            mlp(m, c["intermediate_size"])
        elif model == "deepseek":
            mlp(m + "shared_experts.", c["n_shared_experts"] * c["moe_intermediate_size"])
            experts(m, c["n_routed_experts"], c["moe_intermediate_size"])
        else:
            if model == "qwen35":
                mlp(m + "shared_expert.", c["shared_expert_intermediate_size"])
                out[m + "shared_expert_gate.weight"] = ((1, H), s, 0.0)
            experts(m, c["num_experts"], c["moe_intermediate_size"])
    out["norm.weight"], out["lm_head.weight"] = ((H,), 0.1, norm_mean), ((V, H), s, 0.0)
    return out


def _weight(model, seed, k, spec):
    shape, std, mean = spec
    return _normal(seed, 100 + k, shape, std, mean)


def _tokens(case, seed):
    V = MODELS[case["model"]]["vocab_size"]
    g = _gen(seed, 1)
    ids = torch.randint(0, V, (case["rows"], case["seq"] + 1), device="cuda", generator=g)
    tokens, labels = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    labels[:, -1] = -100  # the last token of a row has no successor
    return tokens, labels


def _packed(case, seed):
    if case.get("docs", 1) <= 1:
        return None
    return [_doc_starts(seed * 31 + r, case["seq"], case["docs"]) for r in range(case["rows"])]


def _expert_inputs(case, seed):
    E, k, H, I, biased = EXPERTS[case["shape"]]
    n = case["tokens"]
    d = dict(x=_normal(seed, 1, (n, H), 1.0), d_out=_normal(seed, 2, (n, H), 1.0),
             logits=_normal(seed, 3, (n, E), 1.0, dtype=torch.float32) + _normal(seed, 4, (1, E), 0.5, dtype=torch.float32),
             w1=_normal(seed, 5, (E, 2 * I, H), 0.02), w2=_normal(seed, 6, (E, H, I), 0.02))
    if biased:
        d["b1"], d["b2"] = _normal(seed, 7, (E, 2 * I), 0.1), _normal(seed, 8, (E, H), 0.1)
    return d


def _attention_inputs(case, seed):
    Hq, Hk, D, window, sinks = ATTENTION[case["shape"]]
    S = case["seq"]
    d = dict(q=_normal(seed, 1, (1, S, Hq, D), 1.0), k=_normal(seed, 2, (1, S, Hk, D), 1.0), v=_normal(seed, 3, (1, S, Hk, D), 1.0),
             d_out=_normal(seed, 4, (1, S, Hq, D), 1.0))
    if sinks:
        d["sinks"] = _normal(seed, 5, (Hq,), 1.0)
    return d


def _optimizer_inputs(case, seed):
    """[(name, weight, gradient, matrix for Muon?)]: a decoder layer with its expert stacks, norms and an embedding."""
    E, H, I, V = case["experts"], case["hidden"], case["intermediate"], case["vocab"]
    shapes = dict(q=(2 * H, H), k=(H // 4, H), v=(H // 4, H), o=(H, 2 * H), gate=(E, I, H), up=(E, I, H), down=(E, H, I),
                  router=(E, H), norm=(H,), embed=(V, H))
    out = []
    for j, (name, shape) in enumerate(shapes.items()):
        w = _normal(seed, 10 + j, shape, 0.02, 1.0 if name == "norm" else 0.0)
        g = _normal(seed, 40 + j, shape, 1e-3, dtype=torch.float32)
        out.append((name, w, g, name not in ("router", "norm", "embed")))
    return out


LR, MOMENTUM, DECAY = 1e-3, 0.95, 0.1


# ------------------------------------------------------------------------------------------------
# the framework's side
# ------------------------------------------------------------------------------------------------
def _prepare_model(case, seed):
    from pithtrain_b200.contexts import distributed, training
    from pithtrain_b200.dualpipe.dualpipev import DualPipeV
    from pithtrain_b200.models import MODEL_CLASSES
    from pithtrain_b200.modules.load_balance import force_balance
    from pithtrain_b200.modules.training import apply_fsdp

    distributed.reset_single_process()
    distributed.device = torch.device("cuda", torch.cuda.current_device())
    cfg = SimpleNamespace(**MODELS[case["model"]], max_position_embeddings=case["seq"])
    before = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device("meta"):
            chunks = torch.nn.Sequential(*[MODEL_CLASSES[cfg.model_type](cfg, phase=f) for f in (0, 1)])
    finally:
        torch.set_default_dtype(before)
    apply_fsdp(chunks, grad_dtype=torch.float32)
    groups = training.shard_groups
    params = {n.split(".", 1)[1]: p for n, p in chunks.named_parameters()}
    shapes = _shapes(case["model"])
    assert {n: tuple(p.shape) for n, p in params.items()} == {n: s[0] for n, s in shapes.items()}
    with torch.no_grad():
        for k, (n, spec) in enumerate(shapes.items()):
            params[n].copy_(_weight(case["model"], seed, k, spec))
    chunks[1].rotary_emb = chunks[0].rotary_emb
    for m in chunks.modules():
        if hasattr(m, "router_replay"):
            m.router_replay = force_balance(m.num_experts)
    tokens, labels = _tokens(case, seed)
    cu = _packed(case, seed)
    cu = None if cu is None else [torch.tensor(c, dtype=torch.int32, device="cuda") for c in cu]
    return dict(kind=case["kind"], model=DualPipeV(chunks), groups=groups, params=params, tokens=tokens, labels=labels,
                cu=cu, rows=case["rows"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "forward"):
        return _prepare_model(case, seed)
    if kind == "attention":
        d = _attention_inputs(case, seed)
        Hq, Hk, D, window, _ = ATTENTION[case["shape"]]
        for n in ("q", "k", "v", "sinks"):
            if n in d:
                d[n].requires_grad_()
        cu = None
        if case["docs"] > 1:
            cu = torch.tensor(_doc_starts(seed, case["seq"], case["docs"]), dtype=torch.int32, device="cuda")
        return dict(d, kind=kind, scale=D ** -0.5, window=(window, 0) if window else (None, None), cu=cu, seq=case["seq"])
    if kind == "experts":
        E, k, H, I, biased = EXPERTS[case["shape"]]
        d = _expert_inputs(case, seed)
        d["x"].requires_grad_()
        d["logits"].requires_grad_()
        grads = {n: torch.zeros(d[n].shape, dtype=torch.float32, device="cuda") for n in ("w1", "w2", "b1", "b2") if n in d}
        for n in ("b1", "b2"):
            if n in d:
                d[n] = torch.nn.Parameter(d[n])
                d[n].main_grad = grads[n]
        return dict(d, kind=kind, k=k, biased=biased, fp8=case["fp8"], grads=grads)
    from pithtrain_b200.modules.optimizer import AdamW, Muon

    muon, adamw, named = [], [], {}
    for name, w, g, matrix in _optimizer_inputs(case, seed):
        p = torch.nn.Parameter(w)
        p.main_grad = g
        named[name] = p
        (muon if matrix else adamw).append(p)
    opts = [Muon(muon, lr=LR, momentum=MOMENTUM, weight_decay=DECAY), AdamW(adamw, lr=LR, weight_decay=DECAY)]
    return dict(kind=kind, optimizers=opts, params=named)


def run(state):
    kind = state["kind"]
    if kind == "train":
        from pithtrain_b200.tasks.pretrain_lm import criterion

        for g in state["groups"]:
            g.zero_grad()
        loss, _ = state["model"].step(state["tokens"], num_chunks=state["rows"], criterion=criterion, labels=state["labels"])
        for g in state["groups"]:
            g.fold_autograd_grads()
        return {"loss": loss, "grads": {n: p.main_grad for n, p in state["params"].items()}}
    if kind == "forward":
        with torch.no_grad():
            _, logits = state["model"].step(state["tokens"], num_chunks=state["rows"], cu_seqlens=state["cu"], return_outputs=True)
        return {"logits": logits}
    if kind == "attention":
        from pithtrain_b200.ops.flash_attn_v4 import flash_attn_func, flash_attn_varlen_func

        q, k, v, sinks = state["q"], state["k"], state["v"], state.get("sinks")
        if state["cu"] is None:
            out = flash_attn_func(q, k, v, state["scale"], True, state["window"], sinks)
        else:
            out = flash_attn_varlen_func(q[0], k[0], v[0], state["cu"], state["seq"], state["scale"], True, state["window"], sinks)[None]
        leaves = (q, k, v) if sinks is None else (q, k, v, sinks)
        return [out, *torch.autograd.grad(out, leaves, state["d_out"])]
    if kind == "experts":
        from pithtrain_b200.dualpipe.utils import FP8WeightCacheControl
        from pithtrain_b200.ops import fp8_linear
        from pithtrain_b200.ops.moe import ExpertWeights, moe_experts
        from pithtrain_b200.ops.router import router_topk

        g = state["grads"]
        for t in g.values():
            t.zero_()
        fp8_linear.enable(state["fp8"])
        FP8WeightCacheControl.step()  # weights change from step to step: quantised copies are made anew
        try:
            if state["biased"]:
                w, idx, _ = router_topk(state["logits"], state["k"], "topk_softmax")
                ew = ExpertWeights(state["w1"], state["w2"], lambda: g["w1"], lambda: g["w2"], b1=state["b1"], b2=state["b2"],
                                   interleaved=True, alpha=1.702, limit=7.0)
            else:
                w, idx, _ = router_topk(state["logits"], state["k"], "softmax_topk", renorm=True)
                ew = ExpertWeights(state["w1"], state["w2"], lambda: g["w1"], lambda: g["w2"])
            out = moe_experts(state["x"], w, idx, ew)
            dx, dl = torch.autograd.grad(out, (state["x"], state["logits"]), state["d_out"])
        finally:
            fp8_linear.enable(False)
            FP8WeightCacheControl.clear()
        return {"out": out, "dx": dx, "dlogits": dl, "idx": idx, **g}
    for opt in state["optimizers"]:
        opt.step()
    muon = state["optimizers"][0].state
    return {"w": dict(state["params"]), "momentum": {n: muon[p]["momentum_buffer"] for n, p in state["params"].items() if p in muon}}


# ------------------------------------------------------------------------------------------------
# work and tolerance
# ------------------------------------------------------------------------------------------------
def _numel(shape):
    return math.prod(shape)


def _pairs(case, window=0):
    """Visible (query, key) pairs of a causal sequence, or of its packed documents taken as equal."""
    S, docs = case["seq"], max(1, case.get("docs", 1))
    n = S / docs
    pairs = docs * n * (n + 1) / 2
    return min(pairs, S * (window + 1)) if window else pairs


def work(case):
    kind = case["kind"]
    if kind in ("train", "forward"):
        c = MODELS[case["model"]]
        shapes = _shapes(case["model"])
        total = sum(_numel(s[0]) for s in shapes.values())
        tokens = case["seq"] * case["rows"]
        active = 0.0
        used = 0.0  # expert weights that some token needs
        for n, (shape, _, _) in shapes.items():
            size = _numel(shape)
            if len(shape) == 3 and ".experts." in n:
                picked = c["num_experts_per_tok"]
                active += size / shape[0] * picked
                used += size * min(1.0, tokens * picked / shape[0])
            elif len(shape) == 2 and n != "embed_tokens.weight":
                active += size
                used += size
        flops = 2 * active * tokens
        for i in range(c["num_hidden_layers"]):
            if case["model"] == "qwen35" and i == 0:
                flops += tokens * c["linear_num_value_heads"] * 128 * 128 * 6  # the recurrence itself
                continue
            dqk, dv = (192, 128) if case["model"] == "deepseek" else (c["head_dim"], c["head_dim"])
            flops += 2 * (dqk + dv) * c["num_attention_heads"] * _pairs(case) * case["rows"]
        if kind == "forward":
            return {"bytes": 2 * used + tokens * (8 + 2 * c["hidden_size"] + 2 * c["vocab_size"]), "flops": flops}
        return {"bytes": 2 * total + 4 * total + 16 * tokens, "flops": 3 * flops}
    if kind == "attention":
        Hq, Hk, D, window, _ = ATTENTION[case["shape"]]
        S = case["seq"]
        return {"bytes": 2 * S * D * (2 * Hq + 2 * Hk) + 2 * S * D * (2 * Hq + 2 * Hk), "flops": 3.5 * 4 * D * Hq * _pairs(case, window)}
    if kind == "experts":
        E, k, H, I, _ = EXPERTS[case["shape"]]
        n = case["tokens"]
        weights = 3 * E * I * H
        return {"bytes": 2 * weights + 4 * weights + 2 * n * H * 4 + 8 * n * E, "flops": 3 * 6 * n * k * H * I}
    E, H, I, V = case["experts"], case["hidden"], case["intermediate"], case["vocab"]
    flops, muon = 0.0, 0
    for count, r, c in ((1, 2 * H, H), (2, H // 4, H), (1, H, 2 * H), (3 * E, min(I, H), max(I, H))):
        m, n = min(r, c), max(r, c)
        flops += count * 5 * (2 * m * m * n + 2 * m * m * m + 2 * m * m * n)
        muon += count * r * c
    adamw = (V + E + 1) * H
    return {"bytes": muon * (2 + 2 + 4 + 4 + 4) + adamw * (2 + 2 + 4 + 16), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "train":
        return {"rel": 0.03, "max": 0.99}
    if kind == "forward":
        return {"rel": 0.03, "max": 0.5}
    if kind == "attention":
        return {"rel": 0.01, "max": 0.3}
    if kind == "experts":
        return {"rel": 0.03, "max": 0.99, "differ": 1e-3} if case["fp8"] else {"rel": 0.015, "max": 0.5, "differ": 1e-3}
    return {"rel": 0.005, "max": 0.2}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------------
def _leaf(t):
    return t.detach().double().requires_grad_()


def _attend(q, k, v, scale, window=0, sinks=None, starts=None):
    """q [S,Hq,D], k [S,Hk,D], v [S,Hk,Dv], causal; documents start at ``starts``."""
    from torch.utils.checkpoint import checkpoint

    S, Hq = q.shape[:2]
    per = Hq // k.shape[1]
    pos = torch.arange(S, device=q.device)
    low = torch.zeros_like(pos)
    if starts is not None:
        s = torch.tensor(starts, device=q.device)
        low = s[torch.bucketize(pos, s[1:], right=True)]
    if window:
        low = torch.maximum(low, pos - window)
    hidden = (pos[None, :] > pos[:, None]) | (pos[None, :] < low[:, None])

    def head(qh, kh, vh, sink):
        s = (qh @ kh.T * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.expand(S, 1)], 1)
        p = s.softmax(-1)
        return p[:, :S] @ vh

    outs = [checkpoint(head, q[:, h], k[:, h // per], v[:, h // per], None if sinks is None else sinks[h], use_reentrant=False)
            for h in range(Hq)]
    return torch.stack(outs, 1)


def _norm(x, w, eps, plus=0.0):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * (w + plus)


def _rotate(x, theta, pos):
    """Rotate-half rotary embedding of x [S, heads, d]."""
    d = x.shape[-1]
    f = torch.outer(pos.double(), 1.0 / theta ** (torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d))
    cos, sin = torch.cat([f.cos()] * 2, -1)[:, None], torch.cat([f.sin()] * 2, -1)[:, None]
    a, b = x[..., : d // 2], x[..., d // 2:]
    return x * cos + torch.cat([-b, a], -1) * sin


def _gated(x, P, p):
    F = torch.nn.functional
    return (F.silu(x @ P[p + "gate_proj.weight"].T) * (x @ P[p + "up_proj.weight"].T)) @ P[p + "down_proj.weight"].T


def _delta_rule(q, k, v, g, beta):
    """Gated delta rule by chunks of 64 tokens; q, k, v [H,S,d], g, beta [H,S]."""
    H, S, dk = q.shape
    C = 64
    n = (S + C - 1) // C
    F = torch.nn.functional
    q, k, v = (F.pad(t, (0, 0, 0, n * C - S)).reshape(H, n, C, -1) for t in (q, k, v))
    g, beta = (F.pad(t, (0, n * C - S)).reshape(H, n, C) for t in (g, beta))
    q = q * dk ** -0.5
    b = g.cumsum(-1)
    low = torch.tril(torch.ones(C, C, dtype=torch.bool, device=q.device))
    decay = (b[..., :, None] - b[..., None, :]).masked_fill(~low, -math.inf).exp()
    eye = torch.eye(C, dtype=q.dtype, device=q.device)
    A = (beta[..., None] * (k @ k.mT) * decay).tril(-1) + eye
    rhs = torch.cat([beta[..., None] * v, beta[..., None] * b.exp()[..., None] * k], -1)
    sol = torch.linalg.solve_triangular(A, rhs, upper=False)
    u, w = sol[..., : v.shape[-1]], sol[..., v.shape[-1]:]
    state = torch.zeros(H, dk, v.shape[-1], dtype=q.dtype, device=q.device)
    outs = []
    for i in range(n):
        new = u[:, i] - w[:, i] @ state
        last = b[:, i, -1:]
        outs.append(b[:, i].exp()[..., None] * (q[:, i] @ state) + ((q[:, i] @ k[:, i].mT) * decay[:, i]) @ new)
        state = last.exp()[..., None] * state + (k[:, i] * (last - b[:, i]).exp()[..., None]).mT @ new
    return torch.stack(outs, 1).reshape(H, n * C, -1)[:, :S]


def _mix(x, P, p, model, c, layer, starts):
    F = torch.nn.functional
    S, eps = x.shape[0], c["rms_norm_eps"]
    pos = torch.arange(S, device=x.device)
    if starts is not None:
        s = torch.tensor(starts, device=x.device)
        pos = pos - s[torch.bucketize(pos, s[1:], right=True)]
    a = p + "self_attn."
    if model in ("small", "qwen3"):
        D, Hq, Hk = c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"]
        q, k, v = ((x @ P[a + n + "_proj.weight"].T).view(S, -1, D) for n in "qkv")
        q, k = (_rotate(_norm(t, P[a + n + "_norm.weight"], eps), c["rope_theta"], pos) for t, n in ((q, "q"), (k, "k")))
        return _attend(q, k, v, D ** -0.5, starts=starts).reshape(S, -1) @ P[a + "o_proj.weight"].T
    if model == "deepseek":
        nh, dn, dr, dv, r = (c[k] for k in ("num_attention_heads", "qk_nope_head_dim", "qk_rope_head_dim", "v_head_dim", "kv_lora_rank"))
        q = (x @ P[a + "q_proj.weight"].T).view(S, nh, dn + dr)
        ckv = x @ P[a + "kv_a_proj_with_mqa.weight"].T
        kv = (_norm(ckv[:, :r], P[a + "kv_a_layernorm.weight"], eps) @ P[a + "kv_b_proj.weight"].T).view(S, nh, dn + dv)
        halves = lambda t: t.unflatten(-1, (dr // 2, 2)).transpose(-1, -2).flatten(-2)  # noqa: E731
        q = torch.cat([q[..., :dn], _rotate(halves(q[..., dn:]), c["rope_theta"], pos)], -1)
        kr = _rotate(halves(ckv[:, None, r:]), c["rope_theta"], pos)
        k = torch.cat([kv[..., :dn], kr.expand(-1, nh, -1)], -1)
        return _attend(q, k, kv[..., dn:], (dn + dr) ** -0.5, starts=starts).reshape(S, -1) @ P[a + "o_proj.weight"].T
    if c["layer_types"][layer] == "full_attention":
        D, Hk = c["head_dim"], c["num_key_value_heads"]
        q, gate = (x @ P[a + "q_proj.weight"].T).view(S, -1, 2 * D).chunk(2, -1)
        k, v = ((x @ P[a + n + "_proj.weight"].T).view(S, Hk, D) for n in "kv")
        q, k = (_norm(t, P[a + n + "_norm.weight"], eps, 1.0) for t, n in ((q, "q"), (k, "k")))
        rd = int(D * c["rope_parameters"]["partial_rotary_factor"])
        q, k = (torch.cat([_rotate(t[..., :rd], c["rope_parameters"]["rope_theta"], pos), t[..., rd:]], -1) for t in (q, k))
        return (_attend(q, k, v, D ** -0.5) * gate.sigmoid()).reshape(S, -1) @ P[a + "o_proj.weight"].T
    a = p + "linear_attn."
    nk, nv, dk, dv = (c["linear_" + k] for k in ("num_key_heads", "num_value_heads", "key_head_dim", "value_head_dim"))
    mixed = x @ P[a + "in_proj_qkv.weight"].T
    w = P[a + "conv1d.weight"]
    taps = w.shape[-1]
    padded = F.pad(mixed, (0, 0, taps - 1, 0))
    mixed = F.silu(sum(padded[j: j + S] * w[:, 0, j] for j in range(taps)))
    q, k, v = mixed.split([nk * dk, nk * dk, nv * dv], -1)
    q, k = (F.normalize(t.view(S, nk, dk), dim=-1).repeat_interleave(nv // nk, 1).transpose(0, 1) for t in (q, k))
    beta = (x @ P[a + "in_proj_b.weight"].T).sigmoid().T
    g = (-P[a + "A_log"].exp() * F.softplus(x @ P[a + "in_proj_a.weight"].T + P[a + "dt_bias"])).T
    o = _delta_rule(q, k, v.view(S, nv, dv).transpose(0, 1), g, beta).transpose(0, 1)
    z = (x @ P[a + "in_proj_z.weight"].T).view(S, nv, dv)
    return (_norm(o, P[a + "norm.weight"], eps) * F.silu(z)).reshape(S, -1) @ P[a + "out_proj.weight"].T


def _feed(x, P, p, model, c, layer):
    F = torch.nn.functional
    if model == "deepseek" and layer < c["first_k_dense_replace"]:
        return _gated(x, P, p)
    n, k = x.shape[0], c["num_experts_per_tok"]
    E = P[p + "gate.weight"].shape[0]
    idx = (torch.arange(n, device=x.device)[:, None] + torch.arange(k, device=x.device) * (E // k)) % E
    w = (x @ P[p + "gate.weight"].T).softmax(-1).gather(1, idx)
    if model != "deepseek":
        w = w / w.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(E):
        tok, slot = torch.where(idx == e)
        if tok.numel() == 0:
            continue
        if model == "qwen35":
            a, b = (x[tok] @ P[p + "experts.gate_up_proj.weight"][e].T).chunk(2, -1)
        else:
            a, b = (x[tok] @ P[p + "experts.%s_proj.weight" % t][e].T for t in ("gate", "up"))
        y = y.index_add(0, tok, (F.silu(a) * b) @ P[p + "experts.down_proj.weight"][e].T * w[tok, slot][:, None])
    if model == "deepseek":
        y = y + _gated(x, P, p + "shared_experts.")
    if model == "qwen35":
        y = y + (x @ P[p + "shared_expert_gate.weight"].T).sigmoid() * _gated(x, P, p + "shared_expert.")
    return y


def _exact_model(case, seed):
    from torch.utils.checkpoint import checkpoint

    model, train = case["model"], case["kind"] == "train"
    c = MODELS[model]
    plus = 1.0 if model == "qwen35" else 0.0
    P = {n: _weight(model, seed, k, spec).double().requires_grad_(train) for k, (n, spec) in enumerate(_shapes(model).items())}
    tokens, labels = _tokens(case, seed)
    packed = _packed(case, seed)
    eps = c["rms_norm_eps"]
    losses, logits = [], []

    def layer(h, i, starts):
        p = "layers.%d." % i
        h = h + _mix(_norm(h, P[p + "input_layernorm.weight"], eps, plus), P, p, model, c, i, starts)
        return h + _feed(_norm(h, P[p + "post_attention_layernorm.weight"], eps, plus), P, p + "mlp.", model, c, i)

    with torch.set_grad_enabled(train):
        for r in range(case["rows"]):
            h = P["embed_tokens.weight"][tokens[r]]
            for i in range(c["num_hidden_layers"]):
                h = checkpoint(layer, h, i, None if packed is None else packed[r], use_reentrant=False)
            out = _norm(h, P["norm.weight"], eps, plus) @ P["lm_head.weight"].T
            if train:
                loss = torch.nn.functional.cross_entropy(out, labels[r], ignore_index=-100, reduction="sum")
                loss.backward()
                losses.append(loss.detach())
            else:
                logits.append(out)
    if train:
        return {"loss": torch.stack(losses), "grads": {n: t.grad for n, t in P.items()}}
    return {"logits": torch.stack(logits)}


def _exact_attention(case, seed):
    Hq, Hk, D, window, _ = ATTENTION[case["shape"]]
    d = _attention_inputs(case, seed)
    q, k, v = (_leaf(d[n][0]) for n in "qkv")
    sinks = _leaf(d["sinks"]) if "sinks" in d else None
    starts = _doc_starts(seed, case["seq"], case["docs"]) if case["docs"] > 1 else None
    out = _attend(q, k, v, D ** -0.5, window, sinks, starts)
    leaves = (q, k, v) if sinks is None else (q, k, v, sinks)
    grads = torch.autograd.grad(out, leaves, d["d_out"][0].double())
    return [out.detach()[None], *(g[None] for g in grads[:3]), *grads[3:]]


def _exact_experts(case, seed):
    E, k, H, I, biased = EXPERTS[case["shape"]]
    d = _expert_inputs(case, seed)
    L = {n: _leaf(t) for n, t in d.items() if n != "d_out"}
    x, d_out = L["x"], d["d_out"].double()
    if biased:
        top, idx = L["logits"].topk(k, -1)
        w = top.softmax(-1)
    else:
        top, idx = L["logits"].softmax(-1).topk(k, -1)
        w = top / top.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(E):
        tok, slot = torch.where(idx == e)
        if tok.numel() == 0:
            continue
        h = x[tok] @ L["w1"][e].T
        if biased:
            h = h + L["b1"][e]
            a, b = h[:, 0::2].clamp(max=7.0), h[:, 1::2].clamp(-7.0, 7.0)
            y = ((b + 1) * a * torch.sigmoid(1.702 * a)) @ L["w2"][e].T + L["b2"][e]
        else:
            a, b = h.chunk(2, -1)
            y = (torch.nn.functional.silu(a) * b) @ L["w2"][e].T
        out = out.index_add(0, tok, y * w[tok, slot][:, None])
    names = [n for n in ("x", "logits", "w1", "w2", "b1", "b2") if n in L]
    g = dict(zip(names, torch.autograd.grad(out, [L[n] for n in names], d_out)))
    res = {"out": out.detach(), "dx": g["x"], "dlogits": g["logits"], "idx": None}
    res.update({n: g[n] for n in ("w1", "w2", "b1", "b2") if n in g})
    return res


def _exact_optimizer(case, seed):
    weights, momenta = {}, {}
    for name, w, g, matrix in _optimizer_inputs(case, seed):
        w, g = w.double(), g.double()
        if not matrix:
            # first step of AdamW: both moments start at zero, so their bias corrections cancel
            weights[name] = w * (1 - LR * DECAY) - LR * g / (g.abs() + 1e-8)
            continue
        m = (1 - MOMENTUM) * g
        momenta[name] = m
        x = g * (1 - MOMENTUM) + m * MOMENTUM
        rows, cols = x.shape[-2:]
        if rows > cols:
            x = x.mT
        x = x / (torch.linalg.vector_norm(x, dim=(-2, -1), keepdim=True) + 1e-7)
        for _ in range(5):
            a = x @ x.mT
            x = 3.4445 * x + (-4.7750 * a + 2.0315 * a @ a) @ x
        if rows > cols:
            x = x.mT
        weights[name] = w * (1 - LR * DECAY) - LR * 0.2 * math.sqrt(max(rows, cols)) * x
    return {"w": weights, "momentum": momenta}


def exact(case, seed):
    return {"train": _exact_model, "forward": _exact_model, "attention": _exact_attention, "experts": _exact_experts,
            "optimizer": _exact_optimizer}[case["kind"]](case, seed)
