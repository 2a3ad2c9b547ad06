"""Workloads by which the speed of this framework is judged: what an RL post-training job has it do on one GPU.

Eight kinds of work, each through the public entry points and over the range of sizes that a job meets:

* ``train``        one GRPO step (``GRPOTrainer.step``): host batch in, forward, loss, backward, AdamW, loss out
* ``moe``          a mixture-of-experts FFN (router, experts, combine), alone or with its backward pass
* ``decode``       one token of a rollout for ``n`` sequences after a shared prompt, up to the logits
* ``score``        log-probs of given completions (``NativeRolloutEngine.score``), forward only
* ``linear_logp``  hidden states x LM head -> selected log-probs (+ entropy), alone or with its backward pass
* ``loss``         GRPO loss over materialised policy / reference logits, forward and backward
* ``sample``       temperature / top-k / top-p sampling of the next token from logits
* ``attention``    the attention operators on their own, forward or forward and backward
"""

import math

import torch

DEV = "cuda"

# (hidden, query heads, key/value heads, FFN) of dense decoders, from the smallest test model to Llama-3-8B
DENSE_WIDTHS = [(512, 4, 2, 1024), (1024, 8, 2, 2816), (2048, 16, 4, 5632), (4096, 32, 8, 14336)]
# (hidden, experts, experts per token, expert FFN) of mixture-of-experts layers, up to Qwen3-30B-A3B
MOE_WIDTHS = [(256, 8, 2, 128), (1024, 32, 4, 384), (2048, 128, 8, 768)]
VOCABS = [4096, 32000, 50257, 128256, 151936]


def _dense(width, layers, vocab):
    h, hq, hkv, f = DENSE_WIDTHS[width]
    return {"hidden": h, "heads": hq, "kv_heads": hkv, "ffn": f, "layers": layers, "vocab": vocab}


def _moe(width):
    h, e, k, f = MOE_WIDTHS[width]
    return {"hidden": h, "experts": e, "top": k, "ffn": f}


def listed():
    return [
        # A unit-test-sized training step: nearly all launches and host work.
        {"name": "train_tiny", "kind": "train", **_dense(0, 2, 4096), "prompt": 192, "group": 4, "length": 128, "micro": 0},
        # A medium decoder with lengths that are no multiple of a tile.
        {"name": "train_ragged", "kind": "train", **_dense(2, 4, 32000), "prompt": 333, "group": 8, "length": 211, "micro": 0},
        # Two layers of the headline step: Llama-3-8B widths, 1024-token prompt run once, completions in two micro-batches.
        {"name": "train_8b_layers", "kind": "train", **_dense(3, 2, 128256), "prompt": 1024, "group": 32, "length": 512,
         "micro": 16},
        # The experts of one Qwen3-30B-A3B layer in a training pass.
        {"name": "moe_train", "kind": "moe", **_moe(2), "tokens": 4500, "backward": True},
        # A decoding step of a full rollout group: 32 completions, 257th token after a 1024-token prompt.
        {"name": "decode_group", "kind": "decode", **_dense(3, 4, 128256), "n": 32, "prompt": 1024, "own": 257, "fp8": False},
        # A few sequences after a longer prompt with fp8 projections: every byte is a weight.
        {"name": "decode_few_fp8", "kind": "decode", **_dense(3, 4, 128256), "n": 3, "prompt": 3001, "own": 50, "fp8": True},
        # Reference-model scoring of a group (old / reference log-probs before a step).
        {"name": "score_group", "kind": "score", **_dense(3, 2, 128256), "prompt": 512, "group": 16, "length": 300},
        # The LM-head operator at the headline width, training direction.
        {"name": "linear_logp_train", "kind": "linear_logp", "tokens": 8192, "hidden": 4096, "vocab": 128256, "bias": False,
         "backward": True, "entropy": False},
        # A short ragged batch over an odd vocabulary with bias and entropy, evaluation direction.
        {"name": "linear_logp_eval", "kind": "linear_logp", "tokens": 777, "hidden": 2048, "vocab": 50257, "bias": True,
         "backward": False, "entropy": True},
        # Drop-in loss for a trainer that materialises its logits (documented benchmark shape).
        {"name": "loss_logits", "kind": "loss", "batch": 32, "tokens": 256, "vocab": 32768, "dtype": "float16", "group": 8},
        # Rollout sampling of a whole group over the largest vocabulary.
        {"name": "sample_group", "kind": "sample", "rows": 256, "vocab": 151936, "dtype": "float32", "top_k": 50,
         "top_p": 0.9, "temperature": 0.7},
        # Documented shared-prefix shape: 64 sequences of 512 queries over one 4096-token key/value prefix.
        {"name": "attention_prefix", "kind": "attention", "form": "prefix", "batch": 1, "group": 64, "length": 512,
         "prompt": 4096, "heads": 1, "kv_heads": 1, "backward": False},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["train", "train", "moe", "decode", "score", "linear_logp", "loss", "sample", "attention"])
    if kind in ("train", "score"):
        group = _log_int(rng, 4, 32)
        case = {"kind": kind, **_dense(rng.randrange(4), rng.randint(1, 2), rng.choice(VOCABS[:4])),
                "prompt": _log_int(rng, 33, 1024), "group": group, "length": _log_int(rng, 32, 512)}
        if kind == "train":
            case["micro"] = rng.choice([0, 0, max(2, group // 2)])
        return case
    if kind == "moe":
        return {"kind": kind, **_moe(rng.randrange(3)), "tokens": _log_int(rng, 1, 8192), "backward": rng.random() < 0.5}
    if kind == "decode":
        return {"kind": kind, **_dense(rng.randrange(4), rng.randint(1, 4), rng.choice(VOCABS[:4])), "n": _log_int(rng, 1, 64),
                "prompt": _log_int(rng, 17, 4096), "own": _log_int(rng, 1, 512), "fp8": rng.random() < 0.3}
    if kind == "linear_logp":
        return {"kind": kind, "tokens": _log_int(rng, 1, 8192), "hidden": rng.choice([512, 1024, 2048, 3584, 4096]),
                "vocab": rng.choice(VOCABS), "bias": rng.random() < 0.3, "backward": rng.random() < 0.5,
                "entropy": rng.random() < 0.3}
    if kind == "loss":
        vocab = _log_int(rng, 1000, 131072)
        group = rng.choice([2, 4, 8])
        batch = group * _log_int(rng, 1, 32 // group)
        most = max(8, min(512, (1 << 28) // (vocab * batch)))
        return {"kind": kind, "batch": batch, "tokens": _log_int(rng, 8, most), "vocab": vocab,
                "dtype": rng.choice(["float16", "bfloat16", "float32"]), "group": group}
    if kind == "sample":
        return {"kind": kind, "rows": _log_int(rng, 1, 256), "vocab": _log_int(rng, 4096, 151936),
                "dtype": rng.choice(["float32", "bfloat16"]), "top_k": rng.choice([0, 1, 20, 50, 200, 1000]),
                "top_p": rng.choice([1.0, 0.95, 0.9]), "temperature": rng.choice([0.7, 1.0])}
    form = rng.choice(["prefix", "causal", "grouped"])
    heads = 1 if form == "prefix" else rng.choice([8, 16, 32])
    return {"kind": kind, "form": form, "batch": rng.randint(1, 4) if form != "grouped" else 1, "group": _log_int(rng, 2, 32),
            "length": _log_int(rng, 33, 1024), "prompt": _log_int(rng, 65, 4096), "heads": heads,
            "kv_heads": 1 if form == "prefix" else rng.choice([heads // 4, heads]), "backward": rng.random() < 0.5}


# ------------------------------------------------------------------------------------------------ inputs
def _config(c):
    from rl_engine.models.config import ModelConfig

    return ModelConfig("case", c["vocab"], c["hidden"], c["layers"], c["heads"], c["kv_heads"], 128, c["ffn"])


def _gen(seed, device=DEV):
    return torch.Generator(device=device).manual_seed(seed)


def _lengths_mask(rows, length, gen):
    """Completions end early at random places, as sampled ones do: between half and all of the positions are real."""
    ends = torch.randint((length + 1) // 2, length + 1, (rows, 1), generator=gen, device=gen.device)
    return torch.arange(length, device=gen.device)[None, :] < ends


def _model(c, seed, **kw):
    from rl_engine.models.llama import LlamaModel

    return LlamaModel(_config(c), dtype=torch.bfloat16, device=DEV, seed=seed, **kw)


def _prepare_train(c, seed):
    from rl_engine.models.grpo import GRPOBatch, GRPOTrainer, policy_logps, synthetic_batch

    trainer = GRPOTrainer(_model(c, seed), lr=1e-6, micro_group=c["micro"] or "auto")
    gen = _gen(seed + 1, "cpu")
    batch = synthetic_batch(c["vocab"], c["prompt"], c["group"], c["length"], seed=seed)
    with torch.no_grad():  # the rollout's own log-probs, with the small drift of an off-policy step
        now = policy_logps(trainer.model, batch.to(DEV)).float().cpu()
    noise = lambda: 0.01 * torch.randn(now.shape, generator=gen)
    batch = GRPOBatch(batch.prompt_ids, batch.completion_ids, batch.rewards, now + noise(), now + noise(),
                      _lengths_mask(c["group"], c["length"], gen))
    return {"trainer": trainer, "batch": batch.pin()}


def _prepare_moe(c, seed):
    from rl_engine.kernels.registry import kernel_registry

    gen = _gen(seed)
    make = lambda std, *shape: torch.empty(*shape, device=DEV, dtype=torch.bfloat16).normal_(0.0, std, generator=gen) \
        .requires_grad_(c["backward"])
    t, h, e, f = c["tokens"], c["hidden"], c["experts"], c["ffn"]
    wanted = [make(1.0, t, h), make(h ** -0.5, e, h), make(0.02, e * 2 * f, h), make(0.02, e * h, f)]
    return {"op": kernel_registry.get_op("moe"), "args": wanted, "top": c["top"],
            "grad": torch.randn(t, h, device=DEV, generator=gen).to(torch.bfloat16) if c["backward"] else None}


def _prepare_decode(c, seed):
    from rl_engine.kernels.registry import kernel_registry

    model = _model(c, seed)
    if c["fp8"]:
        model.enable_fp8_inference()
    gen = _gen(seed + 1)
    n, p, own, rows = c["n"], c["prompt"], c["own"], c["own"] + 16
    cache = model.new_kv_cache(p + n * rows)
    for k, v in cache:
        k.normal_(generator=gen)
        v.normal_(generator=gen)
    tokens = torch.randint(0, c["vocab"], (n,), device=DEV, generator=gen)
    positions = torch.full((n,), p + own - 1, dtype=torch.long, device=DEV)
    slots = p + torch.arange(n, device=DEV) * rows + own - 1
    prefix_layout, own_layout = model.decode_layouts(n, p, rows, own)
    step = lambda: model.decode_step(tokens, positions, cache, slots, prefix_layout, own_layout)
    step()
    # captured once per rollout and replayed for every token, as the rollout engine does
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        hidden = step()
    return {"graph": graph, "hidden": hidden, "head": model.lm_head_weight().detach(), "lm_head": kernel_registry.get_op("lm_head"),
            "keep": (model, cache, tokens, positions, slots, prefix_layout, own_layout)}


def _prepare_score(c, seed):
    from rl_engine.executors.native_rollout import NativeRolloutEngine

    gen = _gen(seed + 1)
    ids = lambda *shape: torch.randint(0, c["vocab"], shape, device=DEV, generator=gen)
    return {"engine": NativeRolloutEngine(_model(c, seed)), "prompt": ids(c["prompt"]), "completions": ids(c["group"], c["length"])}


def _prepare_linear_logp(c, seed):
    from rl_engine.kernels.registry import kernel_registry

    gen = _gen(seed)
    n, d, v = c["tokens"], c["hidden"], c["vocab"]
    hidden = torch.randn(n, d, device=DEV, generator=gen).to(torch.bfloat16)
    weight = torch.empty(v, d, device=DEV, dtype=torch.bfloat16).normal_(0.0, 0.02, generator=gen)
    bias = 0.1 * torch.randn(v, device=DEV, generator=gen) if c["bias"] else None
    wanted = [t for t in (hidden, weight, bias) if t is not None] if c["backward"] else []
    for t in wanted:
        t.requires_grad_(True)
    # policy-gradient weights of the tokens: advantages of a normalised group over the number of tokens
    grad = torch.randn(n, device=DEV, generator=gen) / n
    return {"op": kernel_registry.get_op("linear_logp"), "hidden": hidden, "weight": weight, "bias": bias, "wanted": wanted,
            "targets": torch.randint(0, v, (n,), device=DEV, generator=gen), "grad": grad}


def _prepare_loss(c, seed):
    from rl_engine.kernels.registry import kernel_registry

    gen = _gen(seed)
    b, t, v, dtype = c["batch"], c["tokens"], c["vocab"], getattr(torch, c["dtype"])
    policy = torch.empty(b, t, v, device=DEV, dtype=dtype).normal_(0.0, 2.0, generator=gen)
    ref = torch.empty_like(policy)
    ids = torch.randint(0, v, (b, t), device=DEV, generator=gen)
    old = torch.empty(b, t, device=DEV)
    for i in range(b):  # sequence by sequence: no fp32 copy of all logits
        x = policy[i].float()
        ref[i] = x + 0.05 * torch.randn(x.shape, device=DEV, generator=gen)
        old[i] = x.gather(-1, ids[i, :, None])[:, 0] - torch.logsumexp(x, -1)
    old += 0.01 * torch.randn(old.shape, device=DEV, generator=gen)
    return {"op": kernel_registry.get_op("grpo_loss"), "policy": policy.requires_grad_(True), "ref": ref, "ids": ids, "old": old,
            "rewards": torch.randn(b, device=DEV, generator=gen), "mask": _lengths_mask(b, t, gen), "group": c["group"]}


def _prepare_sample(c, seed):
    from rl_engine.kernels.sampling import SamplerBackend

    logits = (2.0 * torch.randn(c["rows"], c["vocab"], device=DEV, generator=_gen(seed))).to(getattr(torch, c["dtype"]))
    return {"sampler": SamplerBackend(seed=seed), "logits": logits, "top_k": c["top_k"] or None, "top_p": c["top_p"],
            "temperature": c["temperature"]}


def _prepare_attention(c, seed):
    gen = _gen(seed)
    make = lambda *shape: torch.randn(*shape, device=DEV, generator=gen).to(torch.bfloat16).requires_grad_(c["backward"])
    b, g, l, p, hq, hkv = (c[k] for k in ("batch", "group", "length", "prompt", "heads", "kv_heads"))
    if c["form"] == "prefix":
        q, k, v = make(b, g, l, 128), make(b, p, 128), make(b, p, 128)
    elif c["form"] == "causal":
        q, k, v = make(b, p, hq, 128), make(b, p, hkv, 128), make(b, p, hkv, 128)
    else:
        q, k, v = make(p + g * l, hq, 128), make(p + g * l, hkv, 128), make(p + g * l, hkv, 128)
    return {"form": c["form"], "q": q, "k": k, "v": v, "prompt": p, "group": g, "length": l,
            "grad": torch.randn(q.shape, device=DEV, generator=gen).to(torch.bfloat16) if c["backward"] else None}


_PREPARE = {"train": _prepare_train, "moe": _prepare_moe, "decode": _prepare_decode, "score": _prepare_score, "linear_logp": _prepare_linear_logp,
            "loss": _prepare_loss, "sample": _prepare_sample, "attention": _prepare_attention}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["case"] = case
    return state


# ------------------------------------------------------------------------------------------------ one pass
def _run_train(s):
    trainer = s["trainer"]
    loss = trainer.step(s["batch"])
    opt = trainer.opt
    return {"loss": loss, "weights": trainer.model.flat, "grad": trainer.model.flat_grad, "m": opt.m, "v": opt.v}


def _run_moe(s):
    out = s["op"](*s["args"], s["top"])
    grads = torch.autograd.grad(out, s["args"], s["grad"]) if s["grad"] is not None else ()
    return {"out": out.detach(), "grads": list(grads)}


def _run_decode(s):
    s["graph"].replay()
    return s["lm_head"](s["hidden"], s["head"])


def _run_score(s):
    return s["engine"].score(s["prompt"], s["completions"])


def _run_linear_logp(s):
    args = (s["hidden"], s["weight"], s["targets"], s["bias"])
    logp, entropy = s["op"].with_entropy(*args) if s["case"]["entropy"] else (s["op"](*args), None)
    grads = torch.autograd.grad(logp, s["wanted"], s["grad"]) if s["wanted"] else ()
    return {"logp": logp.detach(), "entropy": entropy, "grads": list(grads)}


def _run_loss(s):
    loss, policy_loss, kl = s["op"](s["policy"], s["ref"], s["ids"], s["old"], s["rewards"], s["mask"], clip_eps=0.2, beta=0.04,
                                    samples_per_prompt=s["group"])
    (grad,) = torch.autograd.grad(loss, [s["policy"]])
    return {"loss": loss.detach(), "policy_loss": policy_loss.detach(), "kl": kl.detach(), "grad": grad}


def _run_sample(s):
    return s["sampler"].sample(s["logits"], top_k=s["top_k"], top_p=s["top_p"], temperature=s["temperature"])


def _run_attention(s):
    from rl_engine.kernels.ops.sm100.attention import grouped_prefix_attention
    from rl_engine.kernels.registry import kernel_registry

    q, k, v = s["q"], s["k"], s["v"]
    if s["form"] == "prefix":
        out = kernel_registry.get_op("prefix_shared_attn")(q, k, v)
    elif s["form"] == "causal":
        out = kernel_registry.get_op("attn")(q, k, v, causal=True)
    else:
        out = grouped_prefix_attention(q, k, v, s["prompt"], s["group"], s["length"])
    grads = torch.autograd.grad(out, [q, k, v], s["grad"]) if s["grad"] is not None else ()
    return {"out": out.detach(), "grads": list(grads)}


_RUN = {"train": _run_train, "moe": _run_moe, "decode": _run_decode, "score": _run_score, "linear_logp": _run_linear_logp, "loss": _run_loss,
        "sample": _run_sample, "attention": _run_attention}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------------ what a pass needs
def _layer_params(c):
    h, q, kv = c["hidden"], c["heads"] * 128, c["kv_heads"] * 128
    return h * (q + 2 * kv) + q * h + 3 * h * c["ffn"]


def _pairs(c):
    """Visible (query, key) pairs of a prompt and the completions after it."""
    p, g, l = c["prompt"], c["group"], c["length"]
    return p * (p + 1) / 2 + g * l * p + g * l * (l + 1) / 2


def work(c):
    kind = c["kind"]
    if kind in ("train", "score"):
        layer = _layer_params(c)
        tokens, scored = c["prompt"] + c["group"] * c["length"], c["group"] * c["length"]
        head = c["vocab"] * c["hidden"]
        forward = 2.0 * (c["layers"] * layer * tokens + head * scored) + 4.0 * 128 * c["heads"] * c["layers"] * _pairs(c)
        params = c["layers"] * layer + 2 * head
        if kind == "score":
            return {"bytes": 2.0 * (c["layers"] * layer + head + tokens * c["hidden"]), "flops": forward}
        # read and write of parameter, residual and both moments, write of the gradient; backward is twice the forward
        # (attention: five products against two)
        return {"bytes": 26.0 * params,
                "flops": 3.0 * forward + 2.0 * 128 * c["heads"] * c["layers"] * _pairs(c)}
    if kind == "moe":
        t, h, e, k, f = (c[x] for x in ("tokens", "hidden", "experts", "top", "ffn"))
        hit = e * (1.0 - (1.0 - k / e) ** t)  # experts that receive a token; a training pass writes every expert's gradient
        weights = 3.0 * h * f
        return {"bytes": 2.0 * (2 * t * h + hit * weights) + (2.0 * (2 * t * h + e * weights) if c["backward"] else 0.0),
                "flops": 2.0 * t * (k * weights + e * h) * (3 if c["backward"] else 1)}
    if kind == "decode":
        layer = _layer_params(c)
        n, keys = c["n"], c["prompt"] + c["n"] * c["own"]
        pairs = n * (c["prompt"] + c["own"])
        size = 1.0 if c["fp8"] else 2.0
        return {"bytes": size * c["layers"] * layer + 2.0 * c["vocab"] * c["hidden"]
                + c["layers"] * 2.0 * 2 * keys * c["kv_heads"] * 128 + 2.0 * n * c["vocab"],
                "flops": 2.0 * n * (c["layers"] * layer + c["vocab"] * c["hidden"]) + 4.0 * 128 * c["heads"] * c["layers"] * pairs}
    if kind == "linear_logp":
        n, d, v = c["tokens"], c["hidden"], c["vocab"]
        return {"bytes": 2.0 * (n * d + v * d) * (2 if c["backward"] else 1), "flops": 2.0 * n * d * v * (3 if c["backward"] else 1)}
    if kind == "loss":
        size = 4 if c["dtype"] == "float32" else 2
        return {"bytes": 3.0 * size * c["batch"] * c["tokens"] * c["vocab"], "flops": 0.0}
    if kind == "sample":
        return {"bytes": float((4 if c["dtype"] == "float32" else 2) * c["rows"] * c["vocab"]), "flops": 0.0}
    b, g, l, p, hq, hkv = (c[k] for k in ("batch", "group", "length", "prompt", "heads", "kv_heads"))
    if c["form"] == "prefix":
        queries, keys, pairs = b * g * l, b * p, b * g * l * p
    elif c["form"] == "causal":
        queries, keys, pairs = b * p, b * p, b * p * (p + 1) / 2
    else:
        queries = keys = p + g * l
        pairs = _pairs(c)
    times = 3.5 if c["backward"] else 1.0
    return {"bytes": 2.0 * 128 * (2 * queries * hq + 2 * keys * hkv) * (2 if c["backward"] else 1),
            "flops": times * 4.0 * 128 * hq * pairs}


def tolerance(c):
    """About four times what each path differs from the same path in 32 or 64 bits on its own inputs (never above 3 %)."""
    kind = c["kind"]
    if kind == "sample":
        return {"differ": 0.004}  # a draw at the edge between two tokens, with sums in another order
    if kind == "loss":  # the gradient is rounded to the logits' type; 32-bit sums otherwise
        return {"rel": {"float16": 3.5e-3, "bfloat16": 7.5e-3, "float32": 2e-5}[c["dtype"]], "max": 0.016}
    if kind == "train":  # measured 1.3 % in the gradient, 1.5 % in its square (the second moment)
        return {"rel": 0.03, "max": 0.9}
    if kind == "decode":  # measured 1.3 %
        return {"rel": 0.03, "max": 0.3}
    if kind == "score":
        return {"rel": 4e-3, "max": 0.0125}
    if kind == "linear_logp":
        return {"rel": 0.0096, "max": 0.27}
    if kind == "moe":
        return {"rel": 0.018, "max": 0.38}
    return {"rel": 0.01, "max": 0.24}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _exact_moe(c, seed):
    s = _prepare_moe(c, seed)
    x, router, w1, w2 = (t.detach().double() for t in s["args"])
    t, e, f, top = c["tokens"], c["experts"], c["ffn"], c["top"]
    probs = torch.softmax(x @ router.t(), dim=-1)
    idx = torch.sort(probs, dim=-1, descending=True, stable=True).indices[:, :top]
    picked = probs.gather(1, idx)
    weight = picked / picked.sum(-1, keepdim=True)
    w1, w2 = w1.view(e, 2 * f, -1), w2.view(e, -1, f)
    out, grad = torch.zeros_like(x), None if s["grad"] is None else s["grad"].double()
    if grad is not None:
        dx, dw1, dw2, dweight = torch.zeros_like(x), torch.zeros_like(w1), torch.zeros_like(w2), torch.zeros_like(weight)
    for i in range(e):
        rows, slot = (idx == i).nonzero(as_tuple=True)
        if rows.numel() == 0:
            continue
        gu = x[rows] @ w1[i].t()
        gate, up = gu[:, :f], gu[:, f:]
        sig = torch.sigmoid(gate)
        act = gate * sig * up
        y, w = act @ w2[i].t(), weight[rows, slot][:, None]
        out.index_add_(0, rows, w * y)
        if grad is None:
            continue
        g = grad[rows]
        dweight[rows, slot] = (g * y).sum(-1)
        dy = w * g
        dw2[i] = dy.t() @ act
        da = dy @ w2[i]
        dgu = torch.cat([da * up * sig * (1 + gate * (1 - sig)), da * gate * sig], dim=1)
        dw1[i] = dgu.t() @ x[rows]
        dx.index_add_(0, rows, dgu @ w1[i])
    if grad is None:
        return {"out": out, "grads": []}
    # the renormalised weights are a softmax over the selected logits
    dlogits = torch.zeros_like(probs).scatter_(1, idx, weight * (dweight - (weight * dweight).sum(-1, keepdim=True)))
    return {"out": out, "grads": [dx + dlogits @ router, dlogits.t() @ x, dw1.flatten(0, 1), dw2.flatten(0, 1)]}


def _exact_linear_logp(c, seed):
    s = _prepare_linear_logp(c, seed)
    hidden, weight = s["hidden"].detach(), s["weight"].detach().double()
    bias = None if s["bias"] is None else s["bias"].detach().double()
    logp, entropy, gh, gw, gb = [], [], [], torch.zeros_like(weight) if c["backward"] else None, 0.0
    for i in range(0, c["tokens"], 512):
        h, ids = hidden[i:i + 512].double(), s["targets"][i:i + 512]
        z = h @ weight.t()
        if bias is not None:
            z += bias
        lse = torch.logsumexp(z, -1)
        logp.append(z.gather(1, ids[:, None])[:, 0] - lse)
        p = torch.exp(z - lse[:, None])
        entropy.append(lse - (p * z).sum(-1))
        if c["backward"]:
            g = s["grad"][i:i + 512].double()[:, None]
            dz = (-g * p).scatter_add_(1, ids[:, None], g)
            gh.append(dz @ weight)
            gw += dz.t() @ h
            gb = gb + dz.sum(0)
    grads = [torch.cat(gh), gw] + ([] if bias is None else [gb]) if c["backward"] else []
    return {"logp": torch.cat(logp), "entropy": torch.cat(entropy) if c["entropy"] else None, "grads": grads}


def _exact_loss(c, seed):
    s = _prepare_loss(c, seed)
    rewards, mask = s["rewards"].double().view(-1, c["group"]), s["mask"].double()
    std = rewards.var(-1, correction=0, keepdim=True).clamp_min(1e-12).sqrt()
    adv = ((rewards - rewards.mean(-1, keepdim=True)) / std).view(-1)
    count = mask.sum()
    policy_loss = kl = 0.0
    grad = torch.empty(s["policy"].shape, dtype=torch.float64, device=DEV)
    for i in range(c["batch"]):
        z, r, ids = s["policy"][i].detach().double(), s["ref"][i].double(), s["ids"][i][:, None]
        lse = torch.logsumexp(z, -1, keepdim=True)
        lp = (z.gather(1, ids) - lse)[:, 0]
        lr = r.gather(1, ids)[:, 0] - torch.logsumexp(r, -1)
        ratio, diff = torch.exp(lp - s["old"][i].double()), lr - lp
        free, clipped = ratio * adv[i], ratio.clamp(0.8, 1.2) * adv[i]
        policy_loss += (-torch.minimum(free, clipped) * mask[i]).sum()
        kl += ((torch.exp(diff) - diff - 1) * mask[i]).sum()
        d = torch.where(free <= clipped, -free, torch.zeros_like(free)) + 0.04 * (1 - torch.exp(diff))
        d = (d * mask[i] / count)[:, None]
        grad[i] = (-d * torch.exp(z - lse)).scatter_add_(1, ids, d)
    return {"loss": (policy_loss + 0.04 * kl) / count, "policy_loss": policy_loss / count, "kl": kl / count, "grad": grad}


def _exact_attention(c, seed):
    s = _prepare_attention(c, seed)
    form, p, g, l = c["form"], c["prompt"], c["group"], c["length"]
    q, k, v = (s[n].detach().double() for n in "qkv")
    grad = None if s["grad"] is None else s["grad"].double()
    if form == "prefix":
        q, k, v = q.unsqueeze(3), k.unsqueeze(2), v.unsqueeze(2)  # one head
        spans = [((b, i), [(b, slice(None))], None) for b in range(c["batch"]) for i in range(g)]
    elif form == "causal":
        spans = [((b, slice(None)), [(b, slice(None))], p) for b in range(c["batch"])]
    else:
        spans = [((slice(0, p),), [(slice(0, p),)], p)]
        spans += [((slice(p + i * l, p + (i + 1) * l),), [(slice(0, p),), (slice(p + i * l, p + (i + 1) * l),)], l) for i in range(g)]
    out, grads = torch.empty_like(q), None if grad is None else [torch.zeros_like(t) for t in (q, k, v)]
    rep = c["heads"] // c["kv_heads"]
    for rows, keys, causal in spans:
        for head in range(c["heads"]):
            kh = head // rep
            kk, vv = (torch.cat([t[at][:, kh] for at in keys]) for t in (k, v))
            qq = q[rows][:, head]
            score = qq @ kk.t() * 128 ** -0.5
            if causal is not None:  # the last `causal` keys are the queries' own
                n = kk.shape[0] - causal
                score[:, n:].masked_fill_(torch.ones(causal, causal, dtype=torch.bool, device=DEV).triu(1), -math.inf)
            prob = torch.softmax(score, -1)
            o = out[rows][:, head] = prob @ vv
            if grad is None:
                continue
            do = (grad.unsqueeze(3) if form == "prefix" else grad)[rows][:, head]
            ds = prob * (do @ vv.t() - (do * o).sum(-1, keepdim=True)) * 128 ** -0.5
            grads[0][rows][:, head] = ds @ kk
            at = 0
            for span in keys:
                m = k[span].shape[0]
                grads[1][span][:, kh] += ds[:, at:at + m].t() @ qq
                grads[2][span][:, kh] += prob[:, at:at + m].t() @ do
                at += m
    if form == "prefix":
        out, grads = out.squeeze(3), grads and [grads[0].squeeze(3), grads[1].squeeze(2), grads[2].squeeze(2)]
    return {"out": out, "grads": grads or []}


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w.double()


def _rotate(x, positions):
    half = 64
    freq = (500000.0 ** (-torch.arange(half, dtype=torch.float32, device=DEV) / half)).double()
    ang = (positions.double()[:, None] * freq)[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], dim=-1)


def _exact_layer(model, c, i, x, positions, attend):
    w = {n: model.view("l%d.%s" % (i, n)).detach() for n in ("attn_norm", "wqkv", "wo", "mlp_norm", "w_gate_up", "w_down")}
    hq, hkv = c["heads"], c["kv_heads"]
    qkv = (_rms(x, w["attn_norm"]) @ w["wqkv"].double().t()).view(x.shape[0], hq + 2 * hkv, 128)
    q, k, v = _rotate(qkv[:, :hq], positions), _rotate(qkv[:, hq:hq + hkv], positions), qkv[:, hq + hkv:]
    x = x + attend(q, k, v).reshape(x.shape[0], -1) @ w["wo"].double().t()
    gu = _rms(x, w["mlp_norm"]) @ w["w_gate_up"].double().t()
    gate, up = gu[:, :c["ffn"]], gu[:, c["ffn"]:]
    return x + (gate * torch.sigmoid(gate) * up) @ w["w_down"].double().t()


def _attend(q, k, v, rep, own=0):
    """Queries over all keys; of the last ``own`` keys each query sees those up to its own."""
    k, v = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    score = torch.einsum("qhd,khd->hqk", q, k) * 128 ** -0.5
    if own:
        score[:, :, -own:].masked_fill_(torch.ones(own, own, dtype=torch.bool, device=DEV).triu(1), -math.inf)
    return torch.einsum("hqk,khd->qhd", torch.softmax(score, -1), v)


def _exact_score(c, seed):
    s = _prepare_score(c, seed)
    model, (g, l), p, rep = s["engine"].model, s["completions"].shape, c["prompt"], c["heads"] // c["kv_heads"]
    tokens = torch.cat([s["prompt"], s["completions"].reshape(-1)])
    positions = torch.cat([torch.arange(p, device=DEV), (p + torch.arange(l, device=DEV)).repeat(g)])

    def attend(q, k, v):
        out = [_attend(q[:p], k[:p], v[:p], rep, p)]
        for i in range(g):
            own = slice(p + i * l, p + (i + 1) * l)
            out.append(_attend(q[own], torch.cat([k[:p], k[own]]), torch.cat([v[:p], v[own]]), rep, l))
        return torch.cat(out)

    with torch.no_grad():
        x = model.view("embed")[tokens].double()
        for i in range(c["layers"]):
            x = _exact_layer(model, c, i, x, positions, attend)
        x = _rms(x, model.view("final_norm"))
        before = p + torch.arange(g * l, device=DEV).view(g, l) - 1
        before[:, 0] = p - 1
        head, logp = model.lm_head_weight().detach().double(), []
        for i in range(g):
            z = x[before[i]] @ head.t()
            logp.append(z.gather(1, s["completions"][i, :, None])[:, 0] - torch.logsumexp(z, -1))
    return torch.stack(logp)


def _exact_decode(c, seed):
    if c["fp8"]:
        return None  # the codes are the framework's own
    s = _prepare_decode(c, seed)
    model, cache, tokens, positions, slots = s["keep"][:5]
    n, p, rep, rows = c["n"], c["prompt"], c["heads"] // c["kv_heads"], c["own"] + 16
    with torch.no_grad():
        x = model.view("embed")[tokens].double()
        for i in range(c["layers"]):
            ck, cv = cache[i][0].double(), cache[i][1].double()

            def attend(q, k, v):
                ck[slots], cv[slots] = k, v
                out = []
                for j in range(n):
                    at = slice(p + j * rows, p + j * rows + c["own"])
                    out.append(_attend(q[j:j + 1], torch.cat([ck[:p], ck[at]]), torch.cat([cv[:p], cv[at]]), rep))
                return torch.cat(out)

            x = _exact_layer(model, c, i, x, positions, attend)
        return _rms(x, model.view("final_norm")) @ model.lm_head_weight().detach().double().t()


_EXACT = {"moe": _exact_moe, "linear_logp": _exact_linear_logp, "loss": _exact_loss, "attention": _exact_attention,
          "score": _exact_score, "decode": _exact_decode}


def exact(case, seed):
    """What ``run`` returns, from plain torch in 64 bits.  Not for a training step (its results are the sums of a whole
    step in 16-bit storage) nor for drawn tokens."""
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None
