"""What the performance of this framework is measured on: the passes of an RL post-training step, through the entry points that a
training program calls.

* ``logprob``: :meth:`NativeEngine.forward_logprob` without gradients (old and reference log-probs of packed sequences).
* ``update``: one micro-batch of the actor update: forward, fused policy loss with a KL term, backward into the engine's fp32
  gradient shard.
* ``rollout``: :meth:`NativeRolloutEngine.generate` on a batch of prompts, some of them shared by several samples: prefill, decode
  steps, sampling; bf16 or block-scaled fp8 weights. The prefix cache is dropped after every batch, as a weight update does.
* ``sample``: :func:`verl_b200.ops.sample` with top-k and top-p restrictions on a decode step's logits.

The models are the architectures that the repository names, cut to a few layers; a step's time is layers x the layer plus the head.
"""

from __future__ import annotations

import math
import random

import torch
import torch.utils.checkpoint

from verl_b200 import ops
from verl_b200.models import PackedBatch, build_model, preset
from verl_b200.rollout.engine import NativeRolloutEngine, SamplingParams
from verl_b200.workers.engine.native import NativeEngine

DEV = "cuda"
KL_COEF, CLIP = 0.001, 0.2


def listed() -> list[dict]:
    return [
        # reference log-probs of a handful of short answers (evaluation, a small batch): the model of the example scripts
        dict(name="logprob_few_short", kind="logprob", model="qwen2.5-0.5b", layers=6, n=3, lo=61, hi=233),
        # a micro-batch of the headline benchmark: 16 384 tokens, prompts and answers of up to 1536 together
        dict(name="logprob_micro_batch", kind="logprob", model="qwen2.5-7b", layers=4, n=14, lo=700, hi=1536),
        # long answers: attention is a large part of the work
        dict(name="logprob_long", kind="logprob", model="llama-3-8b", layers=2, n=2, lo=6001, hi=8190),
        # the same pass on a mixture of experts
        dict(name="logprob_experts", kind="logprob", model="qwen3-30b-a3b", layers=2, n=9, lo=300, hi=1100),
        # actor update on short answers
        dict(name="update_few_short", kind="update", model="qwen2.5-0.5b", layers=6, n=5, lo=90, hi=300),
        # actor update of the headline benchmark's model
        dict(name="update_micro_batch", kind="update", model="qwen2.5-7b", layers=4, n=7, lo=700, hi=1536),
        # actor update of a mixture of experts, routed as the rollout was (router replay)
        dict(name="update_experts", kind="update", model="qwen3-30b-a3b", layers=2, n=7, lo=300, hi=900),
        # one prompt: the latency of a decode step
        dict(name="rollout_one", kind="rollout", model="qwen2.5-0.5b", layers=24, n=1, samples=1, lo=61, hi=61, new=48, fp8=False),
        # the headline benchmark's rollout: 16 prompts, 8 samples each
        dict(name="rollout_group", kind="rollout", model="qwen2.5-7b", layers=4, n=16, samples=8, lo=256, hi=512, new=96, fp8=False),
        # fp8 rollout of an ordinary batch
        dict(name="rollout_fp8", kind="rollout", model="qwen2.5-7b", layers=4, n=12, samples=4, lo=100, hi=700, new=64, fp8=True),
        # rollout of a mixture of experts
        dict(name="rollout_experts", kind="rollout", model="qwen3-30b-a3b", layers=4, n=6, samples=4, lo=100, hi=500, new=48, fp8=False),
        # sampling of a decode step with top-k and top-p
        dict(name="sample_restricted", kind="sample", rows=128, vocab=152064, top_k=50, top_p=0.95),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["logprob", "logprob", "update", "update", "rollout", "rollout", "sample"])
    if kind == "sample":  # vocabularies of the repository's architectures, one row to a full decode batch
        return dict(kind=kind, rows=_log_int(rng, 1, 128), vocab=rng.choice([128256, 151936, 152064]),
                    top_k=rng.choice([-1, 20, 50, 200]), top_p=rng.choice([0.8, 0.9, 0.95]))
    # (model, most layers, most tokens of a logprob / update / rollout's prompts): no draw costs more than the largest listed case
    model, layers, *most = rng.choice([("qwen2.5-0.5b", 6, 16000, 8000, 20000), ("qwen2.5-7b", 4, 14000, 7000, 30000),
                                       ("llama-3-8b", 4, 14000, 7000, 30000), ("qwen3-30b-a3b", 2, 8000, 4000, 8000)])
    if kind == "rollout":
        samples, hi = rng.choice([1, 4, 8]), _log_int(rng, 40, 900)
        n = max(1, min(_log_int(rng, 1, 128 // samples), most[2] // (samples * hi)))
        return dict(kind=kind, model=model, layers=layers, n=n, samples=samples, lo=max(1, hi // rng.choice([1, 2, 4])), hi=hi,
                    new=_log_int(rng, 16, 96), fp8=model != "qwen3-30b-a3b" and rng.random() < 0.3)
    most = most[0 if kind == "logprob" else 1]
    hi = _log_int(rng, 60, 8000 if kind == "logprob" else 4000)
    n = max(1, _log_int(rng, 1, max(1, min(48, most // hi))))
    return dict(kind=kind, model=model, layers=layers, n=n, lo=max(8, hi // rng.choice([1, 2, 4])), hi=hi)


# ------------------------------------------------------------------------------------------------------------ inputs
def _config(case: dict):
    return preset(case["model"], num_hidden_layers=case["layers"])


def _lens(case: dict) -> list[int]:
    """Lengths of the case's sequences (rollout: prompts), ragged, the same for every seed."""
    rng = random.Random(7919 * case["n"] + 31 * case["lo"] + case["hi"])
    return [rng.randint(case["lo"], case["hi"]) for _ in range(case["n"])]


def _responses(case: dict) -> list[int]:
    """How many of each sequence's tokens are the answer: most of them, as in training on long answers."""
    return [max(1, (3 * n) // 4) for n in _lens(case)]


def _generator(seed: int, part: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed((seed * 1000003 + part) % (1 << 62))


def _weights(cfg, seed: int) -> dict:
    """Weights in the engine's layout, bf16. Every layer adds about as much to the residual stream as the embedding brought, attention
    scores have a spread of more than one, and the output matrix gives one token (the same one for tied embeddings) a clear lead:
    greedy continuations don't hang on rounding, while log-probs follow every layer."""
    gen = _generator(seed, 1)

    def normal(*shape, std):
        return torch.empty(shape, dtype=torch.bfloat16, device=DEV).normal_(0.0, std, generator=gen)

    H, L, q, kv, V = cfg.hidden_size, cfg.num_hidden_layers, cfg.num_attention_heads * cfg.head_dim, \
        cfg.num_key_value_heads * cfg.head_dim, cfg.vocab_size
    embed_std = 0.02
    wide = 0.02 * math.sqrt(H)  # spread of a projection of a normed row
    act = wide * wide / (1 + wide)  # about that of silu(gate) * up
    per = embed_std * 0.7 / math.sqrt(L)  # what a sublayer adds per element
    w = {"embed_tokens.weight": normal(V, H, std=embed_std)}
    for i in range(L):
        p = f"layers.{i}."
        w[p + "input_layernorm.weight"] = 1 + normal(H, std=0.1)
        w[p + "post_attention_layernorm.weight"] = 1 + normal(H, std=0.1)
        w[p + "self_attn.qkv_proj.weight"] = normal(q + 2 * kv, H, std=0.02)
        if cfg.attention_bias:
            w[p + "self_attn.qkv_proj.bias"] = normal(q + 2 * kv, std=0.1)
        if cfg.qk_norm:
            w[p + "self_attn.q_norm.weight"] = 1 + normal(cfg.head_dim, std=0.1)
            w[p + "self_attn.k_norm.weight"] = 1 + normal(cfg.head_dim, std=0.1)
        w[p + "self_attn.o_proj.weight"] = normal(H, q, std=per / (0.2 * wide * math.sqrt(q)))
        if cfg.is_moe:
            E, I, k = cfg.num_experts, cfg.moe_intermediate_size, cfg.num_experts_per_tok
            w[p + "mlp.gate.weight"] = normal(E, H, std=0.02)
            w[p + "mlp.gate_up_proj"] = normal(E, 2 * I, H, std=0.02)
            w[p + "mlp.down_proj"] = normal(E, H, I, std=per * math.sqrt(k) / (act * math.sqrt(I)))
        else:
            I = cfg.intermediate_size
            w[p + "mlp.gate_up_proj.weight"] = normal(2 * I, H, std=0.02)
            w[p + "mlp.down_proj.weight"] = normal(H, I, std=per / (act * math.sqrt(I)))
    w["norm.weight"] = 1 + normal(H, std=0.1)
    lead = 9.0 / (0.7 * H)  # a lead of about nine in the logits
    if cfg.tie_word_embeddings:
        w["norm.weight"] *= lead / embed_std
    else:
        w["lm_head.weight"] = (w["embed_tokens.weight"] * (lead / embed_std))[_order(cfg, seed)]
    return w


def _order(cfg, seed: int) -> torch.Tensor:
    """Row j of an untied output matrix points at the embedding of token ``order[j]``."""
    return torch.randperm(cfg.vocab_size, device=DEV, generator=_generator(seed, 5))


def _packed(case: dict, cfg, seed: int) -> dict:
    """Packed sequences with the rows that predict answer tokens, and what the policy loss takes beside the log-probs."""
    lens, resp = _lens(case), _responses(case)
    T = sum(lens)
    gen = _generator(seed, 2)
    ids = torch.randint(0, cfg.vocab_size, (T,), device=DEV, generator=gen)
    ends = torch.tensor(lens).cumsum(0).tolist()
    cu = torch.tensor([0] + ends, dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens])
    # the row before every answer token predicts it
    rows = torch.cat([torch.arange(e - r - (r < n), e - 1, device=DEV) for e, n, r in zip(ends, lens, resp)])
    N = rows.numel()
    adv = torch.cat([torch.full((r - (r == n),), 1.0, device=DEV) * a for n, r, a in
                     zip(lens, resp, torch.randn(len(lens), device=DEV, generator=gen))])
    ref = -math.log(cfg.vocab_size) + 0.3 * torch.randn(N, device=DEV, generator=gen)
    out = dict(batch=PackedBatch(ids, pos, cu, max(lens)), rows=rows, labels=ids[rows + 1], adv=adv, ref=ref,
               mask=torch.ones(N, device=DEV), denom=float(N))
    if cfg.is_moe:  # [layers][T, k] experts that the rollout reported
        out["routing"] = [torch.rand(T, cfg.num_experts, device=DEV, generator=gen).topk(cfg.num_experts_per_tok, -1).indices
                          for _ in range(cfg.num_hidden_layers)]
    return out


def _prompts(case: dict, cfg, seed: int) -> list[list[int]]:
    gen = _generator(seed, 3)
    out = []
    for n in _lens(case):
        out += [torch.randint(0, cfg.vocab_size, (n,), device=DEV, generator=gen).tolist()] * case["samples"]
    return out


def _logits(case: dict, seed: int) -> torch.Tensor:
    """fp32 logits with the long tail of a language model's: a few strong tokens per row, the rest spread widely."""
    gen = _generator(seed, 4)
    x = torch.randn(case["rows"], case["vocab"], device=DEV, generator=gen) * 2.0
    top = torch.randint(0, case["vocab"], (case["rows"], 64), device=DEV, generator=gen)
    return x.scatter_add_(1, top, torch.rand(case["rows"], 64, device=DEV, generator=gen) * 8.0 + 4.0)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "sample":
        B = case["rows"]
        full = lambda v, dt: torch.full((B,), v, dtype=dt, device=DEV)  # noqa: E731
        return dict(kind=kind, logits=_logits(case, seed), temperature=full(0.8, torch.float32), top_k=full(case["top_k"], torch.int32),
                    top_p=full(case["top_p"], torch.float32), seed=seed, step=torch.zeros(1, dtype=torch.long, device=DEV))
    cfg = _config(case)
    if kind == "rollout":
        model = build_model(cfg, device=DEV, init=False)
        model.load_state_dict(_weights(cfg, seed))
        prompts = _prompts(case, cfg, seed)
        longest = case["hi"] + case["new"] + 1
        engine = NativeRolloutEngine(model, max_num_seqs=len(prompts), max_model_len=longest, block_size=16,
                                     num_blocks=len(prompts) * (longest // 16 + 2) + 16,
                                     quantization="fp8" if case["fp8"] else None)
        return dict(kind=kind, engine=engine, prompts=prompts,
                    params=SamplingParams(temperature=0.0, max_tokens=case["new"], ignore_eos=True))
    engine = NativeEngine(cfg, {}, {"lr": 1e-6}, device=DEV, trainable=kind == "update", seed=0,
                          state_dict=_weights(cfg, seed)).initialize()
    return dict(kind=kind, engine=engine, **_packed(case, cfg, seed))


# -------------------------------------------------------------------------------------------------------------- passes
def run(state: dict):
    kind = state["kind"]
    if kind == "sample":
        tokens, logprobs = ops.sample(state["logits"], temperature=state["temperature"], top_k=state["top_k"], top_p=state["top_p"],
                                      seed=state["seed"], step=state["step"])
        return dict(tokens=tokens, logprobs=logprobs)
    engine = state["engine"]
    if kind == "rollout":
        outs = engine.generate(state["prompts"], state["params"])
        engine.clear_kv_cache()
        return dict(tokens=torch.tensor([o.token_ids for o in outs]), logprobs=torch.tensor([o.log_probs for o in outs]))
    if kind == "logprob":
        with engine.eval_mode(), torch.no_grad():
            logp, entropy = engine.forward_logprob(state["batch"], state["rows"], state["labels"], 1.0)
        return dict(logp=logp, entropy=entropy)
    if "routing" in state:  # router replay: the actor sets the recorded experts before the pass and takes them away after it
        for layer, experts in zip(engine.model.layers, state["routing"]):
            layer.mlp.replay_routing = experts
    with engine.train_mode():
        engine.optimizer_zero_grad()
        logp, _ = engine.forward_logprob(state["batch"], state["rows"], state["labels"], 1.0)
        loss, _ = ops.ppo_loss_fused(logp, logp.detach(), state["adv"], state["mask"], ref_logp=state["ref"], clip_low=CLIP,
                                     clip_high=CLIP, kl_coef=KL_COEF, denom=state["denom"])
        loss.backward()
    if "routing" in state:
        for layer in engine.model.layers:
            layer.mlp.replay_routing = None
    return dict(loss=loss.detach(), logp=logp.detach(), grads={n: p.main_grad for n, p in engine.model.named_parameters()})


# ---------------------------------------------------------------------------------------------------------------- work
def work(case: dict) -> dict:
    if case["kind"] == "sample":
        return dict(bytes=4 * case["rows"] * case["vocab"] + 24 * case["rows"], flops=0)
    c = _config(case)
    H, D, Hq, Hk, L = c.hidden_size, c.head_dim, c.num_attention_heads, c.num_key_value_heads, c.num_hidden_layers
    attn_w = H * (Hq + 2 * Hk) * D + Hq * D * H
    expert = 3 * H * (c.moe_intermediate_size if c.is_moe else c.intermediate_size)
    used = attn_w + (H * c.num_experts + expert * c.num_experts_per_tok if c.is_moe else expert)  # per token and layer
    held = attn_w + (H * c.num_experts + expert * c.num_experts if c.is_moe else expert)  # per layer
    head = c.vocab_size * H
    lens = _lens(case)
    pairs = sum(n * (n + 1) // 2 for n in lens)  # causal: query, key
    if case["kind"] != "rollout":
        T, N = sum(lens), sum(r - (r == n) for n, r in zip(lens, _responses(case)))
        flops = 2 * T * L * used + 4 * pairs * Hq * D * L + 2 * N * head
        bytes_ = 2 * (L * held + head + T * H) + 8 * N
        if case["kind"] == "update":  # two products of the backward for one of the forward; fp32 gradients written
            return dict(flops=3 * flops, bytes=bytes_ + 4 * (L * held + head * (1 if c.tie_word_embeddings else 2)))
        return dict(flops=flops, bytes=bytes_)
    # a decode step needs the tokens of the one before it: weights and cache are read once per step
    S, B, new = case["samples"], case["n"] * case["samples"], case["new"]
    wb = 1 if case["fp8"] else 2
    touched = held
    if c.is_moe:  # experts that B tokens reach
        touched = attn_w + H * c.num_experts + expert * c.num_experts * (1 - (1 - c.num_experts_per_tok / c.num_experts) ** B)
    cached = sum(S * (n + j) for n in lens for j in range(1, new)) * 2 * Hk * D * 2 * L
    step_bytes = wb * L * touched + 2 * head
    flops = 2 * (sum(lens) + B * (new - 1)) * L * used + 2 * B * new * head
    flops += 4 * Hq * D * L * (pairs + sum(S * (n + j) for n in lens for j in range(1, new)))
    return dict(flops=flops, bytes=wb * L * held + 2 * head + (new - 1) * step_bytes + cached)


def tolerance(case: dict):
    if case["kind"] == "sample":  # fp32 sums over the vocabulary; a token on the edge of the restricted set may change sides
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.01}
    routed = case["model"] == "qwen3-30b-a3b"  # a token near the edge between two experts may take the other one
    if case["kind"] == "update":  # bf16 activations and operands through every layer and back
        return {"rel": 0.03 if routed else 0.02, "max": 0.9}
    if case["kind"] == "rollout":
        return {"rel": 0.015 if routed or case["fp8"] else 0.002, "max": 0.3, "differ": 0.01}
    return {"rel": 0.006, "max": 0.3} if routed else {"rel": 0.001, "max": 0.05}


# ----------------------------------------------------------------------------------------------------------- 64 bits
def _norm64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _rotate64(x, pos, theta):
    half = x.shape[-1] // 2
    a = pos.double()[:, None] * theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attention64(q, k, v):
    """One sequence, causal; a group of query heads at a time."""
    n, Hq, D = q.shape
    G = Hq // k.shape[1]
    mask = torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1)
    outs = []
    for h in range(k.shape[1]):
        s = torch.einsum("qgd,kd->gqk", q[:, h * G : (h + 1) * G], k[:, h]) * D ** -0.5
        outs.append(torch.einsum("gqk,kd->qgd", torch.softmax(s.masked_fill(mask, float("-inf")), -1), v[:, h]))
    return torch.cat(outs, 1)


def _layer64(c, x, pos, lens, routing, w):
    """One decoder layer on packed rows x [T, H] in 64 bits. ``w``: the layer's weights by their short names."""
    D, nq, nk = c.head_dim, c.num_attention_heads, c.num_key_value_heads
    y = _norm64(x, w["input_layernorm.weight"], c.rms_norm_eps)
    qkv = y @ w["self_attn.qkv_proj.weight"].t()
    if c.attention_bias:
        qkv = qkv + w["self_attn.qkv_proj.bias"]
    q, k, v = (t.reshape(x.shape[0], -1, D) for t in qkv.split([nq * D, nk * D, nk * D], -1))
    if c.qk_norm:
        q, k = _norm64(q, w["self_attn.q_norm.weight"], c.rms_norm_eps), _norm64(k, w["self_attn.k_norm.weight"], c.rms_norm_eps)
    q, k = _rotate64(q, pos, c.rope_theta), _rotate64(k, pos, c.rope_theta)
    ckpt = torch.utils.checkpoint.checkpoint if torch.is_grad_enabled() else (lambda f, *a, use_reentrant: f(*a))
    o = [ckpt(_attention64, *t, use_reentrant=False) for t in zip(q.split(lens), k.split(lens), v.split(lens))]
    x = x + torch.cat(o).reshape(x.shape[0], nq * D) @ w["self_attn.o_proj.weight"].t()
    y = _norm64(x, w["post_attention_layernorm.weight"], c.rms_norm_eps)

    def glu(rows, gate_up, down):
        g, u = (rows @ gate_up.t()).chunk(2, -1)
        return (torch.nn.functional.silu(g) * u) @ down.t()

    if not c.is_moe:
        return x + glu(y, w["mlp.gate_up_proj.weight"], w["mlp.down_proj.weight"])
    probs = torch.softmax(y @ w["mlp.gate.weight"].t(), -1)
    top = probs.topk(c.num_experts_per_tok, -1).indices if routing is None else routing
    weight = probs.gather(1, top)
    if c.norm_topk_prob:
        weight = weight / weight.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(c.num_experts):
        t, slot = (top == e).nonzero(as_tuple=True)
        if t.numel():
            out = out.index_add(0, t, glu(y[t], w["mlp.gate_up_proj"][e], w["mlp.down_proj"][e]) * weight[t, slot][:, None])
    return x + out


def _hidden64(c, w, ids, pos, lens, routing=None):
    """Final-norm rows [T, H]; with gradients, layers are recomputed in the backward."""
    x = w["embed_tokens.weight"][ids]
    for i in range(c.num_hidden_layers):
        p = f"layers.{i}."
        lw = {n[len(p):]: t for n, t in w.items() if n.startswith(p)}
        names = sorted(lw)

        def layer(x, *ts, i=i, names=names):
            return _layer64(c, x, pos, lens, None if routing is None else routing[i], dict(zip(names, ts)))

        ts = [lw[n] for n in names]
        x = torch.utils.checkpoint.checkpoint(layer, x, *ts, use_reentrant=False) if torch.is_grad_enabled() else layer(x, *ts)
    return _norm64(x, w["norm.weight"], c.rms_norm_eps)


def _logp64(h, head, labels):
    logits = h @ head.t()
    lse = torch.logsumexp(logits, -1)
    entropy = lse - (torch.softmax(logits, -1) * logits).sum(-1)
    return logits.gather(1, labels[:, None])[:, 0] - lse, entropy


def exact(case: dict, seed: int):
    if case["kind"] == "sample":  # the draws come from the framework's own counter-based generator
        return None
    c = _config(case)
    low = _weights(c, seed)
    w = {n: t.double() for n, t in low.items()}
    del low
    head = w["embed_tokens.weight"] if c.tie_word_embeddings else w["lm_head.weight"]
    if case["kind"] == "rollout":
        return _rollout64(case, c, w, head, seed)
    s = _packed(case, c, seed)
    ids, pos, lens = s["batch"].input_ids, s["batch"].position_ids, _lens(case)
    if case["kind"] == "logprob":
        with torch.no_grad():
            h = _hidden64(c, w, ids, pos, lens)[s["rows"]]
            parts = [_logp64(a, head, b) for a, b in zip(h.split(1024), s["labels"].split(1024))]
        return dict(logp=torch.cat([a for a, _ in parts]), entropy=torch.cat([b for _, b in parts]))
    for t in w.values():
        t.requires_grad_(True)
    with torch.enable_grad():
        h = _hidden64(c, w, ids, pos, lens, s.get("routing"))[s["rows"]]
        logp = torch.cat([torch.utils.checkpoint.checkpoint(lambda a, b: _logp64(a, head, b)[0], a, b, use_reentrant=False)
                          for a, b in zip(h.split(1024), s["labels"].split(1024))])
        # on policy: the ratio is one, and so is its clipped form; KL by exp(d) - d - 1 with d = ref - logp
        ratio = torch.exp(logp - logp.detach())
        d = s["ref"].double() - logp
        loss = (-s["adv"].double() * ratio + KL_COEF * (torch.exp(d) - d - 1)).sum() / s["denom"]
    loss.backward()
    return dict(loss=loss.detach(), logp=logp.detach(), grads={n: w[n].grad for n in w})


@torch.no_grad()
def _rollout64(case, c, w, head, seed):
    """Greedy continuations: guessed by following the leading token, then checked and scored in one pass over the sequences."""
    prompts, new = _prompts(case, c, seed), case["new"]
    if c.tie_word_embeddings:
        follow = lambda t: t  # noqa: E731
    else:
        nxt = _order(c, seed).argsort().tolist()
        follow = lambda t: nxt[t]  # noqa: E731
    tokens, logprobs = [], []
    for i in range(0, len(prompts), case["samples"]):  # samples of a prompt are the same
        seq = list(prompts[i])
        for _ in range(new):
            seq.append(follow(seq[-1]))
        ids = torch.tensor(seq, device=DEV)
        h = _hidden64(c, w, ids[:-1], torch.arange(len(seq) - 1, device=DEV), [len(seq) - 1])[-new:]
        logits = h @ head.t()
        tokens += [logits.argmax(-1)] * case["samples"]
        logprobs += [torch.log_softmax(logits, -1).gather(1, ids[-new:, None])[:, 0]] * case["samples"]
    return dict(tokens=torch.stack(tokens).cpu(), logprobs=torch.stack(logprobs).cpu())
