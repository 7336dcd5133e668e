"""The work whose speed this framework is judged by: requests as a serving program sends them and prompts as a scoring
program replays them, through the engine's public calls (`NativeEngine.generate_sync`, `NativeEngine.trace_step`).

Two kinds of case:

  generate   requests are submitted together, the engine schedules them (chunked prefill, CUDA-graph decode steps), samples
             and reports; the answer is every token with its log-probabilities.
  prompt     given tokens go through the engine's step function in portions of at most 2048 tokens; the answer is the logits
             after the middle and the last token of every prompt.

The models are the repository's presets with their own widths and heads.  Of the 8B Llama preset only some of the 32
equal layers are built, so that three models fit the card beside each other; a decode step of 8 of them spends about a
fifth of its time in the head and the sampler (32 layers: a sixteenth).  Weights are random, of the scale at which a layer's output is about as large as the
stream it is added to.  Random layers predict nothing, so a `generate` case's head knows one successor for every token
(`_peak`): greedy decoding then has a clear winner at every step, as it mostly has with a trained model, and rounding
does not send two correct implementations down different texts.
"""
from __future__ import annotations

import dataclasses
import math
import random

import numpy as np
import torch

from vllm_tgis_adapter_b200.engine import falerax, ponenex
from vllm_tgis_adapter_b200.engine.core import PRESETS, NativeEngine, cache_block_bytes, make_sampling_params

STEP_TOKENS = 2048          # the engine's default token budget of one step
BLOCK = 32                  # tokens of one cache block
TOPN = 5                    # log-probabilities reported beside each token
TILE = 4096                 # rows of a 64-bit head product at a time
F64 = torch.float64


# ------------------------------------------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # one person, one short question to a small model: nothing but latency and launches
        dict(name="chat-125m", kind="generate", model="125m", layers=12, requests=1, prompt_lo=17, prompt_hi=17, new=16, method="greedy"),
        # the headline shape: 32 requests decode together; weights stream from HBM once a step
        dict(name="decode-8b", kind="generate", model="llama3-8b", layers=8, requests=32, prompt_lo=64, prompt_hi=64, new=32, method="greedy"),
        # a busy server: many requests of mixed length, sampled under typical-p, repetition and length penalty
        dict(name="sampled-8b", kind="generate", model="llama3-8b", layers=8, requests=96, prompt_lo=9, prompt_hi=57, new=16, method="sample"),
        # requests that name four LoRA adapters
        dict(name="adapters-8b", kind="generate", model="llama3-8b", layers=4, requests=24, prompt_lo=20, prompt_hi=90, new=24, method="greedy", adapters=4),
        # a full prefill step of mixed prompts
        dict(name="prompts-8b", kind="prompt", model="llama3-8b", layers=4, requests=6, tokens=2048),
        # one long document in four portions: attention over all that came before
        dict(name="document-8b", kind="prompt", model="llama3-8b", layers=4, requests=1, tokens=8003),
        # mixture of experts behind latent attention: prefill and decode in bf16, prefill in float32
        dict(name="prompts-moe", kind="prompt", model="ponenex-2k", layers=4, requests=5, tokens=2048),
        dict(name="decode-moe", kind="generate", model="ponenex-2k", layers=4, requests=32, prompt_lo=64, prompt_hi=64, new=24, method="greedy"),
        dict(name="prompts-moe-f32", kind="prompt", model="ponenex-1k", layers=4, requests=3, tokens=389, dtype="float32"),
        # attention beside a matrix memory, a selective scan and a decayed memory: prefill and decode
        dict(name="prompts-recurrent", kind="prompt", model="falerax-2k", layers=4, requests=7, tokens=2048),
        dict(name="decode-recurrent", kind="generate", model="falerax-2k", layers=4, requests=32, prompt_lo=64, prompt_hi=64, new=24, method="greedy"),
    ]


def _between(rng: random.Random, lo: int, hi: int) -> int:
    """A whole number, spread evenly over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random) -> dict:
    case = dict(rng.choice(listed()))
    name = case.pop("name")
    if case["kind"] == "prompt":
        most = case["requests"]
        lo = 2100 if name == "document-8b" else max(48, case["tokens"] // 12)
        case["tokens"] = _between(rng, lo, case["tokens"])
        case["requests"] = 1 if name == "document-8b" else rng.randint(1, most + 2)
        return case
    case["requests"] = _between(rng, 33 if name == "sampled-8b" else 1, 4 if name == "chat-125m" else case["requests"])
    case["prompt_hi"] = _between(rng, 12, 200 if name == "chat-125m" else 64 if case["prompt_lo"] == 64 else case["prompt_hi"])
    case["prompt_lo"] = rng.randint(3, case["prompt_hi"])
    case["new"] = rng.randint(max(6, case["new"] // 2), case["new"])
    return case


def _config(case: dict):
    presets = PRESETS if case["model"] in PRESETS else ponenex.PRESETS if case["model"].startswith("ponenex") else falerax.PRESETS
    mc = presets[case["model"]]
    return dataclasses.replace(mc, n_layers=case["layers"], layers=mc.layers and mc.layers[: case["layers"]], dtype=case.get("dtype", "bfloat16"))


def _lengths(case: dict, seed: int) -> list[int]:
    rng = random.Random(seed * 7919 + 13)
    if case["kind"] == "generate":
        return [rng.randint(case["prompt_lo"], case["prompt_hi"]) for _ in range(case["requests"])]
    # cut the tokens at random places, no prompt shorter than 4
    n, total = case["requests"], case["tokens"]
    cuts = sorted(rng.sample(range(total - 4 * n + n - 1), n - 1))
    ends = [c - i for i, c in enumerate(cuts)] + [total - 4 * n]
    return [4 + b - a for a, b in zip([0] + ends[:-1], ends)]


# ----------------------------------------------------------------------------------------------------------- weights
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, *shape, scale: float = 1.0, mean: float = 0.0) -> torch.Tensor:
    return (torch.empty(shape, device="cuda", dtype=torch.float32).normal_(mean, scale, generator=gen)).to(torch.bfloat16)


def _peak(gen, embed: torch.Tensor, next_of: torch.Tensor, size: float) -> torch.Tensor:
    """Head rows N(0, 1 / width) plus, in the row of every token's successor, `size` times the token's unit embedding: logits of
    standard deviation one, and one that stands out."""
    v, w = embed.shape
    head = torch.empty((v, w), device="cuda").normal_(0.0, w ** -0.5, generator=gen)
    head[next_of] += embed.float() / embed.float().norm(dim=1, keepdim=True) * size
    return head.to(torch.bfloat16)


def _next_of(vocab: int, gen) -> torch.Tensor:
    return torch.randperm(vocab, device="cuda", generator=gen)


def _llama_weights(mc, seed: int, peak: float) -> tuple[dict, torch.Tensor]:
    gen, w, h = _gen(seed), {}, mc.hidden
    q, kv = mc.n_q_heads * mc.head_dim, mc.n_kv_heads * mc.head_dim
    w["model.embed_tokens.weight"] = _normal(gen, mc.vocab, h, scale=3.0)
    for i in range(mc.n_layers):
        p = f"model.layers.{i}."
        for name, rows, cols in (("self_attn.q_proj", q, h), ("self_attn.k_proj", kv, h), ("self_attn.v_proj", kv, h), ("self_attn.o_proj", h, q),
                                 ("mlp.gate_proj", mc.ffn, h), ("mlp.up_proj", mc.ffn, h), ("mlp.down_proj", h, mc.ffn)):
            w[p + name + ".weight"] = _normal(gen, rows, cols, scale=1.2 * cols ** -0.5)
        w[p + "input_layernorm.weight"] = _normal(gen, h, scale=0.1, mean=1.0)
        w[p + "post_attention_layernorm.weight"] = _normal(gen, h, scale=0.1, mean=1.0)
    w["model.norm.weight"] = _normal(gen, h, scale=0.1, mean=1.0)
    next_of = _next_of(mc.vocab, gen)
    w["lm_head.weight"] = _peak(gen, w["model.embed_tokens.weight"], next_of, peak)
    # cos | sin of every position, rounded to the model's type as the checkpoint's users do
    inv = 1.0 / (mc.rope_theta ** (torch.arange(0, mc.head_dim, 2, dtype=torch.float32) / mc.head_dim))
    angle = torch.outer(torch.arange(mc.max_model_len, dtype=torch.float32), inv)
    w["tgis.rope_cos_sin"] = torch.cat([angle.cos(), angle.sin()], dim=-1).to(torch.bfloat16)
    return w, next_of


def _ponenex_weights(mc, seed: int, peak: float) -> tuple[dict, torch.Tensor]:
    gen, w = _gen(seed), {}
    for name, shape in ponenex.tensor_shapes(mc).items():
        if len(shape) == 1:
            plain = name.endswith(".norm") and name != "final.norm"
            w[name] = _normal(gen, *shape, scale=0.5 if name.endswith("router.b") else 0.1, mean=1.0 if plain else 0.0)
        elif name != "head":
            # a router that has learned to choose: its logits spread over several units
            w[name] = _normal(gen, *shape, scale=2.8 if name == "embed" else (3.0 if name.endswith("router") else 1.0) * shape[1] ** -0.5)
    next_of = _next_of(mc.vocab, gen)
    w["head"] = _peak(gen, w["embed"], next_of, peak)
    return w, next_of


def _falerax_weights(mc, seed: int, peak: float) -> tuple[dict, torch.Tensor]:
    gen, w = _gen(seed), {}
    for name, shape in falerax.tensor_shapes(mc).items():
        leaf = name.rsplit(".", 1)[-1]
        if ".mu." in name:
            t = torch.rand(shape, device="cuda", generator=gen).to(torch.bfloat16)
        elif leaf == "A_log":
            t = torch.log(torch.arange(1, shape[1] + 1, device="cuda").float()).repeat(shape[0], 1).to(torch.bfloat16)
        elif name.endswith("dt.b"):
            t = _normal(gen, *shape, scale=0.5, mean=-3.0)
        elif leaf == "w0":
            t = _normal(gen, *shape, scale=0.5, mean=-1.0)
        elif leaf in ("u", "D"):
            t = _normal(gen, *shape, scale=0.5)
        elif name.endswith("f.b"):
            t = _normal(gen, *shape, scale=0.5, mean=3.0)
        elif name.endswith(("i.b", "conv.b")):
            t = _normal(gen, *shape, scale=0.1)
        elif name == "final.norm":
            # the head is the embedding table (unit rows times `width`): this brings the logits to a standard deviation of one
            t = _normal(gen, *shape, scale=0.1 * mc.hidden ** -0.5, mean=mc.hidden ** -0.5)
        elif len(shape) == 1:
            t = _normal(gen, *shape, scale=0.1, mean=1.0)
        else:
            t = _normal(gen, *shape, scale=1.0 if name == "embed" else shape[1] ** -0.5)
        w[name] = t
    return w, torch.arange(mc.vocab, device="cuda")   # tied head: every token's clear successor is itself


def _weights(case: dict, seed: int):
    mc = _config(case)
    make = {"llama": _llama_weights, "ponenex": _ponenex_weights, "falerax": _falerax_weights}[mc.arch]
    if case["kind"] == "generate":   # size / sqrt(2) / the logits' deviation of one; sampling needs a winner that stays in the nucleus
        peak = (26.0 if case["method"] == "sample" else 18.0) * mc.hidden ** -0.5
    else:
        peak = 0.0
    return make(mc, 1000 + seed, peak)


def _adapters(case: dict, seed: int) -> list[dict]:
    """Rank-16 adapters over all seven projections of every layer, as a PEFT checkpoint gives them (alpha / r folded into B)."""
    mc, gen, out = _config(case), _gen(500_000 + seed), []
    q, kv = mc.n_q_heads * mc.head_dim, mc.n_kv_heads * mc.head_dim
    sizes = dict(q_proj=(q, mc.hidden), k_proj=(kv, mc.hidden), v_proj=(kv, mc.hidden), o_proj=(mc.hidden, q),
                 gate_proj=(mc.ffn, mc.hidden), up_proj=(mc.ffn, mc.hidden), down_proj=(mc.hidden, mc.ffn))
    for _ in range(case["adapters"]):
        out.append({(i, m): (_normal(gen, 16, c, scale=c ** -0.5), _normal(gen, r, 16, scale=0.1))
                    for i in range(mc.n_layers) for m, (r, c) in sizes.items()})
    return out


# -------------------------------------------------------------------------------------------------- what is measured
def _prompts(case: dict, seed: int) -> list[list[int]]:
    rng = np.random.RandomState((seed * 31 + 7) % 2 ** 31)
    return [rng.randint(0, _config(case).vocab, n).tolist() for n in _lengths(case, seed)]


def _params(case: dict, i: int, vocab: int):
    slot = 1 + i % case["adapters"] if case.get("adapters") else 0
    if case["method"] == "greedy":
        return make_sampling_params(greedy=True, eos_token_id=vocab - 1, min_tokens=case["new"], max_tokens=case["new"], num_logprobs=TOPN, lora_slot=slot)
    return make_sampling_params(greedy=False, temperature=0.9, typical_p=0.9, repetition_penalty=1.05, length_penalty=(8, 1.01), eos_token_id=vocab - 1,
                                min_tokens=case["new"], max_tokens=case["new"], num_logprobs=TOPN, seed=100 + i, lora_slot=slot)


def _steps(prompts: list[list[int]]) -> list[tuple[list, list[str]]]:
    """Portions of at most STEP_TOKENS tokens, in order: (entries, finished requests) of every step."""
    steps, entries, ends, room = [], [], [], STEP_TOKENS
    for i, p in enumerate(prompts):
        at, wanted = 0, (len(p) // 2, len(p) - 1)
        while at < len(p):
            n = min(room, len(p) - at)
            entries.append((f"p{i}", p[at: at + n], [x - at for x in wanted if at <= x < at + n]))
            at, room = at + n, room - n
            if at == len(p):
                ends.append(f"p{i}")
            if room == 0:
                steps.append((entries, ends))
                entries, ends, room = [], [], STEP_TOKENS
    if entries:
        steps.append((entries, ends))
    return steps


def prepare(case: dict, seed: int) -> dict:
    mc, prompts = _config(case), _prompts(case, seed)
    new = case.get("new", 0)
    blocks = max(sum(-(-(len(p) + new) // BLOCK) for p in prompts), -(-mc.max_model_len // BLOCK))
    more = dict(max_loras=case["adapters"], max_lora_rank=16) if case.get("adapters") else {}
    engine = NativeEngine(mc, max_num_seqs=max(len(prompts), 4), max_batched_tokens=STEP_TOKENS, kv_cache_bytes=(blocks + 2) * cache_block_bytes(mc), **more)
    engine.load_weights(_weights(case, seed)[0])
    if case.get("adapters"):
        for s, adapter in enumerate(_adapters(case, seed)):
            engine.load_adapter(s + 1, adapter)
    torch.cuda.synchronize()
    if case["kind"] == "generate":
        return dict(kind="generate", engine=engine, prompts=prompts, params=[_params(case, i, mc.vocab) for i in range(len(prompts))])
    return dict(kind="prompt", engine=engine, steps=_steps(prompts))


def run(state: dict) -> dict:
    engine = state["engine"]
    if state["kind"] == "prompt":
        return {"logits": np.concatenate([engine.trace_step(entries, ends) for entries, ends in state["steps"]])}
    answers = engine.generate_sync(state["prompts"], state["params"])
    return {"tokens": np.array([[o.new_token for o in a] for a in answers], dtype=np.int64),
            "logprobs": np.array([[[v for _, v in o.topn] for o in a] for a in answers], dtype=np.float32)}


# ----------------------------------------------------------------------------------------- what it cannot do without
def _layer_cost(mc, layer: int, tokens: float) -> tuple[float, float]:
    """(weights that `tokens` tokens of one step touch, multiply-adds per token) of one layer, without attention and scans."""
    h = mc.hidden
    if mc.arch == "llama":
        n = h * (mc.n_q_heads + 2 * mc.n_kv_heads) * mc.head_dim + mc.n_q_heads * mc.head_dim * h + 3 * h * mc.ffn
        return n, n
    l = mc.layers[layer]
    if mc.arch == "ponenex":
        mix = h * (l.q_rank + l.kv_rank + l.rot_dim + l.heads) + l.q_rank * l.heads * (l.dim + l.rot_dim) + l.heads * (l.dim + l.vdim) * l.kv_rank + l.heads * l.vdim * h
        shared, one = 3 * h * l.shared_ff + h * l.experts, 3 * h * l.expert_ff
        touched = l.experts * (1 - (1 - l.top / l.experts) ** tokens)
        return mix + shared + touched * one, mix + shared + l.top * one
    if l.kind == "parallel":
        n = h * (2 * l.heads * l.dim + l.kv_heads * (l.dim + l.vdim)) + l.heads * l.vdim * h
        n += h * l.mm_heads * (2 * l.mm_dim + 2 * l.mm_vdim) + l.mm_heads * l.mm_vdim * h
    elif l.kind == "mamba1":
        n = h * 2 * l.inner + l.inner * (2 * l.dt_rank + 2 * l.state) + l.inner * h
    else:
        n = 5 * h * l.heads * l.dim + 2 * h * l.decay_rank
    n += 3 * h * l.ff
    return n, n


def _mix_cost(mc, layer: int) -> tuple[float, float, float]:
    """(cache elements of a token, multiply-adds per visible key, multiply-adds per token of a scan) of one layer."""
    if mc.arch == "llama":
        return 2 * mc.n_kv_heads * mc.head_dim, 2 * mc.n_q_heads * mc.head_dim, 0
    l = mc.layers[layer]
    if mc.arch == "ponenex":
        return l.kv_rank + l.rot_dim, l.heads * (l.dim + l.rot_dim + l.vdim), 0
    if l.kind == "parallel":
        return l.kv_heads * (l.dim + l.vdim), l.heads * (l.dim + l.vdim), 2 * l.mm_heads * l.mm_dim * l.mm_vdim
    if l.kind == "mamba1":
        return 0, 0, 3 * l.inner * l.state
    return 0, 0, 2 * l.heads * l.dim * l.dim


def work(case: dict) -> dict:
    mc, lengths = _config(case), _lengths(case, 0)
    esz = 4 if case.get("dtype") == "float32" else 2
    new, total = case.get("new", 0), sum(lengths)
    passes = [min(STEP_TOKENS, total - at) for at in range(0, total, STEP_TOKENS)] + [len(lengths)] * max(0, new - 1)
    seen = sum(n * (n + 1) / 2 for n in lengths) + sum(n + k + 1 for n in lengths for k in range(new - 1))   # keys under all queries
    reread = sum(n + k + 1 for n in lengths for k in range(new - 1)) + total                              # keys that steps read
    if len(lengths) == 1:
        reread += sum(at for at in range(STEP_TOKENS, total, STEP_TOKENS))
    tokens = total + len(lengths) * max(0, new - 1)
    nbytes = flops = 0.0
    for i in range(mc.n_layers):
        cache, per_key, scan = _mix_cost(mc, i)
        for t in passes:
            nbytes += esz * _layer_cost(mc, i, t)[0]
        nbytes += esz * cache * (reread + tokens)
        flops += 2 * (_layer_cost(mc, i, 1)[1] + scan) * tokens + 2 * per_key * seen
    heads = len(lengths) * (new if new else 2)
    nbytes += esz * mc.vocab * mc.hidden * (new if new else 1) + heads * mc.vocab * 4
    flops += 2.0 * mc.vocab * mc.hidden * heads
    if case.get("adapters"):
        per_layer = 16 * (7 * mc.hidden + 2 * mc.n_kv_heads * mc.head_dim + mc.n_q_heads * mc.head_dim + 3 * mc.ffn)
        nbytes += 2.0 * per_layer * mc.n_layers * min(case["adapters"], len(lengths)) * len(passes)
        flops += 2.0 * per_layer * mc.n_layers * tokens
    return {"bytes": nbytes, "flops": flops}


def tolerance(case: dict):
    """Logits and log-probabilities against another correct implementation at the same precision, about four times what this
    engine is away from `exact` (float32 1.4e-6; bf16 logits 0.005 to 0.007, 0.015 with the recurrent layers, whose softmax-free
    memories carry a rounding along; log-probabilities 0.0014 to 0.003, recurrent 0.013, part of which is the same run twice
    differing by 0.004); `differ`: the rest of one text after a token that fell the other way."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] == "prompt" or case["model"].startswith("falerax"):
        return {"rel": 0.03, "max": 0.3, "differ": 0.005}
    return {"rel": 0.012, "max": 0.15, "differ": 0.005}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, ranges, heads_per_kv, window=0, cap=0.0):
    """q [N, H, d], k [N, G, d], v [N, G, dv] of prompts at `ranges`; causal softmax attention inside every prompt."""
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=F64, device=q.device)
    for a, b in ranges:
        for r0 in range(a, b, 2048):   # rows of scores at a time
            r1 = min(b, r0 + 2048)
            i, j = torch.arange(r0, r1, device=q.device)[:, None], torch.arange(a, r1, device=q.device)[None, :]
            hidden = (j > i) | ((i - j >= window) if window > 0 else (j > i))
            for g in range(k.shape[1]):
                h = slice(g * heads_per_kv, (g + 1) * heads_per_kv)
                s = torch.einsum("qhd,kd->hqk", q[r0:r1, h], k[a:r1, g]) * scale
                if cap > 0:
                    s = cap * torch.tanh(s / cap)
                out[r0:r1, h] = torch.einsum("hqk,kd->qhd", torch.softmax(s.masked_fill(hidden, -math.inf), -1), v[a:r1, g])
    return out


def _turn(x, cos, sin):
    """x [N, H, d]: entry i with entry i + d / 2."""
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos[:, None] - b * sin[:, None], b * cos[:, None] + a * sin[:, None]], -1)


def _llama_hidden(mc, w, tok, pos, ranges, adapters=None, slot=None):
    eps = mc.rms_eps
    table = w["tgis.rope_cos_sin"].cuda().to(F64)[pos]
    cos, sin = table.chunk(2, -1)
    x = w["model.embed_tokens.weight"][tok].to(F64)
    for i in range(mc.n_layers):
        p = f"model.layers.{i}."

        def project(v, name):
            y = v @ w[p + name + ".weight"].to(F64).T
            for s, adapter in enumerate(adapters or []):
                a, b = adapter[i, name.split(".")[1]]
                rows = (slot == s + 1).nonzero()[:, 0]
                y[rows] += (v[rows] @ a.to(F64).T) @ b.to(F64).T
            return y

        h = _rms(x, eps) * w[p + "input_layernorm.weight"].to(F64)
        q = _turn(project(h, "self_attn.q_proj").view(-1, mc.n_q_heads, mc.head_dim), cos, sin)
        k = _turn(project(h, "self_attn.k_proj").view(-1, mc.n_kv_heads, mc.head_dim), cos, sin)
        v = project(h, "self_attn.v_proj").view(-1, mc.n_kv_heads, mc.head_dim)
        o = _attend(q, k, v, mc.head_dim ** -0.5, ranges, mc.n_q_heads // mc.n_kv_heads)
        x = x + project(o.flatten(1), "self_attn.o_proj")
        h = _rms(x, eps) * w[p + "post_attention_layernorm.weight"].to(F64)
        x = x + project(torch.nn.functional.silu(project(h, "mlp.gate_proj")) * project(h, "mlp.up_proj"), "mlp.down_proj")
    return _rms(x, eps) * w["model.norm.weight"].to(F64), w["lm_head.weight"]


def _silu_pair(h, gate, up, down):
    return (torch.nn.functional.silu(h @ gate.to(F64).T) * (h @ up.to(F64).T)) @ down.to(F64).T


def _ponenex_hidden(mc, w, tok, pos, ranges):
    eps = mc.rms_eps
    x = w["embed"][tok].to(F64) * mc.embed_scale
    for i, l in enumerate(mc.layers):
        m = {k.split(".mix.")[1]: v.to(F64) for k, v in w.items() if k.startswith(f"l{i}.mix.")}
        f = {k.split(".mlp.")[1]: v for k, v in w.items() if k.startswith(f"l{i}.mlp.")}
        n = {k.split(".")[1]: 1.0 + v.to(F64) for k, v in w.items() if k.startswith(f"l{i}.norm")}
        angle = pos.to(F64)[:, None] * l.rot_base ** (-torch.arange(0, l.rot_dims, 2, device="cuda", dtype=F64) / l.rot_dims)[None]
        cos, sin = angle.cos(), angle.sin()

        def turn(v):
            return torch.cat([_turn(v[..., : l.rot_dims], cos, sin), v[..., l.rot_dims:]], -1)

        h = _rms(x, eps) * n["norm1"]
        q = ((_rms(h @ m["dq"].T, eps) * m["dq.norm"]) @ m["uq"].T).view(-1, l.heads, l.dim + l.rot_dim)
        kv = h @ m["dkv"].T
        c = _rms(kv[:, : l.kv_rank], eps) * m["dkv.norm"]
        k = torch.cat([(c @ m["uk"].T).view(-1, l.heads, l.dim), turn(kv[:, None, l.kv_rank:]).expand(-1, l.heads, -1)], -1)
        o = _attend(torch.cat([q[..., : l.dim], turn(q[..., l.dim:])], -1), k, (c @ m["uv"].T).view(-1, l.heads, l.vdim), l.scale, ranges, 1, l.window)
        o = (o * torch.sigmoid(h @ m["g"].T)[..., None]).flatten(1) @ m["o"].T
        x = x + mc.residual_mult * _rms(o, eps) * n["norm1b"]
        h = _rms(x, eps) * n["norm2"]
        val, ids = torch.topk(h @ f["router"].to(F64).T + f["router.b"].to(F64), l.top, dim=-1)
        share = torch.softmax(val, -1)
        y = torch.sigmoid(h @ f["shared.sg"].to(F64).T) * _silu_pair(h, f["shared.gate"], f["shared.up"], f["shared.down"])
        for e in range(l.experts):
            rows, k_of = (ids == e).nonzero(as_tuple=True)
            if len(rows):
                y[rows] += share[rows, k_of, None] * _silu_pair(h[rows], f[f"e{e}.gate"], f[f"e{e}.up"], f[f"e{e}.down"])
        x = x + mc.residual_mult * _rms(y, eps) * n["norm2b"]
    return _rms(x, eps) * (1.0 + w["final.norm"].to(F64)), w["head"]


def _by_step(ranges):
    """Rows of equal position in all prompts, first positions first: (rows, whether they are first)."""
    for t in range(max(b - a for a, b in ranges)):
        yield t, [i for i, (a, b) in enumerate(ranges) if a + t < b], [a + t for a, b in ranges if a + t < b]


def _memory(q, k, v, ig, fg, ranges):
    n, heads, d = q.shape
    out = torch.zeros(n, heads, v.shape[2], dtype=F64, device="cuda")
    S = torch.zeros(len(ranges), heads, d, v.shape[2], dtype=F64, device="cuda")
    nrm, mx = torch.zeros(len(ranges), heads, d, dtype=F64, device="cuda"), torch.zeros(len(ranges), heads, dtype=F64, device="cuda")
    for t, seqs, rows in _by_step(ranges):
        s, r = torch.tensor(seqs, device="cuda"), torch.tensor(rows, device="cuda")
        top = torch.maximum(fg[r] + mx[s], ig[r])
        a, b = torch.exp(fg[r] + mx[s] - top), torch.exp(ig[r] - top)
        Sn = a[..., None, None] * S[s] + b[..., None, None] * k[r][..., None] * v[r][..., None, :]
        nn = a[..., None] * nrm[s] + b[..., None] * k[r]
        S[s], nrm[s], mx[s] = Sn, nn, top
        den = torch.maximum((nn * q[r]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out[r] = torch.einsum("shd,shdv->shv", q[r], Sn) / den[..., None]
    return out


def _falerax_hidden(mc, w, tok, pos, ranges):
    eps, F = mc.rms_eps, torch.nn.functional
    x = w["embed"][tok].to(F64)
    first = torch.zeros(len(tok), dtype=torch.bool, device="cuda")
    first[[a for a, _ in ranges]] = True
    for i, l in enumerate(mc.layers):
        m = {k.split(".mix.")[1]: v.to(F64) for k, v in w.items() if k.startswith(f"l{i}.mix.")}
        f = {k.split(".mlp.")[1]: v.to(F64) for k, v in w.items() if k.startswith(f"l{i}.mlp.")}
        n = len(tok)
        if l.kind == "parallel":
            q = _rms((x @ m["left.q"].T).view(n, l.heads, l.dim), eps) * m["left.q.norm"]
            q = q * (1.0 + l.qt_coef * torch.log(torch.div(pos + 1, l.qt_every, rounding_mode="floor").to(F64) + 1.0))[:, None, None]
            k = _rms((x @ m["left.k"].T).view(n, l.kv_heads, l.dim), eps) * m["left.k.norm"]
            o = _attend(q, k, (x @ m["left.v"].T).view(n, l.kv_heads, l.vdim), l.scale, ranges, l.heads // l.kv_heads, cap=l.softcap)
            left = (o.flatten(1) * torch.sigmoid(x @ m["left.g"].T)) @ m["left.o"].T
            ig = l.gate_cap * torch.tanh((x @ m["right.i"].T + m["right.i.b"]) / l.gate_cap)
            fg = F.logsigmoid(l.gate_cap * torch.tanh((x @ m["right.f"].T + m["right.f.b"]) / l.gate_cap))
            shape = (n, l.mm_heads, l.mm_dim)
            o = _memory((x @ m["right.q"].T).view(shape) * l.mm_dim ** -0.5, (x @ m["right.k"].T).view(shape), (x @ m["right.v"].T).view(n, l.mm_heads, l.mm_vdim), ig, fg, ranges)
            right = (_rms(o, eps).flatten(1) * m["right.norm"] * torch.sigmoid(x @ m["right.g"].T)) @ m["right.o"].T
            y = 0.5 * (_rms(left, eps) * m["left.out"] + _rms(right, eps) * m["right.out"])
        elif l.kind == "mamba1":
            z = x @ m["in"].T
            u, z = z[:, : l.inner], z[:, l.inner:]
            conv = torch.zeros_like(u)
            for back in range(l.conv):   # tap conv - 1 - back reads the token `back` before
                old = torch.roll(u, back, 0)
                old[pos < back] = 0.0
                conv += old * m["conv"][:, l.conv - 1 - back]
            u = F.silu(conv + m["conv.b"])
            p = u @ m["x"].T
            dt = F.softplus(p[:, : l.dt_rank] @ m["dt"].T + m["dt.b"])
            B, C = p[:, l.dt_rank: l.dt_rank + l.state], p[:, l.dt_rank + l.state:]
            A, S, y = -torch.exp(m["A_log"]), torch.zeros(len(ranges), l.inner, l.state, dtype=F64, device="cuda"), torch.zeros_like(u)
            for t, seqs, rows in _by_step(ranges):
                s, r = torch.tensor(seqs, device="cuda"), torch.tensor(rows, device="cuda")
                S[s] = torch.exp(dt[r][..., None] * A) * S[s] + (dt[r] * u[r])[..., None] * B[r][:, None]
                y[r] = (S[s] * C[r][:, None]).sum(-1) + m["D"] * u[r]
            y = (y * F.silu(z)) @ m["o"].T
        else:
            prev = torch.roll(x, 1, 0)
            prev[first] = 0.0
            mix = {s: x + (prev - x) * m["mu." + s] for s in "rkvgw"}
            r_, k, v = ((mix[s] @ m[s].T).view(n, l.heads, l.dim) for s in "rkv")
            decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ m["w1"].T) @ m["w2"].T + m["w0"])).view(n, l.heads, l.dim)
            S, o = torch.zeros(len(ranges), l.heads, l.dim, l.dim, dtype=F64, device="cuda"), torch.zeros(n, l.heads, l.dim, dtype=F64, device="cuda")
            for t, seqs, rows in _by_step(ranges):
                s, r = torch.tensor(seqs, device="cuda"), torch.tensor(rows, device="cuda")
                kv = k[r][..., None] * v[r][..., None, :]
                o[r] = torch.einsum("shd,shdv->shv", r_[r], S[s] + m["u"][..., None] * kv)
                S[s] = decay[r][..., None] * S[s] + kv
            y = (_rms(o, eps).flatten(1) * m["norm"] * F.silu(mix["g"] @ m["g"].T)) @ m["o"].T
        x = x + _rms(y, eps) * w[f"l{i}.norm1"].to(F64)
        if l.ff:
            x = x + _rms((F.gelu(x @ f["gate"].T, approximate="tanh") * (x @ f["up"].T)) @ f["down"].T, eps) * w[f"l{i}.norm2"].to(F64)
    return _rms(x, eps) * w["final.norm"].to(F64), w["embed"]


def exact(case: dict, seed: int):
    mc, prompts = _config(case), _prompts(case, seed)
    w, next_of = _weights(case, seed)
    new, wanted, texts, after = case.get("new", 0), [], [], []
    next_of = next_of.tolist()
    for p in prompts:
        text, tokens = list(p), []
        for _ in range(new):   # the text that follows: every token's clear successor
            tokens.append(next_of[text[-1]])
            text.append(tokens[-1])
        texts.append(text[:-1] if new else text)
        after.append(tokens)
    ranges, at = [], 0
    for p, text in zip(prompts, texts):
        ranges.append((at, at + len(text)))
        wanted += [at + len(p) - 1 + k for k in range(new)] if new else [at + len(p) // 2, at + len(p) - 1]
        at += len(text)
    tok = torch.tensor([t for text in texts for t in text], device="cuda")
    pos = torch.tensor([k for text in texts for k in range(len(text))], device="cuda")
    if mc.arch == "llama":
        slot = torch.tensor([1 + i % case["adapters"] if case.get("adapters") else 0 for i, text in enumerate(texts) for _ in text], device="cuda")
        hidden, head = _llama_hidden(mc, w, tok, pos, ranges, _adapters(case, seed) if case.get("adapters") else None, slot)
    else:
        hidden, head = (_ponenex_hidden if mc.arch == "ponenex" else _falerax_hidden)(mc, w, tok, pos, ranges)
    hidden = hidden[torch.tensor(wanted, device="cuda")]
    logits = torch.cat([hidden @ head[r: r + TILE].to(F64).T for r in range(0, mc.vocab, TILE)], -1)
    if not new:
        return {"logits": logits}
    return {"tokens": np.array(after, dtype=np.int64), "logprobs": torch.log_softmax(logits, -1).topk(TOPN, -1).values.view(len(prompts), new, TOPN)}
