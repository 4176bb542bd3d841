"""What the speed of this framework is measured on: the three passes of a GRPO step that run on the GPU for seconds -- the
trainer's forward and backward, scoring of given responses, and rollouts -- through their public entry points, from batches where
launches count to the longest prompts of the recipes.  Models have the widths of the presets and few layers; weights are random.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` / ``run`` make and take one pass, ``exact``
is the same pass in 64 bits and plain torch, ``work`` the bytes and operations that a pass cannot do without.
"""
import dataclasses
import math
import random

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from arctic_platform_b200.engine.sampler import SamplerEngine
from arctic_platform_b200.engine.trainer import EngineConfig, TrainEngine
from arctic_platform_b200.models.config import PRESETS
from arctic_platform_b200.models.decoder import DecoderLM, token_logprobs
from arctic_platform_b200.rl.zorro_train.layout import build_packed_batch, build_plain_packed


# ------------------------------------------------------------------------------------------------- the cases
def listed():
    def train(name, model, layers, prompts, samples, prompt, response, shared=True):
        return {"name": name, "kind": "train", "model": model, "layers": layers, "prompts": prompts, "samples": samples,
                "prompt": prompt, "response": response, "shared": shared}

    def score(name, *a, **k):
        return dict(train(name, *a, **k), kind="score")

    def rollout(name, model, layers, prompts, samples, prompt, response):
        return {"name": name, "kind": "rollout", "model": model, "layers": layers, "prompts": prompts, "samples": samples,
                "prompt": prompt, "response": response}

    return [
        # fine-tuning on a handful of short documents of odd lengths: launches and host work
        train("train-short", "qwen3-0.6b", 2, 1, 3, 0, 333, shared=False),
        # the plumbing model's GRPO batch, ragged: 4 prompts of up to 512 tokens, 8 samples of up to 128
        train("train-tiny-grpo", "qwen3-tiny-d128", 2, 4, 8, 512, 128),
        # a supervised batch of whole documents of uneven length
        train("train-documents", "qwen3-1.7b", 2, 1, 7, 0, 4001, shared=False),
        # a micro-batch of the GRPO benchmark: one prompt, 8 of its samples, 2048 + 2048 tokens
        train("train-grpo", "qwen3-4b", 2, 1, 8, 2048, 2048),
        # long-context recipe: one prompt of 32768 tokens whose samples share it, close to 36864 tokens on the GPU
        train("train-long-prompt", "qwen3-4b", 1, 1, 4, 32768, 1024),
        # mixture of experts: 2 prompts, 4 samples each
        train("train-experts", "qwen3-30b-a3b", 1, 2, 4, 1024, 512),
        # reference log-probabilities of ragged responses
        score("score-ragged", "qwen3-8b", 2, 3, 4, 1500, 1111),
        # one prompt, one answer: latency of a decode step
        rollout("rollout-one", "qwen3-4b", 8, 1, 1, 384, 65),
        # the rollout batch of the GRPO benchmark: 8 prompts of 2048 tokens, 16 samples each
        rollout("rollout-grpo", "qwen3-4b", 6, 8, 16, 2048, 33),
        # distinct prompts of uneven length, one sample each (evaluation)
        rollout("rollout-ragged", "qwen3-1.7b", 8, 41, 1, 1500, 33),
        # mixture of experts, 4 prompts of 512 tokens, 8 samples each
        rollout("rollout-experts", "qwen3-30b-a3b", 2, 4, 8, 512, 33),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("train", "train", "score", "rollout", "rollout"))
    model = rng.choice(("qwen3-0.6b", "qwen3-1.7b", "qwen3-4b", "qwen3-8b", "qwen3-30b-a3b"))
    experts = PRESETS[model].is_moe
    while True:
        if kind == "rollout":
            c = {"kind": kind, "model": model, "layers": rng.randint(1, 3 if experts else 6), "prompts": _log(rng, 1, 48),
                 "samples": rng.choice((1, 1, 4, 8, 16)), "prompt": _log(rng, 24, 2500), "response": rng.choice((17, 33, 49))}
            fits = c["prompts"] * c["samples"] <= 128 and c["prompts"] * c["prompt"] <= 20000
        else:
            shared = rng.random() < 0.7
            c = {"kind": kind, "model": model, "layers": rng.randint(1, 1 if experts else 2),
                 "prompts": _log(rng, 1, 6) if shared else 1, "samples": _log(rng, 2, 12),
                 "prompt": _log(rng, 40, 16384) if shared else 0, "response": _log(rng, 48, 4096), "shared": shared}
            tokens = c["prompts"] * (c["prompt"] + c["samples"] * c["response"])
            fits = tokens <= (8000 if experts else 20000)
        if fits and work(c)["flops"] <= 6e13 and work(c)["bytes"] <= 1.2e11:
            return c


# ------------------------------------------------------------------------------------------------- sizes and data
def _cfg(case):
    return dataclasses.replace(PRESETS[case["model"]], num_layers=case["layers"])


def _lengths(case):
    """Prompt lengths and, per prompt, its samples' response lengths: uneven, the same for every seed."""
    rng = random.Random("%d %d %d %d" % (case["prompts"], case["samples"], case["prompt"], case["response"]))
    even = case["prompt"] in (2048, 32768)                    # the benchmark's prompts all have the full length
    some = lambda most, least: most if even else rng.randint(max(least, most // 3), most)
    prompts = [some(case["prompt"], 1) if case["prompt"] else 0 for _ in range(case["prompts"])]
    if case["kind"] == "rollout":
        return prompts, [[case["response"]] * case["samples"] for _ in prompts]
    return prompts, [[some(case["response"], 2) for _ in range(case["samples"])] for _ in prompts]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)


def _weights(case, seed):
    """Weights by name in the model's layouts (bf16).  Sublayer outputs are scaled so that the last token's embedding stays a
    quarter of the final hidden state or so: the next token is then clear, with a log-probability around -1, and greedy decoding
    does not turn on the last bits."""
    cfg, g = _cfg(case), _gen(seed)
    H, I, L = cfg.hidden_size, cfg.intermediate_size, cfg.num_layers
    n = lambda std, *shape: (torch.randn(*shape, device="cuda", generator=g) * std).to(torch.bfloat16)
    gain = lambda size: (1 + 0.1 * torch.randn(size, device="cuda", generator=g)).to(torch.bfloat16)
    cos = min(0.7, math.log(cfg.vocab_size) / (0.02 * H))
    part = 0.02 * math.sqrt(1 / cos ** 2 - 1) / math.sqrt(2 * L)   # standard deviation of one sublayer's output
    w = {"embed": n(0.02, cfg.vocab_size, H), "final_norm": gain(H)}
    if not cfg.tie_word_embeddings:
        w["lm_head"] = w["embed"].roll(1, 0).contiguous()
    for i in range(L):
        b = "blocks.%d." % i
        w.update({b + "ln1": gain(H), b + "wqkv": n(H ** -0.5, cfg.qkv_size, H), b + "q_norm": gain(cfg.head_dim),
                  b + "k_norm": gain(cfg.head_dim), b + "wo": n(part / 0.6 * cfg.q_size ** -0.5, H, cfg.q_size),
                  b + "ln2": gain(H)})
        if cfg.is_moe:
            E, M = cfg.num_experts, cfg.moe_intermediate_size
            w.update({b + "mlp.router": n(1.5 * H ** -0.5, E, H), b + "mlp.wgu": n(H ** -0.5, E, 2 * M, H),
                      b + "mlp.wdown": n(part / 0.25 * M ** -0.5, E, H, M)})
        else:
            w.update({b + "wgu": n(H ** -0.5, 2 * I, H), b + "wdown": n(part / 0.6 * I ** -0.5, H, I)})
    return w


def _tokens(case, seed):
    """``(prompts, responses)`` as lists of token ids; responses per prompt (none for a rollout)."""
    rng = np.random.default_rng([int(seed), 7])
    plens, rlens = _lengths(case)
    take = lambda k: rng.integers(1, _cfg(case).vocab_size, k, dtype=np.int64)
    prompts = [take(p) for p in plens]
    return prompts, [[] if case["kind"] == "rollout" else [take(r) for r in rs] for rs in rlens]


def _grids(case, prompts, responses):
    """The padded batch that a client sends: prompts on the right edge of theirs, responses on the left edge."""
    P, R = case["prompt"], case["response"]
    rows = [(p, r) for p, rs in zip(prompts, responses) for r in rs]
    ids = torch.zeros((len(rows), P + R), dtype=torch.int64)
    mask = torch.zeros_like(ids)
    for i, (p, r) in enumerate(rows):
        ids[i, P - len(p):P], mask[i, P - len(p):P] = torch.from_numpy(p), 1
        ids[i, P:P + len(r)], mask[i, P:P + len(r)] = torch.from_numpy(r), 1
    return ids, mask


def _predictions(case):
    """Scored tokens: all of a response, or all but the first of a document without a prompt."""
    return sum(sum(rs) - (0 if p else len(rs)) for p, rs in zip(*_lengths(case)))


def _advantages(case, seed):
    g = _gen(seed + 17)
    n = _predictions(case)
    return torch.randn(n, device="cuda", generator=g) / n


# ------------------------------------------------------------------------------------------------- one pass
def prepare(case, seed):
    cfg = _cfg(case)
    model = DecoderLM(cfg, "cuda", torch.bfloat16)
    w = _weights(case, seed)
    with torch.no_grad():
        for name, p in model.named_parameters():
            p.copy_(w[name])
    model.rope("cuda")
    prompts, responses = _tokens(case, seed)
    if case["kind"] == "rollout":
        plens, rlens = _lengths(case)
        longest, count = max(plens) + case["response"], sum(len(r) for r in rlens)
        pages = sum((p + 16) // 16 + len(r) * (case["response"] // 16 + 2) for p, r in zip(plens, rlens))
        engine = SamplerEngine(cfg, "cuda", model=model, kv_cache_tokens=16 * (pages + 64), max_batch=max(8, count),
                               max_seq_len=longest + 16)
        return {"case": case, "engine": engine, "prompts": [p.tolist() for p in prompts],
                "params": {"n": case["samples"], "temperature": 0.0, "max_tokens": case["response"], "ignore_eos": True}}
    ids, mask = _grids(case, prompts, responses)
    packed = (build_packed_batch(ids, mask, case["response"]) if case["shared"] else build_plain_packed(ids, mask)).to("cuda")
    state = {"case": case, "model": model, "packed": packed}
    if case["kind"] == "train":
        state["engine"] = TrainEngine(model, EngineConfig.from_ds_config({"gradient_clipping": 1.0}))
        state["advantages"] = _advantages(case, seed)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "rollout":
        out = state["engine"].generate(state["prompts"], state["params"])
        return {"tokens": np.array([r["token_ids"] for r in out]), "logprobs": np.array([r["logprobs"] for r in out])}
    if kind == "score":
        with torch.no_grad():
            lp, entropy = token_logprobs(state["model"], state["packed"])
        return {"logprobs": lp, "entropy": entropy}
    engine = state["engine"]
    engine.zero_grad()
    lp, entropy = token_logprobs(state["model"], state["packed"])
    engine.backward(-(lp * state["advantages"]).sum())
    return {"logprobs": lp.detach(), "entropy": entropy.detach(),
            "grads": {name: p.grad_f32 for name, p in state["model"].named_parameters()}}


def _attended(case):
    """(query, key) pairs of one layer's attention, each prompt once."""
    pairs = 0
    for p, rs in zip(*_lengths(case)):
        pairs += p * (p + 1) // 2
        if case["kind"] != "rollout":
            pairs += sum(r * p + r * (r + 1) // 2 for r in rs)
    return pairs


def work(case):
    cfg, L = _cfg(case), case["layers"]
    H, D = cfg.hidden_size, cfg.head_dim
    plens, rlens = _lengths(case)
    attn = cfg.qkv_size * H + H * cfg.q_size
    expert = 3 * H * cfg.moe_intermediate_size
    active = attn + (cfg.num_experts_per_tok * expert + cfg.num_experts * H if cfg.is_moe else 3 * H * cfg.intermediate_size)
    kept = attn + (cfg.num_experts * (expert + H) if cfg.is_moe else 3 * H * cfg.intermediate_size)
    head = cfg.vocab_size * H
    pairs = 4 * cfg.num_heads * D * _attended(case) * L
    if case["kind"] != "rollout":
        tokens = sum(plens) + sum(sum(r) for r in rlens)
        preds = _predictions(case)
        flops = 2 * (active * L * tokens + head * preds) + pairs
        params = kept * L + head * (1 if cfg.tie_word_embeddings else 2)
        if case["kind"] == "score":
            return {"bytes": 2 * params + 8 * preds, "flops": flops}
        return {"bytes": 6 * params + 8 * preds, "flops": 3 * flops + pairs // 2}
    steps, count, prompt = case["response"] - 1, sum(len(r) for r in rlens), sum(plens)
    kv = 4 * cfg.num_kv_heads * D * L                          # bytes of one token's keys and values
    own = count * steps * (steps + 1) // 2
    used = attn + min(cfg.num_experts, count * cfg.num_experts_per_tok) * expert + cfg.num_experts * H if cfg.is_moe else kept
    return {"bytes": 2 * (kept * L + head) + kv * prompt + steps * (2 * (used * L + head) + kv * prompt) + kv * own,
            "flops": 2 * (active * L * (prompt + count * steps) + head * count * (steps + 1)) + pairs
            + 4 * cfg.num_heads * D * L * (steps * sum(p * len(r) for p, r in zip(plens, rlens)) + own)}


def tolerance(case):
    """About four times the distance to ``exact`` that was measured.  bf16 operands and activations: 1.3e-2 on gradients, 7e-3 on
    entropies, 9e-3 on the small log-probabilities of a rollout.  With experts a few rows choose the other one of two nearly
    equal experts: 5.5e-2 on gradients, 2.5e-2 on log-probabilities."""
    if PRESETS[case["model"]].is_moe:
        return {"rel": 0.25 if case["kind"] == "train" else 0.1}
    return {"rel": {"train": 0.05, "score": 0.03, "rollout": 0.04}[case["kind"]]}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, pos, theta):
    half = x.shape[-1] // 2
    ang = pos.double()[:, None] * theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, first):
    """Rows ``q [n, rep, D]`` of one K/V head; row ``i`` sees the keys up to ``first + i``."""
    s = torch.einsum("nrd,kd->rnk", q, k) / math.sqrt(q.shape[-1])
    seen = torch.arange(k.shape[0], device=q.device)[None] <= first + torch.arange(q.shape[0], device=q.device)[:, None]
    return torch.einsum("rnk,kd->nrd", torch.softmax(s.masked_fill(~seen, -math.inf), -1), v)


def _keep(fn, *args):
    return checkpoint(fn, *args, use_reentrant=False) if torch.is_grad_enabled() else fn(*args)


def _segment(q, k, v, first, rows=1024):
    """Attention of consecutive rows ``q [n, Hq, D]`` whose first one has ``first`` keys before it."""
    n, rep = q.shape[0], q.shape[1] // k.shape[1]
    heads = []
    for h in range(k.shape[1]):
        mine = q[:, h * rep:(h + 1) * rep]
        heads.append(torch.cat([_keep(_attend, mine[a:a + rows], k[:first + min(n, a + rows), h], v[:first + min(n, a + rows), h],
                                      first + a) for a in range(0, n, rows)]))
    return torch.cat(heads, 1)


def _mlp(h, w, b, cfg):
    if not cfg.is_moe:
        gu = h @ w[b + "wgu"].T
        return (torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ w[b + "wdown"].T
    p, e = torch.topk(torch.softmax(h @ w[b + "mlp.router"].T, -1), cfg.num_experts_per_tok, -1)
    p, out = p / p.sum(-1, keepdim=True), torch.zeros_like(h)
    for i in range(cfg.num_experts):
        row, place = (e == i).nonzero(as_tuple=True)
        if len(row):
            gu = h[row] @ w[b + "mlp.wgu"][i].T
            y = (torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ w[b + "mlp.wdown"][i].T
            out = out.index_add(0, row, y * p[row, place][:, None])
    return out


def _layer(x, w, i, cfg, pos, attention):
    b, D, q_size = "blocks.%d." % i, cfg.head_dim, cfg.q_size
    qkv = (_rms(x, w[b + "ln1"], cfg.rms_norm_eps) @ w[b + "wqkv"].T).view(len(x), -1, D)
    q, k, v = qkv.split([cfg.num_heads, cfg.num_kv_heads, cfg.num_kv_heads], 1)
    q = _rotate(_rms(q, w[b + "q_norm"], cfg.rms_norm_eps), pos, cfg.rope_theta)
    k = _rotate(_rms(k, w[b + "k_norm"], cfg.rms_norm_eps), pos, cfg.rope_theta)
    x = x + attention(i, q, k, v).reshape(len(x), q_size) @ w[b + "wo"].T
    return x + _mlp(_rms(x, w[b + "ln2"], cfg.rms_norm_eps), w, b, cfg)


def _head_rows(h, w, labels):
    z = torch.log_softmax(h @ w.T, -1)
    return z.gather(1, labels[:, None])[:, 0], -(z.exp() * z).sum(-1)


def _exact_pass(case, seed):
    """Log-probabilities, entropies and (training) gradients; the packed axis holds every prompt once, then its responses."""
    cfg, train = _cfg(case), case["kind"] == "train"
    w = {k: t.double().requires_grad_(train) for k, t in _weights(case, seed).items()}
    prompts, responses = _tokens(case, seed)
    ids, pos, segments, rows, labels = [], [], [], [], []
    at = 0
    for p, rs in zip(prompts, responses):
        start = at
        if len(p):
            ids.append(p)
            pos.append(np.arange(len(p)))
            segments.append((at, len(p), at, 0))
            at += len(p)
        for r in rs:
            ids.append(r)
            pos.append(len(p) + np.arange(len(r)))
            segments.append((at, len(r), start, len(p)))
            rows.append(np.concatenate([[start + len(p) - 1], at + np.arange(len(r) - 1)]) if len(p) else at + np.arange(len(r) - 1))
            labels.append(r if len(p) else r[1:])
            at += len(r)
    dev = lambda parts: torch.from_numpy(np.concatenate(parts)).cuda()
    ids, pos, rows, labels = dev(ids), dev(pos), dev(rows), dev(labels)

    def attention(i, q, k, v):
        out = []
        for s, n, start, before in segments:
            kk, vv = (torch.cat([t[start:start + before], t[s:s + n]]) for t in (k, v))
            out.append(_segment(q[s:s + n], kk, vv, before))
        return torch.cat(out)

    with torch.set_grad_enabled(train):
        x = w["embed"][ids]
        for i in range(cfg.num_layers):
            x = _keep(lambda x, i=i: _layer(x, w, i, cfg, pos, attention), x)
        h = _rms(x, w["final_norm"], cfg.rms_norm_eps)[rows]
        head = w.get("lm_head", w["embed"])
        parts = [_keep(_head_rows, h[a:a + 2048], head, labels[a:a + 2048]) for a in range(0, len(rows), 2048)]
        lp, entropy = (torch.cat(t) for t in zip(*parts))
    out = {"logprobs": lp.detach(), "entropy": entropy.detach()}
    if train:
        (lp * _advantages(case, seed).double()).sum().neg().backward()
        out["grads"] = {name: t.grad for name, t in w.items()}
    return out


def _exact_rollout(case, seed):
    """Greedy decoding; the samples of a prompt are equal, so each prompt is decoded once."""
    cfg = _cfg(case)
    w = {k: t.double() for k, t in _weights(case, seed).items()}
    prompts, _ = _tokens(case, seed)
    lens = [len(p) for p in prompts]
    steps, kvshape = case["response"], (cfg.num_kv_heads, cfg.head_dim)
    new = lambda p: torch.zeros(p + steps, *kvshape, device="cuda", dtype=torch.float64)
    kc, vc = ([[new(p) for p in lens] for _ in range(cfg.num_layers)] for _ in range(2))
    ids = torch.from_numpy(np.concatenate(prompts)).cuda()
    pos = torch.from_numpy(np.concatenate([np.arange(p) for p in lens])).cuda()
    ends = torch.tensor(lens, device="cuda").cumsum(0)
    head = w.get("lm_head", w["embed"])

    def prompt_attention(i, q, k, v):
        out, at = [], 0
        for s, n in enumerate(lens):
            kc[i][s][:n], vc[i][s][:n] = k[at:at + n], v[at:at + n]
            out.append(_segment(q[at:at + n], k[at:at + n], v[at:at + n], 0))
            at += n
        return torch.cat(out)

    def step_attention(i, q, k, v):
        out = []
        for s, n in enumerate(lens):
            m = n + done - 1
            kc[i][s][m], vc[i][s][m] = k[s], v[s]
            out.append(_segment(q[s:s + 1], kc[i][s][:m + 1], vc[i][s][:m + 1], m))
        return torch.cat(out)

    tokens, logprobs = [], []
    for done in range(steps):
        x = w["embed"][ids]
        for i in range(cfg.num_layers):
            x = _layer(x, w, i, cfg, pos, step_attention if done else prompt_attention)
        if not done:
            x = x[ends - 1]
        lp, ids = torch.log_softmax(_rms(x, w["final_norm"], cfg.rms_norm_eps) @ head.T, -1).max(-1)
        tokens.append(ids)
        logprobs.append(lp)
        pos = torch.tensor(lens, device="cuda") + done
    each = lambda t: torch.stack(t, 1).repeat_interleave(case["samples"], 0)
    return {"tokens": each(tokens), "logprobs": each(logprobs)}


def exact(case, seed):
    if case["kind"] == "rollout":
        with torch.no_grad():
            return _exact_rollout(case, seed)
    return _exact_pass(case, seed)
