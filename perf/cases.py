"""What the speed of this framework is measured on: the phases of a reinforcement-learning step.

    rollout    decode steps (CUDA graph over the paged cache, as the engine replays them) from one row to a full batch, prefill of new
               prompts, prefill that continues cached turns
    training   log-probs of packed sequences, forward + backward with recorded routing and recomputation, the optimizer's update

Sizes are those of `bench.py` and of the presets in `models/config.py`: the MoE model with 16 experts per GPU and the dense ones, cut to
fewer layers so that their share of the vocabulary head stays moderate and several copies fit one GPU.  Everything is bf16 except the
optimizer (fp32 state, bf16 parameters out).

A trained model's residual stream is much larger than what one sublayer adds to it; random initialisation is the other way round.  The
embedding is scaled up for that, which also keeps a near tie between two experts from mattering more than rounding does.
"""
from __future__ import annotations

import math

import torch

from miles_b200 import ops
from miles_b200.engine.kv_cache import KVCache
from miles_b200.models.config import get_config
from miles_b200.models.qwen3 import ForwardMeta, build_model

DEVICE = "cuda"
BLOCK = 64                      # tokens per cache page, the engine's default on a GPU
EMBED_SCALE = 50.0              # embedding rows of unit variance (initialised with 0.02)
MODELS = ("qwen3-30B-A3B", "qwen3-4B", "qwen3-0.6B")
EXPERTS_PER_GPU = 16
LR, BETA1, BETA2, EPS, DECAY, STEP = 1e-6, 0.9, 0.98, 1e-8, 0.1, 7


# ---- the cases ---------------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # the end of a rollout: the longest response of the batch decodes alone (two thirds of a rollout's steps have at most 8 rows)
        dict(name="decode_moe_1", kind="decode", model="qwen3-30B-A3B", layers=12, rows=1, shortest=1801, longest=1801),
        # the tail of a rollout, a handful of responses of unlike length
        dict(name="decode_moe_7", kind="decode", model="qwen3-30B-A3B", layers=12, rows=7, shortest=433, longest=3001),
        # the body of a rollout: 8 prompts x 8 samples minus the first ones that stopped
        dict(name="decode_moe_61", kind="decode", model="qwen3-30B-A3B", layers=12, rows=61, shortest=290, longest=4090),
        # a dense policy with half of its batch still running
        dict(name="decode_dense_19", kind="decode", model="qwen3-4B", layers=12, rows=19, shortest=300, longest=2500),
        # a single short prompt arrives: the latency of the first token
        dict(name="prefill_dense_short", kind="prefill", model="qwen3-4B", layers=6, rows=1, shortest=257, longest=257),
        # the prompts of one rollout batch (256-2048 tokens each)
        dict(name="prefill_moe", kind="prefill", model="qwen3-30B-A3B", layers=12, rows=8, shortest=261, longest=2043),
        # the next turn of multi-turn samples: new tokens behind what the cache holds
        dict(name="extend_moe", kind="extend", model="qwen3-30B-A3B", layers=12, rows=6, shortest=97, longest=900, cached=2500),
        # forward-only log-probs of a packed micro-batch of finished samples
        dict(name="logprob_moe", kind="logprob", model="qwen3-30B-A3B", layers=6, rows=11, shortest=600, longest=3300),
        # forward + backward of a packed micro-batch: recorded routing, full recomputation (the headline recipe)
        dict(name="train_moe", kind="train", model="qwen3-30B-A3B", layers=6, rows=9, shortest=500, longest=2700),
        # long responses of a dense policy
        dict(name="train_dense_long", kind="train", model="qwen3-4B", layers=4, rows=2, shortest=3601, longest=8190),
        # a small policy with a small micro-batch and tied embeddings
        dict(name="train_small", kind="train", model="qwen3-0.6B", layers=4, rows=3, shortest=301, longest=777),
        # the optimizer's update of one rank's shard
        dict(name="adamw", kind="adamw", count=150_000_011),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "extend", "logprob", "train", "train", "adamw"])
    if kind == "adamw":
        return dict(kind=kind, count=_spread(rng, 1_000_003, 150_000_000))
    model = rng.choice(MODELS if kind != "extend" else MODELS[:2])
    if kind == "decode":
        rows, lo = _spread(rng, 1, 64), _spread(rng, 128, 1500)
        return dict(kind=kind, model=model, layers=rng.randint(6, 12), rows=rows, shortest=lo, longest=_spread(rng, lo, 4096))
    if kind == "prefill":
        rows, lo = _spread(rng, 1, 8), _spread(rng, 64, 1000)
        return dict(kind=kind, model=model, layers=rng.randint(4, 8), rows=rows, shortest=lo, longest=_spread(rng, lo, 2048))
    if kind == "extend":
        rows, lo = _spread(rng, 1, 8), _spread(rng, 17, 300)
        return dict(kind=kind, model=model, layers=rng.randint(4, 8), rows=rows, shortest=lo, longest=_spread(rng, lo, 900), cached=_spread(rng, 200, 3000))
    rows, lo = _spread(rng, 2, 8), _spread(rng, 200, 1000)
    return dict(kind=kind, model=model, layers=rng.randint(2, 4), rows=rows, shortest=lo, longest=_spread(rng, lo, 2500))


def _config(case):
    cfg = get_config(case["model"]).with_(num_layers=case["layers"])
    return cfg.with_(num_experts=EXPERTS_PER_GPU) if cfg.is_moe else cfg


def _lengths(case):
    """Ragged lengths from shortest to longest (even over the logarithm), long and short ones mixed."""
    n, a, b = case["rows"], case["shortest"], case["longest"]
    if n == 1:
        return [b]
    ls = [int(round(a * (b / a) ** (i / (n - 1)))) for i in range(n)]
    return [ls[(i * 7 + 3) % n] for i in range(n)] if n % 7 else ls[::-1]


# ---- inputs ------------------------------------------------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _model(case, seed):
    cfg = _config(case)
    model = build_model(cfg, dtype=torch.bfloat16, device=DEVICE, seed=int(seed) % 65521)
    if not cfg.tie_embeddings:
        with torch.no_grad():
            model.embed.mul_(EMBED_SCALE)
    return cfg, model


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEVICE)


def _offsets(lengths):
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    return cu


def _pages(lengths, g):
    """Block tables of sequences whose pages lie in any order: (number of pages, [rows, most pages] int32, flat slots per sequence)."""
    need = [-(-n // BLOCK) for n in lengths]
    order = torch.randperm(sum(need), generator=g, device=DEVICE)
    table = torch.zeros(len(lengths), max(need), dtype=torch.int32, device=DEVICE)
    slots, at = [], 0
    for b, n in enumerate(need):
        mine = order[at:at + n]
        table[b, :n] = mine.to(torch.int32)
        slots.append((mine[:, None] * BLOCK + torch.arange(BLOCK, device=DEVICE)).reshape(-1)[:lengths[b]])
        at += n
    return sum(need), table, slots


def _cache(cfg, pages, g):
    """A paged cache that holds keys and values already: keys of unit variance (they are normed per head), values a little smaller."""
    kv = KVCache(cfg.num_layers, pages, BLOCK, cfg.num_kv_heads, cfg.head_dim, torch.bfloat16, DEVICE)
    for k, v in kv.layers.values():
        k.normal_(0.0, 1.0, generator=g)
        v.normal_(0.0, 0.9, generator=g)
    return kv.layers


def prepare(case, seed):
    g = _generator(seed)
    if case["kind"] == "adamw":
        n = case["count"]
        f32 = dict(dtype=torch.float32, device=DEVICE, generator=g)
        return dict(kind="adamw", master=torch.randn(n, **f32).mul_(0.02), grad=torch.randn(n, **f32).mul_(1e-3), exp_avg=torch.randn(n, **f32).mul_(1e-3),
                    exp_avg_sq=torch.rand(n, **f32).mul_(2e-6), param=torch.empty(n, dtype=torch.bfloat16, device=DEVICE))
    cfg, model = _model(case, seed)
    lengths = _lengths(case)
    kind = case["kind"]
    if kind == "decode":
        # one new token per sequence at position length - 1, everything before it in the cache
        pages, table, slots = _pages(lengths, g)
        tokens = torch.randint(3, cfg.vocab_size, (len(lengths),), generator=g, device=DEVICE, dtype=torch.int32)
        meta = ForwardMeta(positions=_i32([n - 1 for n in lengths]), max_seqlen=1, kv_cache=_cache(cfg, pages, g), block_table=table,
                           seq_lens=_i32(lengths), slot_mapping=torch.stack([s[-1] for s in slots]))
        with torch.no_grad():
            model.logits(model(tokens, meta))        # kernels set up before the capture
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                logits = model.logits(model(tokens, meta))
        return dict(kind=kind, model=model, tokens=tokens, meta=meta, graph=graph, logits=logits)
    total = sum(lengths)
    cu = _offsets(lengths)
    tokens = torch.randint(3, cfg.vocab_size, (total,), generator=g, device=DEVICE, dtype=torch.int32)
    if kind in ("prefill", "extend"):
        before = [0] * len(lengths) if kind == "prefill" else [case["cached"] * (i + 2) // (len(lengths) + 1) for i in range(len(lengths))]
        whole = [a + n for a, n in zip(before, lengths)]
        pages, table, slots = _pages(whole, g)
        meta = ForwardMeta(positions=torch.cat([torch.arange(a, e, dtype=torch.int32, device=DEVICE) for a, e in zip(before, whole)]),
                           max_seqlen=max(lengths), kv_cache=_cache(cfg, pages, g), slot_mapping=torch.cat([s[a:] for s, a in zip(slots, before)]))
        if kind == "prefill":
            meta.cu_seqlens = _i32(cu)
        else:
            meta.block_table, meta.seq_lens, meta.q_lens = table, _i32(whole), _i32(lengths)
            meta.extend = {"cu_q": _i32(cu), "cu_k": _i32(_offsets(whole)), "kv_slots": torch.cat(slots), "max_k": max(whole)}
        return dict(kind=kind, model=model, tokens=tokens, meta=meta, last=torch.tensor([c - 1 for c in cu[1:]], device=DEVICE), before=before)
    meta = ForwardMeta(positions=torch.cat([torch.arange(n, dtype=torch.int32, device=DEVICE) for n in lengths]), cu_seqlens=_i32(cu),
                       max_seqlen=max(lengths), recompute=kind == "train")
    if cfg.is_moe:
        # the experts that the rollout chose, recorded per token and layer
        meta.replay_topk = torch.rand(total, cfg.num_moe_layers, cfg.num_experts, generator=g, device=DEVICE).topk(cfg.moe_topk).indices.to(torch.int32)
    # the responses (the last two thirds of each sequence): row i scores token i + 1
    rows = torch.cat([torch.arange(a + n // 3, a + n - 1, device=DEVICE) for a, n in zip(cu[:-1], lengths)])
    state = dict(kind=kind, model=model, tokens=tokens, meta=meta, rows=rows, targets=tokens[rows + 1].long())
    if kind == "train":
        state["advantage"] = torch.randn(rows.numel(), generator=g, device=DEVICE)
    return state


# ---- one pass ----------------------------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "adamw":
        s = state
        ops.adamw_step(s["master"], s["grad"], s["exp_avg"], s["exp_avg_sq"], lr=LR, beta1=BETA1, beta2=BETA2, eps=EPS, weight_decay=DECAY, step=STEP,
                       param_out=s["param"])
        return {n: s[n] for n in ("master", "exp_avg", "exp_avg_sq", "param")}
    model, meta = state["model"], state["meta"]
    if kind == "decode":
        state["graph"].replay()
        return {"logits": state["logits"], "cache": [list(kv) for kv in meta.kv_cache.values()]}
    if kind in ("prefill", "extend"):
        with torch.no_grad():
            hidden = model(state["tokens"], meta)
            return {"logits": model.logits(hidden[state["last"]]), "cache": [list(kv) for kv in meta.kv_cache.values()]}
    if kind == "logprob":
        with torch.no_grad():
            hidden = model(state["tokens"], meta)
            logp, entropy = model.log_probs(hidden[state["rows"]], state["targets"], 1.0, True)
            return {"logp": logp, "entropy": entropy}
    model.zero_grad(set_to_none=True)
    hidden = model(state["tokens"], meta)
    logp, _ = model.log_probs(hidden[state["rows"]], state["targets"], 1.0)
    loss = -(logp * state["advantage"]).mean()
    loss.backward()
    return {"logp": logp.detach(), "grad": {n: p.grad for n, p in model.named_parameters()}}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------------

def _layer_sizes(cfg):
    """(weights that every token of a layer multiplies, of them those that are read, at one layer)."""
    attn = cfg.hidden_size * (cfg.qkv_size + cfg.q_size)
    if cfg.is_moe:
        expert = 3 * cfg.hidden_size * cfg.moe_ffn_hidden_size
        return attn + cfg.num_experts * cfg.hidden_size + cfg.moe_topk * expert, attn + cfg.num_experts * (cfg.hidden_size + expert)
    ffn = 3 * cfg.hidden_size * cfg.ffn_hidden_size
    return attn + ffn, attn + ffn


def work(case):
    if case["kind"] == "adamw":
        return {"bytes": case["count"] * (4 * 4 + 3 * 4 + 2), "flops": case["count"] * 16}
    cfg, lengths, kind = _config(case), _lengths(case), case["kind"]
    L, head = cfg.num_layers, cfg.hidden_size * cfg.vocab_size
    active, stored = _layer_sizes(cfg)
    row_kv = 2 * 2 * cfg.kv_size                                     # bytes of one token's keys and values in one layer
    if kind == "decode":
        T = len(lengths)
        if cfg.is_moe:
            expert = 3 * cfg.hidden_size * cfg.moe_ffn_hidden_size
            used = cfg.num_experts * (1 - (1 - cfg.moe_topk / cfg.num_experts) ** T)     # experts that some row chooses
            stored -= (cfg.num_experts - used) * expert
        return {"bytes": 2 * (L * stored + head) + L * row_kv * sum(lengths) + 4 * T * cfg.vocab_size,
                "flops": 2 * T * (L * active + head) + 4 * L * cfg.q_size * sum(lengths)}
    T = sum(lengths)
    if kind in ("prefill", "extend"):
        n = len(lengths)
        before = [0] * n if kind == "prefill" else [case["cached"] * (i + 2) // (n + 1) for i in range(n)]
        pairs = sum(q * a + q * (q + 1) / 2 for a, q in zip(before, lengths))
        return {"bytes": 2 * (L * stored + head) + L * row_kv * (T + sum(before)) + 2 * T * cfg.hidden_size + 4 * n * cfg.vocab_size,
                "flops": 2 * (T * L * active + n * head) + 4 * L * cfg.q_size * pairs}
    pairs = sum(n * (n + 1) / 2 for n in lengths)
    scored = sum(n - 1 - n // 3 for n in lengths)
    forward = 2 * (T * L * active + scored * head) + 4 * L * cfg.q_size * pairs
    weights = L * stored + head * (1 if cfg.tie_embeddings else 2)
    if kind == "logprob":
        return {"bytes": 2 * (L * stored + head) + 2 * T * cfg.hidden_size, "flops": forward}
    # the backward's products are twice the forward's (two and a half times for attention); recomputation is the recipe's choice and not counted
    return {"bytes": 2 * 2 * weights + 4 * T * cfg.hidden_size, "flops": 3 * forward + 2 * L * cfg.q_size * pairs}


def tolerance(case):
    # measured against 64 bits, times about four: fp32 sums and a rounded bf16 copy; gradients in bf16 through several layers (up to 0.019, the
    # cap of what can be asked); scores of whole sequences (0.0007); logits and caches after bf16 activations (up to 0.009)
    if case["kind"] == "adamw":
        return {"rel": 1e-5, "max": 1e-2}
    if case["kind"] == "train":
        return {"rel": 0.03, "max": 0.9}
    if case["kind"] == "logprob":
        return {"rel": 0.003, "max": 0.1}
    return {"rel": 0.025, "max": 0.5}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------------

def _norm64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _rope64(x, positions, theta):
    d = x.shape[-1]
    inv = theta ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    ang = positions.double()[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attend64(q, k, v, past):
    """q [n, Hq, D] at positions past, past + 1, ... over k, v [past + n, Hkv, D]."""
    n, hq, d = q.shape
    group = hq // k.shape[1]
    hidden = torch.arange(k.shape[0], device=q.device)[None] > torch.arange(past, past + n, device=q.device)[:, None]
    out = []
    for h in range(k.shape[1]):
        s = q[:, h * group:(h + 1) * group].transpose(0, 1) @ k[:, h].t() / math.sqrt(d)
        out.append(torch.softmax(s.masked_fill(hidden, -math.inf), dim=-1) @ v[:, h])
    return torch.cat(out).transpose(0, 1)


def _ffn64(p, x, cfg, chosen):
    if "mlp.router" not in p:
        gate, up = (x @ p["mlp.w13"].t()).chunk(2, dim=-1)
        return torch.nn.functional.silu(gate) * up @ p["mlp.w2"].t()
    probs = torch.softmax(x @ p["mlp.router"].t(), dim=-1)
    idx = probs.topk(cfg.moe_topk, dim=-1).indices if chosen is None else chosen.long()
    w = probs.gather(1, idx)
    w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(cfg.num_experts):
        token, slot = (idx == e).nonzero(as_tuple=True)
        gate, up = (x[token] @ p["mlp.w13"][e].t()).chunk(2, dim=-1)
        y = torch.nn.functional.silu(gate) * up @ p["mlp.w2"][e].t()
        out = out.index_add(0, token, y * w[token, slot][:, None])
    return out


def _layer64(p, x, cfg, positions, attend, chosen):
    """One layer on the residual stream; `attend(q, k, v)` sees rotated queries and keys."""
    h = _norm64(x, p["ln1"], cfg.rms_eps)
    T = x.shape[0]
    q, k, v = (h @ p["attn.wqkv"].t()).split([cfg.q_size, cfg.kv_size, cfg.kv_size], dim=-1)
    q, k, v = q.view(T, -1, cfg.head_dim), k.view(T, -1, cfg.head_dim), v.view(T, -1, cfg.head_dim)
    q, k = _norm64(q, p["attn.q_norm"], cfg.rms_eps), _norm64(k, p["attn.k_norm"], cfg.rms_eps)
    q, k = _rope64(q, positions, cfg.rope_theta), _rope64(k, positions, cfg.rope_theta)
    x = x + attend(q, k, v).reshape(T, -1) @ p["attn.wo"].t()
    return x + _ffn64(p, _norm64(x, p["ln2"], cfg.rms_eps), cfg, chosen)


def _params64(model):
    """Every parameter in 64 bits by name."""
    return {n: p.detach().double() for n, p in model.named_parameters()}


def _of_layer(params, i):
    pre = f"layers.{i}."
    return {n[len(pre):]: t for n, t in params.items() if n.startswith(pre)}


def exact(case, seed):
    state = prepare(case, seed)
    if case["kind"] == "adamw":
        p, g, m, v = (state[n].double() for n in ("master", "grad", "exp_avg", "exp_avg_sq"))
        m = BETA1 * m + (1 - BETA1) * g
        v = BETA2 * v + (1 - BETA2) * g * g
        p = p * (1 - LR * DECAY) - LR * (m / (1 - BETA1 ** STEP)) / ((v / (1 - BETA2 ** STEP)).sqrt() + EPS)
        return {"master": p, "exp_avg": m, "exp_avg_sq": v, "param": p}
    model, meta, kind = state["model"], state["meta"], case["kind"]
    cfg, lengths = _config(case), _lengths(case)
    if kind in ("decode", "prefill", "extend"):
        with torch.no_grad():
            return _serve64(state, cfg, lengths, model, meta)
    return _score64(state, cfg, lengths, model, meta)


def _serve64(state, cfg, lengths, model, meta):
    new = [1] * len(lengths) if state["kind"] == "decode" else lengths
    before = [n - 1 for n in lengths] if state["kind"] == "decode" else state["before"]
    if state["kind"] == "decode":
        slots = [(meta.block_table[b].long()[:, None] * BLOCK + torch.arange(BLOCK, device=DEVICE)).reshape(-1)[:n] for b, n in enumerate(lengths)]
    elif state["kind"] == "extend":
        slots = list(meta.extend["kv_slots"].split([a + n for a, n in zip(before, new)]))
    else:
        slots = list(meta.slot_mapping.split(new))
    x = model.embed.detach()[state["tokens"].long()].double()
    cache = []
    for i in range(cfg.num_layers):
        p = {n: t.detach().double() for n, t in model.layers[i].named_parameters()}
        kc, vc = (t.double().view(-1, *t.shape[2:]) for t in meta.kv_cache[i])

        def attend(q, k, v, kc=kc, vc=vc):
            kc[meta.slot_mapping], vc[meta.slot_mapping] = k, v
            out, at = [], 0
            for s, a, n in zip(slots, before, new):
                out.append(_attend64(q[at:at + n], kc[s], vc[s], a))
                at += n
            return torch.cat(out)

        x = _layer64(p, x, cfg, meta.positions, attend, None)
        cache.append([t.view(-1, BLOCK, *t.shape[1:]) for t in (kc, vc)])
    if state["kind"] != "decode":
        x = x[state["last"]]
    x = _norm64(x, model.norm.detach().double(), cfg.rms_eps)
    return {"logits": x @ model.head_weight().detach().double().t(), "cache": cache}


def _score64(state, cfg, lengths, model, meta):
    from torch.utils.checkpoint import checkpoint

    train = state["kind"] == "train"
    params = _params64(model)
    del state["model"], model
    for t in params.values():
        t.requires_grad_(train)
    head = params.get("lm_head", params["embed"])

    def attend(q, k, v):
        return torch.cat([_attend64(*qkv, 0) for qkv in zip(q.split(lengths), k.split(lengths), v.split(lengths))])

    def score(h, t, w):
        logits = h @ w.t()
        lse = torch.logsumexp(logits, dim=-1)
        entropy = None if train else lse - (torch.exp(logits - lse[:, None]) * logits).sum(-1)
        return logits.gather(1, t[:, None])[:, 0] - lse, entropy

    with torch.set_grad_enabled(train):
        x = params["embed"][state["tokens"].long()]
        for i in range(cfg.num_layers):
            chosen = meta.replay_topk[:, i] if meta.replay_topk is not None else None
            p = _of_layer(params, i)

            def layer(x, *tensors, names=tuple(p), chosen=chosen):
                return _layer64(dict(zip(names, tensors)), x, cfg, meta.positions, attend, chosen)

            x = checkpoint(layer, x, *p.values(), use_reentrant=False) if train else layer(x, *p.values())
        h = _norm64(x, params["norm"], cfg.rms_eps)[state["rows"]]
        got = [checkpoint(score, a, t, head, use_reentrant=False) if train else score(a, t, head) for a, t in zip(h.split(1024), state["targets"].split(1024))]
        logp = torch.cat([a for a, _ in got])
        if not train:
            return {"logp": logp, "entropy": torch.cat([b for _, b in got])}
        (-(logp * state["advantage"].double()).mean()).backward()
    return {"logp": logp.detach(), "grad": {n: t.grad for n, t in params.items()}}
