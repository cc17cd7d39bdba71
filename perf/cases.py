"""Workloads by which the speed of the framework is followed from change to change.

A case is one call of a user's program: a decode step of `DecodeSession` (inputs from the host, the chosen tokens back), a
prompt through an engine's `prefill`, or one call of the token sampler.  Models are the presets that the benchmarks use,
with random weights and fewer layers than a whole model: "flash" (three layers, so that the window, the compressed source,
the index and its selection all take part), "genesun-1b / -7b" and "belasun-1b / -7b".

Weights are drawn so that a result does not hang on one rounding, as a trained model's do not: the first columns of the
embedding hold a code that only the routers read and nothing writes to, tokens whose routes are nearly tied are left out, and
the output head prefers one successor of every token.  All requests of a decode case are at different places of one stream of
tokens, each with a cache of its own.
"""
from __future__ import annotations

import math

import torch

from ds41rt_b200.models import registry
from ds41rt_b200.ops.sampling import RowParams, pack_params, sample_rows
from ds41rt_b200.runtime.session import DecodeSession

CODE = 64                # columns of the embedding that the routers read
MARGIN = 0.02            # least distance of the last chosen expert from the next one, in standard deviations
LAYERS = {"flash": 3, "genesun-1b": 8, "genesun-7b": 4, "belasun-1b": 8, "belasun-7b": 4}
ACTIVE_BYTES = {"bf16": 2.0, "mxfp8": 1.0, "mxfp4": 0.53125, "nvfp4": 0.5625}


# ---------------------------------------------------------------------------------------------------- the cases
def _prompt(name, model, tokens, chunk, experts="bf16", kv="bf16"):
    return {"name": name, "kind": "prompt", "model": model, "tokens": tokens, "chunk": chunk, "experts": experts, "kv": kv}


def _decode(name, model, requests, context, each=1, experts="bf16", kv="bf16"):
    return {"name": name, "kind": "decode", "model": model, "requests": requests, "context": context, "each": each,
            "experts": experts, "kv": kv}


def listed():
    return [
        # one user's chat: a token at a time, the smallest and most frequent call of the flagship model
        _decode("flash decode 1", "flash", 1, 4096, experts="mxfp8"),
        # the verification pass of a speculative round: the anchor and four drafts of one request
        _decode("flash verify 5", "flash", 1, 4096, each=5, experts="mxfp8"),
        # a small server: sixteen conversations of different lengths, official FP4 experts, FP8 cache
        _decode("flash decode 16", "flash", 16, 3000, experts="mxfp4", kv="fp8"),
        # a busy server: 64 requests, NVFP4 experts and activations, FP8 cache
        _decode("flash decode 64", "flash", 64, 2048, experts="nvfp4", kv="fp8"),
        # a question of a few hundred tokens: one ragged pass
        _prompt("flash prompt 333", "flash", 333, 2048, experts="mxfp8"),
        # a document in one pass, the prompt benchmark's size
        _prompt("flash prompt 8192", "flash", 8192, 8192, experts="mxfp8"),
        # layer-stack models: single decode, batched decode, long and ragged prompts
        _decode("genesun-1b decode 1", "genesun-1b", 1, 4096),
        _decode("belasun-1b decode 8", "belasun-1b", 8, 4096),
        _decode("genesun-7b decode 32", "genesun-7b", 32, 2048),
        _prompt("genesun-7b prompt 4096", "genesun-7b", 4096, 2048),
        _prompt("belasun-7b prompt 3001", "belasun-7b", 3001, 2048),
        # one sampled token for each of sixteen requests over the vocabulary
        {"name": "sample 16", "kind": "sample", "rows": 16, "vocab": 129280},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "sample"])
    if kind == "sample":
        return {"kind": "sample", "rows": _spread(rng, 1, 64), "vocab": rng.choice([129280, 65536, _spread(rng, 30000, 129280)])}
    model = rng.choice(["flash", "flash", "flash", "genesun-1b", "genesun-7b", "belasun-1b", "belasun-7b"])
    experts = rng.choice(["mxfp8", "mxfp8", "mxfp4", "nvfp4"]) if model == "flash" else "bf16"
    kv = rng.choice(["bf16", "fp8"]) if model == "flash" else "bf16"
    if kind == "prompt":
        c = _prompt("", model, _spread(rng, 64, 4096), rng.choice([1024, 2048]), experts, "bf16")
    elif model == "flash" and rng.random() < 0.3:
        c = _decode("", model, 1, _spread(rng, 64, 4096), rng.randint(2, 6), experts, kv)
    else:
        c = _decode("", model, _spread(rng, 1, 64), _spread(rng, 64, 4096), 1, experts, kv)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------------- models
def _config(case):
    family, cfg = registry.preset(case["model"], LAYERS[case["model"]])
    return family, cfg


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _code(embed, gen):
    """Write every token's code into the first columns of the embedding."""
    shape = (embed.shape[0], CODE)
    embed[:, :CODE] = (torch.randint(0, 2, shape, generator=gen, device=embed.device) * 2 - 1).to(embed.dtype)


def _steady(embed, gates, top):
    """Tokens whose routes are decided by a clear margin in every layer."""
    code = embed[:, :CODE].float()
    fine = torch.ones(embed.shape[0], dtype=torch.bool, device=embed.device)
    for g in gates:
        z = code @ g[:, :CODE].float().T
        best = z.topk(top + 1, -1).values
        fine &= (best[:, top - 1] - best[:, top]) > MARGIN * z.std()
    return fine.nonzero().flatten()


def _router(gate, gen):
    """Rows of a router that reads the code alone; its logits have a standard deviation near one."""
    gate.zero_()
    gate[:, :CODE] = (torch.randn(gate.shape[0], CODE, generator=gen, device=gate.device) * CODE ** -0.5).to(gate.dtype)


def _prefer(head, embed, strength, gen):
    """Let the head prefer one successor of every token."""
    successor = torch.randperm(embed.shape[0], generator=gen, device=embed.device)
    for i in range(0, embed.shape[0], 1 << 14):
        at = successor[i:i + (1 << 14)]
        head[at] = (head[at].float() + strength * embed[i:i + (1 << 14)].float()).to(head.dtype)


def _flash_weights(case, seed):
    family, cfg = _config(case)
    w = family.random_weights(cfg, torch.device("cuda", 0), seed=seed % 100003, expert_dtype=case["experts"])
    gen = _gen(seed)
    w.embed.mul_(50.0)                   # rows of unit size: what a layer adds is of the size of what it finds
    _code(w.embed, gen)
    for lw in w.layers:
        _router(lw.w_gate_sh[:cfg.n_experts], gen)
        lw.gate_bias.zero_()
        lw.wo_b[:CODE] = 0
        lw.w2_sh[:CODE] = 0
        lw.w2[:, :CODE].view(torch.uint8).zero_()
    _prefer(w.head, w.embed, 0.005, gen)
    return family, cfg, w, _steady(w.embed, [lw.w_gate_sh[:cfg.n_experts] for lw in w.layers], cfg.topk)


def _stack_tensors(case, seed):
    """name -> tensor of a layer-stack model, and the tokens it is asked about."""
    family, cfg = _config(case)
    gen, out, routers = _gen(seed), {}, []
    for name, shape in family.tensor_shapes(cfg).items():
        out[name] = family.module.random_tensor(cfg, name, shape, gen, torch.device("cuda", 0))
    if case["model"].startswith("genesun"):
        _prefer(out["head"], out["embed"], 0.02, gen)
        return family, cfg, out, torch.arange(cfg.vocab, device="cuda")
    out["final.norm"] = (out["final.norm"].float() * 3.0 * cfg.hidden ** -0.5).bfloat16()   # logits below their cap
    _code(out["embed"], gen)
    for name, t in out.items():
        if name.endswith("mlp.router"):
            _router(t, gen)
            routers.append(t)
        elif name.endswith("mlp.router.b"):
            t.zero_()
        elif name.endswith("norm2"):
            t[:CODE] = 1.0
        elif name.endswith(("mix.o", ".down", "side.proj")):
            t[:CODE] = 0
    return family, cfg, out, _steady(out["embed"], routers, cfg.layers[0].mlp.top)


def _stream(case, seed, steady):
    """The tokens of the case: a prompt, or the stream at whose places the requests of a decode step are."""
    n = case["tokens"] if case["kind"] == "prompt" else case["context"] + case["each"]
    pick = torch.randint(0, steady.numel(), (n,), generator=_gen(seed + 1), device="cuda")
    return steady[pick].tolist()


def _lengths(case, seed):
    """Tokens that each request has behind it: one request all of them, several from a quarter up."""
    n, most = case["requests"], case["context"]
    if n == 1:
        return [most]
    u = torch.rand(n, generator=torch.Generator().manual_seed(seed)).tolist()
    return [most] + [max(1, int(most * 4.0 ** (x - 1.0))) for x in u[1:]]


# ---------------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    dev = torch.device("cuda", 0)
    if case["kind"] == "sample":
        logits = torch.randn(case["rows"], case["vocab"], generator=_gen(seed), device=dev) * 2.5
        # what requests ask for: plain temperature, nucleus, top-k with nucleus, min-p
        asked = [dict(), dict(top_p=0.9), dict(top_k=40, top_p=0.95), dict(min_p=0.05)]
        params = [RowParams(temperature=0.6 + 0.1 * (i % 5), seed=seed + i, position=100 + i, **asked[i % 4])
                  for i in range(case["rows"])]
        return {"case": case, "logits": logits, "params": params}
    if case["model"] == "flash":
        family, cfg, w, steady = _flash_weights(case, seed)
        kv = {"kv_dtype": case["kv"]}
    else:
        family, cfg, tensors, steady = _stack_tensors(case, seed)
        w, kv = family.module.build_weights(cfg, tensors.pop, dev), {}
    stream = _stream(case, seed, steady)
    ctx = len(stream) // 64 * 64 + 128
    if case["kind"] == "prompt":
        e = family.engine(cfg, w, max_rows=case["chunk"], slots=1, max_ctx=ctx, **kv)
        return {"case": case, "engine": e, "tokens": stream}
    n, each = case["requests"], case["each"]
    e = family.engine(cfg, w, max_rows=max(n * each, min(1024, case["context"])), slots=n, max_ctx=ctx, **kv)
    rows = ([], [], [])
    for slot, length in enumerate(_lengths(case, seed)):
        assert e.cache.ensure(slot, length + each + 1)
        e.prefill(slot, stream[:length])
        rows[0].extend(stream[length:length + each])
        rows[1].extend(range(length, length + each))
        rows[2].extend([slot] * each)
    session = DecodeSession(e)
    e.set_rows(*rows)
    session.graph(n * each)
    return {"case": case, "engine": e, "session": session, "rows": rows}


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        logits = state["logits"]
        tokens, status = sample_rows(logits, pack_params(state["params"], logits.device))
        return {"tokens": tokens, "status": status}
    e = state["engine"]
    if case["kind"] == "decode":
        tokens = state["session"].step(*state["rows"])
        return {"tokens": torch.tensor(tokens), "logits": e.logits_rows(len(tokens))}
    token = e.prefill(0, state["tokens"], chunk=case["chunk"])
    out = {"token": token, "logits": e.logits_rows(1)}
    if case["model"] == "flash":
        if case["kv"] == "bf16":
            out["window"] = e.cache.win[:, 0]
    else:
        out["states"] = [e.cache.states[l][0][0] for l in sorted(e.cache.states)]
    return out


# ---------------------------------------------------------------------------------------------------- work and tolerance
def _count(case):
    """(rows, tokens whose keys are read, heads run) of one pass."""
    if case["kind"] == "prompt":
        return case["tokens"], case["tokens"], 1
    rows = case["requests"] * case["each"]
    mean = case["context"] * (1.0 if case["requests"] == 1 else 0.54)
    return rows, mean * case["requests"], rows


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 0.0}
    family, cfg = _config(case)
    rows, keys, heads = _count(case)
    prompt = case["kind"] == "prompt"
    W = cfg.hidden
    b, f = 2.0 * cfg.vocab * W + 4.0 * heads * cfg.vocab, 2.0 * heads * cfg.vocab * W

    def experts(n, top, inter, size):
        used = n * (1.0 - (1.0 - top / n) ** rows)
        return used * 3.0 * W * inter * size, rows * top * 6.0 * W * inter

    if case["model"] == "flash":
        D, ko = cfg.head_dim, cfg.o_groups * cfg.o_lora
        kv_row = 2.0 * D if case["kv"] == "bf16" else D * 33 / 32
        for l in range(cfg.n_layers):
            index, src = l in cfg.index_layers, cfg.source_of(l)
            weights = W * (cfg.q_lora + D + (2 * D if src == l else 0) + (cfg.index_heads if index else 0))
            weights += cfg.q_lora * (cfg.n_heads * D + (cfg.index_heads * cfg.index_dim if index else 0))
            weights += cfg.n_heads * D * cfg.o_lora + ko * W + W * (cfg.n_experts + 3 * cfg.inter)
            eb, ef = experts(cfg.n_experts, cfg.topk, cfg.inter, ACTIVE_BYTES[case["experts"]])
            picked = min(cfg.index_topk, keys / rows / 2 if not prompt else keys / 4) if src is not None else 0
            seen = min(cfg.window, keys) + picked
            b += 2.0 * weights + eb + (min(keys, rows * cfg.window) + (keys / 2 if prompt else rows * picked)) * kv_row
            f += 2.0 * rows * weights + ef + 4.0 * rows * cfg.n_heads * D * seen
            if index:
                pairs = rows * keys / 4 if prompt else rows / case["requests"] * keys / 2
                b += keys / 2 * cfg.index_dim * 2.0
                f += 2.0 * pairs * cfg.index_heads * cfg.index_dim
        return {"bytes": b, "flops": f}
    pairs = rows * (rows + 1) / 2 if prompt else rows / case["requests"] * keys
    for l, spec in enumerate(cfg.layers):
        m = spec.mixer
        shapes = family.layer_shapes(cfg, l)
        weights = sum(s[0] * s[1] for n, s in shapes.items() if len(s) == 2 and ".e" not in n and not n.endswith(".conv"))
        b, f = b + 2.0 * weights, f + 2.0 * rows * weights
        if m.kind == "mlstm":
            state = 4.0 * m.heads * m.dim * m.vdim
            b += 2.0 * state * (1 if prompt else case["requests"])
            f += rows * m.heads * (4.0 * m.dim * m.vdim + (128.0 * (m.dim + m.vdim) if prompt else 0.0))
        elif m.kind == "latent_attention":
            b += 2.0 * keys * (m.kv_rank + m.rot_dim)
            wide = (m.dim + m.rot_dim + m.vdim) if prompt else (2 * m.kv_rank + m.rot_dim)
            f += 2.0 * pairs * m.heads * wide
        else:
            b += 2.0 * keys * m.kv_heads * (m.dim + m.vdim)
            f += 2.0 * pairs * m.heads * (m.dim + m.vdim)
        if spec.mlp is not None and spec.mlp.kind == "moe":
            eb, ef = experts(spec.mlp.experts, spec.mlp.top, spec.mlp.ff, 2.0)
            b, f = b + eb, f + ef
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    # flash rounds activations to 8 or 4 bits (0.03 to 0.05 away from 64 bits), the layer stacks to bf16 (0.004 to 0.013)
    return {"rel": 0.03 if case["model"] == "flash" else 0.02, "max": 0.5}


# ---------------------------------------------------------------------------------------------------- in 64 bits
F64 = torch.float64


def _mm(x, w, step=8192):
    """x @ w.T in 64 bits, the matrix converted in pieces."""
    return torch.cat([x @ w[i:i + step].to(F64).T for i in range(0, w.shape[0], step)], -1)


def _rms(x, w=None, eps=1e-6):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.to(F64)


def _frequencies(rope, dims):
    base = [rope.theta ** (-2.0 * i / dims) for i in range(dims // 2)]
    if rope.factor == 1.0:
        return torch.tensor(base, dtype=F64, device="cuda")
    if rope.bands is not None:
        low, high = rope.bands
        keep = [(rope.original_max_position * f / (2 * math.pi) - low) / (high - low) for f in base]
    else:
        def place(turns):
            return dims * math.log(rope.original_max_position / (turns * 2 * math.pi)) / (2 * math.log(rope.theta))

        a, z = max(math.floor(place(rope.beta_fast)), 0), min(math.ceil(place(rope.beta_slow)), dims - 1)
        keep = [1.0 - (i - a) / max(z - a, 0.001) for i in range(dims // 2)]
    keep = [min(max(k, 0.0), 1.0) for k in keep]
    return torch.tensor([f * k + f / rope.factor * (1 - k) for f, k in zip(base, keep)], dtype=F64, device="cuda")


def _turn(x, pos, freq, back=False):
    """Adjacent pairs of the last dimensions of x [T, ..., D] turned by pos * freq."""
    ang = pos.to(F64)[:, None] * freq
    while ang.dim() < x.dim():
        ang = ang.unsqueeze(1)
    c, s = torch.cos(ang), torch.sin(ang) * (-1 if back else 1)
    n = 2 * freq.numel()
    head, tail = x[..., :x.shape[-1] - n], x[..., x.shape[-1] - n:]
    u, v = tail[..., 0::2], tail[..., 1::2]
    return torch.cat([head, torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)], -1)


def _fp4(t):
    """E2M1 codes, two per byte, the even element in the low half."""
    values = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, 0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=F64, device=t.device)
    return torch.stack([values[(t & 15).long()], values[(t >> 4).long()]], -1).flatten(-2)


def _flash_expert(t, kind):
    return {"mxfp8": lambda: t.to(F64) * 2.0 ** -11, "mxfp4": lambda: _fp4(t) * 2.0 ** -7,
            "bf16": lambda: t.to(F64)}[kind]()


def _swiglu(g, u, limit):
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(g) * u


def _flash_mixes(streams, fn, base, cfg):
    T, m = streams.shape[0], cfg.hc_mult
    flat = streams.reshape(T, -1)
    p = _mm(flat, fn) * torch.rsqrt((flat * flat).mean(-1, keepdim=True) + cfg.norm_eps) + base.to(F64)
    c = torch.softmax(p[:, 2 * m:].view(T, m, m), 2) + cfg.hc_eps
    c = c / (c.sum(1, keepdim=True) + cfg.hc_eps)
    for _ in range(cfg.hc_sinkhorn_iters - 1):
        c = c / (c.sum(2, keepdim=True) + cfg.hc_eps)
        c = c / (c.sum(1, keepdim=True) + cfg.hc_eps)
    return torch.sigmoid(p[:, :m]) + cfg.hc_eps, 2.0 * torch.sigmoid(p[:, m:2 * m]), c


def _flash_attention(cfg, lw, xn, pos, rope, source, select):
    """-> (result, window rows); `select` [T, k] compressed rows per token, -1 where there is none."""
    T, H, D, Q = xn.shape[0], cfg.n_heads, cfg.head_dim, cfg.q_lora
    freq = _frequencies(rope, cfg.rope_dim)
    lat = _rms(_mm(xn, lw.w_qkv[:Q]), lw.q_norm, cfg.norm_eps)
    kv = _turn(_rms(_mm(xn, lw.w_qkv[Q:Q + D]), lw.kv_norm, cfg.norm_eps), pos, freq)
    wq, wo_a = lw.w_qb[:H * D].to(F64), lw.wo_a.to(F64)
    out = torch.empty(T, cfg.o_groups * cfg.o_lora, dtype=F64, device=xn.device)
    for a in range(0, T, 256):
        p = pos[a:a + 256]
        q = _turn((lat[a:a + 256] @ wq.T).view(len(p), H, D), p, freq)
        j = p[:, None] - torch.arange(cfg.window, device=p.device)[None]
        keys, live = kv[j.clamp(min=0)], j >= 0
        if source is not None:
            s = select[a:a + 256]
            keys, live = torch.cat([keys, source[s.clamp(min=0)]], 1), torch.cat([live, s >= 0], 1)
        z = torch.bmm(q, keys.transpose(1, 2)) * cfg.softmax_scale
        z = torch.cat([z.masked_fill(~live[:, None], -math.inf), lw.sink.to(F64)[None, :, None].expand(len(p), H, 1)], -1)
        o = _turn(torch.bmm(torch.softmax(z, -1)[..., :-1], keys), p, freq, back=True)
        o = o.reshape(len(p), cfg.o_groups, -1)
        out[a:a + 256] = torch.einsum("tgk,gok->tgo", o, wo_a).reshape(len(p), -1)
    return _mm(out, lw.wo_b), kv, lat


def _flash_select(cfg, lw, xn, lat, pos, rope, ratio):
    """Compressed rows of the layer and the rows that every token selects."""
    T, D, Q, ID, IH = xn.shape[0], cfg.head_dim, cfg.q_lora, cfg.index_dim, cfg.index_heads
    at = Q + D
    rows = _mm(xn, lw.w_qkv[at:at + D])
    Tc = T // ratio
    first = pos[:Tc * ratio:ratio]
    if ratio == 2:
        gate = torch.softmax(_mm(xn, lw.w_qkv[at + D:at + 2 * D])[:Tc * 2].view(Tc, 2, D), 1)
        rows = (gate * rows[:Tc * 2].view(Tc, 2, D)).sum(1)
    rows = _rms(rows, lw.comp_norm, cfg.norm_eps)
    half = _frequencies(rope, ID // 2)
    keys = _turn(_rms(_mm(rows, lw.wk_idx), lw.k_norm, cfg.norm_eps), first, half)
    weight = _mm(xn, lw.w_qkv[-IH:]) * cfg.index_weight_scale
    wq = lw.w_qb[cfg.n_heads * D:].to(F64)
    k = min(cfg.index_topk, Tc)
    picked = torch.full((T, max(k, 1)), -1, dtype=torch.long, device=xn.device)
    for a in range(0, T, 256):
        p = pos[a:a + 256]
        q = _turn((lat[a:a + 256] @ wq.T).view(len(p), IH, ID), p, half)
        z = torch.zeros(len(p), Tc, dtype=F64, device=xn.device)
        for h in range(IH):
            z += weight[a:a + 256, h:h + 1] * torch.relu(q[:, h] @ keys.T)
        z.masked_fill_(torch.arange(Tc, device=xn.device)[None] >= ((p + 1) // ratio)[:, None], -math.inf)
        if k:
            best = z.topk(k, -1)
            picked[a:a + 256] = best.indices.masked_fill(best.values == -math.inf, -1)
    return _turn(rows, first, _frequencies(rope, cfg.rope_dim)), picked


def _flash_moe(cfg, lw, xn, kind):
    E, I = cfg.n_experts, cfg.inter
    score = torch.sqrt(torch.nn.functional.softplus(_mm(xn, lw.w_gate_sh[:E])))
    ids = (score + lw.gate_bias.to(F64)).topk(cfg.topk, -1).indices
    wt = score.gather(1, ids)
    wt = wt / (wt.sum(-1, keepdim=True) + 1e-20) * cfg.route_scale
    out = _mm(_swiglu(_mm(xn, lw.w_gate_sh[E:E + I]), _mm(xn, lw.w_gate_sh[E + I:]), cfg.swiglu_limit), lw.w2_sh)
    for e in ids.unique().tolist():
        rows, k = torch.where(ids == e)
        w13 = _flash_expert(lw.w13[e], kind)
        act = _swiglu(xn[rows] @ w13[:I].T, xn[rows] @ w13[I:].T, cfg.swiglu_limit) * wt[rows, k][:, None]
        out.index_add_(0, rows, act @ _flash_expert(lw.w2[e], kind).T)
    return out


def _flash_exact(case, seed):
    _, cfg, w, steady = _flash_weights(case, seed)
    tokens = torch.tensor(_stream(case, seed, steady), device="cuda")
    T = len(tokens)
    pos = torch.arange(T, device="cuda")
    streams = w.embed[tokens].to(F64)[:, None].repeat(1, cfg.hc_mult, 1)
    pre = torch.zeros(T, cfg.hc_mult, dtype=F64, device="cuda")
    pre[:, 0] = 1.0
    source = select = None
    windows = []
    for l, lw in enumerate(w.layers):
        rope = cfg.rope_plain if cfg.compress_ratios[l] == 0 else cfg.rope_long
        nxt, post, comb = _flash_mixes(streams, lw.hc_attn_fn, lw.hc_attn_base, cfg)
        xn = _rms((pre[..., None] * streams).sum(1), lw.attn_norm, cfg.norm_eps)
        if lw.ratio:
            lat = _rms(_mm(xn, lw.w_qkv[:cfg.q_lora]), lw.q_norm, cfg.norm_eps)
            source, select = _flash_select(cfg, lw, xn, lat, pos, rope, lw.ratio)
        y, kv, _ = _flash_attention(cfg, lw, xn, pos, rope, source, select)
        windows.append(kv)
        streams, pre = post[:, :, None] * y[:, None] + torch.einsum("tsd,tsh->tdh", comb, streams), nxt
        nxt, post, comb = _flash_mixes(streams, lw.hc_ffn_fn, lw.hc_ffn_base, cfg)
        y = _flash_moe(cfg, lw, _rms((pre[..., None] * streams).sum(1), lw.ffn_norm, cfg.norm_eps), case["experts"])
        streams, pre = post[:, :, None] * y[:, None] + torch.einsum("tsd,tsh->tdh", comb, streams), nxt
    x = _rms((pre[..., None] * streams).sum(1), w.final_norm, cfg.norm_eps)
    out = {"logits": _mm(x[_wanted(case, seed)], w.head)}
    if case["kind"] == "prompt" and case["kv"] == "bf16":
        ring = cfg.window + max(16, case["chunk"])
        win = torch.zeros(cfg.n_layers, ring, cfg.head_dim, dtype=F64, device="cuda")
        for l, kv in enumerate(windows):
            win[l, pos[-ring:] % ring] = kv[-ring:]
        out["window"] = win
    return out


def _wanted(case, seed):
    """Places of the stream whose logits the case returns."""
    if case["kind"] == "prompt":
        return [case["tokens"] - 1]
    return [n + i for n in _lengths(case, seed) for i in range(case["each"])]


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt((d * d).mean(-1, keepdim=True) + eps) * w.to(F64)


def _causal(q, k, v, scale, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, V], one head at a time; `sink` [H] joins every denominator."""
    T, H = q.shape[:2]
    n = H // k.shape[1]
    late = torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1)
    out = []
    for h in range(H):
        z = (q[:, h] @ k[:, h // n].T * scale).masked_fill(late, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink[h].to(F64).expand(T, 1)], 1)
        out.append(torch.softmax(z, -1)[:, :T] @ v[:, h // n])
    return torch.stack(out, 1)


def _latent(m, t, h, pos, eps, shared):
    T, H, D, R = h.shape[0], m.heads, m.dim, m.rot_dim
    freq, mag = _frequencies(m.rope, R), m.magnitude
    q = _mm(_rms(_mm(h, t["mix.dq"]), t["mix.dq.norm"], eps), t["mix.uq"]).view(T, H, D + R)
    if m.kv_from is None:
        kv = _mm(h, t["mix.dkv"])
        shared = _rms(kv[:, :m.kv_rank], t["mix.dkv.norm"], eps), mag * _turn(kv[:, m.kv_rank:], pos, freq)
    lat, rot = shared
    k = torch.cat([_mm(lat, t["mix.uk"]).view(T, H, D), rot[:, None].expand(T, H, R)], -1)
    q = torch.cat([q[..., :D], mag * _turn(q[..., D:], pos, freq)], -1)
    o = _causal(q, k, _mm(lat, t["mix.uv"]).view(T, H, -1), m.scale, t["mix.sink"])
    return _mm(o.reshape(T, -1) * torch.sigmoid(_mm(h, t["mix.g"])), t["mix.o"]), shared


def _mlstm(m, t, h, eps):
    """-> (result, matrix memory after the last token), by the sum over all earlier tokens."""
    T, H = h.shape[0], m.heads
    q, k, v = (_mm(h, t["mix." + n]).view(T, H, -1) for n in "qkv")
    cap = m.gate_cap
    i = cap * torch.tanh((_mm(h, t["mix.i"]) + t["mix.i.b"].to(F64)) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((_mm(h, t["mix.f"]) + t["mix.f.b"].to(F64)) / cap))
    run = f.cumsum(0)
    late = torch.ones(T, T, dtype=torch.bool, device=h.device).triu(1)
    out, memory = [], []
    for a in range(H):
        d = (run[:, a, None] - run[None, :, a] + i[None, :, a]).masked_fill(late, -math.inf)
        top = torch.maximum(d.amax(-1), run[:, a])
        w = torch.exp(d - top[:, None])
        memory.append((w[-1, :, None] * k[:, a]).T @ v[:, a])
        w = w * (q[:, a] @ k[:, a].T) * m.dim ** -0.5
        out.append(w @ v[:, a] / (torch.maximum(w.sum(-1).abs(), torch.exp(-top)) + m.den_eps)[:, None])
    o = _rms(torch.stack(out, 1), None, eps).reshape(T, -1) * t["mix.norm"].to(F64)
    return _mm(o * torch.sigmoid(_mm(h, t["mix.g"])), t["mix.o"]), torch.stack(memory)


def _genesun_exact(case, seed):
    _, cfg, w, steady = _stack_tensors(case, seed)
    tokens = torch.tensor(_stream(case, seed, steady), device="cuda")
    pos, eps = torch.arange(len(tokens), device="cuda"), cfg.norm_eps
    x = w["embed"][tokens].to(F64)
    kept, shared, states = [x], None, []
    for l, spec in enumerate(cfg.layers):
        t = {n[len(f"l{l}."):]: v for n, v in w.items() if n.startswith(f"l{l}.")}
        h = _layer_norm(x, t["norm1"], eps)
        if spec.mixer.kind == "mlstm":
            y, memory = _mlstm(spec.mixer, t, h, eps)
            states.append(memory)
        else:
            y, shared = _latent(spec.mixer, t, h, pos, eps, shared)
        x = x + _layer_norm(y * torch.sigmoid(_mm(h, t["rg1"]) + t["rg1.b"].to(F64)), t["norm1b"], eps)
        if spec.mlp is not None:
            h = _layer_norm(x, t["norm2"], eps)
            z, (a, b, c, d) = _mm(h, t["mlp.up"]), t["mlp.act"].to(F64)
            y = _mm(a * _rms(z, None, eps) + b * _rms(z ** 2, None, eps) + c * _rms(z ** 3, None, eps) + d, t["mlp.down"])
            x = x + _layer_norm(y * torch.sigmoid(_mm(h, t["rg2"]) + t["rg2.b"].to(F64)), t["norm2b"], eps)
        kept.append(x)
        x = sum(c * s for c, s in zip(t["dwa"].to(F64), kept))
    out = {"logits": _mm(_layer_norm(x[_wanted(case, seed)], w["final.norm"], eps), w["head"])}
    if case["kind"] == "prompt":
        out["states"] = states
    return out


def _halves(x, pos, freq):
    ang = (pos.to(F64)[:, None] * freq)[:, None]
    c, s, n = torch.cos(ang), torch.sin(ang), freq.numel()
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], -1)


def _belasun_exact(case, seed):
    _, cfg, w, steady = _stack_tensors(case, seed)
    tokens = torch.tensor(_stream(case, seed, steady), device="cuda")
    T, eps, dim = len(tokens), cfg.norm_eps, cfg.token_side
    pos, x, rings = torch.arange(T, device="cuda"), w["embed"][tokens].to(F64), []
    for l, spec in enumerate(cfg.layers):
        m, ml = spec.mixer, spec.mlp
        t = {n[len(f"l{l}."):]: v for n, v in w.items() if n.startswith(f"l{l}.")}
        h = _rms(x, t["norm1"], eps)
        got, raw = {}, []
        for n in "qkv":
            u, taps = _mm(h, t["mix." + n]), t[f"mix.{n}.conv"].to(F64)
            raw.append(u)
            got[n] = sum(taps[:, -1 - j] * torch.nn.functional.pad(u, (0, 0, j, 0))[:T] for j in range(m.taps))
        ring = torch.zeros(m.taps - 1, sum(u.shape[1] for u in raw), dtype=F64, device="cuda")
        ring[pos[1 - m.taps:] % (m.taps - 1)] = torch.cat(raw, 1)[1 - m.taps:]
        rings.append(ring)
        freq = _frequencies(m.rope, m.rot_dim)
        q = _halves(_rms(got["q"], t["mix.q.norm"], eps).view(T, m.heads, m.dim), pos, freq)
        k = _halves(_rms(got["k"], t["mix.k.norm"], eps).view(T, m.kv_heads, m.dim), pos, freq)
        o = _causal(q, k, got["v"].view(T, m.kv_heads, m.vdim), m.scale)     # every case fits in one chunk
        x = x + _mm((o * torch.sigmoid(_mm(h, t["mix.g"]))[..., None]).reshape(T, -1), t["mix.o"])
        h = _rms(x, t["norm2"], eps)
        best = (_mm(h, t["mlp.router"]) + t["mlp.router.b"].to(F64)).topk(ml.top, -1)
        wt, y = torch.softmax(best.values, -1), torch.zeros_like(x)
        for e in range(ml.experts):
            rows, j = torch.where(best.indices == e)
            g = _mm(h[rows], t[f"mlp.e{e}.gate"]).clamp(max=ml.limit)
            u = _mm(h[rows], t[f"mlp.e{e}.up"]).clamp(-ml.limit, ml.limit)
            act = g * torch.sigmoid(ml.alpha * g) * (u + ml.shift)
            y.index_add_(0, rows, wt[rows, j][:, None] * _mm(act, t[f"mlp.e{e}.down"]))
        x = x + y
        part = w["side.embed"][tokens, l * dim:(l + 1) * dim].to(F64)
        z = torch.nn.functional.gelu(_mm(x, t["side.gate"]), approximate="tanh") * part
        x = x + _rms(_mm(z, t["side.proj"]), t["side.norm"], eps)
    z = _mm(_rms(x[_wanted(case, seed)], w["final.norm"], eps), w["embed"])
    out = {"logits": cfg.logit_softcap * torch.tanh(z / cfg.logit_softcap)}
    if case["kind"] == "prompt":
        out["states"] = rings
    return out


def exact(case, seed):
    if case["kind"] == "sample" or case["experts"] == "nvfp4":      # 4-bit activations: as far off as their rounding is
        return None
    made = {"flash": _flash_exact, "genesun": _genesun_exact, "belasun": _belasun_exact}
    return made[case["model"].split("-")[0]](case, seed)
