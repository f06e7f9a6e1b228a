"""Workloads that time the framework as its users run it, through the engine's public calls.

Two kinds of work. ``generate``: requests handed to an :class:`AttentionEngine` (``add_request``) and stepped to their
last token (``step``), what a serving process does with a batch of arrivals: one prefill of the ragged prompts, then decode
steps of all of them. ``replay``: given tokens through a layered decoder (``open_sequence`` / ``run_given`` /
``close_sequence``), what the trace replay program does: one ragged portion per sequence, then single tokens.

Sizes are those of the model presets, with some layers left out where all layers are alike (a pass is shorter, its
kernels are the same). Weights are random; the LM head is the embedding one token on, so that every model names the next
token id with a clear margin and the tokens do not hang on the rounding of two close logits.
"""

import math

import torch

from crosspool_b200.bench.layered import layered_twin
from crosspool_b200.engine.atn_engine import AttentionEngine, EngineConfig
from crosspool_b200.engine.ffn_local import LocalFfnPort
from crosspool_b200.models.config import LatentMixer, preset
from crosspool_b200.models.layered import layered_attention_weights
from crosspool_b200.models.weights import FfnLayerWeights, random_attention_weights, random_ffn_weights

SMALL, PARTNER, LARGE, EXPERTS = "Qwen/Qwen3-0.6B", "Qwen/Qwen2.5-0.5B", "Qwen/Qwen3-8B", "Qwen/Qwen3-30B-A3B"
CHUNK = 4096        # prompt tokens of a prefill step where a prompt is longer (the engine's default in served deployments)
PAGE = 64           # tokens per cache page in served deployments
HEAD_SCALE = 0.05   # logits of the named token around 30, of the others around +-2


def _generate(name, model, layers, requests, shortest, longest, new, cached=False):
    return {"name": name, "kind": "generate", "model": model, "layers": layers, "requests": requests, "shortest": shortest,
            "longest": longest, "new": new, "cached": cached}


def _replay(name, model, heads, layers, requests, shortest, longest, new, dtype="bfloat16"):
    return {"name": name, "kind": "replay", "model": model, "heads": heads, "layers": layers, "requests": requests,
            "shortest": shortest, "longest": longest, "new": new, "dtype": dtype}


def listed():
    return [
        # one user of an idle small model: short prompt, a short answer; launches and latency
        _generate("chat", SMALL, 28, 1, 45, 45, 12),
        # a handful of users of the same model, ragged short prompts
        _generate("few_users", SMALL, 28, 7, 20, 300, 16),
        # a saturated small model: many running requests over prompts whose pages the prefix cache holds
        _generate("busy_decode", SMALL, 14, 128, 200, 1500, 24, cached=True),
        # arrivals of ordinary prompts up to their first token (time to first token)
        _generate("prompts", SMALL, 28, 8, 130, 900, 1),
        # a long document in chunks, up to its first token
        _generate("document", SMALL, 14, 1, 15987, 15987, 1),
        # a larger model in decode, conversations whose pages are cached
        _generate("large_decode", LARGE, 6, 33, 100, 600, 24, cached=True),
        # ... and in prefill
        _generate("large_prompts", LARGE, 6, 5, 700, 1800, 1),
        # the partner of the small model in a two-model deployment: narrow heads, seven queries to a key head, biases
        _generate("partner", PARTNER, 24, 16, 60, 500, 16),
        # routed experts, decode
        _generate("experts_decode", EXPERTS, 6, 24, 64, 500, 16, cached=True),
        # routed experts, prefill
        _generate("experts_prompts", EXPERTS, 6, 6, 400, 1200, 1),
        # layered decoder (latent attention and linear recurrences): a replayed trace of ragged portions and single tokens
        _replay("layered", SMALL, 16, 8, 16, 200, 700, 12),
        # the same in 32 bits
        _replay("layered_fp32", SMALL, 16, 8, 3, 40, 150, 8, dtype="float32"),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the listed kinds: sizes over the whole range between the smallest and the largest listed ones."""
    most = max(_cost(c) for c in listed())
    while True:
        what = rng.choice(["small", "small", "large", "partner", "experts", "layered", "layered_fp32"])
        new = rng.choice([1, _between(rng, 2, 24)])
        lo = _between(rng, 20, 1200)
        hi = lo + rng.randrange(0, 2 * lo)
        if what == "small":
            if rng.random() < 0.2:          # one long prompt
                n, lo, hi, new = 1, *([_between(rng, 1200, 16000)] * 2), 1
            else:
                n = _between(rng, 1, 128)
            c = _generate(None, SMALL, rng.choice([14, 28]), n, lo, hi, new, cached=new > 1 and rng.random() < 0.5)
        elif what == "large":
            c = _generate(None, LARGE, 6, _between(rng, 1, 48), lo, hi, new, cached=new > 1 and rng.random() < 0.5)
        elif what == "partner":
            c = _generate(None, PARTNER, 24, _between(rng, 1, 64), lo, hi, new, cached=new > 1 and rng.random() < 0.5)
        elif what == "experts":
            c = _generate(None, EXPERTS, 6, _between(rng, 1, 48), lo, hi, new, cached=new > 1 and rng.random() < 0.5)
        elif what == "layered":
            c = _replay(None, SMALL, 16, 8, _between(rng, 1, 32), lo, hi, min(new, 16))
        else:
            c = _replay(None, SMALL, 16, 8, _between(rng, 1, 4), min(lo, 120), min(hi, 200), min(new, 8), dtype="float32")
        del c["name"]
        prompts = sum(_lengths(c))
        if prompts <= (160_000 if c.get("cached") else 8192 if c["requests"] > 1 else 16000) and _cost(c) <= most:
            return c


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 5e12, w["flops"] / (30e12 if case.get("dtype") == "float32" else 5e14)) + 2e-4 * case["new"]


def _lengths(case):
    """Prompt lengths, spread over the case's range; the inputs' seed changes the tokens and not the lengths."""
    lo, hi, n = case["shortest"], case["longest"], case["requests"]
    return [lo + int((hi - lo + 1) * ((i * 0.6180339887498949 + 0.31) % 1.0)) for i in range(n)]


# --------------------------------------------------------------------------------------------------- models


def _config(case):
    c = preset(case["model"]).with_layers(case["layers"])
    return layered_twin(c, case["heads"], case["layers"]) if case["kind"] == "replay" else c


def _tokens(case, seed):
    g = torch.Generator().manual_seed(seed)
    vocab = preset(case["model"]).vocab_size
    return [torch.randint(0, vocab, (n + (case["new"] - 1 if case["kind"] == "replay" else 0),), generator=g).tolist()
            for n in _lengths(case)]


def _classic_weights(case, seed):
    cfg = _config(case)
    w = random_attention_weights(cfg, seed, "cuda", torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    w.embed.normal_(0.0, 1.0, generator=g)
    w.lm_head = w.embed.roll(1, 0) * HEAD_SCALE
    for lw in w.layers:       # trained norm weights are not ones
        for t in (lw.input_norm, lw.post_attn_norm, lw.q_norm, lw.k_norm):
            if t is not None:
                t.uniform_(0.7, 1.3, generator=g)
    ffn = random_ffn_weights(cfg, seed, "cuda", torch.bfloat16)
    for f in ffn:
        if f.is_moe:          # trained routers are decided: the last chosen expert counts for little
            f.router *= 3.0
    return cfg, w, ffn


def _layered_tensors(cfg, seed):
    """The checkpoint tensors of a layered decoder by name, bf16, made where they are first asked for."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    made = {}

    def get(name, shape):
        if name not in made:
            t = torch.empty(shape, device="cuda")
            if name == "embed":
                t.normal_(0.0, 0.5, generator=g)
            elif len(shape) == 2:
                t.normal_(0.0, shape[1] ** -0.5, generator=g)
            elif name.endswith(".b"):
                t.normal_(0.0, 0.1, generator=g)
            else:
                t.uniform_(0.7, 1.3, generator=g)
            made[name] = t.bfloat16()
        return made[name]

    return get, made


def _layered_weights(case, seed):
    cfg = _config(case)
    dt = getattr(torch, case["dtype"])
    get, made = _layered_tensors(cfg, seed)
    w = layered_attention_weights(cfg, lambda n, s: get(n, s).to(dt), "cuda", dt)
    ffn = []
    for i, s in enumerate(cfg.layer_specs):
        f = FfnLayerWeights(get(f"l{i}.mlp.up", (s.ff, cfg.hidden_size)).to(dt), get(f"l{i}.mlp.down", (cfg.hidden_size, s.ff)).to(dt))
        f.extra.update(gated=False, polynorm=(get(f"l{i}.mlp.act", (4,)).float(), cfg.rms_norm_eps))
        ffn.append(f)
    return cfg, w, ffn, made


def _engine_config(case):
    lens, n, new = _lengths(case), case["requests"], case["new"]
    total = sum(lens)
    chunk = min(total, 8192) if n > 1 else min(total, CHUNK)
    pages = sum((l + new) // PAGE + 1 for l in lens) + (2 * n if case.get("cached") else 0)
    return EngineConfig(max_batch=n, prefill_chunk=max(chunk, n), max_seq_len=max(lens) + new + 1, page_size=PAGE, num_pages=pages,
                        max_prefill_seqs=n, decode_buckets=[n], prefix_cache=bool(case.get("cached")), dtype=case.get("dtype", "bfloat16"))


def prepare(case, seed):
    """A warmed-up engine with its weights and the requests' tokens; where prompts are ``cached``, one round of the same
    requests has gone through it, so that the prefix cache holds their full pages."""
    tokens = _tokens(case, seed)
    cfg, w, ffn = (_classic_weights(case, seed) if case["kind"] == "generate" else _layered_weights(case, seed)[:3])
    torch.cuda.synchronize()      # the weights are made on the default stream, the engine works on one of its own
    engine = AttentionEngine(cfg, w, LocalFfnPort(cfg, ffn), _engine_config(case), "cuda")
    torch.cuda.synchronize()
    engine.warmup()
    if case.get("cached"):
        engine.generate(tokens, 1)
    return {"engine": engine, "tokens": tokens, "new": case["new"], "lens": _lengths(case), "kind": case["kind"]}


def run(state):
    e, new = state["engine"], state["new"]
    if state["kind"] == "generate":
        seqs = [e.add_request(t, new) for t in state["tokens"]]
        out = []
        while e.has_work:
            out = e.step()
        # all requests are in every decode step: the last step's logits are theirs, in the order of its results
        return {"tokens": torch.tensor([s.generated for s in seqs], dtype=torch.int32), "logits": e.logits[:len(out)]}
    seqs = [e.open_sequence() for _ in state["tokens"]]
    portions = [t[:n] for t, n in zip(state["tokens"], state["lens"])]
    first = e.run_given(list(zip(seqs, portions)), [[n - 1] for n in state["lens"]])
    later = []
    for i in range(new - 1):
        later.append(e.run_given([(s, [t[n + i]]) for s, t, n in zip(seqs, state["tokens"], state["lens"])], [[0]] * len(seqs)))
    for s in seqs:
        e.close_sequence(s)
    return {"first": first, "later": torch.stack(later)} if later else {"first": first}


# --------------------------------------------------------------------------------------------------- what a pass needs


def _layer_sizes(cfg, case):
    """(weights that every token meets, attention flops per token and cached token, cache bytes per token) of one layer."""
    if case["kind"] == "replay":
        W, H = cfg.hidden_size, cfg.num_q_heads
        m = next(s.mixer for s in cfg.layer_specs if isinstance(s.mixer, LatentMixer))
        lin = W * (4 * H * 128) + H * 128 * W
        lat = W * (H * (m.dim + m.rot_dim) + m.kv_rank + m.rot_dim + H) + m.kv_rank * H * (m.dim + m.vdim) + H * m.vdim * W
        return 2 * W * W + 2 * W * cfg.layer_specs[0].ff + (lin + lat) / 2, H * (m.dim + m.rot_dim + m.vdim), m.kv_rank + m.rot_dim
    a = cfg.hidden_size * (2 * cfg.q_size + 2 * cfg.kv_size)
    return a, 4 * cfg.q_size, 2 * cfg.kv_size


def work(case):
    """Every forward pass reads each weight that its rows use once and the cache of its sequences once, and writes the rows it
    adds to the cache and the logits."""
    cfg, lens, n, new, L = _config(case), _lengths(case), case["requests"], case["new"], case["layers"]
    eb = 4 if case.get("dtype") == "float32" else 2
    shared, pair_flops, kv = _layer_sizes(cfg, case)
    moe = case["kind"] == "generate" and cfg.num_experts > 0
    ffn = 0 if case["kind"] == "replay" else 3 * cfg.hidden_size * (cfg.moe_intermediate_size if moe else cfg.intermediate_size)
    head = cfg.vocab_size * cfg.hidden_size
    fed = [(l - 1) % PAGE + 1 if case.get("cached") else l for l in lens]     # prompt rows that are computed
    chunks = max(1, -(-sum(fed) // CHUNK)) if n == 1 else 1
    passes = [sum(fed) / chunks] * chunks + [n] * (new - 1)
    byts = flops = 0.0
    for rows in passes:
        used = min(cfg.num_experts, rows * cfg.num_experts_per_tok) if moe else 1
        mean = cfg.num_experts * (1 - (1 - cfg.num_experts_per_tok / cfg.num_experts) ** rows) if moe else 1
        byts += L * (shared * eb + min(used, mean) * ffn * eb) + head * eb + n * cfg.vocab_size * (4 if case["kind"] == "replay" else 2)
        flops += 2 * rows * L * (shared + (cfg.num_experts_per_tok if moe else 1) * ffn) + 2 * n * head
    part = 0.5 if case["kind"] == "replay" else 1.0                            # every second layer of the layered decoder caches tokens
    pairs = sum(f * (l - f) + f * (f + 1) / 2 for l, f in zip(lens, fed)) + sum(l + i for l in lens for i in range(1, new))
    cached = sum(lens) + sum(l + i for l in lens for i in range(1, new)) + sum(fed) + n * (new - 1)
    byts += part * L * kv * eb * cached
    flops += part * L * pair_flops * pairs
    if case["kind"] == "replay":                                               # states are read and written once per pass
        state = L / 2 * cfg.num_q_heads * 128 * 128
        byts += n * new * state * 4 * 2
        flops += L / 2 * cfg.num_q_heads * 4 * 128 * 128 * sum(passes)
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    if case.get("dtype") == "float32":        # 5e-6 from 64 bits
        return {"rel": 2.5e-5}
    return {"rel": 0.03, "max": 0.3, "differ": 0.0}      # 1.0e-2 to 1.6e-2 from 64 bits: a bf16 residual stream


# --------------------------------------------------------------------------------------------------- 64 bits


def _rms(x, w, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt() * w.double()


def _mm(x, w):
    return x @ w.double().t()


def _by_rows(fn, x, step=16384):
    return fn(x) if x.shape[0] <= step else torch.cat([fn(p) for p in x.split(step)])


def _angles(cos_at, dims, base):
    f = float(base) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    a = cos_at.double()[:, None] * f
    return a.cos()[:, None], a.sin()[:, None]


def _rotate(x, cos, sin):
    h = x.shape[-1] // 2
    u, v = x[..., :h], x[..., h:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)


def _attend(q, k, v, scale):
    """Causal attention of one sequence, ``[T, H, d]`` queries over ``[T, G, d]`` keys."""
    T, H, _ = q.shape
    G = k.shape[1]
    q = q.view(T, G, H // G, -1).permute(1, 2, 0, 3)
    k, v = k.permute(1, 2, 0)[:, None], v.permute(1, 0, 2)[:, None]
    out, step = [], max(16, (1 << 27) // (T * H))
    for at in range(0, T, step):
        n = min(step, T - at)
        s = q[:, :, at:at + n] @ k[..., :at + n] * scale
        late = torch.ones(n, at + n, dtype=torch.bool, device="cuda").triu(at + 1)
        out.append(s.masked_fill_(late, -math.inf).softmax(-1) @ v[:, :, :at + n])
    return torch.cat(out, 2).permute(2, 0, 1, 3).reshape(T, -1)


def _swiglu(x):
    g, u = x.chunk(2, -1)
    return torch.nn.functional.silu(g) * u


def _experts(x, f, k, renorm):
    p = _mm(x, f.router).softmax(-1)
    w, ids = p.topk(k, -1)
    w = w / w.sum(-1, keepdim=True) if renorm else w
    y = torch.zeros_like(x)
    for e in range(f.router.shape[0]):
        rows, which = (ids == e).nonzero(as_tuple=True)
        if rows.numel():
            y.index_add_(0, rows, _mm(_swiglu(_mm(x[rows], f.gate_up[e])), f.down[e]) * w[rows, which, None])
    return y


def _classic_exact(case, seed):
    cfg, w, ffn = _classic_weights(case, seed)
    prompts, new = _tokens(case, seed), case["new"]
    # the next token is the id one on (checked against the logits below)
    seqs = [p + [(p[-1] + 1 + i) % cfg.vocab_size for i in range(new - 1)] for p in prompts]
    lens = [len(s) for s in seqs]
    ids = torch.tensor([t for s in seqs for t in s], device="cuda")
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    cos, sin = _angles(pos, cfg.head_dim, cfg.rope_theta)
    eps, d = cfg.rms_norm_eps, cfg.head_dim
    x = w.embed[ids].double()
    for lw, f in zip(w.layers, ffn):
        qkv = _by_rows(lambda r: _mm(_rms(r, lw.input_norm, eps), lw.qkv), x)
        if lw.qkv_bias is not None:
            qkv += lw.qkv_bias.double()
        q, k, v = (t.view(len(ids), -1, d) for t in qkv.split([cfg.q_size, cfg.kv_size, cfg.kv_size], -1))
        if lw.q_norm is not None:
            q, k = _rms(q, lw.q_norm, eps), _rms(k, lw.k_norm, eps)
        q, k = _rotate(q, cos, sin), _rotate(k, cos, sin)
        o = torch.cat([_attend(a, b, c, d ** -0.5) for a, b, c in zip(q.split(lens), k.split(lens), v.split(lens))])
        x = x + _by_rows(lambda r: _mm(r, lw.o), o)
        del qkv, q, k, v, o
        if f.is_moe:
            y = _by_rows(lambda r: _experts(_rms(r, lw.post_attn_norm, eps), f, cfg.num_experts_per_tok, cfg.norm_topk_prob), x)
        else:
            y = _by_rows(lambda r: _mm(_swiglu(_mm(_rms(r, lw.post_attn_norm, eps), f.gate_up)), f.down), x)
        x = x + y
    ends = torch.tensor(lens, device="cuda").cumsum(0)
    rows = (ends[:, None] - new + torch.arange(new, device="cuda")).reshape(-1)
    logits = _by_rows(lambda r: _mm(_rms(r, w.final_norm, eps), w.lm_head), x[rows], 512) if new * len(lens) <= 4096 else None
    if logits is None:
        return None
    logits = logits.view(len(lens), new, -1)
    return {"tokens": logits.argmax(-1).to(torch.int32).cpu(), "logits": logits[:, -1].contiguous()}


def _decayed(q, k, v, decay):
    """o_i = q_i sum_{j <= i} decay^(i - j) k_j^T v_j per head, 256 tokens at a time behind a carried state."""
    T, H, d = q.shape
    S = torch.zeros(H, d, v.shape[-1], dtype=torch.float64, device="cuda")
    out = []
    for at in range(0, T, 256):
        a, b, c = (t[at:at + 256].transpose(0, 1) for t in (q, k, v))
        n = a.shape[1]
        i = torch.arange(n, device="cuda", dtype=torch.float64)
        gap = i[:, None] - i
        m = torch.where(gap >= 0, decay[:, None, None] ** gap.clamp_min(0), torch.zeros((), dtype=torch.float64, device="cuda"))
        out.append((a @ b.transpose(1, 2) * m) @ c + (a @ S) * (decay[:, None] ** (i + 1))[..., None])
        S = S * (decay ** n)[:, None, None] + (b * (decay[:, None] ** (n - 1 - i))[..., None]).transpose(1, 2) @ c
    return torch.cat(out, 1).transpose(0, 1)


def _layered_exact(case, seed):
    cfg, _, _, t = _layered_weights(case, seed)
    eps, seqs, new = cfg.rms_norm_eps, _tokens(case, seed), case["new"]
    lens = [len(s) for s in seqs]
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    x = t["embed"][torch.tensor([i for s in seqs for i in s], device="cuda")].double()

    def norm(v, name):
        return torch.tanh(t[name + ".alpha"].double() * v) * t[name].double() + t[name + ".b"].double()

    def gate(h, name):
        return torch.sigmoid(_mm(h, t[name]) + t[name + ".b"].double())

    def unit(z):
        return z * (z.square().mean(-1, keepdim=True) + eps).rsqrt()

    for i, s in enumerate(cfg.layer_specs):
        p, m = f"l{i}.", s.mixer
        h = norm(x, p + "norm1")

        def lin(name, src=h):
            return _mm(src, t[f"{p}mix.{name}"])

        if isinstance(m, LatentMixer):
            H, R = m.heads, m.kv_rank
            cos, sin = _angles(pos, m.rot_dim, m.rot.base)
            q = lin("q").view(-1, H, m.dim + m.rot_dim)
            q = torch.cat([q[..., :m.dim], _rotate(q[..., m.dim:], cos, sin)], -1)
            down = lin("dkv")
            c = unit(down[:, :R]) * t[p + "mix.dkv.norm"].double()
            kr = _rotate(down[:, None, R:], cos, sin).expand(-1, H, -1)
            k = torch.cat([lin("uk", c).view(-1, H, m.dim), kr], -1)
            v = lin("uv", c).view(-1, H, m.vdim)
            o = torch.cat([_attend(a, b, e, m.scale) for a, b, e in zip(q.split(lens), k.split(lens), v.split(lens))])
            o = (o.view(-1, H, m.vdim) * torch.sigmoid(lin("g"))[..., None]).reshape(len(pos), -1)
        else:
            dec = torch.tensor(m.decay, dtype=torch.float64, device="cuda")
            q, k, v = (torch.nn.functional.silu(lin(n)).view(len(pos), m.heads, -1) for n in "qkv")
            o = torch.cat([_decayed(a, b, e, dec) for a, b, e in zip(q.split(lens), k.split(lens), v.split(lens))]).reshape(len(pos), -1)
            o = unit(o) * t[p + "mix.norm"].double() * torch.sigmoid(lin("g"))
        x = x + lin("o", o) * gate(h, p + "rg1")
        h = norm(x, p + "norm2")
        z = _mm(h, t[p + "mlp.up"])
        a, b, c, e = t[p + "mlp.act"].double()
        z = a * unit(z) + b * unit(z * z) + c * unit(z * z * z) + e
        x = x + _mm(z, t[p + "mlp.down"]) * gate(h, p + "rg2")
    ends = torch.tensor(lens, device="cuda").cumsum(0)
    rows = ends[:, None] - new + torch.arange(new, device="cuda")
    logits = _mm(norm(x[rows.reshape(-1)], "final.norm"), t["embed"]).view(len(lens), new, -1).transpose(0, 1)
    return {"first": logits[0], "later": logits[1:]} if new > 1 else {"first": logits[0]}


def exact(case, seed):
    return _classic_exact(case, seed) if case["kind"] == "generate" else _layered_exact(case, seed)
