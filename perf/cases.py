"""The work this framework is used for, as cases that can be timed: sizes, inputs, one pass, what it cannot do without, and what
it should give.

Three kinds of program call the framework, and every case is a pass of one of them:

  * a program with a model of its own that keeps its keys and values in ``TrimKVCache`` (or the budget-sharing class) and
    attends through the attention registry: ``tokens`` (update, attention, eviction check per layer and forward pass, for one
    new token or a piece of a prompt) and ``handoff`` (a whole prompt reduced to its budget);
  * a program that runs a prompt through the mixers of the hybrid decoders: ``retention``, ``mamba2``, ``differential``,
    ``hgrn2``, ``latent`` (new requests, packed prompts of unequal length, result and the state they leave behind);
  * a program that decodes with a whole model: ``qwen3``, ``dafovik``, ``lonulix`` (one token of every request through
    ``GreedyDecoder``, ids supplied by the caller as after sampling).

Sizes are those of the repository's benchmark (layers of width 2048 and 4096, heads of 128 and 64, windows and budgets of 4096)
and what lies around them: one request to 64, a hundred tokens to 32768, budgets from 256.
"""
import math

import torch
import torch.nn.functional as F

DEV = "cuda"
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16}
EPS = 1e-6
VOCAB = 32768


# ---------------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # A chat with one user, a small budget: two layers' update and attention and the eviction check.  Latency and launches.
        dict(name="token 1 request", kind="tokens", batch=1, heads=16, kv_heads=8, memory=512, buffer=128, new=1, layers=2,
             dtype="bf16", budget="head"),
        # Serving 64 requests whose heads share each request's budget: lengths differ from head to head.
        dict(name="token 64 requests shared", kind="tokens", batch=64, heads=32, kv_heads=8, memory=2048, buffer=128, new=1,
             layers=1, dtype="f16", budget="request"),
        # A long prompt fed in pieces of 512 tokens against a full cache; every piece evicts.
        dict(name="piece of 512 8 requests", kind="tokens", batch=8, heads=16, kv_heads=8, memory=4096, buffer=512, new=512,
             layers=1, dtype="bf16", budget="head"),
        # The end of a prompt pass: 8192 tokens of every head reduced to the budget.
        dict(name="hand-off 4 requests", kind="handoff", batch=4, kv_heads=8, tokens=8192, memory=4096, buffer=128, layers=2,
             dtype="bf16"),
        # Prompts through the mixers.  Many long ones, the largest case ...
        dict(name="retention 4 x 8192", kind="retention", width=2048, heads=16, lengths="8192,8192,8192,8192"),
        # ... two of unequal length ...
        dict(name="mamba2 4096 + 2731", kind="mamba2", width=2048, heads=64, lengths="4096,2731"),
        # ... one that is twice the window ...
        dict(name="differential 8192", kind="differential", width=2048, heads=16, kv_heads=8, window=4096, lengths="8192"),
        # ... one short prompt ...
        dict(name="hgrn2 1 x 1500", kind="hgrn2", width=2048, heads=16, lengths="1500"),
        # ... and a wide layer.
        dict(name="latent 2 x 4096 wide", kind="latent", width=4096, heads=32, window=4096, lengths="4096,4096"),
        # Decoding with whole models (four layers of each).
        dict(name="qwen3 32 requests", kind="qwen3", width=2048, heads=16, kv_heads=8, ff=6144, memory=4096, buffer=128, batch=32),
        dict(name="dafovik 32 requests", kind="dafovik", width=2048, heads=16, kv_heads=8, ff=6144, window=4096, batch=32),
        dict(name="lonulix 8 requests", kind="lonulix", width=2048, heads=16, ff=6144, window=4096, batch=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lengths(rng, total):
    """One to four prompts, together at most ``total`` tokens, the shortest of a few hundred."""
    n = rng.choice((1, 1, 2, 3, 4))
    return ",".join(str(_log(rng, 200, total // n)) for _ in range(n))


def draw(rng):
    kind = rng.choice(("tokens", "tokens", "tokens", "handoff", "retention", "mamba2", "differential", "hgrn2", "latent", "qwen3",
                       "dafovik", "lonulix"))
    kv = rng.choice((2, 4, 8))
    if kind == "tokens":
        new = rng.choice((1, 1, 2, 16, 96, 333, 512))
        budget = "head" if new > 1 else rng.choice(("head", "head", "request"))
        memory = _log(rng, 256, 4096)
        room = max(1, 64 * 2048 // (memory * (1 if new == 1 else 4)))
        return dict(kind=kind, batch=_log(rng, 1, min(64, room)), heads=kv * rng.choice((1, 2, 4)), kv_heads=kv, memory=memory,
                    buffer=max(new, rng.choice((32, 128, 200))), new=new, layers=rng.choice((1, 2)),
                    dtype=rng.choice(("bf16", "bf16", "f16")), budget=budget)
    if kind == "handoff":
        tokens = _log(rng, 700, 8192)
        return dict(kind=kind, batch=_log(rng, 1, 4), kv_heads=kv, tokens=tokens, memory=max(200, tokens // rng.choice((2, 3, 5))),
                    buffer=rng.choice((32, 128)), layers=rng.choice((1, 2)), dtype=rng.choice(("bf16", "f16")))
    if kind in ("qwen3", "dafovik", "lonulix"):
        out = dict(kind=kind, width=2048, heads=16, ff=rng.choice((4096, 6144)), batch=_log(rng, 1, 32 if kind != "lonulix" else 16))
        if kind == "qwen3":
            return dict(out, kv_heads=8, memory=_log(rng, 500, 4096), buffer=128)
        return dict(out, window=64 * _log(rng, 8, 64), **(dict(kv_heads=8) if kind == "dafovik" else {}))
    out = dict(kind=kind, width=rng.choice((1024, 2048, 2048)), lengths=_lengths(rng, 8192))
    if kind == "mamba2":
        return dict(out, heads=rng.choice((32, 48, 64)))
    out["heads"] = rng.choice((8, 12, 16))
    if kind == "differential":
        return dict(out, kv_heads=rng.choice((2, 4)), window=_log(rng, 300, 4096))
    if kind == "latent":
        return dict(out, window=_log(rng, 300, 4096))
    return out


# ------------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.bfloat16, scale=1.0):
    return torch.randn(*shape, generator=g, device=DEV, dtype=dtype).mul_(scale)


def _log_beta(g, *shape, dtype, heads_at=None):
    """Log retention gates as a gate biased open gives them; with ``heads_at`` some heads keep longer than others."""
    z = 3.0 + 1.5 * torch.randn(*shape, generator=g, device=DEV)
    if heads_at is not None:
        z += 1.5 * heads_at[None, :, None]
    return F.logsigmoid(z).to(dtype)


def _token_inputs(c, seed):
    """Prompt and new rows of a cache: per layer ``(k, v, log beta)`` of both, and the queries."""
    g, dt = _gen(seed), TYPES[c["dtype"]]
    b, h, m, n = c["batch"], c["kv_heads"], c["memory"], c["new"]
    tilt = None
    prompt = m
    if c["budget"] == "request":
        tilt = torch.randn(h, generator=g, device=DEV)
        prompt = 2 * m
    first, new, q = [], [], []
    for _ in range(c["layers"]):
        for rows, into in ((prompt, first), (n, new)):
            into.append((_randn(g, b, h, rows, 128, dtype=dt), _randn(g, b, h, rows, 128, dtype=dt),
                         _log_beta(g, b, h, rows, dtype=dt, heads_at=tilt)))
        q.append(_randn(g, b, c["heads"], n, 128, dtype=dt))
    return prompt, first, new, q


RANKS = {"q_rank": 1536, "kv_rank": 512}


def _shapes(c):
    """Tensors of a mixer by the names its checkpoint uses, as ``(shape, scale, centre)``."""
    w, h = c["width"], c["heads"]
    m = w ** -0.5
    if c["kind"] == "retention":
        return {**{k: ((h * 128, w), m, 0.0) for k in "qkvg"}, "o": ((w, h * 128), (h * 128) ** -0.5, 0.0)}
    if c["kind"] == "mamba2":
        inner, ch = h * 64, h * 64 + 2 * 8 * 128
        return {"in": ((inner + ch + h, w), m, 0.0), "conv": ((ch, 4), 0.4, 0.0), "conv.b": ((ch,), 0.1, 0.0),
                "dt_bias": ((h,), 1.0, -4.0), "A_log": ((h,), 0.7, 1.5), "D": ((h,), 0.2, 1.0), "norm": ((inner,), 0.1, 1.0),
                "o": ((w, inner), inner ** -0.5, 0.0)}
    if c["kind"] == "differential":
        kv = c["kv_heads"]
        return {"q": ((h * 128, w), m, 0.0), "k": ((kv * 128, w), m, 0.0), "v": ((kv * 128, w), m, 0.0), "g": ((h, w), m, 0.0),
                "q.norm": ((64,), 0.2, 1.0), "k.norm": ((64,), 0.2, 1.0), **{k: ((64,), 0.1, 0.0) for k in ("lq1", "lk1", "lq2", "lk2")},
                "o": ((w, h * 128), (h * 128) ** -0.5, 0.0)}
    if c["kind"] == "hgrn2":
        return {**{k: ((h * 128, w), m, 0.0) for k in "qfv"}, "f.b": ((h * 128,), 1.0, 2.0), "lower": ((h * 128,), 0.12, 0.4),
                "norm": ((128,), 0.1, 1.0), "o": ((w, h * 128), (h * 128) ** -0.5, 0.0)}
    qr, kr = RANKS["q_rank"], RANKS["kv_rank"]
    return {"dq": ((qr, w), m, 0.0), "dq.norm": ((qr,), 0.1, 1.0), "uq": ((h * 192, qr), qr ** -0.5, 0.0), "dkv": ((kr + 64, w), m, 0.0),
            "dkv.norm": ((kr,), 0.1, 1.0), "uk": ((h * 128, kr), kr ** -0.5, 0.0), "uv": ((h * 128, kr), kr ** -0.5, 0.0),
            "o": ((w, h * 128), (h * 128) ** -0.5, 0.0)}


def _decay(heads):
    return [1 - 2.0 ** -(5 + 6 * i / heads) for i in range(heads)]


def _mixer_inputs(c, seed):
    g = _gen(seed)
    lengths = [int(n) for n in c["lengths"].split(",")]
    t = {}
    for name, (shape, scale, centre) in _shapes(c).items():
        t[name] = _randn(g, *shape, scale=scale).add_(centre)
        if name == "lower":
            t[name].clamp_(0.02, 0.8)
    return lengths, t, _randn(g, sum(lengths), c["width"])


def _make_mixer(c):
    from trimkv_b200 import mixers as X
    w, h = c["width"], c["heads"]
    return {"retention": lambda: X.RetentionMixer(w, h, 128, 128, _decay(h), 128, 1e6, EPS),
            "mamba2": lambda: X.SSDMixer(w, h, 64, 128, 8, 4, 8, EPS),
            "differential": lambda: X.DifferentialAttentionMixer(w, h, c["kv_heads"], 64, 128, c["window"], 0.125, 0.5, EPS),
            "hgrn2": lambda: X.HGRN2Mixer(w, h, 128, 128, EPS),
            "latent": lambda: X.LatentAttentionMixer(w, h, 128, 64, 128, RANKS["q_rank"], RANKS["kv_rank"], c["window"], 192 ** -0.5,
                                                     64, 1e6, EPS)}[c["kind"]]()


def _model(c, g):
    """A model of four layers with weights of its own, as the benchmark shapes them."""
    import trimkv_b200 as T
    w, h, ff = c["width"], c["heads"], c["ff"]
    if c["kind"] == "qwen3":
        cls, cfg = T.TrimKVQwen3ForCausalLM, T.TrimKVQwen3Config(
            hidden_size=w, num_hidden_layers=4, num_attention_heads=h, num_key_value_heads=c["kv_heads"], head_dim=128,
            intermediate_size=ff, vocab_size=VOCAB, rope_theta=1e6, retention_gate_intermediate_size=128, retention_gate_bias_init=3.0,
            memory_size=c["memory"], buffer_size=c["buffer"], compress_memory=True, compress_strategy="alpha",
            attn_implementation="tkv_b200")
    elif c["kind"] == "dafovik":
        kinds = {"retention": dict(heads=h, dim=128, vdim=128, rot=dict(base=1e6, dims=128), decay=_decay(h)),
                 "attention": dict(heads=h, kv_heads=c["kv_heads"], dim=64, vdim=128, mask=dict(size=c["window"]), scale=0.125, diff=0.5),
                 "mamba2": dict(heads=w // 32, vdim=64, state=128, groups=8, conv=4, norm_groups=8)}
        cls, cfg = T.DafovikForCausalLM, T.DafovikConfig(
            layers=[{"type": k, "mixer": kinds[k], "mlp": {"kind": "dense", "ff": ff * 3 // 2}}
                    for k in ("retention", "attention", "mamba2", "mamba2")], norm={"eps": EPS}, residual_mult=0.5, vocab=VOCAB, width=w)
    else:
        kinds = {"latent_attention": dict(heads=h, dim=128, rot_dim=64, vdim=128, mask=dict(size=c["window"]), scale=192 ** -0.5,
                                          rot=dict(base=1e6, dims=64), **RANKS),
                 "hgrn2": dict(heads=h, dim=128, vdim=128)}
        ffs = [{"kind": "dense", "ff": ff},
               {"kind": "moe", "expert": {"ff": ff // 4},
                "router": {"experts": 32, "identity": 4, "top": 6, "scale": 1.0, "groups": {"count": 4, "keep": 2}}}]
        types = ("latent_attention", "hgrn2", "hgrn2", "latent_attention")
        cls, cfg = T.LonulixForCausalLM, T.LonulixConfig(
            layers=[{"type": k, "mixer": kinds[k], "mlp": ffs[i % 2]} for i, k in enumerate(types)], norm={"eps": EPS, "groups": 4},
            embedding={"scale": 1.0}, postln_alpha=2.0, vocab=VOCAB, width=w)
    with torch.device("meta"):
        model = cls(cfg)
    model = model.to(torch.bfloat16).to_empty(device=DEV).eval()
    if c["kind"] == "qwen3":
        model.model.rotary_emb = type(model.model.rotary_emb)(cfg).to(DEV)      # its table is no parameter
        named = dict(model.named_parameters())
    else:
        named = model.checkpoint_tensors()
        for p in model.parameters():
            p.data.zero_()
    centre0 = c["kind"] == "dafovik"
    for name, p in named.items():
        p = p.data
        if p.dim() > 1:
            p.normal_(0.0, 1.0 if "embed" in name else 0.4 if name.endswith("conv") else p.shape[-1] ** -0.5, generator=g)
            continue
        stream_norm = name == "final.norm" or name.split(".")[-1] in ("norm1", "norm2")
        centre = 0.0 if centre0 and stream_norm else 1.0 if "norm" in name or name.endswith(".D") else 0.0
        centre, spread = {"dt_bias": (-4.0, 1.0), "A_log": (1.5, 0.7), "lower": (0.4, 0.1), "correction": (0.0, 0.01)}.get(
            name.split(".")[-1], (3.0, 0.3) if "retention_gate" in name else (2.0, 1.0) if name.endswith("f.b") else (centre, 0.1))
        p.normal_(centre, spread, generator=g)
    return model


@torch.no_grad()
def prepare(case, seed):
    c = case
    if c["kind"] == "tokens":
        import trimkv_b200 as T
        prompt, first, new, q = _token_inputs(c, seed)
        cache = T.TrimKVCache(device=DEV) if c["budget"] == "head" else T.BatchedDynamicBudgetTrimKVCache(device=DEV)
        at = torch.arange(prompt, device=DEV)
        for layer, (k, v, beta) in enumerate(first):
            cache.update(k, v, beta, at, layer)
        cache.compress(strategy="alpha", memory_size=c["memory"], buffer_size=c["buffer"])
        return dict(c=c, cache=cache, attend=T.get_attention_interface("tkv_b200"), new=new, q=q,
                    at=torch.arange(prompt, prompt + c["new"], device=DEV))
    if c["kind"] == "handoff":
        g, dt = _gen(seed), TYPES[c["dtype"]]
        b, h, n = c["batch"], c["kv_heads"], c["tokens"]
        rows = [(_randn(g, b, h, n, 128, dtype=dt), _randn(g, b, h, n, 128, dtype=dt), _log_beta(g, b, h, n, dtype=dt))
                for _ in range(c["layers"])]
        return dict(c=c, rows=rows, at=torch.arange(n, device=DEV))
    if c["kind"] in ("qwen3", "dafovik", "lonulix"):
        from trimkv_b200.decoder import GreedyDecoder
        g = _gen(seed)
        model = _model(c, g)
        n = (c["memory"] + c["buffer"] if c["kind"] == "qwen3" else c["window"]) + 37
        ids = torch.randint(0, VOCAB, (c["batch"], n + 1), generator=g, device=DEV)
        if c["kind"] == "qwen3":
            cache = model.new_cache()
            model(input_ids=ids[:, :n], past_key_values=cache, logits_to_keep=1)
        else:
            cache = model.new_cache(DEV, capacity_tokens=n + 64)
            cache.open(c["batch"])
            for lo in range(0, c["batch"], 8):      # the prompts of a few requests at a time
                rows = list(range(lo, min(c["batch"], lo + 8)))
                model.forward_packed(ids[rows, :n].reshape(-1), cache, [n] * len(rows), rows, [len(rows) * n - 1])
        decoder = GreedyDecoder(model, cache)
        next_ids = ids[:, n:].contiguous()
        decoder.step(next_ids, eager=True)
        decoder.step(next_ids)                       # records the step
        return dict(c=c, model=model, cache=cache, decoder=decoder, ids=next_ids)
    from trimkv_b200 import HybridStateCache
    lengths, t, x = _mixer_inputs(c, seed)
    with torch.device(DEV):
        mixer = _make_mixer(c).to(torch.bfloat16).eval()
    for name, p in mixer.checkpoint().items():
        p.data.copy_(t[name])
    cache = HybridStateCache([mixer.state()], DEV, torch.bfloat16, capacity_tokens=max(lengths))
    return dict(c=c, mixer=mixer, cache=cache, x=x, lengths=lengths)


# ----------------------------------------------------------------------------------------------------------------- one pass
@torch.no_grad()
def run(state):
    c = state["c"]
    if c["kind"] == "tokens":
        cache, outs = state["cache"], []
        for layer, ((k, v, beta), q) in enumerate(zip(state["new"], state["q"])):
            keys, values, _, _, kw = cache.update(k, v, beta, state["at"], layer)
            outs.append(state["attend"](None, q, keys, values, None, scaling=128 ** -0.5, flash_attn_kwargs=kw)[0])
        cache.compress(strategy="alpha", memory_size=c["memory"], buffer_size=c["buffer"])
        state["at"] += c["new"]
        if c["budget"] == "head" and c["new"] > 1:
            return outs, list(cache.key_cache), list(cache.value_cache), list(cache.kv_positions)
        return outs, [cache.head_lens[layer] for layer in range(c["layers"])]
    if c["kind"] == "handoff":
        from trimkv_b200 import TrimKVCache
        cache = TrimKVCache(device=DEV, memory_size=c["memory"], buffer_size=c["buffer"], num_layers=c["layers"])
        for layer, (k, v, beta) in enumerate(state["rows"]):
            cache.update(k, v, beta, state["at"], layer)
        cache.compress(strategy="alpha", memory_size=c["memory"], buffer_size=c["buffer"])
        return list(cache.key_cache), list(cache.value_cache), list(cache.kv_positions)
    if c["kind"] in ("qwen3", "dafovik", "lonulix"):
        decoder, cache = state["decoder"], state["cache"]
        decoder.step(state["ids"])
        if c["kind"] == "qwen3":
            n = cache.get_cache_length(0)
            return decoder.logits, [cache.key_cache[layer][:, :, n - 1] for layer in range(4)]
        return decoder.logits, [cache.arrays(layer) for layer in range(4)]
    cache, lengths = state["cache"], state["lengths"]
    if state.get("rows"):
        cache.close(state["rows"])                   # the requests of the pass before are done
    state["rows"] = cache.open(len(lengths))
    batch = cache.begin(lengths)
    y = state["mixer"](state["x"], batch, cache.arrays(0))
    data = cache.arrays(0)
    if "state" in data:
        return y, data["state"]
    kept = {"k": 1, "v": 1, "latent": 0}             # axis of the positions
    return y, {k: [t[i].narrow(kept[k], 0, min(lengths[i] if len(lengths) == 1 else min(lengths), t.shape[kept[k] + 1]))
                   for i in range(len(lengths))] for k, t in data.items()}


# ------------------------------------------------------------------------------------------------------------ work, tolerance
def _pairs(n, window):
    """Pairs (query, key) of a causal window over ``n`` positions."""
    w = min(n, window)
    return w * (w + 1) // 2 + (n - w) * w


def work(case):
    c = case
    if c["kind"] == "tokens":
        b, kv, h, m, n, rows = c["batch"], c["kv_heads"], c["heads"], c["memory"], c["new"], c["memory"] + c["new"]
        evict = b * kv * (m * 8 + m * 520) if n >= c["buffer"] else 0
        return {"bytes": c["layers"] * (b * kv * rows * 512 + b * kv * n * 520 + b * h * n * 512 + evict),
                "flops": c["layers"] * b * h * 4 * 128 * (n * m + n * (n + 1) // 2)}
    if c["kind"] == "handoff":
        return {"bytes": c["layers"] * c["batch"] * c["kv_heads"] * (c["tokens"] * 2 + c["memory"] * 2 * 520), "flops": 0}
    w, h = c["width"], c["heads"]
    if c["kind"] == "qwen3":
        weights = 4 * (w * (h * 128 * 2 + c["kv_heads"] * 256 + 128) + 3 * w * c["ff"]) + w * VOCAB
        kv = 4 * c["batch"] * c["kv_heads"] * (c["memory"] + c["buffer"] // 2) * 512
        return {"bytes": 2 * weights + kv, "flops": 2 * weights * c["batch"] + kv // 512 * (h // c["kv_heads"]) * 512}
    if c["kind"] == "dafovik":
        inner = 2 * w
        weights = 4 * 3 * w * c["ff"] + w * VOCAB + w * (5 * h * 128) + w * (2 * h * 128 + 2 * c["kv_heads"] * 128) + 2 * w * (3 * inner + 2048)
        kv = c["batch"] * (c["kv_heads"] * c["window"] * 512 + 2 * 4 * (h * 128 * 128 + 2 * inner * 128))
        return {"bytes": 2 * weights + kv, "flops": 2 * weights * c["batch"] + c["batch"] * h * c["window"] * 512}
    if c["kind"] == "lonulix":
        qr, kr = RANKS["q_rank"], RANKS["kv_rank"]
        latent = w * (qr + kr + 64) + qr * h * 192 + kr * h * 256 + w * h * 128
        experts = 2 * w * (c["ff"] // 4)
        hit = 32 * (1 - (1 - 6 / 36) ** c["batch"])
        weights = int(2 * latent + 2 * 4 * w * h * 128 + 2 * 4 * w * c["ff"] + 2 * hit * experts + 4 * w * w + w * VOCAB)
        kv = c["batch"] * (2 * c["window"] * (kr + 64) * 2 + 2 * 2 * 4 * h * 128 * 128)
        return {"bytes": 2 * weights + kv, "flops": 2 * weights * c["batch"] + c["batch"] * 2 * h * c["window"] * 2 * (2 * kr + 64)}
    lengths = [int(n) for n in c["lengths"].split(",")]
    T = sum(lengths)
    weights = sum(math.prod(shape) for shape, _, _ in _shapes(c).values())
    bytes_, flops = 2 * (weights + 2 * T * w), 2 * T * weights
    if c["kind"] in ("retention", "mamba2", "hgrn2"):
        p = 64 if c["kind"] == "mamba2" else 128
        return {"bytes": bytes_ + 4 * len(lengths) * h * 128 * p, "flops": flops + 4 * T * h * 128 * p}
    pairs = sum(_pairs(n, c["window"]) for n in lengths)
    per = 2 * (2 * 64 + 2 * 128) if c["kind"] == "differential" else 2 * (192 + 128)
    return {"bytes": bytes_, "flops": flops + pairs * h * per}


def tolerance(case):
    # 16-bit inputs and results, sums in 32 bits.  Copied rows and positions of a cache are equal bit for bit in every correct
    # implementation; only the outputs of attention and of the products differ.
    if case["kind"] == "handoff":
        return "exact"
    return {"rel": 1e-2, "max": 0.3}


# --------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _kept(k, v, beta, age, m):
    """The rows a head keeps: the ``m`` of the largest log beta x age, the lower position first among equals."""
    at = (beta.float() * age).sort(dim=-1, descending=True, stable=True).indices[..., :m].sort(dim=-1).values
    row = at[..., None].expand(*at.shape, k.shape[-1])
    return k.gather(2, row), v.gather(2, row), beta.gather(2, at), at


def _exact_tokens(c, seed):
    prompt, first, new, q = _token_inputs(c, seed)
    if c["layers"] * c["batch"] * c["heads"] * c["new"] * prompt > 2 ** 31:
        return None
    b, kv, n = c["batch"], c["kv_heads"], c["new"]
    group = c["heads"] // kv
    lens = [torch.full((b, kv), prompt, device=DEV) for _ in first]
    if c["budget"] == "request" and prompt > c["memory"] + c["buffer"]:
        age = (prompt + 1 - torch.arange(prompt, device=DEV)).to(first[0][2].dtype)
        scores = torch.cat([(beta * age).flatten(1) for _, _, beta in first], 1)
        top = scores.sort(dim=1, descending=True, stable=True).indices[:, :len(first) * kv * c["memory"]]
        mask = torch.zeros_like(scores, dtype=torch.bool).scatter_(1, top, True).view(b, len(first), kv, prompt)
        lens = [mask[:, i].sum(-1) for i in range(len(first))]
        kept = []
        for i, (k, v, beta) in enumerate(first):
            order = (~mask[:, i]).to(torch.int8).sort(dim=-1, stable=True).indices
            row = order[..., None].expand(*order.shape, 128)
            kept.append((k.gather(2, row), v.gather(2, row), beta.gather(2, order)))
        first = kept
    outs, keys, values = [], [], []
    total = 0
    for (k, v, beta), (k1, v1, beta1), qs, have in zip(first, new, q, lens):
        o = torch.empty(b, n, c["heads"], 128, dtype=torch.float64, device=DEV)
        for i in range(b):
            for h in range(kv):
                live = int(have[i, h])
                kk = torch.cat([k[i, h, :live], k1[i, h]]).double()
                vv = torch.cat([v[i, h, :live], v1[i, h]]).double()
                s = qs[i, h * group:(h + 1) * group].double() @ kk.T * 128 ** -0.5
                s += torch.full((n, live + n), float("-inf"), device=DEV, dtype=torch.float64).triu(live + 1)
                o[i, :, h * group:(h + 1) * group] = (s.softmax(-1) @ vv).transpose(0, 1)
        outs.append(o)
        total += int(have.sum()) + b * kv * n
        if c["budget"] == "head" and n > 1:
            kk, vv, bb = (torch.cat(x, 2) for x in ((k, k1), (v, v1), (beta, beta1)))
            if prompt + n >= c["memory"] + c["buffer"]:
                seen = prompt + n
                kk, vv, bb, _ = _kept(kk, vv, bb, (seen + 1 - torch.arange(seen, device=DEV)).float(), c["memory"])
            keys.append(kk.double())
            values.append(vv.double())
    if c["budget"] == "head" and n > 1:
        return outs, keys, values, [None] * len(keys)
    return outs, [None] * len(outs)


def _recurrence(q, k, v, log_decay, chunk=32):
    """S_t = diag(exp(log_decay_t)) S_(t-1) + k_t v_t^T, o_t = S_t^T q_t; [T, H, .], decays [T, H] or [T, H, N].  In chunks whose
    quotients of decays stay far inside the range of 64 bits."""
    T, H, N = q.shape
    log_decay = log_decay if log_decay.dim() == 3 else log_decay[:, :, None]
    q, k, v, d = (t.transpose(0, 1) for t in (q, k, v, log_decay))
    S = torch.zeros(H, N, v.shape[2], dtype=torch.float64, device=DEV)
    out = torch.empty(H, T, v.shape[2], dtype=torch.float64, device=DEV)
    for a in range(0, T, chunk):
        z = min(T, a + chunk)
        run_ = d[:, a:z].cumsum(1)
        up, down = q[:, a:z] * run_.exp(), k[:, a:z] * (-run_).exp()
        out[:, a:z] = up @ S + (up @ down.transpose(1, 2)).tril() @ v[:, a:z]
        end = run_[:, -1:]
        S = S * end.exp().transpose(1, 2) + (k[:, a:z] * (end - run_).exp()).transpose(1, 2) @ v[:, a:z]
    return out.transpose(0, 1), S


def _softmax_window(q, k, v, scale, window, block=1024):
    """q [T, H, D], k and v [T, H, .]; position i sees j with 0 <= i - j < window."""
    T = q.shape[0]
    out = torch.empty(T, q.shape[1], v.shape[2], dtype=torch.float64, device=DEV)
    for a in range(0, T, block):
        z, lo = min(T, a + block), max(0, a - window + 1)
        gap = torch.arange(a, z, device=DEV)[:, None] - torch.arange(lo, z, device=DEV)[None, :]
        for h in range(q.shape[1]):
            s = (q[a:z, h] @ k[lo:z, h].T * scale).masked_fill_((gap < 0) | (gap >= window), float("-inf"))
            out[a:z, h] = s.softmax(-1) @ v[lo:z, h]
    return out


def _turn(x, base, dims, pairs):
    """Rotary positions: dimension i with i + dims / 2, or neighbours where ``pairs``."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEV)
    a = torch.arange(x.shape[0], dtype=torch.float64, device=DEV)[:, None, None] * base ** (-2.0 * i / dims)
    u, v = (x[..., 0::2], x[..., 1::2]) if pairs else (x[..., :dims // 2], x[..., dims // 2:])
    a, b = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
    return torch.stack([a, b], -1).flatten(-2) if pairs else torch.cat([a, b], -1)


def _exact_request(c, t, x):
    """One request through a mixer: ``(result, state it leaves, by name)``."""
    T, h = x.shape[0], c["heads"]
    if c["kind"] == "retention":
        q, k, v, g = (F.linear(x, t[n]).view(T, h, 128) for n in "qkvg")
        q, k = _turn(q, 1e6, 128, False), _turn(k, 1e6, 128, False) * 128 ** -0.5
        decay = torch.tensor(_decay(h), dtype=torch.float64, device=DEV).log().expand(T, h)
        o, S = _recurrence(q, k, v, decay, 128)
        return (_rms(o) * F.silu(g)).flatten(1) @ t["o"].T, S
    if c["kind"] == "mamba2":
        inner = h * 64
        z, xbc, dt = F.linear(x, t["in"]).split([inner, inner + 2048, h], 1)
        xbc = F.silu(F.conv1d(F.pad(xbc.T, (3, 0))[None], t["conv"][:, None], t["conv.b"], groups=xbc.shape[1])[0].T)
        v, B, C = xbc.split([inner, 1024, 1024], 1)
        v, dt = v.reshape(T, h, 64), F.softplus(dt + t["dt_bias"], threshold=1e9)
        B, C = (y.reshape(T, 8, 128).repeat_interleave(h // 8, 1) for y in (B, C))
        o, S = _recurrence(C, B, v * dt[..., None], -t["A_log"].exp() * dt)
        y = (o + t["D"][:, None] * v).flatten(1) * F.silu(z)
        return (_rms(y.view(T, 8, -1)).flatten(1) * t["norm"]) @ t["o"].T, S
    if c["kind"] == "differential":
        kv = c["kv_heads"]
        q = _rms(F.linear(x, t["q"]).view(T, h, 2, 64)) * t["q.norm"]
        k = _rms(F.linear(x, t["k"]).view(T, kv, 2, 64)) * t["k.norm"]
        v = F.linear(x, t["v"]).view(T, kv, 128)
        wide = [y.repeat_interleave(h // kv, 1) for y in (k[:, :, 0], k[:, :, 1], v)]
        lam = (t["lq1"] @ t["lk1"]).exp() - (t["lq2"] @ t["lk2"]).exp() + 0.5
        a1, a2 = (_softmax_window(q[:, :, m], wide[m], wide[2], 0.125, c["window"]) for m in (0, 1))
        o = _rms(a1 - lam * a2) * 0.5 * F.linear(x, t["g"]).sigmoid()[:, :, None]
        return o.flatten(1) @ t["o"].T, None
    if c["kind"] == "hgrn2":
        q, f, v = (F.linear(x, t[n]) for n in "qfv")
        f = t["lower"] + (1 - t["lower"]) * (f + t["f.b"]).sigmoid()
        o, S = _recurrence(F.silu(q).view(T, h, 128), (1 - f).view(T, h, 128), v.view(T, h, 128), f.log().view(T, h, 128))
        return (_rms(o) * t["norm"]).flatten(1) @ t["o"].T, S
    kr = RANKS["kv_rank"]
    q = F.linear(_rms(F.linear(x, t["dq"])) * t["dq.norm"], t["uq"]).view(T, h, 192)
    down = F.linear(x, t["dkv"])
    lat = _rms(down[:, :kr]) * t["dkv.norm"]
    k, v = F.linear(lat, t["uk"]).view(T, h, 128), F.linear(lat, t["uv"]).view(T, h, 128)
    turned = _turn(down[:, None, kr:], 1e6, 64, True).expand(T, h, 64)
    q = torch.cat([q[..., :128], _turn(q[..., 128:], 1e6, 64, True)], -1)
    o = _softmax_window(q, torch.cat([k, turned], -1), v, 192 ** -0.5, c["window"])
    return o.flatten(1) @ t["o"].T, None


@torch.no_grad()
def exact(case, seed):
    c = case
    if c["kind"] == "tokens":
        return _exact_tokens(c, seed)
    if c["kind"] == "handoff" or work(c)["flops"] > 4e14 or c["kind"] in ("qwen3", "dafovik", "lonulix"):
        return None         # copied rows, compared bit for bit; or too long in 64 bits (whole models: the prompt behind the state)
    lengths, t, x = _mixer_inputs(c, seed)
    t = {k: v.double() for k, v in t.items()}
    ys, states = zip(*(_exact_request(c, t, part.double()) for part in x.split(lengths)))
    y = torch.cat(ys)
    return (y, torch.stack(states)) if states[0] is not None else (y, None)
