"""The work that users of this library have it do, as cases to time and to compare: requests that run from their prompts'
tokens through the decode steps behind them, by `Model.step` on a cache, as the generation loop and trace replay call it.

A case is one batch of requests: open slots, run the prompts in steps of at most 8,192 tokens (the engine's default), then
decode a token a step (the tokens are given, so that a pass can be compared number for number), close the slots. Outputs are
the logits that such a program reads: of each prompt's last token and of every decode step, or of every position where a
text is scored. Weights are random, inputs are drawn from the seed; the model, its cache and its captured steps are what a
serving process keeps.

`exact` restates the models in 64-bit torch: whole sequences, no cache, none of the package's code.
"""
import math
import random

import torch

LFM3_SHAPES = {
    # hidden, heads, feed-forward, context, layers, attention layers at
    "350m": (1024, 16, 6656, 32768, 16, (2, 5, 8, 10, 12, 14)),
    "1.2b": (2048, 32, 8192, 4096, 16, (2, 5, 8, 10, 12, 14)),
    "2.6b": (2048, 32, 10752, 8192, 30, tuple(range(2, 30, 3))),
}
KV_HEADS, HEAD_DIM, VOCAB = 8, 64, 65536
STEP_TOKENS = 8192


def _case(name, model, batch, lo, hi, new, dtype="bfloat16", score=False):
    return {"name": name, "model": model, "batch": batch, "prompt_min": lo, "prompt_max": hi, "new": new, "dtype": dtype,
            "score": score}


def listed():
    return [
        # one short question to the smallest model of the family, a short answer: launches and latency
        _case("chat_350m_b1", "350m", 1, 21, 21, 24),
        # one conversation turn on the 1.2B shape
        _case("chat_1.2b_b1", "1.2b", 1, 128, 128, 64),
        # the benchmark's headline: eight requests with 2,048-token prompts
        _case("decode_1.2b_b8", "1.2b", 8, 2048, 2048, 128),
        # a server full of short chats
        _case("chats_1.2b_b64", "1.2b", 64, 16, 160, 48),
        # a document read once, one answer token (classification, embedding of a prompt, a first token's latency)
        _case("prompt_1.2b_2048", "1.2b", 1, 2048, 2048, 0),
        # the family's large model with unequal prompts
        _case("ragged_2.6b_b16", "2.6b", 16, 256, 4096, 64),
        # the small model on long documents
        _case("long_350m_b12", "350m", 12, 1024, 24576, 32),
        # texts scored at every position (perplexity, reranking): a few unequal ones in a step
        _case("score_1.2b", "1.2b", 6, 40, 700, 0, score=True),
        # the 32-bit option, a few requests
        _case("float32_350m_b4", "350m", 4, 64, 512, 16, dtype="float32"),
        # the reference's own defaults: norms on the branches, a gate per head, seven taps, windowed layers
        _case("options_350m_b5", "options", 5, 100, 1500, 48),
        # latent attention, Mamba-2 and routed experts
        _case("saralix_b8", "saralix", 8, 300, 2048, 64),
        # blocked attention, mLSTM, routed experts with a shared unit, squared ReLU
        _case("nimelorn_b6", "nimelorn", 6, 300, 2048, 64),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    limit = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["chat", "chat", "documents", "documents", "long", "prompt", "score", "float32", "options", "saralix",
                           "nimelorn"])
        new, dtype, score = 0, "bfloat16", False
        if kind == "chat":
            model, batch = rng.choice(sorted(LFM3_SHAPES)), _log_int(rng, 1, 64)
            lo = _log_int(rng, 4, 128)
            hi, new = _log_int(rng, lo, 512), _log_int(rng, 8, 96)
        elif kind == "documents":
            model, batch = rng.choice(sorted(LFM3_SHAPES)), _log_int(rng, 1, 24)
            lo = _log_int(rng, 128, 2048)
            hi, new = _log_int(rng, lo, 3900), _log_int(rng, 16, 128)
        elif kind == "long":
            model, batch, lo, hi, new = "350m", _log_int(rng, 1, 12), 1024, _log_int(rng, 4096, 24576), _log_int(rng, 8, 64)
        elif kind == "prompt":
            model, batch = rng.choice(sorted(LFM3_SHAPES)), 1
            lo = hi = _log_int(rng, 8, 3900)
        elif kind == "score":
            model, batch, score = rng.choice(sorted(LFM3_SHAPES)), _log_int(rng, 1, 8), True
            lo = _log_int(rng, 16, 256)
            hi = _log_int(rng, lo, 800)
        elif kind == "float32":
            model, batch, dtype = "350m", _log_int(rng, 1, 8), "float32"
            lo = _log_int(rng, 8, 256)
            hi, new = _log_int(rng, lo, 700), _log_int(rng, 4, 32)
        else:
            model, batch = kind, _log_int(rng, 1, 12)
            lo = _log_int(rng, 16, 512)
            hi, new = _log_int(rng, lo, 2048), _log_int(rng, 8, 64)
        c = _case("", model, batch, lo, hi, new, dtype, score)
        del c["name"]
        if _cost(c) <= limit:
            return c


def _lengths(case):
    rng = random.Random("%(model)s %(batch)d %(prompt_min)d %(prompt_max)d" % case)
    return [rng.randint(case["prompt_min"], case["prompt_max"]) for _ in range(case["batch"])]


# ------------------------------------------------------------------------------------------- the models
def _lfm3_json(model):
    options = model == "options"
    hidden, heads, ffn, context, layers, attn = LFM3_SHAPES["350m" if options else model]
    kinds = ["full_attention" if i in attn else "conv" for i in range(layers)]
    c = {"model_type": "lfm3", "vocab_size": VOCAB, "hidden_size": hidden, "intermediate_size": ffn, "num_hidden_layers": layers,
         "num_attention_heads": heads, "num_key_value_heads": KV_HEADS, "head_dim": HEAD_DIM, "conv_L_cache": 7 if options else 3,
         "conv_bias": False, "norm_eps": 1e-5, "max_position_embeddings": context, "tie_word_embeddings": True,
         "use_sandwich_norm": options, "attn_head_gate": options, "initializer_range": 0.02}
    if options:
        kinds = ["sliding_attention" if k != "conv" and n % 2 else k for n, k in enumerate(kinds)]
        c["sliding_window"] = 512
    c["layer_types"] = kinds
    c["rope_parameters"] = {k: {"rope_theta": 1000000.0} for k in sorted(set(kinds)) if k != "conv"}
    return c


def _saralix_json():
    rot = {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 1024, "fast": 32.0, "slow": 1.0}}
    latent = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "rot": rot}
    mamba = {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    moe = {"kind": "moe", "expert": {"ff": 1024}, "router": {"experts": 16, "top": 4}}
    layers = [("latent_attention", latent, {"kind": "dense", "ff": 8192, "limit": 7.0}),
              ("mamba2", mamba, moe),
              ("latent_attention_2", dict(latent, mask={"size": 1024}), moe),
              ("mamba2", mamba, moe)]
    return {"architecture": "Saralix", "width": 2048, "vocab": 32768, "norm": {"eps": 1e-5},
            "layers": [{"type": t, "mixer": m, "mlp": f} for t, m, f in layers]}


def _nimelorn_json():
    def attention(heads, kv_heads, vdim):
        return {"heads": heads, "kv_heads": kv_heads, "dim": 64, "vdim": vdim, "mask": {"size": 1024}, "scale": 0.125}

    moe = {"kind": "moe", "expert": {"ff": 1024, "limit": 7.0}, "router": {"experts": 16, "top": 4, "scale": 1.0},
           "shared": {"ff": 1024, "limit": 7.0}}
    mlstm = {"heads": 16, "dim": 64, "vdim": 128, "gate_cap": 15.0}
    layers = [("attention", attention(32, 8, 64), {"kind": "dense", "ff": 8192}), ("mlstm", mlstm, moe),
              ("attention", attention(16, 4, 96), moe), ("mlstm", mlstm, moe)]
    return {"architecture": "Nimelorn", "width": 2048, "vocab": 32768, "norm": {"eps": 1e-5},
            "embedding": {"scale": 2048.0 ** 0.5, "bigram": {"buckets": 65521, "mul_prev": 8191, "mul_cur": 31}},
            "layers": [{"type": t, "mixer": m, "mlp": f} for t, m, f in layers]}


def _json(case):
    return {"saralix": _saralix_json, "nimelorn": _nimelorn_json}.get(case["model"], lambda: _lfm3_json(case["model"]))()


def _shapes(case):
    """name -> (shape, kind): "m" a matrix N(0, 0.02), "b" one that ends a branch (smaller by the square root of the number of
    branches, the usual start of training), "e" the tied table, "t" taps, "v" a norm's weight, "p" the weight of a norm on a
    branch, "u:lo:hi" a vector drawn evenly, "r" a router (spread, as a trained one's: its choices are then few close calls)."""
    c, out = _json(case), {}
    if case["model"] in LFM3_SHAPES or case["model"] == "options":
        H, F, D = c["hidden_size"], c["intermediate_size"], c["head_dim"]
        Hq, Hkv = c["num_attention_heads"], c["num_key_value_heads"]
        out["embed_tokens.weight"] = ((c["vocab_size"], H), "e")
        out["embedding_norm.weight"] = ((H,), "v")
        for i, kind in enumerate(c["layer_types"]):
            p = "layers.%d." % i
            for n in ("operator_norm", "ffn_norm") + (("post_operator_norm", "post_ffn_norm") if c["use_sandwich_norm"] else ()):
                out[p + n + ".weight"] = ((H,), "p" if n.startswith("post") else "v")
            if kind == "conv":
                out[p + "conv.in_proj.weight"] = ((3 * H, H), "m")
                out[p + "conv.conv.weight"] = ((H, 1, c["conv_L_cache"]), "t")
                out[p + "conv.out_proj.weight"] = ((H, H), "b")
            else:
                a = p + "self_attn."
                out[a + "q_proj.weight"], out[a + "o_proj.weight"] = ((Hq * D, H), "m"), ((H, Hq * D), "b")
                out[a + "k_proj.weight"] = out[a + "v_proj.weight"] = ((Hkv * D, H), "m")
                out[a + "q_norm.weight"] = out[a + "k_norm.weight"] = ((D,), "v")
                if c["attn_head_gate"]:
                    out[a + "gate_proj.weight"] = ((Hq, H), "m")
            out[p + "feed_forward.w1.weight"] = out[p + "feed_forward.w3.weight"] = ((F, H), "m")
            out[p + "feed_forward.w2.weight"] = ((H, F), "b")
        return out
    W = c["width"]
    saralix = case["model"] == "saralix"
    out["embed"], out["final.norm"] = ((c["vocab"], W), "e" if saralix else "m"), ((W,), "v")
    if case["model"] == "nimelorn":
        out["bigram"] = ((c["embedding"]["bigram"]["buckets"] + 1, W), "m")
        out["embed.norm"], out["head"] = ((W,), "v"), ((c["vocab"], W), "m")
    for i, layer in enumerate(c["layers"]):
        p, kind, m, f = "l%d." % i, layer["type"], layer["mixer"], layer["mlp"]
        for n in ("norm1", "norm2") + (("norm1b", "norm2b") if saralix else ()):
            out[p + n] = ((W,), "v" if saralix and not n.endswith("b") else "p")
        x = p + "mix."
        if kind.startswith("latent_attention"):
            H = m["heads"]
            out[x + "q"] = ((H * (m["dim"] + m["rot_dim"]), W), "m")
            out[x + "dkv"], out[x + "dkv.norm"] = ((m["kv_rank"] + m["rot_dim"], W), "m"), ((m["kv_rank"],), "v")
            out[x + "uk"], out[x + "uv"] = ((H * m["dim"], m["kv_rank"]), "m"), ((H * m["vdim"], m["kv_rank"]), "m")
            out[x + "o"] = ((W, H * m["vdim"]), "m")
            if kind == "latent_attention":
                out[x + "g"] = ((H, W), "m")
            else:
                out[x + "sink"] = ((H,), "u:-1:1")
        elif kind == "mamba2":
            inner, wide = m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
            out[x + "in"], out[x + "o"] = ((inner + wide + m["heads"], W), "m"), ((W, inner), "m")
            out[x + "conv"], out[x + "conv.b"] = ((wide, m["conv"]), "u:-0.5:0.5"), ((wide,), "u:-0.1:0.1")
            out[x + "dt_bias"], out[x + "A_log"] = ((m["heads"],), "u:-3:0"), ((m["heads"],), "u:-1:1.5")
            out[x + "D"], out[x + "norm"] = ((m["heads"],), "u:0.5:1.5"), ((inner,), "v")
        elif kind == "attention":
            H, G = m["heads"], m["kv_heads"]
            out[x + "q"], out[x + "k"] = ((H * m["dim"], W), "m"), ((G * m["dim"], W), "m")
            out[x + "v"], out[x + "o"], out[x + "g"] = ((G * m["vdim"], W), "m"), ((W, H * m["vdim"]), "m"), ((H, W), "m")
            out[x + "q.norm"] = out[x + "k.norm"] = ((m["dim"],), "v")
        else:
            H, inner = m["heads"], m["heads"] * m["vdim"]
            out[x + "q"] = out[x + "k"] = ((H * m["dim"], W), "m")
            out[x + "v"] = out[x + "g"] = ((inner, W), "m")
            out[x + "o"], out[x + "norm"] = ((W, inner), "m"), ((inner,), "v")
            out[x + "i"] = out[x + "f"] = ((H, W), "m")
            out[x + "i.b"], out[x + "f.b"] = ((H,), "u:-1:1"), ((H,), "u:1:4")
        y = p + "mlp."
        if f["kind"] == "dense":
            for n in ("gate", "up") if saralix else ("up",):
                out[y + n] = ((f["ff"], W), "m")
            out[y + "down"] = ((W, f["ff"]), "m")
        else:
            units = ["e%d." % e for e in range(f["router"]["experts"])] + (["shared."] if f.get("shared") else [])
            for u in units:
                ff = (f["shared"] if u == "shared." else f["expert"])["ff"]
                out[y + u + "gate"] = out[y + u + "up"] = ((ff, W), "m")
                out[y + u + "down"] = ((W, ff), "m")
            out[y + "router"] = ((f["router"]["experts"], W), "r")
            if f.get("shared"):
                out[y + "shared.sg"] = ((1, W), "m")
    return out


def _weights(case, seed):
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    c, out = _json(case), {}
    branches = 2 * (c["num_hidden_layers"] if "num_hidden_layers" in c else len(c["layers"]))
    for name, (shape, kind) in _shapes(case).items():
        if kind in "vp":
            lo, hi = (0.75, 1.25) if kind == "v" else (0.15, 0.35)
            out[name] = torch.empty(shape, device="cuda").uniform_(lo, hi, generator=g)
        elif kind.startswith("u:"):
            out[name] = torch.empty(shape, device="cuda").uniform_(*(float(v) for v in kind.split(":")[1:]), generator=g)
        else:
            std = {"m": 0.02, "b": 0.02 * branches ** -0.5, "e": 0.5, "t": 0.4, "r": 0.1}[kind]
            out[name] = torch.empty(shape, device="cuda", dtype=torch.float32).normal_(0.0, std, generator=g).to(dtype)
    return out


def _tokens(case, seed):
    """Each request's prompt and the tokens its decode steps are fed."""
    g = torch.Generator().manual_seed(7919 * seed + 3)
    vocab = VOCAB if case["model"] not in ("saralix", "nimelorn") else 32768
    return [torch.randint(vocab, (n + case["new"],), generator=g).tolist() for n in _lengths(case)]


# ------------------------------------------------------------------------------------------- the pass
def prepare(case, seed):
    from xpu_serve_b200 import Lfm3Config, NimelornConfig, SaralixConfig
    from xpu_serve_b200.engine.model import Model
    kind = {"saralix": SaralixConfig, "nimelorn": NimelornConfig}.get(case["model"], Lfm3Config)
    config = kind.from_json(_json(case))
    weights = _weights(case, seed)
    if kind is NimelornConfig:               # (its mixers pad theirs on the host, where a folder's weights lie)
        weights = {n: t.cpu() if ".mix." in n else t for n, t in weights.items()}
    model = Model(config.model_spec(), weights, dtype=case["dtype"], device="cuda:0", config=config)
    lens, new = _lengths(case), case["new"]
    held = sum(-(-(n + new) // 64) * 64 for n in lens)
    context = config.max_position_embeddings if kind is Lfm3Config else 4096
    cache = model.new_cache(held + 64 * len(lens), max_slots=len(lens), max_seq_tokens=context)
    vocab = model.spec.vocab
    state = {"model": model, "cache": cache, "new": new, "score": case["score"],
             "prompt_out": torch.empty((len(lens), vocab), device="cuda"),
             "decode_out": torch.empty((new, len(lens), vocab), device="cuda")}
    # a serving process has run a batch before: its steps are captured and its scratch buffers are there
    for s in (seed + 500009, seed):
        tokens = _tokens(case, s)
        state["prompts"] = [t[:n] for t, n in zip(tokens, lens)]
        state["fed"] = [[[t[n + k]] for t, n in zip(tokens, lens)] for k in range(new)]
        if s != seed:
            run(state)
    return state


def run(state):
    model, cache, prompts = state["model"], state["cache"], state["prompts"]
    slots = cache.open(len(prompts))
    if state["score"]:
        logits = model.step(cache, slots, prompts, [list(range(len(p))) for p in prompts])
        cache.close(slots)
        return logits
    at, done = [0] * len(prompts), 0
    while done < len(prompts):
        left, part, pieces, want = STEP_TOKENS, [], [], []
        for i, p in enumerate(prompts):
            take = min(len(p) - at[i], left)
            if take > 0:
                part.append(slots[i])
                pieces.append(p[at[i]:at[i] + take])
                at[i] += take
                left -= take
                want.append([take - 1] if at[i] == len(p) else [])
        logits = model.step(cache, part, pieces, want)
        state["prompt_out"][done:done + logits.shape[0]].copy_(logits)
        done += logits.shape[0]
    for k in range(state["new"]):
        state["decode_out"][k].copy_(model.step(cache, slots, state["fed"][k]))
    cache.close(slots)
    return {"prompt": state["prompt_out"], "decode": state["decode_out"]} if state["new"] else state["prompt_out"]


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Weights once a step (a decode step waits for the one before it and no cache holds them), earlier keys, values and
    state as far as a step reads them, logits written; two operations a weight a token, attention's two products over the
    visible pairs, the recurrences' updates and reads."""
    c, item = _json(case), 4 if case["dtype"] == "float32" else 2
    lens, new, batch = _lengths(case), case["new"], case["batch"]
    tokens, steps = sum(lens), -(-sum(lens) // STEP_TOKENS)
    vocab = c.get("vocab_size", c.get("vocab"))
    wide = c.get("hidden_size", c.get("width"))
    head = vocab * wide
    rows = tokens if case["score"] else batch
    sizes = {n: math.prod(s) for n, (s, _) in _shapes(case).items()}
    experts = c["layers"][1]["mlp"]["router"] if "layers" in c else None
    routed = sum(v for n, v in sizes.items() if ".mlp.e" in n)
    plain = sum(v for n, v in sizes.items() if ".mlp.e" not in n and n not in ("embed", "embed_tokens.weight", "bigram", "head"))
    top, of = (experts["top"], experts["experts"]) if experts else (1, 1)

    def touched(t):              # expected share of the experts that t tokens meet
        return 1.0 - (1.0 - top / of) ** t

    weight = steps * (plain + head + routed) + new * (plain + head + routed * touched(batch))
    flops = 2.0 * (tokens + new * batch) * (plain + routed * top / of) + 2.0 * (rows + new * batch) * head
    moved = 0.0
    for i in range(len(c["layer_types"]) if "layer_types" in c else len(c["layers"])):
        if "layer_types" in c:
            kind, H, G, D = c["layer_types"][i], c["num_attention_heads"], KV_HEADS, HEAD_DIM
            window = c["sliding_window"] if kind == "sliding_attention" else 0
            per_key, per_pair = 2 * G * D * item, 4.0 * H * D
            state = 0 if kind != "conv" else 2 * (c["conv_L_cache"] - 1) * wide * item
            attn, per_token = kind != "conv", 2.0 * c["conv_L_cache"] * wide
        else:
            kind, m = c["layers"][i]["type"], c["layers"][i]["mixer"]
            attn, state, per_token, window = "attention" in kind, 0, 0.0, m.get("mask", {}).get("size", 0)
            if kind.startswith("latent"):
                per_key, per_pair = (m["kv_rank"] + m["rot_dim"]) * item, 2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            elif attn:
                per_key, per_pair = m["kv_heads"] * (m["dim"] + m["vdim"]) * item, 2.0 * m["heads"] * (m["dim"] + m["vdim"])
            else:
                cells = m["heads"] * m["vdim"] * m.get("state", m.get("dim"))
                state, per_token = 8 * cells, 6.0 * cells
        for n in lens:
            if attn:
                w = window or n + new
                pairs = min(n, w) * (min(n, w) + 1) / 2 + max(0, n - w) * w
                seen = sum(min(n + k + 1, w) for k in range(new))
                flops += per_pair * (pairs + seen)
                moved += per_key * (n + seen)
            else:
                flops += per_token * (n + new)
                moved += state * (1 + new)
    moved += 4.0 * vocab * (rows + new * batch) + item * wide * (tokens + new * batch)
    return {"bytes": weight * item + moved, "flops": flops}


def _cost(case):
    w = work(case)
    return w["bytes"] / 4e12 + w["flops"] / (2e13 if case["dtype"] == "float32" else 8e14) + 1e-4 * case["new"]


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 5e-6}         # (measured: 3e-7 off the 64-bit result)
    return {"rel": 0.02}             # (measured: 0.003 to 0.012 off the 64-bit result)


# ------------------------------------------------------------------------------------------- the models in 64 bits
def _rms(x, w, eps):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt((d * d).mean(-1, keepdim=True) + eps) * w


def _mm(x, w):
    return x @ w.double().t()


def _rotate(x, pos, freq, scale=1.0):
    ang = pos.double()[:, None, None] * freq
    n = freq.numel()
    a, b, cos, sin = x[..., :n], x[..., n:2 * n], torch.cos(ang) * scale, torch.sin(ang) * scale
    return torch.cat([a * cos - b * sin, b * cos + a * sin, x[..., 2 * n:]], -1)


def _attend(q, k, v, scale, window=0, block=0, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, E] of one sequence: causal, optionally over the last `window` keys or the query's own
    block of `block` positions, optionally with a sink per head in the denominator."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device=q.device)
    size = max(64, min(2048, (1 << 29) // (T * (H // G))))
    for a in range(0, T, size):
        b = min(T, a + size)
        first = max(0, a - window + 1) if window else (a // block) * block if block else 0
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(first, b, device=q.device)[None, :]
        hide = j > i
        if window:
            hide = hide | (i - j >= window)
        if block:
            hide = hide | (torch.div(i, block, rounding_mode="floor") != torch.div(j, block, rounding_mode="floor"))
        for g in range(G):
            heads = slice(g * (H // G), (g + 1) * (H // G))
            s = torch.einsum("thd,kd->htk", q[a:b, heads], k[first:b, g]) * scale
            s.masked_fill_(hide[None], -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[heads].double()[:, None, None].expand(-1, b - a, 1)], -1)
            s = torch.softmax(s, -1)[..., :b - first]
            out[a:b, heads] = torch.einsum("htk,ke->the", s, v[first:b, g])
    return out


class _Batch:
    """Where each sequence's rows lie among the rows of all."""

    def __init__(self, lens):
        self.lens, self.at = lens, [sum(lens[:i]) for i in range(len(lens))]
        self.pos = torch.cat([torch.arange(n, device="cuda") for n in lens])

    def each(self, f, *xs):
        return torch.cat([f(*(x[a:a + n] for x in xs)) for a, n in zip(self.at, self.lens)])

    def padded(self, x):
        out = torch.zeros(max(self.lens), len(self.lens), *x.shape[1:], dtype=x.dtype, device=x.device)
        for i, (a, n) in enumerate(zip(self.at, self.lens)):
            out[:n, i] = x[a:a + n]
        return out

    def packed(self, x):
        return torch.cat([x[:n, i] for i, n in enumerate(self.lens)])


def _in_parts(f, x, rows=16384):
    return torch.cat([f(x[a:a + rows]) for a in range(0, x.shape[0], rows)])


def _filter(x, taps):
    """Causal, per channel: the last tap belongs to the current row."""
    n = taps.shape[1]
    ext = torch.cat([torch.zeros(n - 1, x.shape[1], dtype=x.dtype, device=x.device), x])
    return sum(taps[:, j].double() * ext[j:j + x.shape[0]] for j in range(n))


def _lfm3_exact(c, w, batch, ids):
    eps, D, Hq, H = c["norm_eps"], HEAD_DIM, c["num_attention_heads"], c["hidden_size"]
    theta = 1000000.0
    freq = torch.tensor([theta ** (-2.0 * i / D) for i in range(D // 2)], dtype=torch.float64, device="cuda")
    h = w["embed_tokens.weight"][ids].double()
    for i, kind in enumerate(c["layer_types"]):
        p = "layers.%d." % i
        x = _rms(h, w[p + "operator_norm.weight"].double(), eps)
        if kind == "conv":
            def conv(x):
                b, g, v = _mm(x, w[p + "conv.in_proj.weight"]).split(H, -1)
                return g * _filter(b * v, w[p + "conv.conv.weight"].reshape(H, -1))
            y = _mm(batch.each(conv, x), w[p + "conv.out_proj.weight"])
        else:
            a = p + "self_attn."
            q = _rms(_mm(x, w[a + "q_proj.weight"]).view(-1, Hq, D), w[a + "q_norm.weight"].double(), eps)
            k = _rms(_mm(x, w[a + "k_proj.weight"]).view(-1, KV_HEADS, D), w[a + "k_norm.weight"].double(), eps)
            v = _mm(x, w[a + "v_proj.weight"]).view(-1, KV_HEADS, D)
            q, k = _rotate(q, batch.pos, freq), _rotate(k, batch.pos, freq)
            window = c["sliding_window"] if kind == "sliding_attention" else 0
            y = batch.each(lambda q, k, v: _attend(q, k, v, D ** -0.5, window), q, k, v)
            if c["attn_head_gate"]:
                y = y * torch.sigmoid(_mm(x, w[a + "gate_proj.weight"]))[..., None]
            y = _mm(y.reshape(-1, Hq * D), w[a + "o_proj.weight"])
        h = h + (_rms(y, w[p + "post_operator_norm.weight"].double(), eps) if c["use_sandwich_norm"] else y)
        f = p + "feed_forward."
        w1, w3, w2 = w[f + "w1.weight"], w[f + "w3.weight"], w[f + "w2.weight"]
        y = _in_parts(lambda x: _mm(torch.nn.functional.silu(_mm(x, w1)) * _mm(x, w3), w2), _rms(h, w[p + "ffn_norm.weight"].double(), eps))
        h = h + (_rms(y, w[p + "post_ffn_norm.weight"].double(), eps) if c["use_sandwich_norm"] else y)
    return h, lambda rows: _mm(_rms(rows, w["embedding_norm.weight"].double(), eps), w["embed_tokens.weight"])


def _experts(f, w, y, x, unit):
    z = _mm(x, w[y + "router"])
    top = torch.topk(z, f["router"]["top"], -1)
    share = torch.zeros_like(z).scatter_(1, top.indices, torch.softmax(top.values, -1) * f["router"].get("scale", 1.0))
    out = torch.zeros_like(x)
    for e in range(z.shape[1]):
        rows = share[:, e].nonzero()[:, 0]
        if rows.numel():
            out[rows] += share[rows, e, None] * unit(x[rows], y + "e%d." % e)
    return out


def _clamped(w, p, x, limit):
    g, u = _mm(x, w[p + "gate"]).clamp(max=limit), _mm(x, w[p + "up"]).clamp(-limit, limit)
    return _mm(g * torch.sigmoid(1.702 * g) * (u + 1.0), w[p + "down"])


def _saralix_latent(m, w, x, h, batch, kind, eps):
    H, D, R, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    rot, sc = m["rot"], m["rot"]["scaling"]
    n = rot["dims"] // 2
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    freq = rot["base"] ** (-2.0 * i / rot["dims"])

    def turn(t):
        return rot["dims"] * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(rot["base"]))

    lo, hi = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), rot["dims"] - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    freq, factor = freq / sc["factor"] * ramp + freq * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    q = _mm(h, w[x + "q"]).view(-1, H, D + R)
    down = _mm(h, w[x + "dkv"])
    latent = _rms(down[:, :rank], w[x + "dkv.norm"].double(), eps)
    q = torch.cat([q[..., :D], _rotate(q[..., D:], batch.pos, freq, factor)], -1)
    k_rot = _rotate(down[:, None, rank:], batch.pos, freq, factor)
    k = torch.cat([_mm(latent, w[x + "uk"]).view(-1, H, D), k_rot.expand(-1, H, -1)], -1)
    v = _mm(latent, w[x + "uv"]).view(-1, H, m["vdim"])
    if kind == "latent_attention":
        y = batch.each(lambda q, k, v: _attend(q, k, v, m["scale"]), q, k, v)
        y = y * torch.sigmoid(_mm(h, w[x + "g"]))[..., None]
    else:
        y = batch.each(lambda q, k, v: _attend(q, k, v, m["scale"], m["mask"]["size"], sink=w[x + "sink"]), q, k, v)
    return _mm(y.reshape(h.shape[0], -1), w[x + "o"])


def _saralix_mamba(m, w, x, h, batch, eps):
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    z, xbc, dt = _mm(h, w[x + "in"]).split([inner, inner + 2 * G * N, H], -1)
    xbc = torch.nn.functional.silu(batch.each(lambda t: _filter(t, w[x + "conv"]), xbc) + w[x + "conv.b"].double())
    dt = torch.nn.functional.softplus(dt + w[x + "dt_bias"].double())
    v, B, C = (batch.padded(t) for t in xbc.split([inner, G * N, G * N], -1))
    T, S = v.shape[:2]
    v = v.view(T, S, G, H // G, P)
    B, C = B.view(T, S, G, 1, N), C.view(T, S, G, 1, N)
    step = batch.padded(dt).view(T, S, G, H // G, 1)
    keep = torch.exp(-torch.exp(w[x + "A_log"].double()).view(G, H // G, 1) * step)
    s = torch.zeros(S, G, H // G, N, P, dtype=torch.float64, device="cuda")
    out = torch.empty_like(v)
    for t in range(T):
        s = s * keep[t][..., None] + (step[t] * B[t])[..., None] * v[t][..., None, :]
        out[t] = (s * C[t][..., None]).sum(-2)
    y = out + w[x + "D"].double().view(G, H // G, 1) * v
    y = batch.packed(y.view(T, S, inner)) * torch.nn.functional.silu(z)
    y = _rms(y.view(-1, m["norm_groups"], inner // m["norm_groups"]), None, eps).reshape(-1, inner) * w[x + "norm"].double()
    return _mm(y, w[x + "o"])


def _saralix_exact(c, w, batch, ids):
    eps = c["norm"]["eps"]

    def unit(x, p):
        return _mm(torch.nn.functional.silu(_mm(x, w[p + "gate"])) * _mm(x, w[p + "up"]), w[p + "down"])

    h = w["embed"][ids].double()
    for i, layer in enumerate(c["layers"]):
        p, kind, m, f = "l%d." % i, layer["type"], layer["mixer"], layer["mlp"]
        x = _layer_norm(h, w[p + "norm1"].double(), eps)
        y = (_saralix_mamba(m, w, p + "mix.", x, batch, eps) if kind == "mamba2"
             else _saralix_latent(m, w, p + "mix.", x, batch, kind, eps))
        h = h + _layer_norm(y, w[p + "norm1b"].double(), eps)
        x = _layer_norm(h, w[p + "norm2"].double(), eps)
        y = _clamped(w, p + "mlp.", x, f["limit"]) if f["kind"] == "dense" else _experts(f, w, p + "mlp.", x, unit)
        h = h + _layer_norm(y, w[p + "norm2b"].double(), eps)
    return h, lambda rows: _mm(_layer_norm(rows, w["final.norm"].double(), eps), w["embed"])


def _nimelorn_mlstm(m, w, x, h, batch, eps):
    H, D, E, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k = (batch.padded(_mm(h, w[x + n]).view(-1, H, D)) for n in ("q", "k"))
    q = q * D ** -0.5
    v = batch.padded(_mm(h, w[x + "v"]).view(-1, H, E))
    gi = batch.padded(cap * torch.tanh((_mm(h, w[x + "i"]) + w[x + "i.b"].double()) / cap))
    gf = batch.padded(torch.nn.functional.logsigmoid(cap * torch.tanh((_mm(h, w[x + "f"]) + w[x + "f.b"].double()) / cap)))
    T, S = q.shape[:2]
    s = torch.zeros(S, H, D, E, dtype=torch.float64, device="cuda")
    n, top = torch.zeros(S, H, D, dtype=torch.float64, device="cuda"), torch.zeros(S, H, dtype=torch.float64, device="cuda")
    out = torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(gf[t] + top, gi[t])
        a, b = torch.exp(gf[t] + top - new)[..., None], torch.exp(gi[t] - new)[..., None]
        s = a[..., None] * s + (b * k[t])[..., None] * v[t][..., None, :]
        n, top = a * n + b * k[t], new
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out[t] = (s * q[t][..., None]).sum(-2) / den[..., None]
    y = batch.packed(_rms(out, None, eps).view(T, S, H * E)) * w[x + "norm"].double()
    return _mm(y * torch.sigmoid(_mm(h, w[x + "g"])), w[x + "o"])


def _nimelorn_exact(c, w, batch, ids):
    eps, e, wide = c["norm"]["eps"], c["embedding"], c["width"]
    b = e["bigram"]
    prev = torch.cat([ids[:1], ids[:-1]])
    rows = torch.where(batch.pos == 0, torch.full_like(ids, b["buckets"]), (prev * b["mul_prev"] + ids * b["mul_cur"]) % b["buckets"])
    ang = batch.pos.double()[:, None] * 10000.0 ** (-2.0 * torch.arange(wide // 2, dtype=torch.float64, device="cuda") / wide)
    h = w["embed"][ids].double() * e["scale"] + w["bigram"][rows].double() + torch.stack([torch.sin(ang), torch.cos(ang)], -1).flatten(1)
    h = _rms(h, w["embed.norm"].double(), eps)
    for i, layer in enumerate(c["layers"]):
        p, m, f = "l%d." % i, layer["mixer"], layer["mlp"]
        x = p + "mix."
        if layer["type"] == "mlstm":
            y = _nimelorn_mlstm(m, w, x, h, batch, eps)
        else:
            q = _rms(_mm(h, w[x + "q"]).view(-1, m["heads"], m["dim"]), w[x + "q.norm"].double(), eps)
            k = _rms(_mm(h, w[x + "k"]).view(-1, m["kv_heads"], m["dim"]), w[x + "k.norm"].double(), eps)
            v = _mm(h, w[x + "v"]).view(-1, m["kv_heads"], m["vdim"])
            y = batch.each(lambda q, k, v: _attend(q, k, v, m["scale"], block=m["mask"]["size"]), q, k, v)
            y = _mm((y * torch.sigmoid(_mm(h, w[x + "g"]))[..., None]).flatten(1), w[x + "o"])
        h = h + _rms(y, w[p + "norm1"].double(), eps)
        x = p + "mlp."
        if f["kind"] == "dense":
            y = _mm(torch.relu(_mm(h, w[x + "up"])) ** 2, w[x + "down"])
        else:
            y = _experts(f, w, x, h, lambda r, u: _clamped(w, u, r, f["expert"]["limit"]))
            y = y + _clamped(w, x + "shared.", h, f["shared"]["limit"]) * torch.sigmoid(_mm(h, w[x + "shared.sg"]))
        h = h + _rms(y, w[p + "norm2"].double(), eps)
    return h, lambda rows: _mm(_rms(rows, w["final.norm"].double(), eps), w["head"])


def exact(case, seed):
    c, w, tokens, lens, new = _json(case), _weights(case, seed), _tokens(case, seed), _lengths(case), case["new"]
    batch = _Batch([n + new for n in lens])
    ids = torch.tensor([t for s in tokens for t in s], device="cuda")
    kind = {"saralix": _saralix_exact, "nimelorn": _nimelorn_exact}.get(case["model"], _lfm3_exact)
    h, head = kind(c, w, batch, ids)
    if case["score"]:
        return head(h)
    last = torch.tensor([a + n - 1 for a, n in zip(batch.at, lens)], device="cuda")
    prompt = head(h[last])
    if not new:
        return prompt
    return {"prompt": prompt, "decode": torch.stack([head(h[last + k + 1]) for k in range(new)])}
