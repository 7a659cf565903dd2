"""The work that users of this framework have it do, as cases that can be timed and checked: decode steps and prompts of the
`Transformer` (Mistral-7B / Nemo / Mixtral layer shapes), prompt scoring, mixture-of-experts layers, and prompts, experts and decode steps
of layered decoders in both of their data types.  Every case goes through the package's public entry points (`Transformer.forward`,
`forward_partial`, `forward_logprobs`, `MoeLayer.forward`, `LayeredTransformer.hidden` / `forward`, a feed-forward's `run`).

Weights are random with the scale of trained ones (matrices 1 / sqrt(inputs), norm weights around one); caches of earlier tokens are filled
with random keys and values.  `exact` states the same computation in float64 with plain torch."""
import math
import types
import zlib

import torch

import mistral_inference_b200 as mi
from mistral_inference_b200.args import LayeredArgs, MoeArgs
from mistral_inference_b200.layered import LayeredTransformer
from mistral_inference_b200.transformer import Transformer

DEV = "cuda"
EPS = 1e-5
THETA = 1e6  # rotation base of the Transformer when params.json names none
HD = 128

# Layer shapes of the models in the repository's configurations.
SHAPES = {
    "7b": dict(dim=4096, hidden=14336, heads=32, kv=8, vocab=32000, window=4096),
    "nemo": dict(dim=5120, hidden=14336, heads=32, kv=8, vocab=131072, window=0),
    "8x7b": dict(dim=4096, hidden=14336, heads=32, kv=8, vocab=32000, window=0, experts=8, top=2),
    "8x22b": dict(dim=6144, hidden=16384, heads=48, kv=8, vocab=32768, window=0, experts=8, top=2),
}
# Sizes of layered decoders (attention / lightning layers with a dense feed-forward; experts of a mixture).
LAYERED = {
    "w2048": dict(width=2048, heads=16, kv=4, dim=128, ff=8192, vocab=32768),
    "w4096": dict(width=4096, heads=32, kv=8, dim=128, ff=14336, vocab=32768),
}
EXPERTS = {
    "w2048": dict(width=2048, experts=16, identity=4, top=4, groups=4, keep=2, ff=1408),
    "w4096": dict(width=4096, experts=8, identity=0, top=2, groups=1, keep=1, ff=14336),
}
REL_ROWS = 32


def listed():
    return [
        # chat with one user: the next token of the whole Mistral-7B at a full 4096-token window (batch 1 is the smallest decode step)
        {"name": "decode_7b_b1", "kind": "decode", "shape": "7b", "layers": 32, "batch": 1, "ctx": 4096},
        # a server's decode step: 32 sequences of about 1100 tokens through layers of the Nemo shape and its 131072-entry head
        {"name": "decode_nemo_b32", "kind": "decode", "shape": "nemo", "layers": 8, "batch": 32, "ctx": 1106},
        # the first pass over a long prompt, one layer of the 7B shape
        {"name": "prompt_7b_4k", "kind": "prompt", "shape": "7b", "batch": 1, "tokens": 4096, "past": 0},
        # prompts that are taken in portions (generate's chunk_size): the fourth portion of three sequences, keys from the ring and the portion
        {"name": "prompt_portion_7b", "kind": "prompt", "shape": "7b", "batch": 3, "tokens": 777, "past": 2331},
        # a handful of short questions that arrive together: few tokens, ragged, too many for a decode step and too few to fill the GPU
        {"name": "prompt_short_7b", "kind": "prompt", "shape": "7b", "batch": 5, "tokens": 41, "past": 0},
        # scoring given text: log-probabilities of every token of two texts, head of the Nemo shape
        {"name": "score_nemo", "kind": "score", "shape": "nemo", "batch": 2, "tokens": 601},
        # experts of Mixtral-8x7B for the tokens of a prompt, and for one decode step of eight sequences
        {"name": "moe_8x7b_prompt", "kind": "moe", "shape": "8x7b", "tokens": 2048},
        {"name": "moe_8x7b_decode", "kind": "moe", "shape": "8x7b", "tokens": 8},
        # a long prompt through a layered decoder: one attention layer and one lightning layer at the larger size
        {"name": "layered_prompt_w4096", "kind": "layered_prompt", "size": "w4096", "mixers": "attention,lightning", "dtype": "bf16", "batch": 1, "tokens": 4096},
        # the same design in true 32-bit arithmetic, three ragged prompts of a few hundred tokens
        {"name": "layered_prompt_fp32", "kind": "layered_prompt", "size": "w2048", "mixers": "attention,lightning", "dtype": "fp32", "batch": 3, "tokens": 301},
        # experts with a grouped choice for the tokens of a prompt
        {"name": "layered_moe_w2048", "kind": "layered_moe", "size": "w2048", "dtype": "bf16", "tokens": 2500},
        # a layered decoder's decode step, eight sequences of about 2000 tokens
        {"name": "layered_decode_b8", "kind": "layered_decode", "size": "w2048", "layers": 8, "dtype": "bf16", "batch": 8, "ctx": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "score", "moe", "layered_prompt", "layered_prompt", "layered_moe", "layered_decode"])
    if kind == "decode":
        batch = rng.choice([1, _log(rng, 2, 64), _log(rng, 2, 64)])
        return {"kind": kind, "shape": rng.choice(["7b", "nemo"]), "layers": rng.randint(2, 8), "batch": batch, "ctx": _log(rng, 16, 4096 if batch <= 32 else 1024)}
    if kind == "prompt":
        total, past = _log(rng, 20, 4096), rng.choice([0, 0, 1])
        batch = rng.randint(1, min(8, max(1, total // 8)))
        tokens = max(2, total // batch)
        return {"kind": kind, "shape": rng.choice(["7b", "nemo"]), "batch": batch, "tokens": tokens, "past": _log(rng, 16, 4000 - tokens) if past and tokens < 3900 else 0}
    if kind == "score":
        return {"kind": kind, "shape": rng.choice(["7b", "nemo"]), "batch": rng.randint(1, 4), "tokens": _log(rng, 20, 300)}
    if kind == "moe":
        return {"kind": kind, "shape": rng.choice(["8x7b", "8x22b"]), "tokens": _log(rng, 2, 2048)}
    if kind == "layered_prompt":
        dtype = rng.choice(["bf16", "bf16", "fp32"])
        size = "w2048" if dtype == "fp32" else rng.choice(["w2048", "w4096"])
        total = _log(rng, 20, 900 if dtype == "fp32" else 4096)
        batch = rng.randint(1, min(6, max(1, total // 10)))
        return {"kind": kind, "size": size, "mixers": rng.choice(["attention", "lightning", "attention,lightning"]), "dtype": dtype, "batch": batch,
                "tokens": max(2, total // batch)}
    if kind == "layered_moe":
        return {"kind": kind, "size": rng.choice(["w2048", "w4096"]), "dtype": "bf16", "tokens": _log(rng, 2, 2500)}
    return {"kind": kind, "size": rng.choice(["w2048", "w4096"]), "layers": rng.choice([4, 8]), "dtype": "bf16", "batch": _log(rng, 1, 16), "ctx": _log(rng, 16, 3000)}


# ------------------------------------------------------------------------------------------------------------------ inputs
def _dtype(case):
    return torch.float32 if case.get("dtype") == "fp32" else torch.bfloat16


def _normal(seed, name, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed((seed * 1000003) ^ zlib.crc32(name.encode()))
    return torch.empty(shape, dtype=dtype, device=DEV).normal_(mean, std, generator=g)


def _matrix(seed, name, rows, cols, dtype=torch.bfloat16, gain=1.0):
    return _normal(seed, name, (rows, cols), gain / math.sqrt(cols), 0.0, dtype)


def _tokens(seed, n, vocab):
    g = torch.Generator(device=DEV).manual_seed(seed * 7919 + 5)
    return torch.randint(0, vocab, (n,), device=DEV, generator=g)


def _lengths(case):
    """Ragged lengths around case["tokens"]: the first sequence has exactly that many, the others up to a third fewer."""
    n, b = case["tokens"], case["batch"]
    return [max(1, n - (i * n) // (3 * b)) for i in range(b)]


def _contexts(case):
    """Tokens that each sequence of a decode step has in the cache: up to a quarter fewer than case["ctx"]."""
    n, b = case["ctx"], case["batch"]
    return [max(1, n - (i * n) // (4 * b)) for i in range(b)]


def _transformer_weight(case, seed, key):
    """The checkpoint's tensor of one key (reference names)."""
    s = SHAPES[case["shape"]]
    d, h = s["dim"], s["hidden"]
    last = key.rsplit(".", 2)[-2] if key.endswith(".weight") else key
    if last in ("attention_norm", "ffn_norm", "norm"):
        return _normal(seed, key, (d,), 0.15, 1.0)
    shape = {"tok_embeddings": (s["vocab"], d), "output": (s["vocab"], d), "wq": (s["heads"] * HD, d), "wk": (s["kv"] * HD, d), "wv": (s["kv"] * HD, d),
             "wo": (d, s["heads"] * HD), "w1": (h, d), "w3": (h, d), "w2": (d, h), "gate": (s.get("experts", 1), d)}[last]
    if last == "tok_embeddings":
        return _normal(seed, key, shape)
    return _matrix(seed, key, *shape)


def _transformer(case, seed, layers, moe=False):
    s = SHAPES[case["shape"]]
    args = mi.TransformerArgs(dim=s["dim"], n_layers=layers, head_dim=HD, hidden_dim=s["hidden"], n_heads=s["heads"], n_kv_heads=s["kv"], norm_eps=EPS,
                              vocab_size=s["vocab"], sliding_window=s["window"] or None, max_batch_size=max(1, case.get("batch", 1)),
                              moe=MoeArgs(num_experts=s["experts"], num_experts_per_tok=s["top"]) if moe else None)
    model = Transformer.empty(args, DEV, torch.bfloat16)
    for key in model.state_dict():
        model.load_state_dict({key: _transformer_weight(case, seed, key)}, strict=False)
    model.rope_table  # the table is made once per model
    return model


def _ring(seed, i, name, batch, rows, kv, dim, dtype):
    return _normal(seed, f"ring.{i}.{name}", (batch, rows, kv, dim), 0.7, 0.0, dtype)


def _fesenex_layers(case):
    if case["kind"] == "layered_decode":
        return ["lightning" if i % 4 == 3 else "attention" for i in range(case["layers"])]
    return case["mixers"].split(",")


def _fesenex_config(case):
    s = LAYERED[case["size"]]
    att = {"type": "attention", "mixer": {"heads": s["heads"], "kv_heads": s["kv"], "dim": s["dim"], "vdim": s["dim"], "scale": s["dim"] ** -0.5,
                                          "bias_max": 4096, "q_temp": {"coef": 0.1, "every": 1024}, "v_mix": True},
           "mlp": {"kind": "dense", "ff": s["ff"], "limit": 7.0}}
    lin = {"type": "lightning", "mixer": {"heads": s["heads"], "dim": s["dim"], "vdim": s["dim"], "decay": [math.exp(-1.0 / (4 + 8 * h)) for h in range(s["heads"])]},
           "mlp": {"kind": "dense", "ff": s["ff"], "limit": 7.0}}
    return {"architecture": "Fesenex", "vocab": s["vocab"], "width": s["width"], "embedding": {"scale": 1.0}, "norm": {"eps": EPS},
            "layers": [att if k == "attention" else lin for k in _fesenex_layers(case)]}


def _fesenex_weights(case, seed):
    cfg, dt = _fesenex_config(case), _dtype(case)
    W, out = cfg["width"], {}

    def mat(name, rows, cols):
        out[name] = _matrix(seed, name, rows, cols, dt)

    def vec(name, n, mean=0.0, std=0.1):
        out[name] = _normal(seed, name, (n,), std, mean, dt)

    out["embed"] = _normal(seed, "embed", (cfg["vocab"], W), 1.0, 0.0, dt)
    vec("final.norm", W, 1.0)
    mat("head", cfg["vocab"], W)
    for i, L in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", L["mixer"], L["mlp"]["ff"]
        vec(p + "norm1", W, 1.0)
        vec(p + "norm2", W, 1.0)
        if L["type"] == "attention":
            for n, r in (("q", m["heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]), ("v", m["kv_heads"] * m["vdim"])):
                mat(p + "mix." + n, r, W)
                vec(p + "mix." + n + ".b", r)
            vec(p + "mix.q.norm", m["dim"], 1.0)
            vec(p + "mix.k.norm", m["dim"], 1.0)
            out[p + "mix.rel"] = _normal(seed, p + "mix.rel", (REL_ROWS, m["heads"]), 1.0, 0.0, dt)
            out[p + "mix.vmix"] = torch.tensor(0.3, dtype=dt, device=DEV)
            mat(p + "mix.o", W, m["heads"] * m["vdim"])
        else:
            for n, r in (("q", m["heads"] * m["dim"]), ("k", m["heads"] * m["dim"]), ("v", m["heads"] * m["vdim"]), ("g", m["heads"] * m["vdim"])):
                mat(p + "mix." + n, r, W)
            vec(p + "mix.norm", m["heads"] * m["vdim"], 1.0)
            mat(p + "mix.o", W, m["heads"] * m["vdim"])
        mat(p + "mlp.gate", ff, W)
        mat(p + "mlp.up", ff, W)
        mat(p + "mlp.down", W, ff)
    return out


def _experts_config(case):
    s = EXPERTS[case["size"]]
    mix = {"heads": 4, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 256, "kv_rank": 512, "scale": 192 ** -0.5, "rot": {"base": 10000.0, "dims": 64}}
    mlp = {"kind": "moe", "expert": {"ff": s["ff"]},
           "router": {"experts": s["experts"], "identity": s["identity"], "top": s["top"], "groups": {"count": s["groups"], "keep": s["keep"]}}}
    return {"architecture": "Taruvik", "vocab": 256, "width": s["width"], "norm": {"eps": EPS}, "layers": [{"type": "latent_attention", "mixer": mix, "mlp": mlp}]}


def _experts_weights(case, seed):
    s, dt = EXPERTS[case["size"]], _dtype(case)
    p, n = "l0.mlp.", s["experts"] + s["identity"]
    out = {p + "router": _matrix(seed, p + "router", n, s["width"], dt, gain=2.0), p + "correction": _normal(seed, p + "correction", (n,), 0.01, 0.0, dt)}
    for e in range(s["experts"]):
        for name, r, c in (("gate", s["ff"], s["width"]), ("up", s["ff"], s["width"]), ("down", s["width"], s["ff"])):
            out[f"{p}e{e}.{name}"] = _matrix(seed, f"{p}e{e}.{name}", r, c, dt)
    return out


def prepare(case, seed):
    st = types.SimpleNamespace(case=case)
    kind = case["kind"]
    if kind in ("decode", "prompt", "score"):
        s = SHAPES[case["shape"]]
        st.model = _transformer(case, seed, case.get("layers", 1))
        B = case["batch"]
        if kind == "decode":
            st.past, st.seqlens = _contexts(case), [1] * B
        else:
            st.seqlens = _lengths(case)
            st.past = [case.get("past", 0)] * B
        longest = max(p + n for p, n in zip(st.past, st.seqlens))
        st.cache = st.model.make_cache(B, longest)
        for i, W in enumerate(st.cache.cache_sizes):
            for name, ring in (("k", st.cache.cache_k[i]), ("v", st.cache.cache_v[i])):
                if max(st.past):
                    ring.copy_(_ring(seed, i, name, B, W, s["kv"], HD, torch.bfloat16))
                else:
                    ring.zero_()
        st.ids = _tokens(seed, sum(st.seqlens), s["vocab"])
        if max(st.past):
            st.cache.init_kvseqlens(B)
            st.cache.update_seqlens(st.past)
        if kind == "score":
            st.targets = torch.roll(st.ids, -1)
            st.targets[torch.tensor(st.seqlens, device=DEV).cumsum(0) - 1] = -1
    elif kind == "moe":
        s = SHAPES[case["shape"]]
        st.model = _transformer(case, seed, 1, moe=True)
        st.layer = st.model.layers["0"].feed_forward
        st.x = _normal(seed, "x", (case["tokens"], s["dim"]))
        st.ws = st.model.workspace(case["tokens"])
    elif kind in ("layered_prompt", "layered_decode"):
        st.model = LayeredTransformer.empty(LayeredArgs.from_dict(_fesenex_config(case)), DEV, _dtype(case))
        st.model.load_state_dict(_fesenex_weights(case, seed))
        s, B = LAYERED[case["size"]], case["batch"]
        decode = kind == "layered_decode"
        st.past = _contexts(case) if decode else [0] * B
        st.seqlens = [1] * B if decode else _lengths(case)
        st.cache = st.model.make_cache(B, max(p + n for p, n in zip(st.past, st.seqlens)))
        st.states = {}
        for i in st.cache.cache_k:
            for name, ring in (("k", st.cache.cache_k[i]), ("v", st.cache.cache_v[i])):
                if decode:
                    ring.copy_(_ring(seed, i, name, B, ring.shape[1], s["kv"], s["dim"], ring.dtype))
                else:
                    ring.zero_()
        for i, t in st.cache.cache_state.items():
            t.copy_(_normal(seed, f"state.{i}", tuple(t.shape), 0.5, 0.0, torch.float32))
            if decode:
                st.states[i] = t.clone()
        st.ids = _tokens(seed, sum(st.seqlens), s["vocab"])
        if decode:
            st.cache.init_kvseqlens(B)
            st.cache.update_seqlens(st.past)
    elif kind == "layered_moe":
        s = EXPERTS[case["size"]]
        st.model = LayeredTransformer.empty(LayeredArgs.from_dict(_experts_config(case)), DEV, _dtype(case))
        st.model.load_state_dict(_experts_weights(case, seed), strict=False)
        st.layer = st.model.layers[0].mlp
        st.hn = _normal(seed, "hn", (case["tokens"], s["width"]), dtype=_dtype(case))
        st.x32 = _normal(seed, "x32", (case["tokens"], s["width"]), 0.05, dtype=torch.float32)
    else:
        raise ValueError(kind)
    return st


def run(st):
    kind = st.case["kind"]
    if kind == "decode":
        logits = st.model.forward(st.ids, st.seqlens, st.cache)
        st.cache.update_seqlens([-1] * len(st.seqlens))  # a drafted token taken back: the next pass decodes the same position
        last = len(st.cache.cache_sizes) - 1
        return {"logits": logits, "k": st.cache.cache_k[last], "v": st.cache.cache_v[last]}
    if kind == "prompt":
        if not max(st.past):
            st.cache.reset()
        h = st.model.forward_partial(st.ids, st.seqlens, st.cache)
        if max(st.past):
            st.cache.update_seqlens([-n for n in st.seqlens])
        return {"hidden": h, "k": st.cache.cache_k[0], "v": st.cache.cache_v[0]}
    if kind == "score":
        st.cache.reset()
        lp, last = st.model.forward_logprobs(st.ids, st.seqlens, st.cache, st.targets)
        return {"logprobs": lp, "last": last}
    if kind == "moe":
        return st.layer.forward(st.x, st.ws)
    if kind == "layered_prompt":
        st.cache.reset()
        out = {"hidden": st.model.hidden(st.ids, st.seqlens, st.cache)}
        for i in st.cache.cache_k:
            out[f"k{i}"], out[f"v{i}"] = st.cache.cache_k[i], st.cache.cache_v[i]
        for i, t in st.cache.cache_state.items():
            out[f"state{i}"] = t
        return out
    if kind == "layered_decode":
        logits = st.model.forward(st.ids, st.seqlens, st.cache)
        st.cache.update_seqlens([-1] * len(st.seqlens))  # a drafted token taken back, recurrent states with it
        for i, t in st.states.items():
            st.cache.cache_state[i].copy_(t)
        return {"logits": logits}
    x = st.x32.clone()
    st.layer.run(st.hn, x)
    return x


# ------------------------------------------------------------------------------------------------------------------ work
def _visible(past, n, window):
    """Keys that the n queries behind `past` cached tokens see, in all."""
    w = window or (past + n)
    return sum(min(past + i + 1, w) for i in range(n)) if n < 64 else int(sum(min(past + (j + 0.5) * n / 64, w) for j in range(64)) * n / 64)


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prompt", "score"):
        s = SHAPES[case["shape"]]
        d, q, kv = s["dim"], s["heads"] * HD, s["kv"] * HD
        layer = d * (2 * q + 2 * kv) + 3 * d * s["hidden"]
        layers = case.get("layers", 1)
        past = _contexts(case) if kind == "decode" else [case.get("past", 0)] * case["batch"]
        n = [1] * case["batch"] if kind == "decode" else _lengths(case)
        T = sum(n)
        W = s["window"]
        seen = sum(_visible(p, m, W) for p, m in zip(past, n))
        old = sum(min(p, W or p) for p in past)
        new = sum(min(m, W or m) for m in n)
        bytes_ = layers * (2 * layer + 2 * 2 * kv * (old + new)) + 2 * T * d
        flops = layers * (2 * T * layer + 4 * q * seen)
        if kind == "prompt":
            return {"bytes": bytes_ + 2 * T * d, "flops": flops}
        # one row of the head per token; scoring gives logits of each sequence's last token only
        out = 4 * T * s["vocab"] if kind == "decode" else 4 * T + 4 * len(n) * s["vocab"]
        return {"bytes": bytes_ + 2 * s["vocab"] * d + out, "flops": flops + 2 * T * s["vocab"] * d}
    if kind == "moe":
        s = SHAPES[case["shape"]]
        T = case["tokens"]
        used = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** T)
        return {"bytes": 2 * used * 3 * s["dim"] * s["hidden"] + 2 * 2 * T * s["dim"], "flops": 2 * T * s["top"] * 3 * s["dim"] * s["hidden"]}
    size = 4 if case["dtype"] == "fp32" else 2
    if kind == "layered_moe":
        s = EXPERTS[case["size"]]
        T = case["tokens"]
        share = s["top"] / (s["experts"] + s["identity"])
        used = s["experts"] * (1 - (1 - share) ** T)
        return {"bytes": size * (used * 3 * s["width"] * s["ff"] + T * s["width"]) + 8 * T * s["width"],
                "flops": 2 * T * share * s["experts"] * 3 * s["width"] * s["ff"]}
    s = LAYERED[case["size"]]
    d, q, kv = s["width"], s["heads"] * s["dim"], s["kv"] * s["dim"]
    decode = kind == "layered_decode"
    past = _contexts(case) if decode else [0] * case["batch"]
    n = [1] * case["batch"] if decode else _lengths(case)
    T = sum(n)
    bytes_, flops = size * T * d + 4 * T * d, 0
    for k in _fesenex_layers(case):
        params = 3 * d * s["ff"] + (d * (2 * q + 2 * kv) if k == "attention" else 5 * d * q)
        bytes_ += size * params
        flops += 2 * T * params
        if k == "attention":
            seen = sum(_visible(p, m, 0) for p, m in zip(past, n))
            bytes_ += 2 * size * kv * (sum(past) + T)
            flops += 4 * q * seen
        else:
            state = s["heads"] * s["dim"] * s["dim"]
            bytes_ += 4 * state * len(n) * (2 if decode else 1)
            flops += 4 * state * T
    if decode:
        bytes_ += size * s["vocab"] * d + 4 * T * s["vocab"]
        flops += 2 * T * s["vocab"] * d
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times the relative error against `exact` that was measured over listed and drawn cases."""
    kind = case["kind"]
    if case.get("dtype") == "fp32":
        return {"rel": 8e-6}
    if kind in ("decode", "layered_decode"):
        return {"rel": 0.03}  # every layer's roundings travel through all that follow
    if kind == "layered_moe":
        return {"rel": 0.012}
    return {"rel": 0.02}


# ------------------------------------------------------------------------------------------------------------------ exact
def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _rotate(x, pos):
    """x [n, heads, HD]: neighbouring pairs turned by pos * THETA^(-2i / HD)."""
    f = THETA ** (-torch.arange(0, HD, 2, dtype=torch.float64, device=DEV) / HD)
    a = pos.double()[:, None] * f
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack((u * c - v * s, u * s + v * c), -1).flatten(-2)


def _softmax_attention(q, k, v, qpos, kpos, scale, window, bias=None):
    """q [n, H, d] over k, v [m, G, d]: causal, at most `window` positions back (0: all); bias(distances, head) is added to the scores."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64, device=DEV)
    dist = qpos[:, None] - kpos[None]
    hidden = (dist < 0) | ((dist >= window) if window else (dist < 0))
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // G)].T * scale
        if bias is not None:
            s = s + bias(dist, h)
        out[:, h] = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ v[:, h // (H // G)]
    return out.flatten(1)


def _exact_transformer(case, seed):
    s = SHAPES[case["shape"]]
    kind, B, W = case["kind"], case["batch"], s["window"]
    past = _contexts(case) if kind == "decode" else [case.get("past", 0)] * B
    n = [1] * B if kind == "decode" else _lengths(case)
    start = [0]
    for m in n:
        start.append(start[-1] + m)
    longest = max(p + m for p, m in zip(past, n))
    rows = W or longest
    ids = _tokens(seed, sum(n), s["vocab"])
    w = lambda key: _transformer_weight(case, seed, key).double()  # noqa: E731
    x = _transformer_weight(case, seed, "tok_embeddings.weight")[ids].double()
    pos = [torch.arange(p, p + m, device=DEV) for p, m in zip(past, n)]
    rings = None
    for i in range(case.get("layers", 1)):
        p = f"layers.{i}."
        hn = _rms(x, w(p + "attention_norm.weight"))
        q = (hn @ w(p + "attention.wq.weight").T).view(-1, s["heads"], HD)
        k = (hn @ w(p + "attention.wk.weight").T).view(-1, s["kv"], HD)
        v = (hn @ w(p + "attention.wv.weight").T).view(-1, s["kv"], HD)
        if max(past):
            rings = [_ring(seed, i, name, B, rows, s["kv"], HD, torch.bfloat16).double() for name in ("k", "v")]
        else:
            rings = [torch.zeros(B, rows, s["kv"], HD, dtype=torch.float64, device=DEV) for _ in range(2)]
        att = []
        for b in range(B):
            a, z = start[b], start[b + 1]
            qb, kb, vb = _rotate(q[a:z], pos[b]), _rotate(k[a:z], pos[b]), v[a:z]
            have = min(past[b], rows)
            old = torch.arange(past[b] - have, past[b], device=DEV)
            ka, va = torch.cat((rings[0][b, old % rows], kb)), torch.cat((rings[1][b, old % rows], vb))
            # one new token: the ring's window; a portion: (p - W, p]
            att.append(_softmax_attention(qb, ka, va, pos[b], torch.cat((old, pos[b])), HD ** -0.5, rows if W else 0))
            keep = slice(max(0, n[b] - rows), n[b])
            rings[0][b, pos[b][keep] % rows] = kb[keep]
            rings[1][b, pos[b][keep] % rows] = vb[keep]
        x = x + torch.cat(att) @ w(p + "attention.wo.weight").T
        hn = _rms(x, w(p + "ffn_norm.weight"))
        x = x + (torch.nn.functional.silu(hn @ w(p + "feed_forward.w1.weight").T) * (hn @ w(p + "feed_forward.w3.weight").T)) @ w(p + "feed_forward.w2.weight").T
    x = _rms(x, w("norm.weight"))
    if kind == "prompt":
        return {"hidden": x, "k": rings[0], "v": rings[1]}
    head = w("output.weight")
    if kind == "decode":
        return {"logits": x @ head.T, "k": rings[0], "v": rings[1]}
    lp = torch.zeros(len(ids), dtype=torch.float64, device=DEV)
    last = []
    for b in range(B):
        a, z = start[b], start[b + 1]
        for r in range(a, z - 1, 256):
            e = min(r + 256, z - 1)
            lp[r:e] = torch.log_softmax(x[r:e] @ head.T, -1).gather(1, ids[r + 1:e + 1, None])[:, 0]
        last.append(x[z - 1] @ head.T)
    return {"logprobs": lp, "last": torch.stack(last)}


def _exact_moe(case, seed):
    s = SHAPES[case["shape"]]
    x = _normal(seed, "x", (case["tokens"], s["dim"])).double()
    w = lambda key: _transformer_weight(case, seed, "layers.0.feed_forward." + key).double()  # noqa: E731
    scores = (x @ w("gate.weight").T).bfloat16().double()  # the router's scores are numbers of the model's type: ties go to the lower expert
    idx = torch.sort(scores, dim=-1, descending=True, stable=True).indices[:, : s["top"]]
    wts = torch.softmax(scores.gather(1, idx), -1)
    out = torch.zeros_like(x)
    for e in range(s["experts"]):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        xe = x[t]
        y = (torch.nn.functional.silu(xe @ w(f"experts.{e}.w1.weight").T) * (xe @ w(f"experts.{e}.w3.weight").T)) @ w(f"experts.{e}.w2.weight").T
        out.index_add_(0, t, wts[t, j][:, None] * y)
    return out


def _exact_experts(case, seed):
    s, w = EXPERTS[case["size"]], _experts_weights(case, seed)
    p, n = "l0.mlp.", s["experts"] + s["identity"]
    h = _normal(seed, "hn", (case["tokens"], s["width"]), dtype=_dtype(case)).double()
    out = _normal(seed, "x32", (case["tokens"], s["width"]), 0.05, dtype=torch.float32).double()
    score = torch.softmax(h @ w[p + "router"].double().T, -1)
    choice = score + w[p + "correction"].double()
    best = choice.view(-1, s["groups"], n // s["groups"]).max(-1).values
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(s["keep"], -1).indices, True)
    idx = choice.masked_fill(~kept.repeat_interleave(n // s["groups"], 1), float("-inf")).topk(s["top"], -1).indices
    wts = score.gather(1, idx)
    for e in range(n):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        y = h[t]
        if e < s["experts"]:
            y = (torch.nn.functional.silu(y @ w[f"{p}e{e}.gate"].double().T) * (y @ w[f"{p}e{e}.up"].double().T)) @ w[f"{p}e{e}.down"].double().T
        out.index_add_(0, t, wts[t, j][:, None] * y)
    return out


def _buckets(rows, far):
    """Row of the distance table for every distance up to the first one in the last row."""
    half, out, n = rows // 2, [], 0
    while not out or out[-1] != rows - 1:
        out.append(n if n < half else min(rows - 1, half + int(math.floor(math.log(n / half) / math.log(far / half) * (rows - half)))))
        n += 1
    return torch.tensor(out, device=DEV)


def _exact_fesenex(case, seed):
    cfg, weights = _fesenex_config(case), _fesenex_weights(case, seed)
    decode, B, s = case["kind"] == "layered_decode", case["batch"], LAYERED[case["size"]]
    past = _contexts(case) if decode else [0] * B
    n = [1] * B if decode else _lengths(case)
    start = [0]
    for m in n:
        start.append(start[-1] + m)
    rows = max(p + m for p, m in zip(past, n))
    w = lambda key: weights[key].double()  # noqa: E731
    x = weights["embed"][_tokens(seed, sum(n), s["vocab"])].double()
    pos = torch.cat([torch.arange(p, p + m, device=DEV) for p, m in zip(past, n)])
    first, out = None, {}
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", L["mixer"]
        h = _rms(x, w(f"l{i}.norm1"))
        if L["type"] == "attention":
            q = _rms((h @ w(p + "q").T + w(p + "q.b")).view(-1, m["heads"], m["dim"]), w(p + "q.norm"))
            k = _rms((h @ w(p + "k").T + w(p + "k.b")).view(-1, m["kv_heads"], m["dim"]), w(p + "k.norm"))
            v = (h @ w(p + "v").T + w(p + "v.b")).view(-1, m["kv_heads"], m["vdim"])
            qt = m["q_temp"]
            q = q * (1.0 + qt["coef"] * torch.log((torch.div(pos + 1, qt["every"], rounding_mode="floor") + 1).double()))[:, None, None]
            if first is None:
                first = v
            else:
                v = (1.0 - w(p + "vmix")) * v + w(p + "vmix") * first
            if decode:
                kr, vr = (_ring(seed, i, name, B, rows, m["kv_heads"], m["dim"], _dtype(case)).double() for name in ("k", "v"))
            else:
                kr, vr = (torch.zeros(B, rows, m["kv_heads"], m["dim"], dtype=torch.float64, device=DEV) for _ in range(2))
            table = w(p + "rel")[_buckets(REL_ROWS, m["bias_max"])]
            bias = lambda dist, head: table[dist.clamp(0, len(table) - 1), head]  # noqa: E731
            ys = []
            for b in range(B):
                a, z, e = start[b], start[b + 1], past[b] + n[b]
                kr[b, past[b]:e], vr[b, past[b]:e] = k[a:z], v[a:z]
                ys.append(_softmax_attention(q[a:z], kr[b, :e], vr[b, :e], pos[a:z], torch.arange(e, device=DEV), m["scale"], 0, bias))
            y = torch.cat(ys)
            if not decode:
                out[f"k{i}"], out[f"v{i}"] = kr, vr
        else:
            silu = torch.nn.functional.silu
            q, k, v = (silu(h @ w(p + c).T).view(-1, m["heads"], m["dim"]) for c in "qkv")
            state = torch.zeros(B, m["heads"], m["dim"], m["vdim"], dtype=torch.float64, device=DEV)
            if decode:
                state = _normal(seed, f"state.{i}", tuple(state.shape), 0.5, 0.0, torch.float32).double()
            decay = torch.tensor(m["decay"], dtype=torch.float64, device=DEV)[:, None, None]
            y = torch.empty(len(x), m["heads"], m["vdim"], dtype=torch.float64, device=DEV)
            for b in range(B):
                for t in range(start[b], start[b + 1]):
                    state[b] = decay * state[b] + k[t, :, :, None] * v[t, :, None, :]
                    y[t] = (state[b] * q[t, :, :, None]).sum(1)
            y = _rms(y.flatten(1), w(p + "norm")) * torch.sigmoid(h @ w(p + "g").T)
            if not decode:
                out[f"state{i}"] = state
        x = x + y @ w(p + "o").T
        h, p, lim = _rms(x, w(f"l{i}.norm2")), f"l{i}.mlp.", L["mlp"]["limit"]
        g, u = (h @ w(p + "gate").T).clamp(max=lim), (h @ w(p + "up").T).clamp(-lim, lim)
        x = x + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + "down").T
    if decode:
        return {"logits": _rms(x, w("final.norm")) @ w("head").T}
    return {"hidden": x, **out}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("decode", "prompt", "score"):
            return _exact_transformer(case, seed)
        if kind == "moe":
            return _exact_moe(case, seed)
        if kind == "layered_moe":
            return _exact_experts(case, seed)
        return _exact_fesenex(case, seed)
