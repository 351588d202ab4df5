"""Cases of the engine's own work, for measuring it: what `Engine.step` is called with, over the range it is used in.

A case is a model (by name, see `_model`), a kind of step and its sizes:

* ``prefill``: `rows` prompts of `tokens` tokens in all, brought whole in one step, the last row's logits wanted.
* ``decode``: one token for each of `rows` live requests that hold up to `tokens` tokens each.
* ``mixed``: a request joins `rows` live ones that hold up to `tokens` tokens each: its prompt of three portions of
  `portion` tokens is brought beside their decoded tokens (three steps), then it leaves.

Lengths within a batch differ, as they do in a server. Weights are random (matrices N(0, 0.02), norm weights
1 + N(0, 0.1), biases N(0, 0.1)) and made on the GPU from the seed, token ids are random, and so is what requests hold.
`exact` restates the four designs in 64-bit torch from their equations; it uses nothing of the engine.

Designs with a mixture of experts are left out, and Nisotar runs with its dense feed-forward in every layer: a router's
choice between two nearly equal experts is a coin toss at 16 bits, so that two correct implementations differ by more than
any bound worth stating.
"""

import math

import torch

from dynalm_b200 import Engine, StepEntry

DEVICE = "cuda:0"

# ----------------------------------------------------------------------------------------------------
# models
# ----------------------------------------------------------------------------------------------------


def _llama(hidden, layers, heads, kv_heads, head_dim, inner, vocab, tied, scaling, theta=500000.0, eps=1e-5, context=131072):
    cfg = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": vocab, "hidden_size": hidden,
           "intermediate_size": inner, "num_hidden_layers": layers, "num_attention_heads": heads,
           "num_key_value_heads": kv_heads, "head_dim": head_dim, "max_position_embeddings": context, "rms_norm_eps": eps,
           "rope_theta": theta, "tie_word_embeddings": tied}
    if scaling:
        factor, original = scaling
        cfg["rope_scaling"] = {"rope_type": "llama3", "factor": factor, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                               "original_max_position_embeddings": original}
    return cfg


def _todupel(width, layers, heads, kv_heads, dim, ff):
    mixer = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": 2 * dim, "scale": dim ** -0.5, "softcap": 30.0,
             "diff": 0.4, "q_temp": {"coef": 0.2, "every": 256}}
    return {"architecture": "Todupel", "vocab": 32000, "width": width, "norm": {"eps": 1e-5},
            "layers": [{"type": "attention", "mixer": dict(mixer), "mlp": {"kind": "dense", "ff": ff}} for _ in range(layers)]}


def _rematar(width, kinds, ssd, latent, ff):
    heads, vdim, state, groups, conv, parts = ssd
    s = {"heads": heads, "vdim": vdim, "state": state, "groups": groups, "conv": conv, "norm_groups": parts}
    heads, dim, rot, vdim, q_rank, kv_rank, window = latent
    a = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "q_rank": q_rank, "kv_rank": kv_rank,
         "scale": (dim + rot) ** -0.5, "rot": {"base": 10000.0, "dims": rot}, "mask": {"size": window}}
    return {"architecture": "Rematar", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "postln_alpha": 2.0,
            "embedding": {"scale": 8.0},
            "layers": [{"type": "mamba2" if k == "s" else "latent_attention", "mixer": dict(s if k == "s" else a),
                        "mlp": {"kind": "dense", "ff": ff}} for k in kinds]}


def _nisotar(width, kinds, attention, latent, delta, ff):
    heads, kv_heads, dim, turned, size = attention
    att = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "mask": {"size": size}}
    stretch = {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    heads, dim, rot, vdim, kv_rank, window = latent
    lat = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": kv_rank, "scale": (dim + rot) ** -0.5,
           "mask": {"size": window}, "rot": {"base": 10000.0, "dims": rot}}
    heads, kv_heads, dim, vdim, conv, inner = delta
    right = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "conv": conv, "decay_rank": inner,
             "gate_rank": inner}
    mixers = {"l": ("latent_attention", lat),
              "a": ("attention", dict(att, rot={"base": 50000.0, "dims": turned, "scaling": stretch})),
              "p": ("parallel", {"left": dict(att, rot={"base": 500000.0, "dims": turned}), "right": right})}
    return {"architecture": "Nisotar", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "embedding": {"scale": 8.0},
            "layers": [{"type": mixers[k][0], "mixer": mixers[k][1], "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}}
                       for k in kinds]}


_MODELS = {
    "tiny-a": lambda: _llama(64, 2, 4, 2, 16, 192, 256, True, None, 10000.0, 1e-5, 16384),
    "tiny-b": lambda: _llama(96, 3, 6, 2, 32, 160, 384, False, (8.0, 32), 500000.0, 1e-6, 16384),
    "llama-1b": lambda: _llama(2048, 16, 32, 8, 64, 8192, 128256, True, (32.0, 8192)),
    "llama-3b": lambda: _llama(3072, 28, 24, 8, 128, 8192, 128256, True, (32.0, 8192)),
    # (twelve of the 8B shape's layers: with random weights each layer adds to the rounding of the 16-bit activations, and
    # behind all 32 two correct implementations lie 3.5 % apart)
    "llama-8b": lambda: _llama(4096, 12, 32, 8, 128, 14336, 128256, False, (8.0, 8192)),
    "todupel-2048-d64": lambda: _todupel(2048, 4, 16, 4, 64, 12288),
    "todupel-4096-d64": lambda: _todupel(4096, 2, 32, 8, 64, 21504),
    "todupel-2048-d32": lambda: _todupel(2048, 4, 32, 8, 32, 12288),
    "rematar-2048-n128": lambda: _rematar(2048, "sass", (64, 64, 128, 8, 4, 8), (16, 128, 64, 128, 768, 512, 1024), 12288),
    "rematar-4096-n128": lambda: _rematar(4096, "sa", (128, 64, 128, 8, 4, 8), (32, 128, 64, 128, 1536, 512, 2048), 21504),
    "rematar-2048-n64": lambda: _rematar(2048, "sass", (32, 128, 64, 1, 4, 1), (16, 64, 32, 64, 512, 256, 512), 12288),
    "nisotar-2048-d128": lambda: _nisotar(2048, "lpap", (16, 4, 128, 128, 1024), (16, 128, 64, 128, 512, 1024),
                                          (16, 16, 128, 128, 4, 128), 8192),
    "nisotar-4096-d128": lambda: _nisotar(4096, "lp", (32, 8, 128, 128, 2048), (32, 128, 64, 128, 512, 2048),
                                          (32, 16, 128, 128, 4, 128), 14336),
    "nisotar-2048-d64": lambda: _nisotar(2048, "lpap", (32, 8, 64, 32, 512), (32, 64, 32, 64, 256, 512),
                                         (32, 8, 64, 64, 4, 64), 8192),
}


def _model(case):
    return _MODELS[case["model"]]()


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _matrix(name, *shape):
    return name, shape, "matrix"


def _around_one(name, *shape):
    return name, shape, "norm"


def _bias(name, *shape):
    return name, shape, "bias"


def _tensors(cfg):
    """(name in a model file, shape, kind) of every tensor of the design."""
    out = []
    if "architectures" in cfg:
        H, F, V, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["head_dim"]
        q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
        out += [_matrix("model.embed_tokens.weight", V, H), _around_one("model.norm.weight", H)]
        if not cfg["tie_word_embeddings"]:
            out.append(_matrix("lm_head.weight", V, H))
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out += [_around_one(p + "input_layernorm.weight", H), _around_one(p + "post_attention_layernorm.weight", H),
                    _matrix(p + "self_attn.q_proj.weight", q, H), _matrix(p + "self_attn.k_proj.weight", kv, H),
                    _matrix(p + "self_attn.v_proj.weight", kv, H), _matrix(p + "self_attn.o_proj.weight", H, q),
                    _matrix(p + "mlp.gate_proj.weight", F, H), _matrix(p + "mlp.up_proj.weight", F, H),
                    _matrix(p + "mlp.down_proj.weight", H, F)]
        return out
    V, W = cfg["vocab"], cfg["width"]
    out += [_matrix("embed", V, W), _matrix("head", V, W), _around_one("final.norm", W)]
    for i, layer in enumerate(cfg["layers"]):
        m, kind, p, ff = layer["mixer"], layer["type"], f"l{i}.mix.", layer["mlp"]["ff"]
        out += [_around_one(f"l{i}.norm1", W), _around_one(f"l{i}.norm2", W), _matrix(f"l{i}.mlp.up", ff, W),
                _matrix(f"l{i}.mlp.down", W, ff)]
        if cfg["architecture"] == "Todupel":
            H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            out += [_matrix(p + "q", H * 2 * d, W), _matrix(p + "k", G * 2 * d, W), _matrix(p + "v", G * e, W),
                    _matrix(p + "o", W, H * e), _around_one(p + "q.norm", d), _around_one(p + "k.norm", d)]
            out += [_bias(p + n, d) for n in ("lq1", "lk1", "lq2", "lk2")]
        elif cfg["architecture"] == "Rematar":
            out += [_around_one(f"l{i}.ls1", W), _around_one(f"l{i}.ls2", W)]
            if kind == "mamba2":
                H, inner, C = m["heads"], m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
                out += [_matrix(p + "in", inner + C + H, W), _bias(p + "conv", C, m["conv"]), _bias(p + "conv.b", C),
                        _bias(p + "dt_bias", H), _bias(p + "A_log", H), _around_one(p + "D", H), _around_one(p + "norm", inner),
                        _matrix(p + "o", W, inner)]
            else:
                H, d, r, e, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
                out += [_matrix(p + "dq", m["q_rank"], W), _around_one(p + "dq.norm", m["q_rank"]),
                        _matrix(p + "uq", H * (d + r), m["q_rank"]), _matrix(p + "dkv", R + r, W), _around_one(p + "dkv.norm", R),
                        _matrix(p + "uk", H * d, R), _matrix(p + "uv", H * e, R), _bias(p + "sink", H),
                        _matrix(p + "g", H * e, W), _matrix(p + "o", W, H * e)]
        else:
            out += [_matrix(f"l{i}.mlp.gate", ff, W), _bias(f"l{i}.mlp.gate.b", ff), _bias(f"l{i}.mlp.up.b", ff),
                    _bias(f"l{i}.mlp.down.b", W)]
            if kind == "latent_attention":
                H, d, r, e, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
                out += [_matrix(p + "q", H * (d + r), W), _matrix(p + "dkv", R + r, W), _around_one(p + "dkv.norm", R),
                        _matrix(p + "uk", H * d, R), _matrix(p + "uv", H * e, R), _matrix(p + "o", W, H * e)]
            a, pa = (m["left"], p + "left.") if kind == "parallel" else (m, p)
            if kind in ("parallel", "attention"):
                H, G, d, e = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
                out += [_matrix(pa + "q", H * d, W), _matrix(pa + "k", G * d, W), _matrix(pa + "o", W, H * e),
                        _around_one(pa + "q.norm", d), _around_one(pa + "k.norm", d)]
                out += [_around_one(pa + "out", W)] if kind == "parallel" else [_matrix(pa + "v", G * e, W)]
            if kind == "parallel":
                m, p = m["right"], p + "right."
                H, G, d, e, K = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
                for n, size in (("q", G * d), ("k", G * d), ("v", H * e)):
                    out += [_matrix(p + n, size, W), _bias(p + n + ".conv", size, K)]
                out += [_matrix(p + "b", H, W), _matrix(p + "a1", m["decay_rank"], W), _matrix(p + "a2", H * d, m["decay_rank"]),
                        _matrix(p + "g1", m["gate_rank"], W), _matrix(p + "g2", H * e, m["gate_rank"]), _bias(p + "A_log", H),
                        _bias(p + "dt_bias", H * d), _around_one(p + "norm", e), _matrix(p + "o", W, H * e),
                        _around_one(p + "out", W)]
    return out


def _weights(case, seed):
    """Tensors on the GPU in the case's type: what a model file of this seed holds."""
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    gen = torch.Generator(device=DEVICE)
    out = {}
    for i, (name, shape, kind) in enumerate(_tensors(_model(case))):
        gen.manual_seed(seed * 65537 + i)
        t = torch.randn(shape, generator=gen, device=DEVICE, dtype=dtype)
        if kind == "norm":
            t.mul_(0.1).add_(1.0)
        else:
            t.mul_(0.02 if kind == "matrix" else 0.1)
        out[name] = t
    return out


# ----------------------------------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------------------------------

ROOM = {"tiny-a": 8192, "tiny-b": 8192}       # tokens a live request may still grow by before it is ended and begun again
DEFAULT_ROOM = 2048
STEP_TOKENS = 2048                            # the most prompt tokens that the preparation brings in one step


def listed():
    return [
        # The smallest model and a few live requests, in 32 bits: every step is launches and host work.
        {"name": "tiny decode", "model": "tiny-b", "dtype": "float32", "kind": "decode", "rows": 5, "tokens": 100},
        # One user talking to the 1B model: a chain of short kernels that stream the weights.
        {"name": "1b decode, 1 user", "model": "llama-1b", "dtype": "bfloat16", "kind": "decode", "rows": 1, "tokens": 2048},
        # A few users: the benchmark's default workload.
        {"name": "1b decode, 8 users", "model": "llama-1b", "dtype": "bfloat16", "kind": "decode", "rows": 8, "tokens": 2048},
        # A busy server: weights and as many bytes of cache again, products of 64 rows.
        {"name": "1b decode, 64 users", "model": "llama-1b", "dtype": "bfloat16", "kind": "decode", "rows": 64, "tokens": 2048},
        # A document to read before the first token.
        {"name": "1b prompt of 2048", "model": "llama-1b", "dtype": "bfloat16", "kind": "prefill", "rows": 1, "tokens": 2048},
        # Continuous batching: a new request's prompt in portions of 512 beside the others' tokens, on the 3B model.
        {"name": "3b joined by a request", "model": "llama-3b", "dtype": "bfloat16", "kind": "mixed", "rows": 31, "tokens": 1500,
         "portion": 512},
        # The largest products: three prompts of different lengths at once at the 8B model's sizes.
        {"name": "8b three prompts", "model": "llama-8b", "dtype": "bfloat16", "kind": "prefill", "rows": 3, "tokens": 2499},
        # The true 32-bit path, which answers are checked against: a prompt, and a few users' tokens.
        {"name": "1b prompt of 700, 32-bit", "model": "llama-1b", "dtype": "float32", "kind": "prefill", "rows": 1, "tokens": 700},
        {"name": "1b decode, 4 users, 32-bit", "model": "llama-1b", "dtype": "float32", "kind": "decode", "rows": 4, "tokens": 500},
        # The other designs: differential attention, state-space layers with latent attention, the delta rule beside
        # chunked attention. Odd lengths, as prompts have.
        {"name": "todupel prompt of 2048", "model": "todupel-2048-d64", "dtype": "bfloat16", "kind": "prefill", "rows": 1,
         "tokens": 2048},
        {"name": "rematar two prompts", "model": "rematar-2048-n128", "dtype": "bfloat16", "kind": "prefill", "rows": 2,
         "tokens": 1777},
        {"name": "nisotar joined by a request", "model": "nisotar-2048-d128", "dtype": "bfloat16", "kind": "mixed", "rows": 8,
         "tokens": 1500, "portion": 700},
    ]


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / (5e13 if case["dtype"] == "float32" else 1.6e15))


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    most = max(_cost(c) for c in listed())
    while True:
        model = rng.choice(sorted(_MODELS))
        dtype = "bfloat16"
        if model.startswith("tiny") or (model == "llama-1b" and rng.random() < 0.35):
            dtype = "float32"
        kind = rng.choice(("prefill", "decode", "mixed"))
        case = {"model": model, "dtype": dtype, "kind": kind, "rows": spread(1, 64), "tokens": spread(16, 4096)}
        if kind == "prefill":
            case["rows"] = rng.choice((1, 1, 2, 3, 5))
        if kind == "mixed":
            case["portion"] = spread(16, 700)
        if model == "llama-8b" and kind != "prefill":
            case["rows"] = min(case["rows"], 16)
        if _cost(case) <= most and case["tokens"] >= case["rows"]:
            return case


def _lengths(case):
    """Tokens of every prompt, or tokens every live request holds at first."""
    rows, tokens = case["rows"], case["tokens"]
    if case["kind"] != "prefill":
        return [max(1, tokens - (i * 7919) % (tokens // 8 + 1)) for i in range(rows)]
    lengths = [max(1, tokens * (2 + i % 3) // (3 * rows + 3)) for i in range(rows)]
    lengths[-1] += tokens - sum(lengths)
    return lengths


def _ids(case, seed, lengths):
    """One list of token ids per length."""
    gen = torch.Generator().manual_seed(seed * 65537 + 17)
    flat = torch.randint(0, _vocab(_model(case)), (sum(lengths),), generator=gen).tolist()
    out, at = [], 0
    for n in lengths:
        out.append(flat[at:at + n])
        at += n
    return out


FED = 64              # ids a live request is fed, over and over


def _all_ids(case, seed):
    """(what every request holds or brings, what the live ones are fed, the joining request's prompt)."""
    lengths = _lengths(case)
    live = 0 if case["kind"] == "prefill" else case["rows"]
    joining = 3 * case["portion"] if case["kind"] == "mixed" else 0
    ids = _ids(case, seed, lengths + [FED] * live + [joining])
    return ids[:len(lengths)], ids[len(lengths):len(lengths) + live], ids[-1]


class _Session:
    """A user's program around an engine: its live requests and what it feeds them."""

    def __init__(self, case, seed):
        self.case = case
        self.held, self.fed, self.joining = _all_ids(case, seed)
        self.room = ROOM.get(case["model"], DEFAULT_ROOM)
        prefill, mixed = case["kind"] == "prefill", case["kind"] == "mixed"
        pages = sum(-(-(len(h) + (0 if prefill else self.room)) // 16) for h in self.held) + -(-len(self.joining) // 16) + 8
        per_step = sum(map(len, self.held)) if prefill else max(STEP_TOKENS, case["rows"] + case.get("portion", 0))
        self.engine = Engine(config=_model(case), tensors=_weights(case, seed), dtype=case["dtype"], ctx=16 * pages,
                             batch=per_step, max_running=case["rows"] + (1 if mixed else 0), device=DEVICE)
        self.given = 0
        if not prefill:
            self._begin()

    def _begin(self):
        for r, ids in enumerate(self.held):
            for at in range(0, len(ids), STEP_TOKENS):
                self.engine.step([StepEntry(r, ids[at:at + STEP_TOKENS])])
        self.given = 0

    def _tokens(self):
        """The live requests' next tokens; requests that have grown to their limit are ended and begun again first."""
        if self.given >= self.room:
            for r in range(len(self.held)):
                self.engine.end(r)
            self._begin()
        at = self.given % FED
        self.given += 1
        return [StepEntry(r, [ids[at]], [0]) for r, ids in enumerate(self.fed)]

    def prefill(self):
        logits = self.engine.step([StepEntry(r, ids, [len(ids) - 1]) for r, ids in enumerate(self.held)])
        for r in range(len(self.held)):
            self.engine.end(r)
        return logits

    def decode(self):
        return self.engine.step(self._tokens())

    def join(self):
        if self.given + 3 > self.room:
            self.given = self.room
        n, out = self.case["portion"], []
        for i in range(3):
            new = StepEntry("new", self.joining[i * n:(i + 1) * n], [n - 1] if i == 2 else [])
            logits = self.engine.step(self._tokens() + [new])
            out.append(logits.clone() if i < 2 else logits)      # (the next step writes its logits where these stand)
        self.engine.end("new")
        return out


def prepare(case, seed):
    return _Session(case, seed)


def run(state):
    return {"prefill": state.prefill, "decode": state.decode, "mixed": state.join}[state.case["kind"]]()


# ----------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------------

def _runs(case):
    """(first position, tokens) of every run of tokens a pass brings."""
    if case["kind"] == "prefill":
        return [(0, n) for n in _lengths(case)]
    if case["kind"] == "decode":
        return [(n, 1) for n in _lengths(case)]
    return [(n, 3) for n in _lengths(case)] + [(0, 3 * case["portion"])]


def _pairs(start, n, window=0, chunk=0):
    """Pairs of a query and a key it sees, over n queries from position `start` on."""
    total = 0
    if chunk:
        for p in range(start, start + n):
            total += p % chunk + 1
        return total
    full = start + n
    total = (full * (full + 1) - start * (start + 1)) // 2
    if window:
        lo = max(start, window)
        if full > lo:
            total -= (full - window) * (full - window + 1) // 2 - (lo - window) * (lo - window + 1) // 2
    return total


def _mixers(cfg):
    """Per layer: a list of (flops per query-key pair, window, chunk, cache numbers a token leaves) of its attention, and a
    list of (flops per token, numbers of 32-bit state) of its recurrences."""
    if "architectures" in cfg:
        h, g, d = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        return [([(4 * h * d, 0, 0, 2 * g * d)], []) for _ in range(cfg["num_hidden_layers"])]
    out = []
    for layer in cfg["layers"]:
        m, kind, att, rec = layer["mixer"], layer["type"], [], []
        if cfg["architecture"] == "Todupel":
            att.append((m["heads"] * 4 * (m["dim"] + m["vdim"]), 0, 0, m["kv_heads"] * (2 * m["dim"] + m["vdim"])))
        elif kind == "mamba2":
            rec.append((6 * m["heads"] * m["vdim"] * m["state"], m["heads"] * m["vdim"] * m["state"]))
        elif kind == "latent_attention":
            att.append((2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), m["mask"]["size"], 0, m["kv_rank"] + m["rot_dim"]))
        else:
            a = m["left"] if kind == "parallel" else m
            size = a["mask"]["size"]
            att.append((4 * a["heads"] * a["dim"], 0 if kind == "parallel" else size, size if kind == "parallel" else 0,
                        (1 if kind == "parallel" else 2) * a["kv_heads"] * a["dim"]))
            if kind == "parallel":
                r = m["right"]
                rec.append((7 * r["heads"] * r["dim"] * r["vdim"], r["heads"] * r["dim"] * r["vdim"]))
        out.append((att, rec))
    return out


def work(case):
    cfg = _model(case)
    size = 4 if case["dtype"] == "float32" else 2
    runs, steps = _runs(case), 3 if case["kind"] == "mixed" else 1
    tokens = sum(n for _, n in runs)
    wanted = len(runs) if steps == 1 else 3 * case["rows"] + 1
    vocab, width = _vocab(cfg), cfg.get("hidden_size") or cfg["width"]
    matrices = sum(math.prod(shape) for name, shape, kind in _tensors(cfg)
                   if kind == "matrix" and name not in ("embed", "head", "model.embed_tokens.weight", "lm_head.weight"))
    flops = 2.0 * matrices * tokens + 2.0 * vocab * width * wanted
    moved = float(size) * steps * (matrices + vocab * width) + size * tokens * width + 4.0 * vocab * wanted
    for att, rec in _mixers(cfg):
        for per_pair, window, chunk, numbers in att:
            flops += per_pair * sum(_pairs(s, n, window, chunk) for s, n in runs)
            read = sum(min(s, window) if window else (s % chunk if chunk else s) for s, _ in runs) * steps
            moved += size * numbers * (read + tokens)
        for per_token, state in rec:
            flops += per_token * tokens
            moved += 2.0 * 4 * state * len(runs) * steps
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """32-bit: logits lie up to 2e-5 of their size from the 64-bit ones. 16-bit: activations are rounded to 8 bits of mantissa
    in every part of a layer; the 16-layer model's logits lie 1.9 % from the 64-bit ones, and 1.8 % apart when another
    attention kernel of the engine computes them (largest single difference 0.14 of the root mean square)."""
    if case["dtype"] == "float32":
        return {"rel": 8e-5, "max": 1e-3}
    return {"rel": 3e-2, "max": 0.3}


# ----------------------------------------------------------------------------------------------------
# the designs in 64 bits
# ----------------------------------------------------------------------------------------------------

_MOST_WORK = 2.0e14          # operations in 64 bits that take about ten seconds on the GPU
_MOST_TOKENS = 20000         # tokens through recurrences that are walked one by one


def _rms(x, weight=None, eps=1e-5):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _layer_norm(x, weight, eps):
    dev = x - x.mean(-1, keepdim=True)
    return dev / torch.sqrt((dev * dev).mean(-1, keepdim=True) + eps) * weight


def _silu(z):
    return z * torch.sigmoid(z)


def _attend(q, k, v, scale, window=0, chunk=0, cap=0.0, sink=None):
    """Causal attention of a whole sequence. q [n, H, d], k [n, G, d], v [n, G, e]; `sink` [H]: one more score per head in the
    denominator. Queries go in runs so that the scores of one fit the memory."""
    n, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    pos = torch.arange(n, device=q.device)
    for lo in range(0, n, 512):
        hi = min(n, lo + 512)
        first = max(0, lo - window + 1) if window else 0
        seen = pos[None, first:hi] <= pos[lo:hi, None]
        if window:
            seen &= pos[lo:hi, None] - pos[None, first:hi] < window
        if chunk:
            seen &= (pos[lo:hi, None] // chunk) == (pos[None, first:hi] // chunk)
        kk = k[first:hi].repeat_interleave(H // G, 1)
        vv = v[first:hi].repeat_interleave(H // G, 1)
        s = torch.einsum("qhd,khd->hqk", q[lo:hi], kk) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~seen, -torch.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[:, None, None])
        w = torch.exp(s - top)
        den = w.sum(-1, keepdim=True)
        if sink is not None:
            den = den + torch.exp(sink[:, None, None] - top)
        out[lo:hi] = torch.einsum("hqk,khe->qhe", w / den, vv)
    return out


def _turn(x, cos, sin, interleaved=False):
    """x [n, ..., d] with its first 2 * len(cos[0]) numbers turned in pairs: (i, i + half), or (2i, 2i + 1)."""
    half = cos.shape[-1]
    shape = (cos.shape[0],) + (1,) * (x.dim() - 2) + (half,)
    c, s = cos.reshape(shape), sin.reshape(shape)
    y = x.clone()
    a, b = (x[..., 0:2 * half:2], x[..., 1:2 * half:2]) if interleaved else (x[..., :half], x[..., half:2 * half])
    u, w = a * c - b * s, b * c + a * s
    if interleaved:
        y[..., 0:2 * half:2], y[..., 1:2 * half:2] = u, w
    else:
        y[..., :half], y[..., half:2 * half] = u, w
    return y


def _conv(u, taps):
    n, K = u.shape[0], taps.shape[1]
    full = torch.cat([torch.zeros(K - 1, u.shape[1], dtype=u.dtype, device=u.device), u])
    return sum(full[j:j + n] * taps[:, j] for j in range(K))


def _llama_angles(cfg, n):
    """The design's rotary angles are numbers of 32 bits: position times frequency, rounded."""
    d, base = cfg["head_dim"], torch.tensor(cfg["rope_theta"], dtype=torch.float32)
    i = torch.arange(d // 2, dtype=torch.float32)
    inv = base ** (-2.0 * i / d)
    scaling = cfg.get("rope_scaling")
    if scaling:
        factor, low, high = scaling["factor"], scaling["low_freq_factor"], scaling["high_freq_factor"]
        old, div = scaling["original_max_position_embeddings"], []
        for j in range(d // 2):
            wave = 2.0 * math.pi * float(base) ** (2.0 * j / d)
            smooth = (old / wave - low) / (high - low)
            div.append(1.0 if wave < old / high else factor if wave > old / low else 1.0 / ((1.0 - smooth) / factor + smooth))
        inv = inv / torch.tensor(div, dtype=torch.float32)
    angle = (torch.arange(n, dtype=torch.float32)[:, None] * inv[None, :]).double().to(DEVICE)
    return angle.cos(), angle.sin()


def _llama_rows(cfg, w, ids):
    n, heads, groups, d, eps = len(ids), cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    cos, sin = _llama_angles(cfg, n)
    x = w("model.embed_tokens.weight", ids)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w(p + "input_layernorm.weight"), eps)
        q = _turn((h @ w(p + "self_attn.q_proj.weight").T).view(n, heads, d), cos, sin)
        k = _turn((h @ w(p + "self_attn.k_proj.weight").T).view(n, groups, d), cos, sin)
        v = (h @ w(p + "self_attn.v_proj.weight").T).view(n, groups, d)
        x = x + _attend(q, k, v, d ** -0.5).reshape(n, -1) @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, w(p + "post_attention_layernorm.weight"), eps)
        x = x + (_silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    return _rms(x, w("model.norm.weight"), eps)


def _todupel_rows(cfg, w, ids):
    n, eps = len(ids), cfg["norm"]["eps"]
    x = w("embed", ids)
    pos = torch.arange(n, device=DEVICE, dtype=torch.float64)
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        H, G, d, e, init = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["diff"]
        h = _rms(x, w(f"l{i}.norm1"), eps)
        warm = 1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1) / m["q_temp"]["every"]) + 1.0)
        q = _rms((h @ w(p + "q").T).view(n, H, 2, d), w(p + "q.norm"), eps) * warm[:, None, None, None]
        k = _rms((h @ w(p + "k").T).view(n, G, 2, d), w(p + "k.norm"), eps)
        v = (h @ w(p + "v").T).view(n, G, e)
        lam = torch.exp(w(p + "lq1") @ w(p + "lk1")) - torch.exp(w(p + "lq2") @ w(p + "lk2")) + init
        a, b = (_attend(q[:, :, j], k[:, :, j], v, m["scale"], cap=m["softcap"]) for j in (0, 1))
        mix = (_rms(a - lam * b, None, eps) * (1.0 - init)).reshape(n, -1) @ w(p + "o").T
        z = torch.relu(_rms(x, w(f"l{i}.norm2"), eps) @ w(f"l{i}.mlp.up").T)
        x = x + mix + (z * z) @ w(f"l{i}.mlp.down").T
    return _rms(x, w("final.norm"), eps)


def _plain_angles(base, dims, n, scaling=None):
    """(cos, sin) with frequencies stretched where `scaling` says so, and lengths with them."""
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / dims)
    mag = 1.0
    if scaling:
        s, L = scaling["factor"], scaling["original"]
        lo, hi = (dims * math.log(L / (2.0 * math.pi * t)) / (2.0 * math.log(base)) for t in (scaling["fast"], scaling["slow"]))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, mag = f / s * ramp + f * (1.0 - ramp), 0.1 * math.log(s) + 1.0
    angle = (torch.arange(n, dtype=torch.float64)[:, None] * f[None, :]).to(DEVICE)
    return angle.cos() * mag, angle.sin() * mag


def _latent(m, w, p, q, h, n, eps, interleaved, sink=None):
    H, d, r, e, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    cos, sin = _plain_angles(m["rot"]["base"], m["rot"]["dims"], n)
    q = torch.cat([q[..., :d], _turn(q[..., d:], cos, sin, interleaved)], -1)
    low = h @ w(p + "dkv").T
    c, kr = _rms(low[:, :R], w(p + "dkv.norm"), eps), _turn(low[:, R:], cos, sin, interleaved)
    k = torch.cat([(c @ w(p + "uk").T).view(n, H, d), kr[:, None].expand(n, H, r)], -1)
    return _attend(q, k, (c @ w(p + "uv").T).view(n, H, e), m["scale"], window=m["mask"]["size"], sink=sink).reshape(n, H * e)


def _state_space(m, w, p, h, n, eps):
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    z, u, dt = (h @ w(p + "in").T).split([inner, inner + 2 * G * N, H], -1)
    act = _silu(_conv(u, w(p + "conv")) + w(p + "conv.b"))
    x, B, C = act.split([inner, G * N, G * N], -1)
    x = x.reshape(n, H, P)
    B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    dt = torch.nn.functional.softplus(dt + w(p + "dt_bias"), threshold=1e3)
    decay = torch.exp(-torch.exp(w(p + "A_log")) * dt)
    xd = x * dt[..., None]
    S = torch.zeros(H, N, P, dtype=torch.float64, device=DEVICE)
    y = torch.empty(n, H, P, dtype=torch.float64, device=DEVICE)
    for t in range(n):
        S.mul_(decay[t][:, None, None]).baddbmm_(B[t][:, :, None], xd[t][:, None, :])
        torch.bmm(C[t][:, None, :], S, out=y[t].unsqueeze(1))
    y = y + w(p + "D")[:, None] * x
    g = (y.reshape(n, inner) * _silu(z)).view(n, m["norm_groups"], -1)
    return (_rms(g, None, eps).reshape(n, inner) * w(p + "norm")) @ w(p + "o").T


def _rematar_rows(cfg, w, ids):
    n, eps, alpha = len(ids), cfg["norm"]["eps"], cfg["postln_alpha"]
    x = w("embed", ids) * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        if layer["type"] == "mamba2":
            y = _state_space(m, w, p, x, n, eps)
        else:
            q = (_rms(x @ w(p + "dq").T, w(p + "dq.norm"), eps) @ w(p + "uq").T).view(n, m["heads"], m["dim"] + m["rot_dim"])
            y = _latent(m, w, p, q, x, n, eps, True, w(p + "sink"))
            y = (y * torch.sigmoid(x @ w(p + "g").T)) @ w(p + "o").T
        x = _rms(alpha * x + y * w(f"l{i}.ls1"), w(f"l{i}.norm1"), eps)
        f = torch.nn.functional.gelu(x @ w(f"l{i}.mlp.up").T, approximate="tanh") @ w(f"l{i}.mlp.down").T
        x = _rms(alpha * x + f * w(f"l{i}.ls2"), w(f"l{i}.norm2"), eps)
    return _rms(x, w("final.norm"), eps)


def _delta(m, w, p, h, n, eps):
    H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_silu(_conv(h @ w(p + c).T, w(p + c + ".conv"))) for c in "qkv")
    q, k, v = q.view(n, G, d), k.view(n, G, d), v.view(n, H, e)
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (q * d ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    beta = torch.sigmoid(h @ w(p + "b").T)
    step = torch.nn.functional.softplus(h @ w(p + "a1").T @ w(p + "a2").T + w(p + "dt_bias"), threshold=1e3).view(n, H, d)
    g = torch.exp(-torch.exp(w(p + "A_log"))[None, :, None] * step)
    gate = torch.sigmoid(h @ w(p + "g1").T @ w(p + "g2").T)
    S = torch.zeros(H, d, e, dtype=torch.float64, device=DEVICE)
    o = torch.empty(n, H, e, dtype=torch.float64, device=DEVICE)
    for t in range(n):
        S.mul_(g[t][:, :, None])
        u = beta[t][:, None, None] * (v[t][:, None, :] - torch.bmm(k[t][:, None, :], S))
        S.baddbmm_(k[t][:, :, None], u)
        torch.bmm(q[t][:, None, :], S, out=o[t].unsqueeze(1))
    return (_rms(o, w(p + "norm"), eps).reshape(n, H * e) * gate) @ w(p + "o").T


def _normed_attention(m, w, p, h, n, eps, chunked):
    H, G, d = m["heads"], m["kv_heads"], m["dim"]
    k = (h @ w(p + "k").T).view(n, G, d)
    v = k if chunked else (h @ w(p + "v").T).view(n, G, d)
    cos, sin = _plain_angles(m["rot"]["base"], m["rot"]["dims"], n, m["rot"].get("scaling"))
    q = _turn(_rms((h @ w(p + "q").T).view(n, H, d), w(p + "q.norm"), eps), cos, sin)
    k = _turn(_rms(k, w(p + "k.norm"), eps), cos, sin)
    size, zero = m["mask"]["size"], torch.zeros(H, dtype=torch.float64, device=DEVICE)
    return _attend(q, k, v, m["scale"], 0 if chunked else size, size if chunked else 0, sink=zero).reshape(n, -1) @ w(p + "o").T


def _nisotar_rows(cfg, w, ids):
    n, eps = len(ids), cfg["norm"]["eps"]
    x = w("embed", ids) * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        m, p, kind = layer["mixer"], f"l{i}.mix.", layer["type"]
        h = _layer_norm(x, w(f"l{i}.norm1"), eps)
        if kind == "parallel":
            a = _normed_attention(m["left"], w, p + "left.", h, n, eps, True)
            b = _delta(m["right"], w, p + "right.", h, n, eps)
            y = 0.5 * (_rms(a, w(p + "left.out"), eps) + _rms(b, w(p + "right.out"), eps))
        elif kind == "attention":
            y = _normed_attention(m, w, p, h, n, eps, False)
        else:
            q = (h @ w(p + "q").T).view(n, m["heads"], m["dim"] + m["rot_dim"])
            y = _latent(m, w, p, q, h, n, eps, False) @ w(p + "o").T
        x = x + y
        h, p, limit = _layer_norm(x, w(f"l{i}.norm2"), eps), f"l{i}.mlp.", layer["mlp"]["limit"]
        g = torch.clamp(h @ w(p + "gate").T + w(p + "gate.b"), max=limit)
        u = torch.clamp(h @ w(p + "up").T + w(p + "up.b"), -limit, limit)
        x = x + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + "down").T + w(p + "down.b")
    return _layer_norm(x, w("final.norm"), eps)


def exact(case, seed):
    """`run`'s logits in 64 bits, every sequence worked out whole; None where that takes too long."""
    cfg = _model(case)
    held, fed, joining = _all_ids(case, seed)
    if case["kind"] == "prefill":
        sequences, wanted = held, [1] * len(held)
    else:
        steps = 1 if case["kind"] == "decode" else 3
        sequences, wanted = [h + f[:steps] for h, f in zip(held, fed)], [steps] * len(held)
        if joining:
            sequences, wanted = sequences + [joining], wanted + [1]
    tokens = sum(map(len, sequences))
    matrices = sum(math.prod(shape) for name, shape, kind in _tensors(cfg) if kind == "matrix" and "embed" not in name)
    recurrent = any(rec for _, rec in _mixers(cfg))
    if 2.0 * matrices * tokens > _MOST_WORK or (recurrent and tokens > _MOST_TOKENS):
        return None
    tensors = _weights(case, seed)

    def w(name, rows=None):
        t = tensors[name]
        return t.double() if rows is None else t[torch.tensor(rows, device=t.device)].double()
    rows = {"Todupel": _todupel_rows, "Rematar": _rematar_rows, "Nisotar": _nisotar_rows}.get(cfg.get("architecture"), _llama_rows)
    head = next(n for n in ("lm_head.weight", "head", "model.embed_tokens.weight") if n in tensors)
    last = [rows(cfg, w, ids)[-n:] for ids, n in zip(sequences, wanted)]
    last = [x @ w(head).T for x in last]
    if case["kind"] != "mixed":
        return torch.cat(last)
    live = case["rows"]
    return [torch.stack([last[r][i] for r in range(live)] + ([last[live][0]] if i == 2 else [])) for i in range(3)]
