"""The work that users of this library have it do, as cases that can be timed.

A case names a model (layer sizes of this repository's benchmark, random
weights), a dtype, and what is done with it:

* ``decode``: a server's steady state: ``batch`` sequences with about ``tokens`` cached positions each, one more token
  of each per pass, chosen on the device.  The contexts grow from pass to pass, as they do in use.
* ``session``: ``batch`` prompts arrive together, ``later`` more join while the first ones decode, and ``steps`` further
  steps bring one token each: prefill of whole prompts, the mixed step of continuous batching, and decode.
* ``generate``: the Python entry point, prompts in and tokens out, beside the logits that a caller may ask it for.

``tokens`` is the length of the longest prompt; with ``ragged`` the others are shorter, down to a fifth.
"""
from __future__ import annotations

import gc
import math
import zlib

import numpy as np
import torch

from esp_b200.config import config_from_dict
from esp_b200.engine import Engine, StepEntry
from esp_b200.provider import DecoderProvider, GenerationRequest

# ---------------------------------------------------------------------------------------------------------
# models: layer sizes of bench.py
_QWEN = {
    "architectures": ["Qwen2MoeForCausalLM"], "model_type": "qwen2_moe", "hidden_act": "silu", "head_dim": 128,
    "vocab_size": 151936, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "norm_topk_prob": False, "decoder_sparse_step": 1,
    "mlp_only_layers": [], "use_sliding_window": False, "sliding_window": None, "tie_word_embeddings": False,
}
_A27B = dict(_QWEN, num_hidden_layers=24, hidden_size=2048, num_attention_heads=16, num_key_value_heads=16,
             max_position_embeddings=8192, intermediate_size=5632, num_experts=60, num_experts_per_tok=4,
             moe_intermediate_size=1408, shared_expert_intermediate_size=5632)
_Q57B = dict(_QWEN, num_hidden_layers=28, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4,
             max_position_embeddings=32768, intermediate_size=18944, num_experts=64, num_experts_per_tok=8,
             moe_intermediate_size=2560, shared_expert_intermediate_size=20480)
_VOCAB, _WINDOW = 32768, 4096


def _galirax(width, ff, layers):
    """Attention over all keys, windowed attention that keeps the first tokens, linear attention, routed experts."""
    heads = width // 128
    att = {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
           "rot": {"dims": 128, "base": 1e6}}
    scaled = dict(att, rot=dict(att["rot"], scaling={"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}))
    kept = dict(att, mask={"size": _WINDOW, "keep_first": 4})
    linear = {"heads": heads, "dim": 128, "vdim": 128, "decay": [1 - 2.0 ** -(3 + 6 * h / heads) for h in range(heads)]}
    pattern = [("attention", scaled), ("attention_2", kept), ("lightning", linear), ("attention_2", kept)]
    moe = {"kind": "moe", "router": {"experts": 16, "top": 4, "scale": 2.5, "groups": {"count": 4, "keep": 2}},
           "expert": {"ff": ff // 4}}
    return {"architecture": "Galirax", "vocab": _VOCAB, "width": width, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "layers": [{"type": t, "mixer": dict(m), "mlp": dict(moe)} for t, m in (pattern[i % 4] for i in range(layers))]}


def _zusepel(width, ff, layers):
    """Gated linear recurrences, time mixing with token shift, attention through a cached latent, dense feed-forwards."""
    heads = width // 128
    lat = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 3 * width // 8, "kv_rank": min(512, width // 4),
           "scale": (128 + 64) ** -0.5, "mask": {"size": _WINDOW},
           "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "fast": 32.0, "original": 4096, "slow": 1.0}}}
    pattern = [("hgrn2", {"heads": heads, "dim": 128, "vdim": 128}), ("wkv", {"heads": width // 64, "dim": 64}),
               ("latent_attention", lat), ("latent_attention", dict(lat, kv_from=-1))]
    out = []
    for i in range(layers):
        t, m = pattern[i % 4][0], dict(pattern[i % 4][1])
        if "kv_from" in m:
            m["kv_from"] = i - 1
        out.append({"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": ff}})
    return {"architecture": "Zusepel", "vocab": _VOCAB, "width": width, "norm": {"eps": 1e-6}, "residual_mult": 0.7,
            "layers": out, "decay_ranks": {str(i): 64 for i in range(layers) if out[i]["type"] == "wkv"}}


def _config(case):
    model, layers = case["model"], case["layers"]
    if model == "a2.7b":
        return dict(_A27B, num_hidden_layers=layers)
    if model == "57b-a14b":
        return dict(_Q57B, num_hidden_layers=layers)
    kind, width = model.split("-w")
    return {"galirax": _galirax, "zusepel": _zusepel}[kind](int(width), {"1024": 2816, "2048": 5632}[width], layers)


def _is_qwen(c):
    return "hidden_size" in c


def _vocab(c):
    return c["vocab_size"] if _is_qwen(c) else c["vocab"]


# ---------------------------------------------------------------------------------------------------------
# cases
def listed():
    def case(name, model, layers, kind, batch, tokens, *, dtype="bfloat16", ragged=False, later=0, steps=0):
        return {"name": name, "model": model, "layers": layers, "dtype": dtype, "kind": kind, "batch": batch,
                "tokens": tokens, "ragged": ragged, "later": later, "steps": steps}

    return [
        # one user waiting for the next token: launches and latency count
        case("a2.7b decode 1", "a2.7b", 24, "decode", 1, 1024),
        # the headline of bench.py: eight sequences at a context of 4,096
        case("a2.7b decode 8", "a2.7b", 24, "decode", 8, 4000),
        # a busy server with unequal contexts: nearly every expert at work
        case("a2.7b decode 64", "a2.7b", 24, "decode", 64, 500, ragged=True),
        # a question of one line: time to the first token
        case("a2.7b prompt of 19", "a2.7b", 24, "session", 1, 19),
        # one long prompt (the prefill of bench.py)
        case("a2.7b prompt of 2048", "a2.7b", 24, "session", 1, 2048),
        # continuous batching: odd prompts, more that join while the first ones decode, two steps more
        case("a2.7b mixed batch", "a2.7b", 24, "session", 5, 613, ragged=True, later=3, steps=2),
        # the larger shape, cut to the layers that leave room for three of it: the longest prompt here
        case("57b-a14b prompt of 4096", "57b-a14b", 4, "session", 1, 4096),
        # the larger shape at a long context, grouped queries
        case("57b-a14b decode 8", "57b-a14b", 4, "decode", 8, 7900),
        # the true 32-bit path: an unequal batch of prompts, then tokens one by one
        case("a2.7b 32-bit batch", "a2.7b", 4, "session", 6, 381, dtype="float32", ragged=True, steps=3),
        # the designs with other layers: windowed and linear attention beside experts; recurrences and latents
        case("galirax-w2048 prompt of 2048", "galirax-w2048", 8, "session", 1, 2048),
        case("zusepel-w2048 decode 8", "zusepel-w2048", 8, "decode", 8, 2000),
        # the smallest call: the entry point with one short prompt and few tokens on a small model
        case("galirax-w1024 generate", "galirax-w1024", 8, "generate", 1, 13, steps=8),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model, layers, dtype = rng.choice([
        ("a2.7b", 24, "bfloat16"), ("a2.7b", 24, "bfloat16"), ("a2.7b", 24, "bfloat16"), ("a2.7b", 4, "float32"),
        ("57b-a14b", 4, "bfloat16"), ("galirax-w2048", 8, "bfloat16"), ("zusepel-w2048", 8, "bfloat16"),
        ("galirax-w1024", 8, "bfloat16"), ("zusepel-w1024", 8, "bfloat16")])
    kind = rng.choice(["decode", "decode", "session", "session", "session", "generate"])
    if dtype == "float32" and kind == "decode":
        kind = "session"                # the 32-bit path's use: whole batches, compared
    case = {"model": model, "layers": layers, "dtype": dtype, "kind": kind, "batch": 1, "tokens": 1, "ragged": True,
            "later": 0, "steps": 0}
    if kind == "decode":
        case["batch"] = log(1, 64)
        case["tokens"] = log(24, min(4000, 32000 // case["batch"]))
    elif kind == "session":
        total = log(12, 1000 if dtype == "float32" else 4000)
        case["batch"] = min(log(1, 16), max(1, total // 4))
        if rng.random() < 0.4:
            case["later"], case["steps"] = rng.randint(0, 4), rng.randint(1, 2)
        case["tokens"] = max(3, total // (case["batch"] + case["later"]))
    else:
        case["batch"], case["tokens"], case["steps"] = rng.randint(1, 3), log(5, 300), rng.randint(3, 7)
    return case


# ---------------------------------------------------------------------------------------------------------
# weights: every tensor from (seed, name), so that they can be made again one by one
def _stored(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _make(name, shape, seed, dtype):
    """Random values in the ranges that keep every mechanism at work.  The head's row for token t is the embedding of
    token t - 1, so that the model has a next token it is sure of, as a trained one mostly has."""
    if name in ("head", "lm_head.weight"):
        table = _make("embed" if name == "head" else "model.embed_tokens.weight", shape, seed, dtype)
        return torch.roll(table, 1, 0).mul_(0.02 if name == "lm_head.weight" else 1 / (0.7 * math.sqrt(shape[1])))
    g = torch.Generator(device="cuda").manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & ((1 << 62) - 1))
    t = torch.empty(shape, dtype=dtype, device="cuda")
    leaf = name.rsplit(".", 1)[-1]
    if name.startswith("model.") or name.startswith("lm_head"):
        if name == "model.embed_tokens.weight":
            return t.normal_(0.0, 1.0, generator=g)
        if "norm" in name:
            return t.normal_(1.0, 0.02, generator=g)
        if ".experts." in name and "down_proj" in name:
            # the last expert that a token takes scores hardly more than the next one: small beside the residual stream,
            # so that a token whose experts change places by rounding stays the same token
            return t.normal_(0.0, 0.007, generator=g)
        return t.normal_(0.0, 0.02, generator=g)
    if name == "embed":
        return t.normal_(0.0, 0.7, generator=g)
    if leaf == "down" and ".e" in name:
        # as above; here the four chosen scores are nearly equal
        return t.normal_(0.0, 0.05 / math.sqrt(shape[1]), generator=g)
    if len(shape) == 2 and leaf != "u":
        return t.normal_(0.0, 1 / math.sqrt(shape[1]), generator=g)
    if leaf in ("norm", "norm1", "norm2"):
        return t.normal_(1.0, 0.2, generator=g)
    if leaf == "dwa":
        return t.normal_(1 / shape[0], 0.1 / shape[0], generator=g)
    if leaf in ("ls1", "ls2"):
        return t.uniform_(0.4, 1.2, generator=g)
    if leaf == "lower":
        return t.uniform_(0.0, 0.95, generator=g)
    if ".mu." in name:
        return t.uniform_(0.0, 1.0, generator=g)
    mean, std = {"b": (0.0, 0.2), "sink": (0.0, 1.5), "correction": (0.0, 0.05), "w0": (-1.5, 1.0), "u": (0.0, 0.5),
                 "act": (0.0, 0.5)}[leaf]
    return t.normal_(mean, std, generator=g)


class _Source:
    """A checkpoint as the loader sees one."""

    def __init__(self, specs, seed, dtype):
        self._shapes = {s.name: tuple(s.shape) for s in specs if not s.optional}
        self._seed, self._dtype = seed, dtype

    def names(self):
        return list(self._shapes)

    def dtype(self, name):
        return self._dtype

    def shape(self, name):
        return self._shapes[name]

    def read_into(self, name, view):
        view.copy_(_make(name, self._shapes[name], self._seed, self._dtype))


# ---------------------------------------------------------------------------------------------------------
# inputs
_WARM = 3        # decode steps ahead of the first pass: a server that has been running


def _inputs(case, seed):
    """Token lists of every sequence: prompts, and what follows them."""
    rng = np.random.default_rng([seed, 17])
    n = case["batch"] + case["later"]
    lens = [case["tokens"]] + [int(rng.integers(max(1, case["tokens"] // 5), case["tokens"] + 1)) if case["ragged"]
                               else case["tokens"] for _ in range(n - 1)]
    vocab = _vocab(_config(case))
    prompts = [rng.integers(0, vocab, k).tolist() for k in lens]
    room = _room(case) if case["kind"] == "decode" else 1 + case["steps"]
    return prompts, rng.integers(0, vocab, (room, n)).tolist()


def _room(case):
    """Decode passes before the sequences of a state are done and others like them take their places."""
    return 640 if case["batch"] * case["tokens"] > 4096 else 2048


def _pages(n):
    return (n + 63) // 64 * 64


class _State:
    pass


def prepare(case, seed):
    gc.collect()
    torch.cuda.empty_cache()
    s = _State()
    s.case = case
    s.prompts, s.follow = _inputs(case, seed)
    config = config_from_dict(_config(case))
    n = len(s.prompts)
    tokens = sum(_pages(len(p) + len(s.follow) + 1) for p in s.prompts) + 64 * n
    s.engine = Engine(config, lambda specs: _Source(specs, seed, _stored(case)), dtype=case["dtype"], max_tokens=tokens,
                      max_slots=n + 1)
    if case["kind"] == "generate":
        s.provider = DecoderProvider(s.engine, None, max_batch=8)
        # the first request is greedy, the others draw
        s.requests = [GenerationRequest(prompt_ids=p, max_tokens=case["steps"], temperature=0.8 if i else 0.0,
                                        top_p=0.95 if i else None, seed=i + 1 if i else None) for i, p in enumerate(s.prompts)]
    elif case["kind"] == "decode":
        _arrive(s)
        for _ in range(_WARM):
            run(s)
    return s


def _arrive(s):
    """The sequences of a decode case enter: every second one draws its tokens, the others take the likeliest."""
    e, room = s.engine, 4096
    s.slots = [e.open() for _ in s.prompts]
    waiting = []
    for slot, p in list(zip(s.slots, s.prompts)) + [(None, [])]:
        if waiting and (slot is None or sum(len(w.tokens) for w in waiting) + len(p) > room):
            e.step(waiting)
            waiting = []
        if slot is not None:
            waiting.append(StepEntry(slot, p, []))
    for i, slot in enumerate(s.slots):
        e.seed_slot(slot, 7 + i)
    s.temperatures = [0.8 if i % 2 else 0.0 for i in range(len(s.slots))]
    s.top_ps = [0.95 if i % 2 else None for i in range(len(s.slots))]
    s.at = 0


def run(s):
    case, e = s.case, s.engine
    if case["kind"] == "generate":
        logits = s.provider.next_token_logits(s.prompts[0])
        return [[list(g.token_ids) for g in s.provider.generate(s.requests)], logits]
    if case["kind"] == "decode":
        if s.at == len(s.follow):
            for slot in s.slots:
                e.close(slot)
            _arrive(s)
        tokens, logits = e.step_and_pick([StepEntry(slot, [t], [0]) for slot, t in zip(s.slots, s.follow[s.at])],
                                         s.temperatures, s.top_ps)
        s.at += 1
        return [tokens, logits]
    n, first = len(s.prompts), case["batch"]
    slots = [e.open() for _ in range(n)]
    out = [e.step([StepEntry(slots[i], s.prompts[i], [len(s.prompts[i]) - 1]) for i in range(first)])]
    if case["later"]:
        entries = [StepEntry(slots[i], [s.follow[0][i]], [0]) for i in range(first)]
        entries += [StepEntry(slots[i], s.prompts[i], [len(s.prompts[i]) - 1]) for i in range(first, n)]
        out.append(e.step(entries))
    for j in range(case["steps"]):
        out.append(e.step([StepEntry(slots[i], [s.follow[1 + j][i]], [0]) for i in range(n)]))
    for slot in slots:
        e.close(slot)
    return out


# ---------------------------------------------------------------------------------------------------------
# what a pass cannot do without: every weight it uses, every cached key it sees and every input read once, outputs and
# new keys written once
def _steps(case):
    """(new tokens, cached tokens) per sequence, and the rows of logits, for every step of a pass; the lengths of a
    ragged batch at their mean."""
    n, b, t = case["batch"] + case["later"], case["batch"], case["tokens"]
    other = 0.6 * t if case["ragged"] else t
    lens = [t] + [other] * (n - 1)
    if case["kind"] == "decode":
        return [([1] * b, lens, b)]
    if case["kind"] == "generate":
        return ([([t], [0], 1), (lens, [0] * n, n)]
                + [([1] * n, [k + j for k in lens], n) for j in range(case["steps"] - 1)])
    out = [(lens[:b], [0] * b, b)]
    if case["later"]:
        out.append(([1] * b + lens[b:], lens[:b] + [0] * (n - b), n))
    return out + [([1] * n, [k + 1 + j for k in lens], n) for j in range(case["steps"])]


def _layer_sizes(c):
    """Per layer: weights that every token uses, weights of one expert, experts, experts a token takes, multiplications
    per visible key, cached numbers per position, the state's numbers per sequence."""
    if _is_qwen(c):
        H, nh, nkv, hd = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        fixed = H * (nh + 2 * nkv) * hd + nh * hd * H + c["num_experts"] * H + H + 3 * H * c["shared_expert_intermediate_size"]
        return [(fixed, 3 * H * c["moe_intermediate_size"], c["num_experts"], c["num_experts_per_tok"], 2 * nh * hd,
                 2 * nkv * hd, 0)] * c["num_hidden_layers"]
    out, D = [], c["width"]
    for layer in c["layers"]:
        m, f, t = layer["mixer"], layer["mlp"], layer["type"]
        H, K = m["heads"], m["dim"]
        keys = kept = state = 0
        if t == "wkv":
            fixed, state = 5 * D * H * K + 64 * (D + H * K), H * K * K
        elif t in ("hgrn2", "lightning"):
            fixed = D * H * (2 * K + (2 if t == "hgrn2" else 3) * m["vdim"])
            state = H * K * m["vdim"]
        elif t == "latent_attention":
            fixed = m["q_rank"] * (D + H * (K + m["rot_dim"])) + m["kv_rank"] * H * (K + m["vdim"]) + D * H * m["vdim"]
            keys = H * (K + m["rot_dim"] + m["vdim"])
            if m.get("kv_from") is None:
                fixed += D * (m["kv_rank"] + m["rot_dim"])
            kept = m["kv_rank"] + m["rot_dim"]
        else:
            fixed = D * (H * K + m["kv_heads"] * (K + m["vdim"]) + H * m["vdim"])
            keys, kept = H * (K + m["vdim"]), m["kv_heads"] * (K + m["vdim"])
        if f["kind"] == "dense":
            out.append((fixed + 2 * D * f["ff"], 0, 1, 0, keys, kept, state))
        else:
            r = f["router"]
            out.append((fixed + r["experts"] * D, 3 * D * f["expert"]["ff"], r["experts"], r["top"], keys, kept, state))
    return out


def work(case):
    c = _config(case)
    el = 4 if case["dtype"] == "float32" else 2
    width, vocab = (c["hidden_size"], c["vocab_size"]) if _is_qwen(c) else (c["width"], c["vocab"])
    total_bytes = total_flops = 0.0
    for news, pasts, rows in _steps(case):
        n = sum(news)
        seen = sum(a * (p + (a + 1) / 2) for a, p in zip(news, pasts))
        for fixed, expert, experts, top, keys, kept, state in _layer_sizes(c):
            used = experts * (1 - (1 - top / experts) ** n) if expert else 0
            total_bytes += el * (fixed + used * expert) + el * kept * sum(a + p for a, p in zip(news, pasts))
            total_bytes += 2 * 4 * state * len(news)
            total_flops += 2 * n * (fixed + top * expert) + 2 * keys * seen + 4 * state * n
        total_bytes += el * vocab * width + el * width * n + 4 * rows * vocab
        total_flops += 2 * rows * vocab * width
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    # bfloat16 activations between the layers (relative step 2^-8) through 4 to 24 layers, where two experts that score
    # alike may also change places for some token; 32-bit sums in another order
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-2, "differ": 0.01}
    return {"rel": 0.03, "max": 0.5, "differ": 0.01}


# ---------------------------------------------------------------------------------------------------------
# the same in 64 bits, by plain formulas, over packed rows of all sequences at once
class _Weights:
    def __init__(self, case, seed):
        self.seed, self.dtype = seed, _stored(case)

    def __call__(self, name, *shape):
        return _make(name, shape, self.seed, self.dtype).double()


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, b, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


def _silu(z):
    return z * torch.sigmoid(z)


def _attend(q, k, v, scale, spans, mask=None, sink=None):
    """q [N, H, K], k [N, G, K], v [N, G, V]: causal attention within every span of rows, 512 queries at a time."""
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    rep = q.shape[1] // k.shape[1]
    for lo, hi in spans:
        for a in range(lo, hi, 512):
            b = min(hi, a + 512)
            i, j = torch.arange(a, b, device="cuda")[:, None], torch.arange(lo, b, device="cuda")[None, :]
            seen = j <= i
            if mask is not None:
                seen = seen & ((i - j < mask["size"]) | (j - lo < mask.get("keep_first", 0)))
            qs = q[a:b].view(b - a, k.shape[1], rep, -1)
            s = torch.einsum("tgrk,sgk->grts", qs, k[lo:b]) * scale
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                none = sink.view(k.shape[1], rep, 1, 1).expand(-1, -1, b - a, 1)
                p = torch.softmax(torch.cat([s, none], -1), -1)[..., :-1]
            else:
                p = torch.softmax(s, -1)
            out[a:b] = torch.einsum("grts,sgv->tgrv", p, v[lo:b]).reshape(b - a, q.shape[1], -1)
    return out


def _by_rows(fn, x, step=8192):
    return torch.cat([fn(x[i:i + step]) for i in range(0, x.shape[0], step)])


def _gated(x, gate, up, down):
    return _by_rows(lambda r: (_silu(r @ gate.T) * (r @ up.T)) @ down.T, x)


def _experts(x, ids, weights, count, matrices):
    y = torch.zeros_like(x)
    for e in range(count):
        t, j = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            y[t] += weights[t, j][:, None] * _gated(x[t], *matrices(e))
    return y


def _angles(positions, freq):
    ang = positions.double()[:, None, None] * freq[None, None, :]
    return torch.cos(ang), torch.sin(ang)


def _exact_qwen(c, W, x, positions, spans, rows):
    H, nh, nkv, hd, eps = (c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"],
                           c["rms_norm_eps"])
    E, Im, Is = c["num_experts"], c["moe_intermediate_size"], c["shared_expert_intermediate_size"]
    half = hd // 2
    freq = c["rope_theta"] ** (-2.0 * torch.arange(half, dtype=torch.float64, device="cuda") / hd)
    cos, sin = _angles(positions, freq)

    def rotated(z):
        a, b = z[..., :half], z[..., half:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for i in range(c["num_hidden_layers"]):
        p, a, f = f"model.layers.{i}.", f"model.layers.{i}.self_attn.", f"model.layers.{i}.mlp."
        h = _rms(x, eps) * W(p + "input_layernorm.weight", H)
        q, k, v = (h @ W(f"{a}{t}_proj.weight", m * hd, H).T + W(f"{a}{t}_proj.bias", m * hd)
                   for t, m in (("q", nh), ("k", nkv), ("v", nkv)))
        o = _attend(rotated(q.view(-1, nh, hd)), rotated(k.view(-1, nkv, hd)), v.view(-1, nkv, hd), hd ** -0.5, spans)
        x = x + o.reshape(-1, nh * hd) @ W(a + "o_proj.weight", H, nh * hd).T
        if i + 1 == c["num_hidden_layers"]:
            x = x[rows]                      # nothing below mixes rows
        h = _rms(x, eps) * W(p + "post_attention_layernorm.weight", H)
        prob = torch.softmax(h @ W(f + "gate.weight", E, H).T, -1)
        top, ids = torch.topk(prob, c["num_experts_per_tok"], -1)
        y = _experts(h, ids, top, E, lambda e: [W(f"{f}experts.{e}.{t}_proj.weight", *s)
                                                for t, s in (("gate", (Im, H)), ("up", (Im, H)), ("down", (H, Im)))])
        s = f + "shared_expert."
        y += torch.sigmoid(h @ W(f + "shared_expert_gate.weight", 1, H).T) * _gated(
            h, W(s + "gate_proj.weight", Is, H), W(s + "up_proj.weight", Is, H), W(s + "down_proj.weight", H, Is))
        x = x + y
    return (_rms(x, eps) * W("model.norm.weight", H)) @ W("lm_head.weight", c["vocab_size"], H).T


def _recurrence(spans, steps, read):
    """Runs ``steps(state, rows)`` -> state and ``read`` along all spans side by side: rows are the spans' t-th rows."""
    longest = max(hi - lo for lo, hi in spans)
    order = sorted(range(len(spans)), key=lambda s: spans[s][0] - spans[s][1])
    state = None
    for t in range(longest):
        live = [spans[s][0] + t for s in order if spans[s][1] - spans[s][0] > t]
        rows = torch.tensor(live, device="cuda") if len(live) > 1 else slice(live[0], live[0] + 1)
        state = steps(state if state is None else state[:len(live)], rows)
        read(state, rows)


def _exact_galirax(c, W, x, positions, spans, rows):
    D, eps = c["width"], c["norm"]["eps"]

    def rotated(z, rot):
        i = torch.arange(rot["dims"] // 2, dtype=torch.float64, device="cuda")
        freq = float(rot["base"]) ** (-2.0 * i / rot["dims"])
        sc = rot.get("scaling")
        if sc:
            turns = sc["original"] * freq / (2 * math.pi)
            share = ((turns - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
            freq = freq / sc["factor"] * (1 - share) + freq * share
        cos, sin = _angles(positions, freq)
        a, b = z[..., 0::2], z[..., 1::2]
        return torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)

    for i, layer in enumerate(c["layers"]):
        p, m, r, ff = f"l{i}.mix.", layer["mixer"], layer["mlp"]["router"], layer["mlp"]["expert"]["ff"]
        heads, K, V = m["heads"], m["dim"], m["vdim"]
        h = _layer_norm(x, W(f"l{i}.norm1", D), W(f"l{i}.norm1.b", D), eps)
        if layer["type"] == "lightning":
            q, k, v = (_silu(h @ W(p + t, heads * n, D).T).view(-1, heads, n) for t, n in (("q", K), ("k", K), ("v", V)))
            decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[:, None, None]
            o = torch.empty_like(v)

            def steps(S, at):
                kv = k[at][..., :, None] * v[at][..., None, :]
                return kv if S is None else decay * S + kv

            def read(S, at):
                o[at] = (S * q[at][..., :, None]).sum(-2)
            _recurrence(spans, steps, read)
            o = _rms(o.reshape(-1, heads * V), eps) * W(p + "norm", heads * V) * torch.sigmoid(h @ W(p + "g", heads * V, D).T)
        else:
            G = m["kv_heads"]
            q, k, v = h @ W(p + "q", heads * K, D).T, h @ W(p + "k", G * K, D).T, h @ W(p + "v", G * V, D).T
            if layer["type"] == "attention_2":
                q = _rms(q + W(p + "q.b", heads * K), eps) * W(p + "q.norm", heads * K)
                k = _rms(k + W(p + "k.b", G * K), eps) * W(p + "k.norm", G * K)
                v = v + W(p + "v.b", G * V)
            o = _attend(rotated(q.view(-1, heads, K), m["rot"]), rotated(k.view(-1, G, K), m["rot"]), v.view(-1, G, V),
                        m["scale"], spans, m.get("mask"), W(p + "sink", heads)).reshape(-1, heads * V)
        y = o @ W(p + "o", D, heads * V).T
        f = f"l{i}.mlp."
        score = torch.sigmoid(h @ W(f + "router", r["experts"], D).T)
        groups, per = r["groups"]["count"], r["experts"] // r["groups"]["count"]
        choice = (score + W(f + "correction", r["experts"])).view(-1, groups, per)
        best = choice.topk(2, -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
        allowed = torch.zeros_like(choice[..., 0], dtype=torch.bool).scatter_(1, best, True)
        ids = choice.masked_fill(~allowed[..., None], -math.inf).flatten(1).topk(r["top"], -1).indices
        wts = score.gather(1, ids)
        wts = wts / (wts.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        x = x + y + _experts(h, ids, wts, r["experts"], lambda e: [W(f"{f}e{e}.{t}", *s) for t, s in (
            ("gate", (ff, D)), ("up", (ff, D)), ("down", (D, ff)))])
    h = _layer_norm(x[rows], W("final.norm", D), W("final.norm.b", D), eps)
    return c["logit_softcap"] * torch.tanh(h @ W("head", c["vocab"], D).T / c["logit_softcap"])


def _exact_zusepel(c, W, x, positions, spans, rows):
    D, eps, mult = c["width"], c["norm"]["eps"], c["residual_mult"]
    starts = torch.tensor([lo for lo, _hi in spans], device="cuda")
    streams, kept = [x], {}

    def rotated(z, rot):
        dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
        i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
        f = base ** (-2 * i / dims)
        lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * sc[t])) / (2 * math.log(base)) for t in ("fast", "slow"))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        cos, sin = _angles(positions, f / sc["factor"] * ramp + f * (1 - ramp))
        mag = 0.1 * math.log(sc["factor"]) + 1
        a, b = z[..., :dims // 2], z[..., dims // 2:dims]
        return torch.cat([(a * cos - b * sin) * mag, (b * cos + a * sin) * mag, z[..., dims:]], -1)

    for i, layer in enumerate(c["layers"]):
        p, m, ff = f"l{i}.mix.", layer["mixer"], layer["mlp"]["ff"]
        H, K = m["heads"], m["dim"]
        V = m.get("vdim", K)
        h = _rms(x, eps) * W(f"l{i}.norm1", D)
        if layer["type"] == "hgrn2":
            q = _silu(h @ W(p + "q", H * K, D).T).view(-1, H, K)
            v = (h @ W(p + "v", H * V, D).T).view(-1, H, V)
            low = W(p + "lower", H * K)
            f = (low + (1 - low) * torch.sigmoid(h @ W(p + "f", H * K, D).T + W(p + "f.b", H * K))).view(-1, H, K)
            o = torch.empty_like(v)

            def steps(S, at):
                new = (1 - f[at])[..., :, None] * v[at][..., None, :]
                return new if S is None else f[at][..., :, None] * S + new

            def read(S, at):
                o[at] = (S * q[at][..., :, None]).sum(-2)
            _recurrence(spans, steps, read)
            o = (_rms(o, eps) * W(p + "norm", V)).reshape(-1, H * V)
        elif layer["type"] == "wkv":
            prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
            prev[starts] = 0
            mixed = {s: h + (prev - h) * W(f"{p}mu.{s}", D) for s in "rkvgw"}
            r, k, v = ((mixed[s] @ W(p + s, H * K, D).T).view(-1, H, K) for s in "rkv")
            gate = _silu(mixed["g"] @ W(p + "g", H * K, D).T)
            low = torch.tanh(mixed["w"] @ W(p + "w1", 64, D).T) @ W(p + "w2", H * K, 64).T + W(p + "w0", H * K)
            decay, u = torch.exp(-torch.exp(low)).view(-1, H, K), W(p + "u", H, K)[..., None]
            o = torch.empty_like(v)

            def steps(S, at):
                kv = k[at][..., :, None] * v[at][..., None, :]
                o[at] = (((0 if S is None else S) + u * kv) * r[at][..., :, None]).sum(-2)
                return kv if S is None else decay[at][..., :, None] * S + kv
            _recurrence(spans, steps, lambda S, at: None)
            o = _rms(o, eps).reshape(-1, H * K) * W(p + "norm", H * K) * gate
        else:
            R, rank = m["rot_dim"], m["kv_rank"]
            if m.get("kv_from") is None:
                d = h @ W(p + "dkv", rank + R, D).T
                kept[i] = (_rms(d[:, :rank], eps) * W(p + "dkv.norm", rank), rotated(d[:, None, rank:], m["rot"]))
            lat, key_rot = kept[i if m.get("kv_from") is None else m["kv_from"]]
            q = (_rms(h @ W(p + "dq", m["q_rank"], D).T, eps) * W(p + "dq.norm", m["q_rank"])) @ W(
                p + "uq", H * (K + R), m["q_rank"]).T
            q = q.view(-1, H, K + R)
            q = torch.cat([q[..., :K], rotated(q[..., K:], m["rot"])], -1)
            k = torch.cat([(lat @ W(p + "uk", H * K, rank).T).view(-1, H, K), key_rot.expand(-1, H, -1)], -1)
            v = (lat @ W(p + "uv", H * V, rank).T).view(-1, H, V)
            o = _attend(q, k, v, m["scale"], spans, m.get("mask")).reshape(-1, H * V)
        x = x + mult * ((o @ W(p + "o", D, o.shape[1]).T) * W(f"l{i}.ls1", D))
        h = _rms(x, eps) * W(f"l{i}.norm2", D)
        ap, aq = (torch.nn.functional.softplus(z) for z in W(f"l{i}.mlp.act", 2))
        up, down = W(f"l{i}.mlp.up", ff, D), W(f"l{i}.mlp.down", D, ff)

        def feed(r):
            z = r @ up.T
            neg = (0.5 + aq) * (torch.expm1(z.clamp(max=0)) - z)
            return (torch.where(z > 0, ap * z * z, neg) + 0.5 * z) @ down.T
        x = x + mult * (_by_rows(feed, h) * W(f"l{i}.ls2", D))
        streams.append(x)
        mixw = W(f"l{i}.dwa", i + 2)
        x = sum(mixw[j] * s for j, s in enumerate(streams))
    return (_rms(x[rows], eps) * W("final.norm", D)) @ W("head", c["vocab"], D).T


def exact(case, seed):
    """64-bit logits of the first pass on a new state."""
    c = _config(case)
    prompts, follow = _inputs(case, seed)
    n, first = len(prompts), case["batch"]
    seqs, wanted = [], []                        # tokens of every sequence, and the step of each of its logits rows
    for i, p in enumerate(prompts):
        if case["kind"] == "decode":
            extra = [follow[j][i] for j in range(_WARM + 1)]
            seqs.append(p + extra)
            wanted.append({len(p) + _WARM: 0})
        elif case["kind"] == "generate":
            seqs.append(p)
            wanted.append({len(p) - 1: 0} if i == 0 else {})
        else:
            joined = 0 if i < first else 1
            extra = ([follow[0][i]] if case["later"] and not joined else []) + [follow[1 + j][i] for j in range(case["steps"])]
            seqs.append(p + extra)
            wanted.append({len(p) - 1 + k: joined + k for k in range(len(extra) + 1)})
    spans, rows, step_of, at = [], [], [], 0
    for s, w in zip(seqs, wanted):
        spans.append((at, at + len(s)))
        rows += [at + k for k in w]
        step_of += list(w.values())
        at += len(s)
    W = _Weights(case, seed)
    vocab, width = (c["vocab_size"], c["hidden_size"]) if _is_qwen(c) else (c["vocab"], c["width"])
    x = W("model.embed_tokens.weight" if _is_qwen(c) else "embed", vocab, width)[
        torch.tensor([t for s in seqs for t in s], device="cuda")]
    positions = torch.cat([torch.arange(hi - lo, device="cuda") for lo, hi in spans])
    fn = _exact_qwen if _is_qwen(c) else _exact_galirax if c["architecture"] == "Galirax" else _exact_zusepel
    logits = fn(c, W, x, positions, spans, torch.tensor(rows, device="cuda"))
    if case["kind"] == "decode":
        return [None, logits]
    if case["kind"] == "generate":
        return [None, logits[0]]
    steps = torch.tensor(step_of)
    return [logits[(steps == k).nonzero()[:, 0].cuda()] for k in range(int(steps.max()) + 1)]
