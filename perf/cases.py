"""What a user has this engine do, as cases that can be timed and checked one by one.

A case is a dict of plain values.  ``kind`` says which use it stands for:

* ``prompt``: whole prompts arrive together and run as one step (time to the first token);
* ``decode``: live requests get one token each, from a CUDA graph (the steady state of a long generation);
* ``generate``: short prompts arrive and a few tokens follow, then the requests end (a chat turn);
* ``mixed``: prompts beside requests that decode, in one step (continuous batching);
* ``sample``: rows of logits become token ids (the end of every step).

``model`` and ``size`` name a design and its layer sizes: Qwen3 at its published 0.6B and 8B layer sizes, the other
designs at widths of 1,024 and 4,096, each with a few layers (one of every kind the design has) and random weights.
The designs whose feed-forwards are chosen by a learned router are left out, or run with dense feed-forwards: there the
rounding of an activation alone may send a token to another expert, so two correct runs need not agree.
Token ids are given, not generated, so that every run sees the same tokens; the logits of every step are the result.

``exact`` is the same computation in 64 bits in plain torch, whole sequences at once.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from xinfer_b200.config import config_from_dict
from xinfer_b200.engine.runner import ModelRunner, StepInput
from xinfer_b200.models.decoder import model_weight_specs
from xinfer_b200.sampling import SamplingParams
from xinfer_b200.sampling.sampler import Sampler
from xinfer_b200.weights.random_init import RandomWeightStore

DEVICE = "cuda:0"
PAGE = 16
VOCAB = {"qwen3": 151936}      # the others: 32,000
LIFE = 1024                    # tokens a decoding request lives before another one takes its place
NEW_TOKENS = 16                # decoded tokens of a "generate" case

SIZES = {
    "0.6b": dict(hidden=1024, heads=16, kv_heads=8, dim=128, ff=3072),
    "8b": dict(hidden=4096, heads=32, kv_heads=8, dim=128, ff=12288),
    "1k": dict(hidden=1024, heads=16, kv_heads=8, dim=128, ff=3072, expert_ff=768, rank=256, rot=32),
    "4k": dict(hidden=4096, heads=32, kv_heads=8, dim=128, ff=12288, expert_ff=3072, rank=512, rot=64),
}


def listed():
    return [
        # one user, a small model: a step is launches and latency
        dict(name="qwen3-0.6b-decode-1", model="qwen3", size="0.6b", layers=28, dtype="bf16", kind="decode", requests=1, tokens=1024),
        # the headline workload: eight users at context 4,096, bound by weights and cache
        dict(name="qwen3-8b-decode-8", model="qwen3", size="8b", layers=8, dtype="bf16", kind="decode", requests=8, tokens=4096),
        # a chat turn of many users with prompts of uneven length
        dict(name="qwen3-0.6b-generate-32", model="qwen3", size="0.6b", layers=8, dtype="bf16", kind="generate", requests=32, tokens=97),
        # one prompt of the headline's length, bound by matrix products
        dict(name="qwen3-8b-prompt-2048", model="qwen3", size="8b", layers=4, dtype="bf16", kind="prompt", requests=1, tokens=2048),
        # continuous batching: three ragged prompts beside sixteen decoding requests
        dict(name="qwen3-0.6b-mixed", model="qwen3", size="0.6b", layers=8, dtype="bf16", kind="mixed", requests=3, tokens=777, live=16),
        # the float32 engine, as one runs it to check a model
        dict(name="qwen3-0.6b-f32-prompt", model="qwen3", size="0.6b", layers=2, dtype="f32", kind="prompt", requests=2, tokens=301),
        # sampling for a full batch
        dict(name="sample-64", model="qwen3", kind="sample", requests=64, top_k=20, top_p=0.95, temperature=0.6),
        # a long prompt of the design with talking heads beside a recurrence
        dict(name="tidarax-4k-prompt-2048", model="tidarax", size="4k", layers=4, dtype="bf16", kind="prompt", requests=1, tokens=2048),
        # its decode, at the small size
        dict(name="tidarax-1k-decode-8", model="tidarax", size="1k", layers=4, dtype="bf16", kind="decode", requests=8, tokens=2048),
        # ragged prompts of the design with latent attention
        dict(name="dufitar-4k-prompt-2", model="dufitar", size="4k", layers=4, dtype="bf16", kind="prompt", requests=2, tokens=1275),
        # ragged prompts of the design with state-space and delta-rule layers
        dict(name="gulipel-1k-prompt-3", model="gulipel", size="1k", layers=4, dtype="bf16", kind="prompt", requests=3, tokens=901),
        # decode over linear attention and two kinds of latent attention
        dict(name="napuzen-4k-decode-4", model="napuzen", size="4k", layers=4, dtype="bf16", kind="decode", requests=4, tokens=2000),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["prompt", "decode", "generate", "mixed", "sample"], [36, 30, 14, 10, 10])[0]
    if kind == "sample":
        return dict(model="qwen3", kind=kind, requests=_spread(rng, 1, 64), temperature=rng.choice([0.0, 0.6, 0.8, 1.0]),
                    top_k=rng.choice([0, 20, 50, 200]), top_p=rng.choice([1.0, 0.9, 0.95]))
    model = rng.choices(["qwen3", "tidarax", "dufitar", "gulipel", "napuzen"], [40, 15, 15, 15, 15])[0]
    dtype = "f32" if model == "qwen3" and kind in ("prompt", "generate") and rng.random() < 0.25 else "bf16"
    size = rng.choice(["0.6b", "8b"] if model == "qwen3" else ["1k", "4k"])
    layers = 4
    if dtype == "f32":
        size, layers = "0.6b", 2
    most = {"prompt": 256 if dtype == "f32" else 2048, "decode": 3000, "generate": 1024, "mixed": 1500}[kind]
    if kind == "generate" and dtype == "f32":
        most = 64
    requests = _spread(rng, 1, {"prompt": 8, "decode": 32, "generate": 32, "mixed": 4}[kind])
    if dtype == "f32":
        requests = min(requests, 4)
    if kind == "decode":
        tokens = _spread(rng, 1000, max(1000, min(most, 16000 // requests)))
    else:
        tokens = _spread(rng, 16, most)
        requests = max(1, min(requests, most // tokens))
    case = dict(model=model, size=size, layers=layers, dtype=dtype, kind=kind, requests=requests, tokens=tokens)
    if kind == "mixed":
        case["live"] = _spread(rng, 1, 24)
    return case


# ---- configurations: the layer sizes above in each design's own keys ------------------------------------------------
def _vocab(case):
    return VOCAB.get(case["model"], 32000)


def _longest(case):
    return (max(case["tokens"], 512) if case["kind"] == "mixed" else case["tokens"]) + LIFE + 64


def _config(case):
    z, n, vocab = SIZES[case["size"]], case["layers"], _vocab(case)
    d, H, G = z["dim"], z["heads"], z["kv_heads"]
    if case["model"] == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], vocab_size=vocab, hidden_size=z["hidden"], intermediate_size=z["ff"],
                    num_hidden_layers=n, num_attention_heads=H, num_key_value_heads=G, head_dim=d, rms_norm_eps=1e-6,
                    rope_theta=1000000.0, max_position_embeddings=40960, tie_word_embeddings=case["size"] == "0.6b",
                    sliding_window=None)
    dense = dict(kind="dense", ff=z["ff"])
    layers = []
    if case["model"] == "tidarax":
        left = dict(heads=H, kv_heads=G, dim=d, vdim=d, scale=d ** -0.5,
                    rot=dict(dims=d, base=500000.0, scaling=dict(factor=8.0, low=1.0, high=4.0, original=8192)))
        mixer = dict(left=left, left_scale=1.0, right=dict(width=z["hidden"]), right_scale=1.0)
        moe = dict(kind="moe", expert=dict(ff=z["expert_ff"]), router=dict(experts=8, top=2))
        layers = [dict(type="parallel", mixer=mixer, mlp=moe if i % 2 else dense) for i in range(n)]
        return dict(architecture="Tidarax", vocab=vocab, width=z["hidden"], norm=dict(eps=1e-6), layers=layers)
    if case["model"] == "dufitar":
        attn = dict(type="attention", mlp=dense, mixer=dict(
            heads=H, kv_heads=G, dim=d, vdim=d, scale=d ** -0.5, mask=dict(size=4096),
            rot=dict(dims=d // 2, base=1000000.0, scaling=dict(factor=8.0, original=8192, fast=16.0, slow=2.0))))
        for i in range(n):
            m = dict(heads=H, dim=d, rot_dim=z["rot"], vdim=d, kv_rank=z["rank"], scale=(d + z["rot"]) ** -0.5,
                     mask=dict(size=4096), rot=dict(dims=z["rot"], base=100000.0))
            if i % 4 == 3:
                m["kv_from"] = i - 2
            layers.append(dict(type="latent_attention", mixer=m, mlp=dense) if i % 2 else attn)
        return dict(architecture="Dufitar", vocab=vocab, width=z["hidden"], norm=dict(eps=1e-6), residual_mult=0.5,
                    embedding=dict(scale=2.0), layers=layers)
    if case["model"] == "gulipel":
        ss = 2 * z["hidden"] // 64
        ssm = dict(heads=ss, vdim=64, state=128, groups=max(1, ss // 16), conv=4, norm_groups=max(1, ss // 16))
        par = dict(left=dict(heads=H, kv_heads=G, dim=d, vdim=d, scale=d ** -0.5, q_temp=dict(coef=0.25, every=512)),
                   right=dict(heads=H, kv_heads=H, dim=d, vdim=d, conv=4, decay_rank=64, gate_rank=64))
        layers = [dict(type="parallel", mixer=par, mlp=dense) if i % 2 else
                  dict(type="mamba2_2" if i % 4 else "mamba2", mixer=ssm, mlp=dense) for i in range(n)]
        return dict(architecture="Gulipel", vocab=vocab, width=z["hidden"], norm=dict(eps=1e-6), max_positions=_longest(case),
                    logit_softcap=40.0, embedding=dict(scale=z["hidden"] ** 0.5, bigram=dict(buckets=100003, mul_prev=8191, mul_cur=31)),
                    token_side=dict(dim=64), layers=layers)
    if case["model"] == "napuzen":
        gla = dict(type="gla", mixer=dict(heads=H, dim=d, vdim=d, tau=8.0))
        rot = dict(dims=z["rot"], base=100000.0, scaling=dict(factor=4.0, original=8192, fast=16.0, slow=2.0))
        one = dict(type="latent_attention", mixer=dict(heads=H, dim=d, rot_dim=z["rot"], vdim=d, q_rank=3 * z["rank"],
                                                       kv_rank=z["rank"], scale=(d + z["rot"]) ** -0.5, rot=rot))
        two = dict(type="latent_attention_2", mixer=dict(heads=H, dim=d, vdim=d, kv_rank=z["rank"], scale=d ** -0.5, mask=dict(size=4096)))
        layers = [dict(gla if i % 2 == 0 else (one if i % 4 == 3 else two), mlp=dict(dense, limit=7.0)) for i in range(n)]
        return dict(architecture="Napuzen", vocab=vocab, width=z["hidden"], norm=dict(eps=1e-6), canon=dict(taps=4), logit_scale=0.8,
                    layers=layers)
    raise ValueError(case["model"])


# ---- what a program has in hand -------------------------------------------------------------------------------------
def _lengths(case):
    """Prompt lengths of the case's requests: the longest is ``tokens``, the others fall off unevenly."""
    return [max(1, case["tokens"] * (case["requests"] - i) // case["requests"] - (5 * i) % 7) for i in range(case["requests"])]


def _tokens(case, seed):
    """(prompts of the case, prompts of the live requests, decode tokens): seeded uniform token ids."""
    rng, vocab = np.random.default_rng(seed), _vocab(case)
    lens = [case["tokens"]] * case["requests"] if case["kind"] == "decode" else _lengths(case)
    live = [257 + 13 * (i % 11) for i in range(case.get("live", 0))]
    prompts = [rng.integers(0, vocab, size=n, dtype=np.int32) for n in lens]
    return prompts, [rng.integers(0, vocab, size=n, dtype=np.int32) for n in live], \
        rng.integers(0, vocab, size=(LIFE + 1, max(case["requests"], len(live))), dtype=np.int32)


class _Live:
    """Requests that decode: each takes the given tokens one by one, and starts anew from its prompt after ``LIFE`` of them."""

    def __init__(self, runner, prompts, tokens):
        self.runner, self.prompts, self.tokens = runner, prompts, tokens
        self.slots = []
        self.open()

    def open(self):
        for s in self.slots:
            self.runner.close_request(s)
        self.slots = [self.runner.open_request() for _ in self.prompts]
        self.at = 0
        for s, p in zip(self.slots, self.prompts):
            self.runner.step([StepInput(s, p, [])])

    def entries(self):
        if self.at == LIFE:
            self.open()
        row = self.tokens[self.at]
        self.at += 1
        return [StepInput(s, row[j:j + 1], (0,)) for j, s in enumerate(self.slots)]


def prepare(case, seed):
    if case["kind"] == "sample":
        g = torch.Generator(device=DEVICE)
        g.manual_seed(seed)
        n = case["requests"]
        params = SamplingParams(temperature=case["temperature"], top_k=case["top_k"] or None, top_p=case["top_p"])
        return dict(case=case, logits=torch.randn(n, _vocab(case), generator=g, device=DEVICE) * 3.0, params=[params] * n,
                    seeds=[seed + i for i in range(n)], sampler=Sampler(DEVICE, n))
    prompts, live, toks = _tokens(case, seed)
    longest = _longest(case)
    most = len(prompts) + len(live)
    runner = ModelRunner.random(_config(case), seed, dtype=case["dtype"], block_size=PAGE, device=DEVICE, max_num_seqs=most,
                                num_blocks=most * (longest // PAGE + 2), max_model_len=longest)
    state = dict(case=case, runner=runner, prompts=prompts, toks=toks)
    if case["kind"] == "decode":
        state["live"] = _Live(runner, prompts, toks)
        runner.step(state["live"].entries(), allow_graph=True)      # the loop is under way
    elif case["kind"] == "mixed":
        state["live"] = _Live(runner, live, toks)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sample":
        return state["sampler"].sample(state["logits"], state["params"], state["seeds"], [3] * case["requests"])
    runner = state["runner"]
    if kind == "decode":
        return runner.step(state["live"].entries(), allow_graph=True)
    slots = [runner.open_request() for _ in state["prompts"]]
    first = [StepInput(s, p, (len(p) - 1,)) for s, p in zip(slots, state["prompts"])]
    if kind == "mixed":
        first = state["live"].entries() + first
    logits = runner.step(first)
    if kind == "generate":
        logits = [logits.clone()]
        for i in range(NEW_TOKENS):
            row = state["toks"][i]
            logits.append(runner.step([StepInput(s, row[j:j + 1], (0,)) for j, s in enumerate(slots)], allow_graph=True).clone())
    for s in slots:
        runner.close_request(s)
    return logits


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "sample":
        n = case["requests"] * _vocab(case)
        return {"bytes": 4.0 * n, "flops": 4.0 * n}
    z, size = SIZES[case["size"]], 4 if case["dtype"] == "f32" else 2
    cfg = _config(case)
    entry, parsed = config_from_dict(cfg)
    tables = ("embed", "bigram", "pos", "side.embed", "table")
    read = mult = 0.0
    for s in model_weight_specs(entry.plan_of(parsed)):
        if s.name.split(".")[-1] in tables or "embed" in s.name or len(s.shape) < 2:
            continue
        if "lm_head" in s.name or s.name == "head":
            continue
        n = float(np.prod(s.concrete_shape()))
        read += n
        mult += n / 4 if ".mlp.e" in s.name else n     # two of eight experts per token
    head = float(z["hidden"] * _vocab(case))
    steps = [(_lengths(case) if case["kind"] != "decode" else [1] * case["requests"], 0 if case["kind"] != "decode" else case["tokens"])]
    if case["kind"] == "mixed":
        steps[0] = (steps[0][0] + [1] * case["live"], 0)
    total_bytes = total_flops = 0.0
    attn_layers = case["layers"] if case["model"] in ("qwen3", "tidarax", "dufitar") else case["layers"] / 2
    row = (z["rank"] + z["rot"]) if case["model"] == "napuzen" else 2 * z["kv_heads"] * z["dim"]
    if case["model"] == "dufitar":
        row = (row + z["rank"] + z["rot"]) / 2
    state = {"gulipel": z["heads"] * 128 * 128 + 2 * z["hidden"] * 128, "napuzen": z["heads"] * 128 * 128 * 1.0}.get(case["model"], 0) * case["layers"] / 2
    for counts, before in steps:
        T, R = float(sum(counts)), float(len(counts))
        pairs = sum(c * before + c * (c + 1) / 2.0 for c in counts)
        total_bytes += size * (read + head + attn_layers * row * (T + sum(before for _ in counts))) + 4 * R * _vocab(case) + 8 * R * state
        total_flops += 2 * T * mult + 2 * R * head + attn_layers * 4 * z["heads"] * z["dim"] * pairs + 8 * T * state
    if case["kind"] == "generate":
        R, k = float(case["requests"]), float(NEW_TOKENS)
        total_bytes += k * (size * (read + head + attn_layers * row * sum(_lengths(case))) + 4 * R * _vocab(case) + 8 * R * state)
        total_flops += k * R * (2 * (mult + head) + attn_layers * 4 * z["heads"] * z["dim"] * case["tokens"] / 2 + 8 * state)
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    # float32: 1e-6 away from 64 bits was seen over 2 layers of sums over 1,024 to 3,072 terms; bfloat16: 0.004 to 0.026
    # over 4 to 28 layers of activations of 8 bits, and two such runs differ by less than both of them
    if case["dtype"] == "f32":
        return {"rel": 4e-6, "max": 1e-4}
    return {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, scale, window=None, sink=None, mix=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv]: causal softmax attention; ``sink``: one more score per head without a
    value; ``mix``: scores mixed across heads before the softmax."""
    T, H, _ = q.shape
    k, v = (t.repeat_interleave(H // t.shape[1], 1).transpose(0, 1) for t in (k, v))
    pos = torch.arange(T, device=q.device)
    out = []
    for a in range(0, T, 256):
        s = q[a:a + 256].transpose(0, 1) @ k.transpose(1, 2) * scale
        if mix is not None:
            s = torch.einsum("hg,gij->hij", mix, s)
        far = pos[a:a + 256, None] - pos[None, :]
        s = s.masked_fill((far < 0) if window is None else (far < 0) | (far >= window), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, s.shape[1], 1)], -1)
        p = torch.softmax(s, -1)[..., :T]
        out.append((p @ v).transpose(0, 1))
    return torch.cat(out).reshape(T, -1)


def _rotate(x, freqs, magnitude, neighbours):
    """x [T, heads, d]: the first channels turn by position * frequency (float32, as rotary tables hold it)."""
    half = len(freqs)
    f = torch.tensor(freqs, dtype=torch.float64).float().to(x.device)
    a = (torch.arange(x.shape[0], device=x.device).float()[:, None] * f).double()
    c, s = torch.cos(a)[:, None] * magnitude, torch.sin(a)[:, None] * magnitude
    out = x.clone()
    one, two = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if neighbours else (slice(0, half), slice(half, 2 * half))
    out[..., one] = x[..., one] * c - x[..., two] * s
    out[..., two] = x[..., two] * c + x[..., one] * s
    return out


def _frequencies(rot):
    """(frequencies, magnitude) of a rotary description: plain, slowed for long wavelengths, or YaRN."""
    dims, base, sc = rot["dims"], rot["base"], rot.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not sc:
        return f, 1.0
    if "low" in sc:
        out = []
        for x in f:
            wave = 2.0 * math.pi / x
            s = min(max((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"]), 0.0), 1.0)
            out.append((1.0 - s) * x / sc["factor"] + s * x)
        return out, 1.0

    def at(turns):
        return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [x / sc["factor"] * r + x * (1.0 - r) for x, r in zip(f, ramp)], 0.1 * math.log(sc["factor"]) + 1.0


def _conv(x, taps, bias=None):
    n, K = x.shape[0], taps.shape[1]
    padded = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    y = sum(padded[j:j + n] * taps[:, j] for j in range(K))
    return y if bias is None else y + bias


def _qwen3(cfg, w, ids):
    T, eps, H, G, d = len(ids), cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    f32 = [float(np.float32(1.0) / np.float32(cfg["rope_theta"] ** (2.0 * j / d))) for j in range(d // 2)]
    x = w["model.embed_tokens.weight"][ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a, m = p + "self_attn.", p + "mlp."
        h = _unit(x, eps) * w[p + "input_layernorm.weight"]
        q = _unit((h @ w[a + "q_proj.weight"].T).view(T, H, d), eps) * w[a + "q_norm.weight"]
        k = _unit((h @ w[a + "k_proj.weight"].T).view(T, G, d), eps) * w[a + "k_norm.weight"]
        v = (h @ w[a + "v_proj.weight"].T).view(T, G, d)
        q, k = _rotate(q, f32, 1.0, False), _rotate(k, f32, 1.0, False)
        x = x + _attend(q, k, v, 1.0 / math.sqrt(d)) @ w[a + "o_proj.weight"].T
        h = _unit(x, eps) * w[p + "post_attention_layernorm.weight"]
        x = x + (_silu(h @ w[m + "gate_proj.weight"].T) * (h @ w[m + "up_proj.weight"].T)) @ w[m + "down_proj.weight"].T
    head = w["model.embed_tokens.weight"] if cfg["tie_word_embeddings"] else w["lm_head.weight"]
    return (_unit(x, eps) * w["model.norm.weight"]), head, None


def _tidarax(cfg, w, ids):
    T, eps = len(ids), cfg["norm"]["eps"]
    x = w["embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        a, b = m["left"], m["right"]
        l, r = p + "mix.left.", p + "mix.right."
        h = _unit(x, eps) * (1.0 + w[p + "norm1"])
        f, mag = _frequencies(a["rot"])
        q, k = (_unit(_rotate((h @ w[l + n].T).view(T, -1, a["dim"]), f, mag, False), eps) for n in ("q", "k"))
        v = (h @ w[l + "v"].T).view(T, -1, a["vdim"])
        o = _attend(q, k, v, a["scale"], sink=q.new_zeros(a["heads"]), mix=w[l + "talk"])
        z = torch.sigmoid(h @ w[r + "z"].T + w[r + "z.b"])
        u = h @ w[r + "x"].T + w[r + "x.b"]
        u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u)) * z
        s, states = x.new_zeros(b["width"]), []
        for t in range(T):
            s = (1.0 - z[t]) * s + u[t]
            states.append(s)
        x = x + m["left_scale"] * (o @ w[l + "o"].T) + m["right_scale"] * ((torch.stack(states) * _silu(h @ w[r + "g"].T)) @ w[r + "o"].T)
        h, g = _unit(x, eps) * (1.0 + w[p + "norm2"]), p + "mlp."
        if layer["mlp"]["kind"] == "dense":
            y, c = h @ w[g + "up"].T, w[g + "act"]
            x = x + (c[0] * _unit(y, eps) + c[1] * _unit(y ** 2, eps) + c[2] * _unit(y ** 3, eps) + c[3]) @ w[g + "down"].T
        else:
            chosen = w[g + "table"][ids].long()
            add = torch.zeros_like(x)
            for e in range(layer["mlp"]["router"]["experts"]):
                rows = (chosen == e).any(1).nonzero()[:, 0]
                q = f"{g}e{e}."
                add[rows] += (_silu(h[rows] @ w[q + "gate"].T) * (h[rows] @ w[q + "up"].T)) @ w[q + "down"].T / chosen.shape[1]
            x = x + add
    return _unit(x, eps) * (1.0 + w["final.norm"]), w["head"], None


def _dufitar(cfg, w, ids):
    T, eps, rows = len(ids), cfg["norm"]["eps"], {}

    def norm(x, n):
        return torch.tanh(w[n + ".alpha"] * x) * w[n] + w[n + ".b"]
    x = w["embed"][ids] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p, m, mult = f"l{i}.", layer["mixer"], cfg["residual_mult"]
        a, H, d = p + "mix.", m["heads"], m["dim"]
        h = norm(x, p + "norm1")
        f, mag = _frequencies(m["rot"])
        if layer["type"] == "attention":
            q, k = (_rotate((h @ w[a + n].T).view(T, -1, d), f, mag, True) for n in ("q", "k"))
            o = _attend(q, k, (h @ w[a + "v"].T).view(T, -1, m["vdim"]), m["scale"], m["mask"]["size"])
        else:
            src = m.get("kv_from", i)
            if src == i:
                c = h @ w[a + "dkv"].T
                rows[i] = (_unit(c[:, :m["kv_rank"]], eps) * w[a + "dkv.norm"], _rotate(c[:, None, m["kv_rank"]:], f, mag, True))
            c, kr = rows[src]
            q = (h @ w[a + "q"].T).view(T, H, -1)
            q = torch.cat([q[..., :d], _rotate(q[..., d:], f, mag, True)], -1)
            k = torch.cat([(c @ w[a + "uk"].T).view(T, H, d), kr.expand(T, H, -1)], -1)
            o = _attend(q, k, (c @ w[a + "uv"].T).view(T, H, -1), m["scale"], m["mask"]["size"], sink=w[a + "sink"])
            o = o * torch.sigmoid(h @ w[a + "g"].T)
        x = x + mult * norm(o @ w[a + "o"].T, p + "norm1b")
        h, g = norm(x, p + "norm2"), p + "mlp."
        x = x + mult * norm((F.gelu(h @ w[g + "gate"].T, approximate="tanh") * (h @ w[g + "up"].T)) @ w[g + "down"].T, p + "norm2b")
    return norm(x, "final.norm"), w["embed"], None


def _gulipel(cfg, w, ids):
    n, eps, emb = len(ids), cfg["norm"]["eps"], cfg["embedding"]
    b = emb["bigram"]
    pair = (torch.cat([ids[:1], ids[:-1]]) * b["mul_prev"] + ids * b["mul_cur"]) % b["buckets"]
    pair[0] = b["buckets"]
    x = w["embed"][ids] * emb["scale"] + w["bigram"][pair]
    if "pos" in w:
        x = x + w["pos"][:n]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        h = _unit(x, eps) * w[p + "norm1"]
        if layer["type"] == "parallel":
            a, c, l, r = m["left"], m["right"], p + "mix.left.", p + "mix.right."
            H, d, dv = a["heads"], a["dim"], a["vdim"]
            q, k, v = ((h @ w[l + t].T + w[l + t + ".b"]).view(n, -1, d) for t in ("q", "k", "v"))
            steps = torch.div(torch.arange(n, device=x.device) + 1, a["q_temp"]["every"], rounding_mode="floor").double()
            q = _unit(q, eps) * w[l + "q.norm"] * (1.0 + a["q_temp"]["coef"] * torch.log(steps + 1.0))[:, None, None]
            o = _attend(q, _unit(k, eps) * w[l + "k.norm"], v, a["scale"]) * torch.sigmoid(h @ w[l + "g"].T)
            left = o @ w[l + "o"].T
            H, d, dv = c["heads"], c["dim"], c["vdim"]
            q, k, v = (_silu(_conv(h @ w[r + t].T, w[r + t + ".conv"])).view(n, -1, s) for t, s in (("q", d), ("k", d), ("v", dv)))
            q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
            k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            q, k = (t.repeat_interleave(H // t.shape[1], 1) for t in (q, k))
            beta = torch.sigmoid(h @ w[r + "b"].T)[..., None]
            decay = F.softplus(h @ w[r + "a1"].T @ w[r + "a2"].T + w[r + "dt_bias"]).view(n, H, d)
            decay = torch.exp(-torch.exp(w[r + "A_log"])[None, :, None] * decay)
            S, out = x.new_zeros(H, d, dv), []
            for t in range(n):
                S = S * decay[t][:, :, None]
                S = S + k[t][:, :, None] * (beta[t] * (v[t] - (k[t][:, None] @ S)[:, 0]))[:, None]
                out.append((q[t][:, None] @ S)[:, 0])
            o = _unit(torch.stack(out), eps) * w[r + "norm"] * torch.sigmoid(h @ w[r + "g1"].T @ w[r + "g2"].T).view(n, H, dv)
            right = o.reshape(n, -1) @ w[r + "o"].T
            y = 0.5 * (_unit(left, eps) * w[p + "mix.left.out"] + _unit(right, eps) * w[p + "mix.right.out"])
        else:
            r, H, P, N, G = p + "mix.", m["heads"], m["vdim"], m["state"], m["groups"]
            z, xbc, dt = (h @ w[r + "in"].T).split([H * P, H * P + 2 * G * N, H], -1)
            xs, B, C = _silu(_conv(xbc, w[r + "conv"], w[r + "conv.b"])).split([H * P, G * N, G * N], -1)
            xs, B, C = xs.view(n, H, P), *(t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
            dt = F.softplus(dt + w[r + "dt_bias"])
            keep = torch.exp(-torch.exp(w[r + "A_log"]) * dt)
            S, out = x.new_zeros(H, N, P), []
            for t in range(n):
                S = S * keep[t][:, None, None] + (dt[t][:, None] * B[t])[:, :, None] * xs[t][:, None]
                out.append((C[t][:, None] @ S)[:, 0])
            y = (torch.stack(out) + w[r + "D"][:, None] * xs).reshape(n, -1) * _silu(z)
            y = _unit(y.view(n, m["norm_groups"], -1), eps).reshape(n, -1) * w[r + "norm"] @ w[r + "o"].T
        x = x + _unit(y, eps) * w[p + "norm1b"] * w[p + "ls1"]
        h, g = _unit(x, eps) * w[p + "norm2"], p + "mlp."
        y = (_silu(h @ w[g + "gate"].T + w[g + "gate.b"]) * (h @ w[g + "up"].T + w[g + "up.b"])) @ w[g + "down"].T + w[g + "down.b"]
        x = x + _unit(y, eps) * w[p + "norm2b"] * w[p + "ls2"]
        dim, g = cfg["token_side"]["dim"], p + "side."
        y = (F.gelu(x @ w[g + "gate"].T, approximate="tanh") * w["side.embed"][ids, i * dim:(i + 1) * dim]) @ w[g + "proj"].T
        x = x + _unit(y, eps) * w[g + "norm"]
    return _unit(x, eps) * w["final.norm"], w["head"], lambda z: cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def _napuzen(cfg, w, ids):
    T, eps = len(ids), cfg["norm"]["eps"]
    x = w["embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        a, H, d, dv = p + "mix.", m["heads"], m["dim"], m["vdim"]
        h = x + _conv(x, w[p + "canon1"])
        if layer["type"] == "gla":
            q, k, v = ((h @ w[a + t].T).view(T, H, -1) for t in ("q", "k", "v"))
            keep = torch.sigmoid(h @ w[a + "a1"].T @ w[a + "a2"].T + w[a + "a2.b"]).view(T, H, d) ** (1.0 / m["tau"])
            S, out = x.new_zeros(H, d, dv), []
            for t in range(T):
                S = keep[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
                out.append((q[t][:, None] @ S)[:, 0])
            o = _unit(torch.stack(out) * d ** -0.5, eps) * w[a + "norm"]
            o = o.reshape(T, -1) * _silu(h @ w[a + "g"].T)
        else:
            r = m["kv_rank"]
            kv = h @ w[a + "dkv"].T
            c = _unit(kv[:, :r], eps) * w[a + "dkv.norm"]
            k, v = (c @ w[a + "uk"].T).view(T, H, d), (c @ w[a + "uv"].T).view(T, H, dv)
            if layer["type"] == "latent_attention":
                f, mag = _frequencies(m["rot"])
                q = ((_unit(h @ w[a + "dq"].T, eps) * w[a + "dq.norm"]) @ w[a + "uq"].T).view(T, H, -1)
                q = torch.cat([q[..., :d], _rotate(q[..., d:], f, mag, True)], -1)
                k = torch.cat([k, _rotate(kv[:, None, r:], f, mag, True).expand(T, H, -1)], -1)
                o = _attend(q, k, v, m["scale"])
            else:
                o = _attend((h @ w[a + "q"].T).view(T, H, d), k, v, m["scale"], m["mask"]["size"])
                o = (o.view(T, H, dv) * torch.sigmoid(h @ w[a + "g"].T)[:, :, None]).reshape(T, -1)
        x = x + _unit(o @ w[a + "o"].T, eps) * w[p + "norm1"]
        g, limit = p + "mlp.", layer["mlp"]["limit"]
        one, two = (x @ w[g + "gate"].T).clamp(max=limit), (x @ w[g + "up"].T).clamp(-limit, limit)
        x = x + _unit((one * torch.sigmoid(1.702 * one) * (two + 1.0)) @ w[g + "down"].T, eps) * w[p + "norm2"]
    return _unit(x, eps) * w["final.norm"], w["embed"], lambda z: z * cfg["logit_scale"]


_EXACT = {"qwen3": _qwen3, "tidarax": _tidarax, "dufitar": _dufitar, "gulipel": _gulipel, "napuzen": _napuzen}


def exact(case, seed):
    if case["kind"] == "sample":
        return None      # token ids
    cfg = _config(case)
    entry, parsed = config_from_dict(cfg)
    plan = entry.plan_of(parsed)
    specs = model_weight_specs(plan)
    store = RandomWeightStore(specs, seed, plan.init_std, plan.norm_init_std)
    dtype = torch.float32 if case["dtype"] == "f32" else torch.bfloat16
    w = {s.name: store.get(s.name, DEVICE, dtype) for s in specs}
    w = {n: t.double() if t.is_floating_point() else t for n, t in w.items()}
    prompts, live, toks = _tokens(case, seed)

    def logits(seq, last):
        """Logits of the last ``last`` positions of a sequence, [last, vocab]."""
        y, head, post = _EXACT[case["model"]](cfg, w, torch.from_numpy(np.concatenate(seq).astype(np.int64)).to(DEVICE))
        z = y[-last:] @ head.T
        return post(z) if post else z
    if case["kind"] == "decode":
        return torch.cat([logits([p, toks[:2, j]], 1) for j, p in enumerate(prompts)])
    if case["kind"] == "generate":
        per = torch.stack([logits([p, toks[:NEW_TOKENS, j]], NEW_TOKENS + 1) for j, p in enumerate(prompts)])
        return [per[:, i] for i in range(NEW_TOKENS + 1)]
    return torch.cat([logits([p, toks[:1, j]], 1) for j, p in enumerate(live)] + [logits([p], 1) for p in prompts])
