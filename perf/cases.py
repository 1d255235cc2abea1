"""The work a program has this framework do, as cases that can be timed and compared: prompts through ``Engine.step``, whole
requests through ``Engine.generate``, and batches decoded step by step through ``Engine.session``.

Models have the layer sizes of the repository's own configurations: Llama 3.2 1B and 3B, Llama 3.1 8B (eight of its 32 layers), the
tiny Llama of the tests, and Zirivik and Saluzen at width 2,048 as ``bench.py --compare`` builds them (Zirivik with dense
feed-forwards: a choice between experts near a tie changes a row by more than any rounding does).  Weights are random, made with
torch: every matrix ~ N(0, 0.81 / inputs), the ones that write the residual stream divided by the root of their number, and an
embedding strong enough that the most likely token stands out as it does in a trained model (it is the token itself), so that what
is generated does not hang on the last bit of a logit.

``prepare`` keeps the loaded engine of the model used last, as a serving program does; the tokens come from the seed.
"""
from __future__ import annotations

import gc
import json
import math
import random
import zlib

import torch

from fastgguf_b200 import Engine, SamplingParams, StepEntry
from fastgguf_b200.registry import config_from_dict
from fastgguf_b200.weights import expected_tensors

LLAMA3_ROPE = {"rope_type": "llama3", "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}


def _llama(width, layers, heads, kv_heads, head_dim, ff, vocab, tied, factor, positions, eps=1e-5, theta=500000.0):
    return {"architectures": ["LlamaForCausalLM"], "hidden_size": width, "num_hidden_layers": layers, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "head_dim": head_dim, "intermediate_size": ff, "vocab_size": vocab, "rms_norm_eps": eps,
            "rope_theta": theta, "rope_scaling": dict(LLAMA3_ROPE, factor=factor) if factor else None,
            "tie_word_embeddings": tied, "max_position_embeddings": positions, "bos_token_id": 1, "eos_token_id": 2}


def _zirivik():
    E = 2048
    ret = {"heads": 16, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - 6 * h / 15) for h in range(16)],
           "rot": {"base": 1000000.0, "dims": 64}}
    att = {"heads": 32, "kv_heads": 8, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 1024, "keep_first": 4}}
    dense = {"kind": "dense", "ff": 8192}
    layers = []
    for _ in range(2):
        at = len(layers) + 2
        layers += [{"type": "retention", "mixer": ret, "mlp": dense}, {"type": "retention", "mixer": ret, "mlp": dense},
                   {"type": "attention", "mixer": att, "mlp": dense}, {"type": "attention", "mixer": dict(att, kv_from=at), "mlp": dense}]
    return {"architecture": "Zirivik", "vocab": 32768, "width": E, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
            "logit_softcap": 30.0, "layers": layers}


def _saluzen():
    E, hd = 2048, 64
    lat = {"heads": 32, "dim": 64, "rot_dim": 64, "vdim": hd, "kv_rank": 512, "q_rank": E * 3 // 4, "scale": 128 ** -0.5,
           "rot": {"base": 10000.0, "dims": 64}}
    left = {"heads": 32, "kv_heads": 8, "dim": hd, "vdim": hd, "scale": hd ** -0.5}
    causal = dict(left, rot={"base": 500000.0, "dims": hd // 2, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}})
    chunked = dict(left, rot={"base": 1000000.0, "dims": hd // 2}, mask={"size": 1024})
    ssm = {"heads": E // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
    delta = {"heads": E // 128, "kv_heads": E // 256, "dim": 128, "vdim": 128, "conv": 4}
    dense = {"kind": "dense", "ff": 8192}
    layers = []
    for _ in range(2):
        at = len(layers)
        layers += [{"type": "latent_attention", "mixer": lat, "mlp": dense}, {"type": "latent_attention", "mixer": dict(lat, kv_from=at), "mlp": dense},
                   {"type": "parallel", "mixer": {"left": causal, "right": ssm}, "mlp": dense},
                   {"type": "parallel_2", "mixer": {"left": chunked, "right": delta, "left_scale": 0.7, "right_scale": 0.6}, "mlp": dense}]
    return {"architecture": "Saluzen", "vocab": 32768, "width": E, "norm": {"eps": 1e-6}, "layers": layers}


MODELS = {
    "tiny": _llama(64, 2, 4, 2, 16, 192, 256, True, None, 128, theta=10000.0),
    "1b": _llama(2048, 16, 32, 8, 64, 8192, 128256, True, 32.0, 131072),
    "3b": _llama(3072, 28, 24, 8, 128, 8192, 128256, True, 32.0, 131072),
    "8b": _llama(4096, 8, 32, 8, 128, 14336, 128256, False, 8.0, 131072),
    "zirivik": _zirivik(),
    "saluzen": _saluzen(),
}
#: model -> (sequence slots, tokens the cache holds, longest sequence)
ROOM = {"tiny": (4, 512, 128), "1b": (64, 98304, 4096), "3b": (8, 32768, 4096), "8b": (8, 65536, 8192),
        "zirivik": (16, 32768, 4096), "saluzen": (16, 32768, 4096)}
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# ------------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest call: the tiny float32 Llama of the tests, three prompts of 5, 9 and 1 tokens, eight greedy tokens each, then
        # the logits of every position (what trace replay writes): launches and host work, no arithmetic to speak of
        {"name": "tiny-f32-generate", "kind": "generate", "model": "tiny", "dtype": "float32", "lengths": "5,9,1", "steps": 8, "all": True},
        # the benchmark's prompt: time to the first token of one request of 2,048 tokens
        {"name": "1b-prompt-2048", "kind": "prompt", "model": "1b", "dtype": "bfloat16", "lengths": "2048"},
        # a few short requests that arrive together, odd lengths
        {"name": "1b-prompts-short", "kind": "prompt", "model": "1b", "dtype": "bfloat16", "lengths": "197,61,333"},
        # one user waiting: a request of 512 tokens answered with 64, greedy, and the log-probabilities of the answer
        {"name": "1b-generate-1", "kind": "generate", "model": "1b", "dtype": "bfloat16", "lengths": "512", "steps": 64, "all": False},
        # the headline: eight sequences of unequal lengths decoded together, greedy
        {"name": "1b-decode-8", "kind": "decode", "model": "1b", "dtype": "bfloat16", "lengths": "128,1024,301,777,530,211,645,958", "steps": 64, "temp": 0.0},
        # a full server: 64 sequences, the default sampler (temperature 1, top-k 64, top-p 0.95)
        {"name": "1b-decode-64", "kind": "decode", "model": "1b", "dtype": "bfloat16", "batch": 64, "shortest": 128, "longest": 512, "steps": 64, "temp": 1.0},
        # the true 32-bit path: a prompt, and a batch of eight decoded
        {"name": "1b-f32-prompt-2048", "kind": "prompt", "model": "1b", "dtype": "float32", "lengths": "2048"},
        {"name": "1b-f32-decode-8", "kind": "decode", "model": "1b", "dtype": "float32", "lengths": "33,128,64,100,17,81,57,120", "steps": 32, "temp": 0.0},
        # the 3B shapes with head size 128: prompts from 64 to 2,048 tokens, decoded together
        {"name": "3b-decode-8", "kind": "decode", "model": "3b", "dtype": "bfloat16", "lengths": "64,2048,333,1200,96,1777,640,411", "steps": 48, "temp": 0.0},
        # a full context of the 8B shapes
        {"name": "8b-prompt-8192", "kind": "prompt", "model": "8b", "dtype": "bfloat16", "lengths": "8191"},
        # the other architectures: recurrent layers beside windowed attention, pairs of mixers and latent attention
        {"name": "zirivik-decode-8", "kind": "decode", "model": "zirivik", "dtype": "bfloat16", "lengths": "256,1024,611,333,800,512,419,970", "steps": 32, "temp": 0.0},
        {"name": "saluzen-decode-8", "kind": "decode", "model": "saluzen", "dtype": "bfloat16", "lengths": "256,1024,611,333,800,512,419,970", "steps": 32, "temp": 0.0},
    ]


def _spread(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    model, dtype = rng.choice([("1b", "bfloat16"), ("1b", "bfloat16"), ("1b", "bfloat16"), ("1b", "float32"), ("1b", "float32"), ("3b", "bfloat16"),
                               ("8b", "bfloat16"), ("zirivik", "bfloat16"), ("saluzen", "bfloat16"), ("tiny", rng.choice(["float32", "bfloat16"]))])
    if model == "tiny":
        return {"kind": "generate", "model": model, "dtype": "float32", "lengths": ",".join(str(rng.randint(1, 60)) for _ in range(rng.randint(1, 4))),
                "steps": rng.randint(2, 24), "all": True}
    slots, _, longest = ROOM[model]
    kind = rng.choice(["prompt", "decode", "decode", "generate"] if model == "1b" else ["prompt", "decode"])
    most = 2048 if dtype == "float32" else 8000 if model == "8b" else 6000
    if kind == "prompt":
        total, n = _spread(rng, 24, most), rng.choice([1, 1, 2, 3, 5])
        parts = [max(1, int(total / n * rng.uniform(0.4, 1.0))) for _ in range(n)]
        return {"kind": kind, "model": model, "dtype": dtype, "lengths": ",".join(str(min(p, longest)) for p in parts)}
    if kind == "generate":
        return {"kind": kind, "model": model, "dtype": dtype, "lengths": str(_spread(rng, 16, 1024)), "steps": rng.randint(8, 48), "all": False}
    batch = _spread(rng, 1, 16 if dtype == "float32" else slots)
    top = max(32, min(1500, (1000 if dtype == "float32" else 12000) // batch))
    return {"kind": kind, "model": model, "dtype": dtype, "batch": batch, "shortest": max(8, top // rng.randint(2, 8)), "longest": top,
            "steps": rng.randint(12, 40 if dtype == "bfloat16" else 24), "temp": rng.choice([0.0, 1.0])}


def _lengths(case):
    if "lengths" in case:
        return [int(n) for n in case["lengths"].split(",")]
    rng = random.Random(case["batch"] * 7919 + case["longest"])
    return [rng.randint(case["shortest"], case["longest"]) for _ in range(case["batch"])]


def _prompts(case, seed):
    rng = random.Random(seed)
    cfg = MODELS[case["model"]]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    return [[rng.randrange(3, vocab) for _ in range(n)] for n in _lengths(case)]


# ------------------------------------------------------------------------------ weights and engines
def _weights(model, dtype):
    """Checkpoint name -> a maker of its tensor on the GPU, in the type it is stored in."""
    cfg = MODELS[model]
    decls = expected_tensors(config_from_dict(cfg))
    layers = cfg.get("num_hidden_layers") or len(cfg["layers"])
    llama = "architectures" in cfg

    def make(name):
        d = decls[name if not (name == "head" and model == "saluzen") else "embed"]
        seeded = "embed" if name == "head" or name == "lm_head.weight" else "embed" if "embed" in name else name
        g = torch.Generator(device="cuda").manual_seed(zlib.crc32((model + ":" + seeded).encode()))
        shape = tuple(d["shape"])
        z = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
        if seeded == "embed":
            t = (0.15 if llama else 0.06) * z                # the head's rows too: a token's own logit is the largest
        elif name.endswith(("norm1b", "norm2b")):            # what a sublayer adds is small beside the stream, as after training
            t = 0.06 * (1.0 + d["std"] * z) - (1.0 if model == "zirivik" else 0.0)
        elif d["init"] == "one_plus_normal":
            t = 1.0 + d["std"] * z
        elif len(shape) == 2 and "conv" not in name:
            t = z * (0.9 / math.sqrt(shape[1]))
            if llama and name.endswith(("o_proj.weight", "down_proj.weight")):
                t = t / math.sqrt(2.0 * layers)
        else:
            t = d["std"] * z
        return t.to(DTYPES[dtype])

    return decls, make


_loaded = {}


def _engine(model, dtype):
    key = (model, dtype)
    if key not in _loaded:
        _loaded.clear()
        gc.collect()
        decls, make = _weights(model, dtype)
        tensors = {name: make(name).cpu() for name in decls}
        torch.cuda.empty_cache()
        slots, tokens, longest = ROOM[model]
        _loaded[key] = Engine.from_tensors(config_from_dict(MODELS[model]), tensors, dtype=dtype, max_tokens=tokens, max_batch=slots, max_seq_len=longest)
    return _loaded[key]


def prepare(case, seed):
    return {"engine": _engine(case["model"], case["dtype"]), "prompts": _prompts(case, seed), "kind": case["kind"], "steps": case.get("steps", 0),
            "all": case.get("all", False), "sampling": SamplingParams(temp=case.get("temp", 0.0), top_k=64, top_p=0.95, seed=7)}


# ------------------------------------------------------------------------------ one pass
def _score(engine, sequences, want_from):
    """Logits of every sequence's rows from want_from on: one step over all of them."""
    slots = [engine.acquire() for _ in sequences]
    try:
        return engine.step([StepEntry(s, t, range(a, len(t))) for s, t, a in zip(slots, sequences, want_from)])
    finally:
        for s in slots:
            engine.release(s)


def run(state):
    engine, prompts = state["engine"], state["prompts"]
    if state["kind"] == "prompt":
        return _score(engine, prompts, [len(p) - 1 for p in prompts])
    if state["kind"] == "generate":
        done = engine.generate(prompts, temp=0.0, max_tokens=state["steps"], ignore_eos=True)
        whole = [p + c.tokens for p, c in zip(prompts, done)]
        logits = _score(engine, whole, [0 if state["all"] else len(p) - 1 for p in prompts])
        return {"tokens": torch.tensor([c.tokens for c in done]), "logits": logits}
    session = engine.session(prompts, state["sampling"])
    try:
        live = range(len(prompts))
        for _ in range(state["steps"]):
            session.advance(live)
        return engine.step([StepEntry(s, [p[-1]], [0]) for s, p in zip(session.slots, prompts)])
    finally:
        session.close()


# ------------------------------------------------------------------------------ what a pass cannot do without
def _layer_weights(model):
    """(numbers of the matrices every row meets, numbers of the head)."""
    cfg = MODELS[model]
    decls = expected_tensors(config_from_dict(cfg))
    head = (cfg.get("vocab_size") or cfg["vocab"]) * (cfg.get("hidden_size") or cfg["width"])
    body = sum(math.prod(d["shape"]) for n, d in decls.items() if "embed" not in n and n not in ("head", "lm_head.weight") and len(d["shape"]) > 1)
    return body, head


def _attention_costs(model):
    """[(flops a (row, key) pair, bytes-numbers a cached key, most keys a row sees)] and the numbers of a sequence's recurrent state."""
    cfg = MODELS[model]
    if "architectures" in cfg:
        q = cfg["num_attention_heads"] * cfg["head_dim"]
        kv = cfg["num_key_value_heads"] * cfg["head_dim"]
        return [(4 * q, 2 * kv, 1 << 30)] * cfg["num_hidden_layers"], 0
    out, state = [], 0
    for layer in cfg["layers"]:
        m = layer["mixer"]
        sides = [m] if "left" not in m else [m["left"], m["right"]]
        for s in sides:
            if "kv_rank" in s:
                out.append((2 * s["heads"] * (s["dim"] + s["rot_dim"] + s["vdim"]), s["kv_rank"] + s["rot_dim"], 1 << 30))
            elif "state" in s:
                state += s["heads"] * s["vdim"] * s["state"]
            elif "scale" in s:
                size = s["mask"]["size"] if s.get("mask") else 1 << 30
                out.append((2 * s["heads"] * (s["dim"] + s["vdim"]), s["kv_heads"] * (s["dim"] + s["vdim"]), size))
            else:
                state += s["heads"] * s["dim"] * s["vdim"]
    return out, state


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    body, head = _layer_weights(case["model"])
    att, state = _attention_costs(case["model"])
    cfg = MODELS[case["model"]]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    bytes_ = flops = 0.0

    def step(starts, news, want):
        nonlocal bytes_, flops
        rows = sum(news)
        bytes_ += size * (body + head) + 4.0 * want * vocab
        flops += 2.0 * rows * body + 2.0 * want * head + 6.0 * rows * state
        for f, numbers, most in att:
            for a, n in zip(starts, news):
                seen = sum(min(most, a + i + 1) for i in ((0,) if n == 1 else range(n)))
                flops += f * seen
                bytes_ += size * numbers * (min(most, a) + n)
        bytes_ += 4.0 * 2 * state * len(news)

    lengths = _lengths(case)
    zero = [0] * len(lengths)
    step(zero, lengths, len(lengths))
    if case["kind"] == "prompt":
        return {"bytes": bytes_, "flops": flops}
    steps = case["steps"] - 1 if case["kind"] == "generate" else case["steps"] + 1
    for s in range(steps):
        step([n + s for n in lengths], [1] * len(lengths), len(lengths))
    if case["kind"] == "generate":
        whole = [n + case["steps"] for n in lengths]
        step(zero, whole, sum(whole) if case["all"] else len(lengths) * (case["steps"] + 1))
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5, "max": 3e-4, "differ": 0.0}      # seen: up to 4e-6 from the float64 result
    return {"rel": 0.03, "max": 0.5, "differ": 0.0}             # seen: 6e-3 to 1e-2 from the float64 result


# ------------------------------------------------------------------------------ the same in 64 bits
F64 = torch.float64


class _Plain:
    """The models in float64, written from their equations: rows of all sequences side by side, mixers sequence by sequence."""

    def __init__(self, case):
        self.cfg = MODELS[case["model"]]
        self.decls, self.make = _weights(case["model"], case["dtype"])
        self.kept = {}

    def w(self, name):
        return self.make(name).to(F64)

    @staticmethod
    def norm(x, w, eps):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w

    @staticmethod
    def frequencies(base, dims, sc=None):
        f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64) / dims)
        if sc:
            factor, low, high = sc["factor"], sc.get("low", sc.get("low_freq_factor")), sc.get("high", sc.get("high_freq_factor"))
            orig = sc.get("original", sc.get("original_max_position_embeddings"))
            wave = 2.0 * math.pi / f
            blend = (orig / wave - low) / (high - low)
            mid = (1.0 - blend) * f / factor + blend * f
            f = torch.where(wave > orig / low, f / factor, torch.where(wave < orig / high, f, mid))
        return f.cuda()

    @staticmethod
    def rotate(x, f, adjacent=False):
        """x [T, heads, d] turned by position * f, pairs (i, i + n) or (2i, 2i + 1) of its first 2 n numbers."""
        n, out = len(f), x.clone()
        ang = torch.arange(x.shape[0], dtype=F64, device="cuda")[:, None, None] * f
        c, s = torch.cos(ang), torch.sin(ang)
        one, two = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if adjacent else (slice(0, n), slice(n, 2 * n))
        out[..., one], out[..., two] = x[..., one] * c - x[..., two] * s, x[..., two] * c + x[..., one] * s
        return out

    @staticmethod
    def attend(q, k, v, scale, size=None, keep=0, chunk=None, sink=None):
        """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv]; a few heads at a time."""
        T, H, G = q.shape[0], q.shape[1], k.shape[1]
        i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
        seen = j <= i
        if size:
            seen = seen & ((i - j < size) | (j < keep))
        if chunk:
            seen = seen & (i // chunk == j // chunk)
        out = torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
        for h in range(H):
            g = h // (H // G)
            s = (q[:, h] @ k[:, g].T).mul_(scale).masked_fill_(~seen, -math.inf)
            m = s.max(-1, keepdim=True).values
            if sink is not None:
                m = torch.clamp(m, min=float(sink[h]))
            e = torch.exp_(s.sub_(m))
            z = e.sum(-1, keepdim=True)
            if sink is not None:
                z = z + torch.exp(sink[h] - m)
            out[:, h] = (e @ v[:, g]) / z
        return out

    @staticmethod
    def conv(u, w, bias=None):
        T, taps = u.shape[0], w.shape[1]
        u = torch.cat([torch.zeros(taps - 1, u.shape[1], dtype=F64, device="cuda"), u])
        y = sum(u[j:j + T] * w[:, j] for j in range(taps))
        return y if bias is None else y + bias

    # -------------------------------------------------------------- mixers: h is one sequence's normalised rows, W its weights by name
    def grouped(self, h, m, W):
        T, dims = h.shape[0], m["dim"]
        q, k, v = (h @ W["q"].T + W.get("q.b", 0.0), h @ W["k"].T + W.get("k.b", 0.0), h @ W["v"].T + W.get("v.b", 0.0))
        q, k, v = q.view(T, m["heads"], dims), k.view(T, m["kv_heads"], dims), v.view(T, m["kv_heads"], -1)
        if m.get("rot"):
            f = self.frequencies(m["rot"]["base"], m["rot"]["dims"], m["rot"].get("scaling"))
            q, k = self.rotate(q, f), self.rotate(k, f)
        return q, k, v

    def retention(self, h, m, W, eps):
        T, H, d = h.shape[0], m["heads"], m["dim"]
        q, k, v = (h @ W["q"].T).view(T, H, d), (h @ W["k"].T).view(T, H, d), (h @ W["v"].T).view(T, H, -1)
        f = self.frequencies(m["rot"]["base"], m["rot"]["dims"])
        q, k = self.rotate(q, f), self.rotate(k, f) * d ** -0.5
        decay = torch.tensor(m["decay"], dtype=F64, device="cuda")
        i = torch.arange(T, dtype=F64, device="cuda")
        o = torch.empty_like(v)
        for n in range(H):                                   # o_i = sum over j <= i of decay^(i - j) (q_i . k_j) v_j
            o[:, n] = ((q[:, n] @ k[:, n].T) * torch.tril(decay[n] ** (i[:, None] - i[None, :]).clamp(min=0.0))) @ v[:, n]
        o = self.norm(o, 1.0, eps).reshape(T, -1)
        return (o * torch.nn.functional.silu(h @ W["g"].T)) @ W["o"].T

    def state_space(self, h, m, W, eps):
        T, H, dv, N, G, R = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"], m["norm_groups"]
        silu, inner = torch.nn.functional.silu, m["heads"] * m["vdim"]
        u = h @ W["in"].T
        z, xbc, dt = u[:, :inner], u[:, inner:2 * inner + 2 * G * N], u[:, 2 * inner + 2 * G * N:]
        xbc = silu(self.conv(xbc, W["conv"], W["conv.b"]))
        x = xbc[:, :inner].view(T, H, dv)
        B, C = (xbc[:, inner + a * G * N:inner + (a + 1) * G * N].view(T, G, N).repeat_interleave(H // G, 1) for a in (0, 1))
        dt = torch.nn.functional.softplus(dt + W["dt_bias"].view(-1), threshold=30.0)
        log_a = torch.cumsum(-torch.exp(W["A_log"].view(-1)) * dt, 0)
        y = torch.empty(T, H, dv, dtype=F64, device="cuda")
        lower = torch.ones(T, T, dtype=torch.bool, device="cuda").tril()
        for n in range(H):                                   # y_i = sum over j <= i of a_(j+1) .. a_i dt_j (C_i . B_j) x_j
            fall = torch.exp((log_a[:, n, None] - log_a[None, :, n]).masked_fill(~lower, -math.inf))
            y[:, n] = ((C[:, n] @ B[:, n].T) * fall * dt[None, :, n]) @ x[:, n] + W["D"].view(-1)[n] * x[:, n]
        y = (y.reshape(T, inner) * silu(z)).view(T, R, inner // R)
        return (self.norm(y, 1.0, eps).reshape(T, inner) * W["norm"].view(-1)) @ W["o"].T

    def gated_delta(self, h, m, W, eps):
        T, H, G, d, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        silu = torch.nn.functional.silu
        q, k = (silu(self.conv(h @ W[n].T, W[n + ".conv"])).view(T, G, d) for n in "qk")
        v = silu(self.conv(h @ W["v"].T, W["v.conv"])).view(T, H, dv)
        q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(H // G, 1)
        k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
        beta = torch.sigmoid(h @ W["b"].T)
        g = torch.exp(-torch.exp(W["A_log"].view(-1)) * torch.nn.functional.softplus(h @ W["a"].T + W["dt_bias"].view(-1), threshold=30.0))
        S = torch.zeros(H, d, dv, dtype=F64, device="cuda")
        o = torch.empty(T, H, dv, dtype=F64, device="cuda")
        for t in range(T):
            S = S * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = self.norm(o, W["norm"].view(-1), eps) * silu(h @ W["g"].T).view(T, H, dv)
        return o.reshape(T, H * dv) @ W["o"].T

    def latent(self, h, m, W, eps, i, seq):
        T, r = h.shape[0], m["kv_rank"]
        f = self.frequencies(m["rot"]["base"], m["rot"]["dims"])
        if m.get("kv_from") is None:
            u = h @ W["dkv"].T
            self.kept[i, seq] = (self.norm(u[:, :r], W["dkv.norm"].view(-1), eps), self.rotate(u[:, None, r:], f, True))
        c, kr = self.kept[i if m.get("kv_from") is None else m["kv_from"], seq]
        q = (self.norm(h @ W["dq"].T, W["dq.norm"].view(-1), eps) @ W["uq"].T).view(T, m["heads"], -1)
        q = torch.cat([q[..., :m["dim"]], self.rotate(q[..., m["dim"]:], f, True)], -1)
        k = torch.cat([(c @ W["uk"].T).view(T, m["heads"], m["dim"]), kr.expand(T, m["heads"], m["rot_dim"])], -1)
        return self.attend(q, k, (c @ W["uv"].T).view(T, m["heads"], m["vdim"]), m["scale"]).reshape(T, -1) @ W["o"].T

    def mixer(self, h, i, layer, W, eps, seq):
        m, T = layer["mixer"], h.shape[0]
        side = lambda s: {n[len(s):]: t for n, t in W.items() if n.startswith(s)}  # noqa: E731
        if layer["type"] == "retention":
            return self.retention(h, m, W, eps)
        if layer["type"] == "latent_attention":
            return self.latent(h, m, W, eps, i, seq)
        if layer["type"] == "attention":
            if "kv_from" not in m:
                q, k, v = self.grouped(h, m, W)
                self.kept[i, seq] = (k, v)
            else:
                q, (k, v) = (h @ W["q"].T).view(T, m["heads"], -1), self.kept[m["kv_from"], seq]
            return self.attend(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"]).reshape(T, -1) @ W["o"].T
        L, R, ml = side("left."), side("right."), m["left"]
        one = layer["type"] == "parallel"
        q, k, v = self.grouped(h, ml, L)
        sink = torch.zeros(ml["heads"], dtype=F64, device="cuda") if one else L["sink"].view(-1)
        o = self.attend(q, k, v, ml["scale"], chunk=ml["mask"]["size"] if ml.get("mask") else None, sink=sink)
        g = torch.sigmoid(h @ L["g"].T)
        left = (o * (g.view(o.shape) if one else g.view(T, -1, 1))).reshape(T, -1) @ L["o"].T
        if one:
            right = self.state_space(h, m["right"], R, eps)
            return 0.5 * (self.norm(left, L["out"].view(-1), eps) + self.norm(right, R["out"].view(-1), eps))
        return m["left_scale"] * left + m["right_scale"] * self.gated_delta(h, m["right"], R, eps)

    # -------------------------------------------------------------- models
    def forward(self, sequences, want_from):
        at = [0]
        for t in sequences:
            at.append(at[-1] + len(t))
        tokens = torch.tensor([t for s in sequences for t in s], device="cuda")
        parts = [slice(a, b) for a, b in zip(at, at[1:])]
        want = torch.tensor([a + r for a, t, f in zip(at, sequences, want_from) for r in range(f, len(t))], device="cuda")
        x, head = self.llama(tokens, parts) if "architectures" in self.cfg else self.others(tokens, parts)
        x = x[want]
        out = torch.cat([x @ rows.to(F64).T for rows in head.split(16384)], -1)
        cap = self.cfg.get("logit_softcap")
        return cap * torch.tanh(out / cap) if cap else out

    def llama(self, tokens, parts):
        c = self.cfg
        eps, d, silu = c["rms_norm_eps"], c["head_dim"], torch.nn.functional.silu
        f = self.frequencies(c["rope_theta"], d, c["rope_scaling"])
        embed = self.make("model.embed_tokens.weight")
        x = embed[tokens].to(F64)
        for i in range(c["num_hidden_layers"]):
            w = lambda n: self.w("model.layers.%d.%s.weight" % (i, n))  # noqa: B023, E731
            h = self.norm(x, w("input_layernorm"), eps)
            q, k, v = (h @ w("self_attn.%s_proj" % n).T for n in "qkv")
            o = torch.empty_like(q)
            for p in parts:
                T = p.stop - p.start
                o[p] = self.attend(self.rotate(q[p].view(T, -1, d), f), self.rotate(k[p].view(T, -1, d), f), v[p].view(T, -1, d), d ** -0.5).reshape(T, -1)
            x = x + o @ w("self_attn.o_proj").T
            h = self.norm(x, w("post_attention_layernorm"), eps)
            for p in torch.arange(x.shape[0], device="cuda").split(16384):
                x[p] += (silu(h[p] @ w("mlp.gate_proj").T) * (h[p] @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
        return self.norm(x, self.w("model.norm.weight"), eps), embed if c["tie_word_embeddings"] else self.make("lm_head.weight")

    def others(self, tokens, parts):
        eps = self.cfg["norm"]["eps"]
        zirivik = self.cfg["architecture"] == "Zirivik"
        weight = lambda n: self.w(n).view(-1) + (1.0 if zirivik else 0.0)  # noqa: E731
        embed = self.make("embed")
        x = embed[tokens].to(F64)
        for i, layer in enumerate(self.cfg["layers"]):
            p = "l%d." % i
            W = {n[len(p) + 4:]: self.w(n) for n in self.decls if n.startswith(p + "mix.")}
            h = self.norm(x, weight(p + "norm1"), eps)
            y = torch.cat([self.mixer(h[s], i, layer, W, eps, n) for n, s in enumerate(parts)])
            x = x + self.norm(y, weight(p + "norm1b"), eps)
            h = self.norm(x, weight(p + "norm2"), eps)
            u = h @ self.w(p + "mlp.up").T
            u = torch.relu(u) ** 2 if zirivik else torch.nn.functional.silu(h @ self.w(p + "mlp.gate").T) * u
            x = x + self.norm(u @ self.w(p + "mlp.down").T, weight(p + "norm2b"), eps)
        return self.norm(x, weight("final.norm"), eps), embed if zirivik else self.make("head")


def exact(case, seed):
    prompts = _prompts(case, seed)
    last = [len(p) - 1 for p in prompts]
    steps = case.get("steps", 0)
    with torch.no_grad():
        plain = _Plain(case)
        if case["kind"] == "prompt":
            return plain.forward(prompts, last)
        if case["kind"] == "decode":
            # the tokens fed: the most likely one each time, which is the prompt's last token again, then that token once more
            return plain.forward([p + [p[-1]] * (steps + 1) for p in prompts], [n + steps + 1 for n in last])
        whole = [p + [p[-1]] * steps for p in prompts]       # a guess, put right token by token until it is what is chosen
        while True:
            logits = plain.forward(whole, last)
            best = logits.argmax(-1).view(len(prompts), steps + 1)[:, :steps].tolist()
            wrong = [next((k for k in range(steps) if best[s][k] != whole[s][len(p) + k]), None) for s, p in enumerate(prompts)]
            if all(k is None for k in wrong):
                break
            for s, k in enumerate(wrong):
                if k is not None:
                    whole[s][len(prompts[s]) + k:] = [best[s][k]] * (steps - k)
        if case["all"]:
            logits = plain.forward(whole, [0] * len(prompts))
        return {"tokens": None, "logits": logits}
