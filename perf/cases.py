"""The work that a user of this library has it do, as measurable cases.

A case is one batch of requests on a model that is already loaded, through ``Engine``'s public
calls.  Its ``kind`` says which part of a request's life one pass covers:

* ``prompt``: open the sequences, run all prompts as one step, read the logits behind each, close;
* ``decode``: ``steps`` single-token steps of sequences whose prompts lie in the cache (they keep
  growing from pass to pass and start anew when they have grown by a fixed length);
* ``serve``: open, prompts, ``steps`` single-token steps, close.

Every step draws a token for each sequence, as a serving loop does; the tokens that the next step
takes are given (as ``bin/trace_run`` gives them), because with random weights a drawn token hangs
on the last bits of 16-bit arithmetic and everything behind it with it.  For the same reason the drawn
tokens are outputs only where the arithmetic is 32-bit; the last step's logits depend on everything
that was cached and are outputs everywhere.  The steps before the last are read one behind, as
``Engine.generate`` reads them.

Sizes are those of the benchmark: Llama-3.2-1B layer sizes whole; 3B sizes with half their layers and 8B sizes with a
quarter of theirs (a layer more is the same work once more); the 2,048-wide comparison sizes of the other
decoders with dense feed-forwards (where experts are chosen, a rounding now and then turns a choice, and logits
cannot be compared), and the same Llama in 32-bit.  Weights are random, drawn by torch from
each tensor's name; one engine per model serves every case, as one loaded model serves all requests."""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

from libllm_b200.engine import Engine, SamplingParams, StepItem

ROPE3 = dict(rope_type="llama3", low_freq_factor=1.0, high_freq_factor=4.0, original_max_position_embeddings=8192)
LLAMA = dict(model_type="llama", rope_theta=500000.0, rms_norm_eps=1e-5, max_position_embeddings=131072, hidden_act="silu",
             num_attention_heads=32, num_key_value_heads=8)


def _sinezen():
    mixer = dict(heads=32, kv_heads=8, dim=64, vdim=64, scale=0.125, mask=dict(size=1024), rot=dict(base=500000.0, dims=64))
    layer = dict(type="attention", mixer=mixer, mlp=dict(kind="dense", ff=8192))
    return dict(architecture="Sinezen", vocab=32000, width=2048, norm=dict(eps=1e-5), layers=[layer] * 4, loop=dict(start=2, stop=4, times=3))


def _sesuzen():
    attention = dict(heads=32, kv_heads=8, dim=64, vdim=64, scale=0.125, mask=dict(size=1024, keep_first=4))
    mlp = dict(kind="dense", ff=8192)
    return dict(architecture="Sesuzen", vocab=32000, width=2048, max_positions=4096, norm=dict(eps=1e-5), canon=dict(taps=4),
                logit_softcap=30.0, loop=dict(start=0, stop=2, times=4),
                layers=[dict(type="general_delta", mixer=dict(heads=32, dim=64, rank=64), mlp=mlp),
                        dict(type="attention", mixer=attention, mlp=mlp)])


def _sobezen():
    rot = dict(dims=64, base=1e4)
    ramp = dict(dims=32, base=1e4, scaling=dict(factor=4.0, original=2048, fast=16.0, slow=2.0))
    mlp = dict(kind="dense", ff=8192, limit=7.0)
    latent = dict(heads=32, dim=64, rot_dim=32, vdim=64, kv_rank=512, q_rank=768, scale=96 ** -0.5, rot=ramp)
    layers = []
    for i in range(0, 8, 4):
        layers += [dict(type="channel_delta", mixer=dict(heads=32, kv_heads=8, dim=64, vdim=64, conv=4), mlp=mlp),
                   dict(type="attention", mixer=dict(heads=32, kv_heads=8, dim=64, vdim=64, scale=0.125, rot=rot), mlp=mlp),
                   dict(type="latent_attention", mixer=dict(latent), mlp=mlp),
                   dict(type="latent_attention", mixer=dict(latent, kv_from=i + 2), mlp=mlp)]
    return dict(architecture="Sobezen", vocab=32000, width=2048, norm=dict(eps=1e-5), embedding=dict(scale=1.0), logit_scale=1.0, layers=layers)


# model -> (configuration, type of the engine, tokens its cache holds, longest sequence, widest prompt step drawn)
MODELS = {
    "llama-1b": (dict(LLAMA, num_hidden_layers=16, hidden_size=2048, head_dim=64, intermediate_size=8192, vocab_size=128256,
                      rope_scaling=dict(ROPE3, factor=32.0), tie_word_embeddings=True), "bfloat16", 655360, 16384, 16384),
    "llama-3b-half": (dict(LLAMA, num_hidden_layers=14, hidden_size=3072, num_attention_heads=24, head_dim=128, intermediate_size=8192,
                           vocab_size=128256, rope_scaling=dict(ROPE3, factor=32.0), tie_word_embeddings=True), "bfloat16", 393216, 8192, 8192),
    "llama-8b-quarter": (dict(LLAMA, num_hidden_layers=8, hidden_size=4096, head_dim=128, intermediate_size=14336, vocab_size=128256,
                              rope_scaling=dict(ROPE3, factor=8.0), tie_word_embeddings=False), "bfloat16", 655360, 8192, 8192),
    "llama-2k-32bit": (dict(LLAMA, num_hidden_layers=8, hidden_size=2048, head_dim=64, intermediate_size=8192, vocab_size=32000,
                            rope_scaling=None, tie_word_embeddings=True), "float32", 32768, 4096, 384),
    "sinezen-2k": (_sinezen(), "bfloat16", 262144, 4096, 8192),
    "sesuzen-2k": (_sesuzen(), "bfloat16", 262144, 4096, 8192),
    "sobezen-2k": (_sobezen(), "bfloat16", 262144, 4096, 8192),
}


def _case(name, model, kind, batch, length, ragged=False, steps=0, sampled=False):
    c = dict(model=model, kind=kind, batch=batch, length=length, ragged=ragged, steps=steps, sampled=sampled)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a chat's short turn: the first token's latency, odd length, launches count
        _case("1b-prompt-37", "llama-1b", "prompt", 1, 37),
        # the benchmark's prompt
        _case("1b-prompt-2048", "llama-1b", "prompt", 1, 2048),
        # one user reading along: greedy, latency alone
        _case("1b-decode-b1", "llama-1b", "decode", 1, 1100, steps=16),
        # the benchmark's decode point, drawn with the reference's default sampling
        _case("1b-decode-b8", "llama-1b", "decode", 8, 2048, steps=16, sampled=True),
        # a loaded server: many sequences of unequal length
        _case("1b-decode-b64", "llama-1b", "decode", 64, 2048, True, steps=32, sampled=True),
        # unequal prompts and their first answers' tokens, heads of 128 channels
        _case("3b-serve-16", "llama-3b-half", "serve", 16, 2048, True, steps=16, sampled=True),
        # long documents in one batch
        _case("8b-prompt-4x4096", "llama-8b-quarter", "prompt", 4, 4096),
        # their answers
        _case("8b-decode-b32", "llama-8b-quarter", "decode", 32, 4096, steps=16, sampled=True),
        # the 32-bit engine, which one checks a checkpoint with: two short prompts, a few tokens
        _case("32bit-serve-2", "llama-2k-32bit", "serve", 2, 150, True, steps=6),
        # the other decoders: a prompt's whole life each
        _case("sinezen-serve-4", "sinezen-2k", "serve", 4, 2000, True, steps=12),
        _case("sesuzen-serve-2", "sesuzen-2k", "serve", 2, 2000, True, steps=12),
        _case("sobezen-serve-2", "sobezen-2k", "serve", 2, 2000, True, steps=12),
    ]


def draw(rng):
    model = rng.choice(["llama-1b"] * 6 + ["llama-3b-half"] * 2 + ["llama-8b-quarter"] * 2 + ["llama-2k-32bit", "sinezen-2k", "sesuzen-2k", "sobezen-2k"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["prompt", "decode", "serve"])
    widest = MODELS[model][4]
    small = model == "llama-2k-32bit"
    batch = log(1, 3 if small else 64 if kind == "decode" else 16)
    most = (8 if kind == "decode" else 1) * widest // batch
    length = log(16, max(17, min(most, 300 if small else 3000 if model.startswith("s") else 4096)))
    steps = 0 if kind == "prompt" else rng.randint(3, 6 if small else 24)
    return _case(None, model, kind, batch, length, batch > 1 and rng.random() < 0.6, steps, rng.random() < 0.5)


def lengths(case):
    """Prompt lengths: all alike, or spread evenly over [length / 16, length] in a mixed order."""
    n, top = case["batch"], case["length"]
    if not case["ragged"]:
        return [top] * n
    return [max(1, int(round(top * (1 - 15 / 16 * ((i * 0.6180339887498949) % 1.0))))) for i in range(n)]


# ---------------------------------------------------------------- weights
def _shapes(c):
    """name -> (shape, law) of every tensor; law: (mean, deviation)."""
    out = {}
    mat = lambda n, k, s=1.0: ([n, k], (0.0, s / math.sqrt(k)))  # noqa: E731
    vec = lambda n, mean=1.0, dev=0.1: ([n], (mean, dev))  # noqa: E731
    if c.get("model_type") == "llama":
        H, I, V, d = c["hidden_size"], c["intermediate_size"], c["vocab_size"], c["head_dim"]
        q, kv = c["num_attention_heads"] * d, c["num_key_value_heads"] * d
        out["model.embed_tokens.weight"] = ([V, H], (0.0, 0.02))
        out["model.norm.weight"] = vec(H)
        if not c["tie_word_embeddings"]:
            out["lm_head.weight"] = ([V, H], (0.0, 0.02))
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out.update({p + "input_layernorm.weight": vec(H), p + "post_attention_layernorm.weight": vec(H)})
            for n, a, b in (("self_attn.q_proj", q, H), ("self_attn.k_proj", kv, H), ("self_attn.v_proj", kv, H), ("self_attn.o_proj", H, q),
                            ("mlp.gate_proj", I, H), ("mlp.up_proj", I, H), ("mlp.down_proj", H, I)):
                out[p + n + ".weight"] = ([a, b], (0.0, 0.02))
        return out
    W, V = c["width"], c["vocab"]
    arch = c["architecture"]
    out["embed"] = ([V, W], (0.0, 1.0 if arch != "Sesuzen" else 1.0 / math.sqrt(W) * 4))
    out["final.norm"] = vec(W)
    if arch == "Sesuzen":
        out.update({"pos": ([c["max_positions"], W], (0.0, 0.05)), "final.norm.b": vec(W, 0.0)})
    else:
        out["head"] = mat(V, W)
    if arch == "Sinezen":
        out["loop.in"] = mat(W, 2 * W)
    for i, L in enumerate(c["layers"]):
        m, p, ff = L["mixer"], f"l{i}.", L["mlp"]["ff"]
        x = p + "mix."
        H, d = m["heads"], m["dim"]
        out[p + "norm1"] = vec(W)
        if arch == "Sinezen":
            G, dv = m["kv_heads"], m["vdim"]
            out.update({x + "q": mat(H * d, W), x + "k": mat(G * d, W), x + "v": mat(G * dv, W), x + "q.norm": vec(H * d), x + "k.norm": vec(G * d),
                        x + "g": mat(H, W), x + "o": mat(W, H * dv)})
            out.update({p + "mlp.gate": mat(ff, W), p + "mlp.up": mat(ff, W), p + "mlp.down": mat(W, ff)})
            continue
        out[p + "norm2"] = vec(W)
        if arch == "Sesuzen":
            out.update({p + "norm1.b": vec(W, 0.0), p + "norm2.b": vec(W, 0.0), p + "canon1": ([W, c["canon"]["taps"]], (0.0, 0.3))})
            if L["type"] == "attention":
                G, dv = m["kv_heads"], m["vdim"]
                out.update({x + "q": mat(H * d, W), x + "q.b": vec(H * d, 0.0), x + "k": mat(G * d, W), x + "k.b": vec(G * d, 0.0),
                            x + "v": mat(G * dv, W), x + "v.b": vec(G * dv, 0.0), x + "g": mat(H * dv, W), x + "o": mat(W, H * dv)})
            else:
                N, r = H * d, m["rank"]
                out.update({x + n: mat(N, W) for n in ("r", "k", "v", "g", "a")})
                out.update({x + "a.b": vec(N, 0.0, 0.5), x + "w1": mat(r, W), x + "w2": mat(N, r), x + "w0": vec(N, -2.0, 1.0), x + "norm": vec(N), x + "o": mat(W, N)})
            out.update({p + "mlp.up": mat(ff, W), p + "mlp.down": mat(W, ff)})
            continue
        out.update({p + "ls1": vec(W, 0.6), p + "ls2": vec(W, 0.6)})
        if L["type"] == "attention":
            G = m["kv_heads"]
            out.update({x + "q": mat(H * d, W), x + "q.b": vec(H * d, 0.0), x + "k": mat(G * d, W), x + "k.b": vec(G * d, 0.0), x + "o": mat(W, H * d)})
        elif L["type"] == "latent_attention":
            r, dv, R, Q = m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
            out.update({x + "dq": mat(Q, W), x + "dq.norm": vec(Q), x + "uq": mat(H * (d + r), Q), x + "uk": mat(H * d, R), x + "uv": mat(H * dv, R), x + "o": mat(W, H * dv)})
            if "kv_from" not in m:
                out.update({x + "dkv": mat(R + r, W), x + "dkv.norm": vec(R)})
        else:
            G, dv, taps, r = m["kv_heads"], m["vdim"], m["conv"], 16
            out.update({x + n: mat(k, W) for n, k in (("q", G * d), ("k", G * d), ("v", H * dv), ("b", H), ("a1", r), ("g1", r))})
            out.update({x + n + ".conv": ([k, taps], (0.0, 0.5)) for n, k in (("q", G * d), ("k", G * d), ("v", H * dv))})
            out.update({x + "A_log": vec(H, -1.5, 0.8), x + "norm": vec(dv), x + "a2": mat(H * d, r), x + "dt_bias": vec(H * d, 0.0, 0.5),
                        x + "g2": mat(H * dv, r), x + "o": mat(W, H * dv)})
        for n, a, b in (("gate", ff, W), ("up", ff, W), ("down", W, ff)):
            out[p + "mlp." + n] = mat(a, b)
            out[p + "mlp." + n + ".b"] = vec(a, 0.0)
    return out


def _tensor(name, shape, law):
    """The tensor of that name on the GPU: matrices in bfloat16, vectors in 32-bit, the same on every call."""
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()))
    t = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(law[0], law[1], generator=g)
    return t if len(shape) == 1 else t.to(torch.bfloat16)


_engines = {}


def _engine(model):
    if model not in _engines:
        config, dtype, tokens, longest, _ = MODELS[model]
        weights = {n: _tensor(n, *s).cpu() for n, s in _shapes(config).items()}
        _engines[model] = Engine.from_tensors(config, weights, dtype=dtype, max_tokens=tokens, max_seq_len=longest, max_slots=512)
    return _engines[model]


# ---------------------------------------------------------------- the passes
def _tokens(case, seed):
    """(prompts, the tokens of each step, uniform numbers of each step and of the prompts)."""
    c = MODELS[case["model"]][0]
    vocab = c.get("vocab_size") or c["vocab"]
    rng = np.random.default_rng([seed, 77])
    prompts = [rng.integers(0, vocab, n).tolist() for n in lengths(case)]
    steps = rng.integers(0, vocab, (case["steps"], case["batch"])).tolist()
    uniforms = rng.random((case["steps"] + 1, case["batch"])).tolist()
    return prompts, steps, uniforms


class _Requests:
    """A batch of requests with the engine that serves them; decode keeps the sequences open."""

    def __init__(self, case, seed):
        self.kind = case["kind"]
        self.engine = _engine(case["model"])
        self.prompts, self.steps, self.uniforms = _tokens(case, seed)
        # the reference's defaults, or the greedy choice
        self.sampling = SamplingParams() if case["sampled"] else SamplingParams(temperature=0.0, top_k=1, top_p=1.0)
        self.whole = MODELS[case["model"]][1] == "float32"
        self.longest = min(self.engine.max_seq_len, max(len(p) for p in self.prompts) + min(4096, 65536 // len(self.prompts)))
        self.slots = []
        if self.kind == "decode":
            self.begin().result()

    def begin(self):
        self.slots = [self.engine.open_sequence() for _ in self.prompts]
        return self.engine.step_tokens([StepItem(s, p, [len(p) - 1]) for s, p in zip(self.slots, self.prompts)], self.sampling, self.uniforms[-1])

    def end(self):
        for s in self.slots:
            self.engine.close_sequence(s)
        self.slots = []

    def __del__(self):
        self.end()


def prepare(case, seed):
    return _Requests(case, seed)


def run(state):
    e = state.engine
    if state.kind == "prompt":
        state.slots = [e.open_sequence() for _ in state.prompts]
        logits = e.step([StepItem(s, p, [len(p) - 1]) for s, p in zip(state.slots, state.prompts)])
        state.end()
        return _outputs(logits)
    pending, drawn = [], []
    if state.kind == "serve":
        pending.append(state.begin())
    elif max(e.sequence_length(s) for s in state.slots) + len(state.steps) > state.longest:
        state.end()
        pending.append(state.begin())
    for tokens, uniforms in zip(state.steps[:-1], state.uniforms):
        pending.append(e.step_tokens([StepItem(s, [t], [0]) for s, t in zip(state.slots, tokens)], state.sampling, uniforms))
        if len(pending) > 1:
            drawn.append(pending.pop(0).result())
    items = [StepItem(s, [t], [0]) for s, t in zip(state.slots, state.steps[-1])]
    logits, last = e.step(items, state.sampling, state.uniforms[len(state.steps) - 1])
    drawn += [p.result() for p in pending]
    if state.kind == "serve":
        state.end()
    return _outputs(logits, np.array(drawn + [last.tolist()]) if state.whole and state.kind == "serve" else None)


CHECKED = 3        # sequences of a batch that are computed in 64 bits


def _outputs(logits, drawn=None):
    out = {"first": logits[:CHECKED]}
    if len(logits) > CHECKED:
        out["others"] = logits[CHECKED:]
    if drawn is not None:
        out["tokens"] = drawn
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def _runs(c):
    """The layers in running order."""
    if c.get("model_type") == "llama":
        return list(range(c["num_hidden_layers"]))
    n, loop = len(c["layers"]), c.get("loop")
    if not loop:
        return list(range(n))
    return list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))


def _parts(c):
    """Per layer run: (values of matrices in the mixer, in the feed-forward, flops a (query, key) pair, cached values a
    position, visible keys at a position, 32-bit values of state, flops a token of the recurrence); the output matrix;
    values of matrices between layers."""
    out = []
    if c.get("model_type") == "llama":
        H, I, d, nH, nKV = c["hidden_size"], c["intermediate_size"], c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"]
        layer = (H * (2 * nH + 2 * nKV) * d, 3 * H * I, 4 * nH * d, 2 * nKV * d, lambda p: p + 1, 0, 0)
        return [layer] * c["num_hidden_layers"], c["vocab_size"] * H, 0
    shapes = _shapes(c)
    size = lambda prefix: sum(math.prod(s) for n, (s, _) in shapes.items() if n.startswith(prefix) and len(s) == 2)  # noqa: E731
    for i in _runs(c):
        L = c["layers"][i]
        m, kind = L["mixer"], L["type"]
        mix, ff = size(f"l{i}.mix."), size(f"l{i}.mlp.")
        if kind == "attention":
            mask = m.get("mask")
            if not mask:
                seen = lambda p: p + 1  # noqa: E731
            elif c["architecture"] == "Sinezen":
                seen = lambda p, b=mask["size"]: p % b + 1  # noqa: E731
            else:
                seen = lambda p, w=mask["size"], k=mask["keep_first"]: min(p + 1, w) + max(0, min(k, p + 1 - w))  # noqa: E731
            out.append((mix, ff, 2 * m["heads"] * (m["dim"] + m["vdim"]), m["kv_heads"] * (m["dim"] + m["vdim"]), seen, 0, 0))
        elif kind == "latent_attention":
            row = m["kv_rank"] + m["rot_dim"]
            out.append((mix, ff, 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), row, lambda p: p + 1, 0, 0))
        else:
            dv = m.get("vdim", m["dim"])
            out.append((mix, ff, 0, 0, lambda p: 0, m["heads"] * m["dim"] * dv, 8 * m["heads"] * m["dim"] * dv))
    return out, c["vocab"] * c["width"], (c["loop"]["times"] * 2 * c["width"] ** 2 if c["architecture"] == "Sinezen" else 0)


def work(case):
    """Prompts: every matrix once, what is cached written, a product's flops for every token (the last feed-forward and the
    output matrix for the wanted rows alone).  A single-token step: every matrix, the visible cached rows, the state read
    and written.  Layers that run several times are read as often: more than the L2 holds lies between."""
    c, dtype, _, _, _ = MODELS[case["model"]]
    b = 4 if dtype == "float32" else 2
    parts, head, between = _parts(c)
    lens, n = lengths(case), case["batch"]
    matrices = sum(p[0] + p[1] for p in parts) + head + between
    total = dict(bytes=0.0, flops=0.0)
    vocab = head // (c.get("hidden_size") or c["width"])
    if case["kind"] != "decode":
        T = sum(lens)
        total["bytes"] += b * matrices + sum(b * p[3] * T + 4 * p[5] * n for p in parts)
        total["flops"] += 2.0 * T * (matrices - head) - 2.0 * (T - n) * parts[-1][1] + 2.0 * n * head
        for p in parts:
            total["flops"] += sum(p[2] * p[4](t) for m in lens for t in range(m)) + float(p[6]) * T
    for k in range(case["steps"]):
        total["bytes"] += b * matrices + sum(b * p[3] * sum(p[4](m + k) for m in lens) + 8 * p[5] * n for p in parts)
        total["flops"] += 2.0 * n * matrices + sum(p[2] * sum(p[4](m + k) for m in lens) + float(p[6]) * n for p in parts)
    total["bytes"] += 4 * n * vocab
    return total


def tolerance(case):
    """Measured between the library's own ways of computing the same (products on the older tensor-core path, attention
    kernels on the older one): Llama sizes 0.008 to 0.017 (0.04 to 0.085 at the worst value), the others 0.0032 to 0.0056
    (0.026), and each as far from 64 bits; 32-bit: 6e-6 from 64 bits."""
    if MODELS[case["model"]][1] == "float32":
        return {"rel": 3e-5, "max": 3e-4, "differ": 0.01}
    return {"rel": 0.03, "max": 0.3} if case["model"].startswith("llama") else {"rel": 0.02, "max": 0.1}


# ---------------------------------------------------------------- the same in 64 bits, in plain torch
F64 = torch.float64


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, b, eps):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], w, b, eps)


def _attend(q, k, v, scale, visible):
    """q [T, H, d], k [T, G, d], v [T, G, dv]: softmax over the visible keys, a key head at a time."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=q.device)
    for g in range(G):
        h = slice(g * (H // G), (g + 1) * (H // G))
        s = torch.einsum("ihd,jd->hij", q[:, h], k[:, g]) * scale
        out[:, h] = torch.einsum("hij,jd->ihd", s.masked_fill_(~visible, -math.inf).softmax(-1), v[:, g])
    return out


def _turn(x, angles, magnitude=1.0, pairs=False):
    """Rotates the first 2 * angles.shape[1] channels of x [T, heads, d]: halves, or neighbouring pairs."""
    n = 2 * angles.shape[1]
    c, s = (angles.cos() * magnitude)[:, None], (angles.sin() * magnitude)[:, None]
    out = x.clone()
    a, b = (slice(0, n, 2), slice(1, n, 2)) if pairs else (slice(0, n // 2), slice(n // 2, n))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _frequencies(n, base, scaling):
    f = [float(base) ** (-2.0 * i / n) for i in range(n // 2)]
    if scaling and "low_freq_factor" in scaling:          # slow turns are divided, fast ones kept, a blend between
        lo, hi, orig = scaling["low_freq_factor"], scaling["high_freq_factor"], scaling["original_max_position_embeddings"]
        blend = [min(max((orig * x / (2 * math.pi) - lo) / (hi - lo), 0.0), 1.0) for x in f]
        f = [(1 - s) * x / scaling["factor"] + s * x for x, s in zip(f, blend)]
    elif scaling:                                         # a ramp over the pair's index
        where = lambda turns: n * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(where(scaling["fast"])), 0), min(math.ceil(where(scaling["slow"])), n - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(n // 2)]
        f = [x / scaling["factor"] * r + x * (1 - r) for x, r in zip(f, ramp)]
    return torch.tensor(f, dtype=F64, device="cuda")


def _short_conv(x, w):
    """x [T, C], w [C, taps], the last tap on the token itself, zeros before the first."""
    taps = w.shape[1]
    xp = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(xp[j:j + x.shape[0]] * w[:, j] for j in range(taps))


def _llama64(c, w, ids):
    H, G, d, T, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], len(ids), c["rms_norm_eps"]
    visible = torch.ones(T, T, dtype=torch.bool, device="cuda").tril()
    angles = torch.arange(T, dtype=F64, device="cuda")[:, None] * _frequencies(d, c["rope_theta"], c["rope_scaling"])
    x = w("model.embed_tokens.weight")[ids]
    for i in range(c["num_hidden_layers"]):
        lw = lambda n: w(f"model.layers.{i}.{n}.weight")  # noqa: E731, B023
        h = _rms(x, lw("input_layernorm"), eps)
        q, k, v = ((h @ lw(f"self_attn.{n}_proj").T).view(T, -1, d) for n in "qkv")
        o = _attend(_turn(q, angles), _turn(k, angles), v, d ** -0.5, visible)
        x = x + o.reshape(T, H * d) @ lw("self_attn.o_proj").T
        h = _rms(x, lw("post_attention_layernorm"), eps)
        x = x + (torch.nn.functional.silu(h @ lw("mlp.gate_proj").T) * (h @ lw("mlp.up_proj").T)) @ lw("mlp.down_proj").T
    return w("model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight") @ _rms(x[-1], w("model.norm.weight"), eps)


def _sinezen64(c, w, ids):
    T, eps, pos = len(ids), c["norm"]["eps"], torch.arange(len(ids), device="cuda")
    x0 = x = w("embed")[ids]
    loop, runs = c["loop"], _runs(c)
    for r, i in enumerate(runs):
        if i == loop["start"]:
            x = torch.cat([x, x0], -1) @ w("loop.in").T
        m, lw = c["layers"][i]["mixer"], lambda n: w(f"l{i}.{n}")  # noqa: E731, B023
        h = _rms(x, lw("norm1"), eps)
        angles = pos.to(F64)[:, None] * _frequencies(m["rot"]["dims"], m["rot"]["base"], None)
        block = pos // m["mask"]["size"]
        visible = (pos[None] <= pos[:, None]) & (block[None] == block[:, None])
        q = _turn(_rms(h @ lw("mix.q").T, lw("mix.q.norm"), eps).view(T, -1, m["dim"]), angles)
        k = _turn(_rms(h @ lw("mix.k").T, lw("mix.k.norm"), eps).view(T, -1, m["dim"]), angles)
        o = _attend(q, k, (h @ lw("mix.v").T).view(T, -1, m["vdim"]), m["scale"], visible) * torch.sigmoid(h @ lw("mix.g").T)[:, :, None]
        x = x + o.reshape(T, -1) @ lw("mix.o").T + (torch.nn.functional.silu(h @ lw("mlp.gate").T) * (h @ lw("mlp.up").T)) @ lw("mlp.down").T
    return w("head") @ _rms(x[-1], w("final.norm"), eps)


def _sesuzen64(c, w, ids):
    T, eps, pos = len(ids), c["norm"]["eps"], torch.arange(len(ids), device="cuda")
    x = w("embed")[ids] + w("pos")[:T]
    one = lambda z: z / torch.sqrt((z * z).mean(-1, keepdim=True) + eps)  # noqa: E731
    for i in _runs(c):
        L, lw = c["layers"][i], lambda n: w(f"l{i}.{n}")  # noqa: E731, B023
        m = L["mixer"]
        H, d = m["heads"], m["dim"]
        h = _layer_norm(x, lw("norm1"), lw("norm1.b"), eps)
        h = h + _short_conv(h, lw("canon1"))
        if L["type"] == "attention":
            near = pos[:, None] - pos[None] < m["mask"]["size"]
            visible = (pos[None] <= pos[:, None]) & (near | (pos[None] < m["mask"]["keep_first"]))
            q, k, v = ((h @ lw("mix." + n).T + lw(f"mix.{n}.b")).view(T, -1, d) for n in "qkv")
            o = _attend(q, k, one(v), m["scale"], visible).reshape(T, -1)
        else:
            r, k, v = ((h @ lw("mix." + n).T).view(T, H, d) for n in "rkv")
            decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ lw("mix.w1").T) @ lw("mix.w2").T + lw("mix.w0"))).view(T, H, d, 1)
            rate = torch.sigmoid(h @ lw("mix.a").T + lw("mix.a.b")).view(T, H, d)
            unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            S, o = x.new_zeros(H, d, d), x.new_empty(T, H, d)
            cut, add = (rate * unit)[..., None], k[..., None] * v[:, :, None]
            for t in range(T):
                S = decay[t] * S - cut[t] * (unit[t][:, None] @ S) + add[t]
                o[t] = (r[t][:, None] @ S)[:, 0]
            o = one(o).reshape(T, -1) * lw("mix.norm")
        x = x + (o * torch.sigmoid(h @ lw("mix.g").T)) @ lw("mix.o").T
        h = _layer_norm(x, lw("norm2"), lw("norm2.b"), eps)
        x = x + torch.relu(h @ lw("mlp.up").T) ** 2 @ lw("mlp.down").T
    z = w("embed") @ _layer_norm(x[-1:], w("final.norm"), w("final.norm.b"), eps)[0]
    return c["logit_softcap"] * torch.tanh(z / c["logit_softcap"])


def _sobezen64(c, w, ids):
    T, eps, pos = len(ids), c["norm"]["eps"], torch.arange(len(ids), device="cuda").to(F64)
    silu, visible, rows = torch.nn.functional.silu, torch.ones(T, T, dtype=torch.bool, device="cuda").tril(), {}
    x = w("embed")[ids] * c["embedding"]["scale"]
    for i, L in enumerate(c["layers"]):
        m, lw = L["mixer"], lambda n: w(f"l{i}.{n}")  # noqa: E731, B023
        H, d = m["heads"], m["dim"]
        h = _rms(x, lw("norm1"), eps)
        if L["type"] == "channel_delta":
            G, dv = m["kv_heads"], m["vdim"]
            q, k, v = (silu(_short_conv(h @ lw("mix." + n).T, lw(f"mix.{n}.conv"))).view(T, -1, d) for n in "qkv")
            unit = lambda z: (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)  # noqa: E731, B023
            q, k = unit(q) * d ** -0.5, unit(k)
            step = torch.nn.functional.softplus(h @ lw("mix.a1").T @ lw("mix.a2").T + lw("mix.dt_bias")).view(T, H, d)
            decay = torch.exp(-torch.exp(lw("mix.A_log"))[None, :, None] * step)[..., None]
            beta = torch.sigmoid(h @ lw("mix.b").T)[:, :, None]
            S, o = x.new_zeros(H, d, dv), x.new_empty(T, H, dv)
            for t in range(T):
                S = decay[t] * S
                S = S + k[t][..., None] * (beta[t] * (v[t] - (k[t][:, None] @ S)[:, 0]))[:, None]
                o[t] = (q[t][:, None] @ S)[:, 0]
            o = _rms(o, lw("mix.norm"), eps) * torch.sigmoid(h @ lw("mix.g1").T @ lw("mix.g2").T).view(T, H, dv)
        else:
            rot = m["rot"]
            angles = pos[:, None] * _frequencies(rot["dims"], rot["base"], rot.get("scaling"))
            if L["type"] == "attention":
                q, k = ((h @ lw("mix." + n).T + lw(f"mix.{n}.b")).view(T, -1, d) for n in "qk")
                o = _attend(_turn(q, angles, pairs=True), _turn(k, angles, pairs=True), k, m["scale"], visible)
            else:
                mag = 0.1 * math.log(rot["scaling"]["factor"]) + 1.0
                if "kv_from" not in m:
                    both = h @ lw("mix.dkv").T
                    rows[i] = _rms(both[:, :m["kv_rank"]], lw("mix.dkv.norm"), eps), _turn(both[:, None, m["kv_rank"]:], angles, mag, True)
                latent, shared = rows[m.get("kv_from", i)]
                q = (_rms(h @ lw("mix.dq").T, lw("mix.dq.norm"), eps) @ lw("mix.uq").T).view(T, H, -1)
                q = torch.cat([q[..., :d], _turn(q[..., d:], angles, mag, True)], -1)
                k = torch.cat([(latent @ lw("mix.uk").T).view(T, H, d), shared.expand(T, H, m["rot_dim"])], -1)
                o = _attend(q, k, (latent @ lw("mix.uv").T).view(T, H, m["vdim"]), m["scale"], visible)
        x = x + (o.reshape(T, -1) @ lw("mix.o").T) * lw("ls1")
        h, lim = _rms(x, lw("norm2"), eps), L["mlp"]["limit"]
        g = torch.clamp(h @ lw("mlp.gate").T + lw("mlp.gate.b"), max=lim)
        u = torch.clamp(h @ lw("mlp.up").T + lw("mlp.up.b"), -lim, lim)
        x = x + ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ lw("mlp.down").T + lw("mlp.down.b")) * lw("ls2")
    return c["logit_scale"] * (w("head") @ _rms(x[-1], w("final.norm"), eps))


def exact(case, seed):
    """The first sequences' logits in 64 bits; the others', and drawn tokens, have no value here."""
    c = MODELS[case["model"]][0]
    prompts, steps, _ = _tokens(case, seed)
    shapes = _shapes(c)
    kept = {}                                   # the matrices in 64 bits, as far as they leave room for the rest

    def w(name):
        if name in kept:
            return kept[name]
        t = _tensor(name, *shapes[name]).to(F64)
        if torch.cuda.mem_get_info()[0] > 60e9:
            kept[name] = t
        return t

    forward = {"Sinezen": _sinezen64, "Sesuzen": _sesuzen64, "Sobezen": _sobezen64}.get(c.get("architecture"), _llama64)
    rows = []
    for i, p in enumerate(prompts[:CHECKED]):
        ids = torch.tensor(p + [s[i] for s in steps], device="cuda")
        rows.append(forward(c, w, ids))
    out = {"first": torch.stack(rows).cpu().numpy()}
    if case["batch"] > CHECKED:
        out["others"] = None
    if MODELS[case["model"]][1] == "float32" and case["kind"] == "serve":
        out["tokens"] = None
    return out
