"""The work whose speed this repository answers for: steps of an engine through ``Session``.

A case is one step of a running engine, as the scheduler or a user's own loop issues it:

``prefill``
    Prompts come whole: the requests are opened, run as one step, asked for the logits of their last token (or of
    every token) and closed again.
``decode``
    ``batch`` requests whose contexts are in the cache bring one token each and want its logits.  The step is the
    scheduler's call (``step_reserved``), which leaves recording the progress to the caller, so that every pass is
    the same step; a recurrent layer's state moves on from pass to pass.
``mixed``
    What continuous batching makes of a busy server: requests that decode beside portions of longer prompts.

The models have the sizes that ``bench.py`` and ``bench_arch.py`` measure (Qwen3-0.6B and 8B; Binupel and Bikadra with
width 2,048 and 12 layers) and random weights.  The 8B model has 6 of its 36 layers: at its width the rounding of
bfloat16 activations grows from layer to layer with random weights, and after 12 or 36 of them two correct
implementations' outputs are too far apart to be compared (0.022 and 0.036 from 64 bits).  The architectures with routed experts are left out:
where two experts tie, a rounding decides which one runs.  Weights and tokens come from the seed alone.
"""

from __future__ import annotations

import gc
import hashlib
import json
import math
import os
import tempfile

import torch

from qwen3_from_scratch_b200.engine.batch import Entry
from qwen3_from_scratch_b200.engine.session import Session

PAGE = 16
PORTION = 2048  # tokens of a step while contexts are filled


# ---------------------------------------------------------------------- models
def _qwen3(hidden, heads, inter, layers, tied):
    return dict(architectures=["Qwen3ForCausalLM"], vocab_size=151936, hidden_size=hidden, hidden_act="silu",
                num_hidden_layers=layers, max_position_embeddings=40960, num_key_value_heads=8,
                num_attention_heads=heads, head_dim=128, intermediate_size=inter, rms_norm_eps=1e-6,
                rope_theta=1000000.0, tie_word_embeddings=tied)


def _binupel():
    ff = {"kind": "dense", "ff": 6144}
    scan = {"type": "mamba1", "mixer": {"inner": 4096, "state": 16, "dt_rank": 128, "conv": 4}, "mlp": ff}
    rec = {"type": "rglru", "mixer": {"width": 2048, "blocks": 8, "conv": 4}, "mlp": ff}
    att = {"type": "attention", "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                          "q_temp": {"coef": 0.3, "every": 256}}, "mlp": ff}
    return {"architecture": "Binupel", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "postln_alpha": 2.0,
            "layers": [scan, rec, att] * 4}


def _bikadra():
    ff = {"kind": "dense", "ff": 6144}
    ssm = {"type": "mamba2", "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "norm_groups": 8, "conv": 4},
           "mlp": ff}
    att = {"type": "latent_attention",
           "mixer": {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 1536,
                     "scale": 192 ** -0.5,
                     "rot": {"base": 10000.0, "dims": 64,
                             "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}},
           "mlp": ff}
    return {"architecture": "Bikadra", "vocab": 32000, "width": 2048, "embedding": {"scale": 1.0}, "streams": 4,
            "norm": {"eps": 1e-6}, "logit_softcap": 30.0, "layers": [ssm, att] * 6}


MODELS = {
    "qwen3-0.6b": _qwen3(1024, 16, 3072, 28, True),
    "qwen3-8b": _qwen3(4096, 32, 12288, 6, False),
    "binupel": _binupel(),
    "bikadra": _bikadra(),
}


# ---------------------------------------------------------------------- cases
def listed():
    return [
        # one user in a chat: the smallest call, where the chain of launches counts
        {"name": "decode_1", "model": "qwen3-0.6b", "dtype": "bfloat16", "kind": "decode", "batch": 1, "low": 517, "high": 517},
        # the benchmark's headline: batch 8 at a context of 4,096
        {"name": "decode_8", "model": "qwen3-0.6b", "dtype": "bfloat16", "kind": "decode", "batch": 8, "low": 4096, "high": 4096},
        # a loaded server: contexts of all lengths
        {"name": "decode_64", "model": "qwen3-0.6b", "dtype": "bfloat16", "kind": "decode", "batch": 64, "low": 130, "high": 2048},
        # a short question
        {"name": "prefill_300", "model": "qwen3-0.6b", "dtype": "bfloat16", "kind": "prefill", "batch": 1, "low": 300, "high": 300, "want": "last"},
        # the benchmark's prompt step
        {"name": "prefill_2048", "model": "qwen3-0.6b", "dtype": "bfloat16", "kind": "prefill", "batch": 1, "low": 2048, "high": 2048, "want": "last"},
        # continuous batching: 23 requests decode while three prompts go on
        {"name": "mixed", "model": "qwen3-0.6b", "dtype": "bfloat16", "kind": "mixed", "batch": 23, "low": 200, "high": 1500, "portions": "37,411,700", "history": 512},
        # the serving configuration's decode step
        {"name": "decode_8b_8", "model": "qwen3-8b", "dtype": "bfloat16", "kind": "decode", "batch": 8, "low": 1024, "high": 2048},
        # its prompt step: the largest call
        {"name": "prefill_8b_2048", "model": "qwen3-8b", "dtype": "bfloat16", "kind": "prefill", "batch": 1, "low": 2048, "high": 2048, "want": "last"},
        # scoring a text in float32: the logits of every token (trace replay, --dtype float32)
        {"name": "score_f32", "model": "qwen3-0.6b", "dtype": "float32", "kind": "prefill", "batch": 2, "low": 203, "high": 310, "want": "all"},
        # generating in float32
        {"name": "decode_f32_4", "model": "qwen3-0.6b", "dtype": "float32", "kind": "decode", "batch": 4, "low": 400, "high": 900},
        # the other designs: a recurrent one's decode step, one with a latent cache in its prompt step
        {"name": "binupel_decode_8", "model": "binupel", "dtype": "bfloat16", "kind": "decode", "batch": 8, "low": 2048, "high": 2048},
        {"name": "bikadra_prefill_2048", "model": "bikadra", "dtype": "bfloat16", "kind": "prefill", "batch": 1, "low": 2048, "high": 2048, "want": "last"},
    ]


def _spread(rng, low, high):
    """A whole number from ``low`` to ``high``, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    model, dtype, kinds, most = rng.choice([
        ("qwen3-0.6b", "bfloat16", ("decode", "prefill", "mixed"), 4096),
        ("qwen3-0.6b", "bfloat16", ("decode", "prefill", "mixed"), 4096),
        ("qwen3-8b", "bfloat16", ("decode", "prefill"), 2048),
        ("qwen3-0.6b", "float32", ("decode", "prefill"), 700),
        ("binupel", "bfloat16", ("decode", "prefill"), 2048),
        ("bikadra", "bfloat16", ("decode", "prefill"), 2048),
    ])
    kind = rng.choice(kinds)
    case = {"model": model, "dtype": dtype, "kind": kind}
    if kind == "prefill":
        case["batch"] = rng.choice([1, 1, 1, 2, 3])
        case["high"] = _spread(rng, 40, most // case["batch"])
        case["low"] = case["high"] if case["batch"] == 1 else _spread(rng, 33, case["high"])
        case["want"] = "all" if dtype == "float32" and case["high"] <= 400 else "last"
        return case
    small = dtype == "float32" or model != "qwen3-0.6b"
    case["batch"] = _spread(rng, 1, 16 if small else 64)
    case["high"] = _spread(rng, 64, min(most, 60000 // case["batch"], 16384 // case["batch"] if small else most))
    case["low"] = case["high"] if case["batch"] == 1 else _spread(rng, 33, case["high"])
    if kind == "mixed":
        case["portions"] = ",".join(str(_spread(rng, 17, 900)) for _ in range(rng.choice([1, 2, 3])))
        case["history"] = rng.choice([0, 160, 512, 1003])
    return case


def _lengths(case):
    """Tokens of each request after the step (for ``mixed``: of those that decode)."""
    n, low, high = case["batch"], case["low"], case["high"]
    return [high if n == 1 else low + (high - low) * i // (n - 1) for i in range(n)]


def _sequences(case):
    """(tokens in the cache before the step, tokens that the step brings) of every request, in the step's order."""
    if case["kind"] == "prefill":
        return [(0, n) for n in _lengths(case)]
    rows = [(n - 1, 1) for n in _lengths(case)]
    if case["kind"] == "mixed":
        rows += [(case["history"], int(n)) for n in case["portions"].split(",")]
    return rows


def _wanted(case, new):
    return list(range(new)) if case.get("want") == "all" else [new - 1]


def _ids(case, seed):
    vocab = MODELS[case["model"]].get("vocab_size") or MODELS[case["model"]]["vocab"]
    g = torch.Generator().manual_seed(int(seed) * 2 + 1)
    return [torch.randint(0, vocab, (before + new,), generator=g).tolist() for before, new in _sequences(case)]


# ---------------------------------------------------------------------- one pass
def prepare(case, seed):
    gc.collect()  # an engine holds itself in a cycle: one that is done with gives its memory back here
    rows, ids = _sequences(case), _ids(case, seed)
    with tempfile.TemporaryDirectory(prefix="q3b200-perf-") as folder:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(MODELS[case["model"]], f)
        session = Session(folder, dtype=case["dtype"], page_size=PAGE, max_seqs=max(2, len(rows)),
                          num_pages=sum(-(-(b + n) // PAGE) for b, n in rows) + 2,
                          max_step_tokens=max(PORTION, sum(n for _, n in rows)), random_weights=int(seed))
    session.step([Entry("first use", ids[0][:2], (1,))])  # what ``SyncEngine.warmup`` is for
    session.step([Entry("first use", ids[0][2:3], (0,))])
    session.end("first use")
    entries = [Entry(i, ids[i][b:], tuple(_wanted(case, n))) for i, (b, n) in enumerate(rows)]
    if case["kind"] != "prefill":
        for i, (before, _) in enumerate(rows):
            for at in range(0, before, PORTION):
                session.step([Entry(i, ids[i][at:min(before, at + PORTION)])])
        session.prepare(entries)
    return {"session": session, "entries": entries, "whole": case["kind"] == "prefill"}


def run(state):
    session, entries = state["session"], state["entries"]
    if not state["whole"]:
        return session.step_reserved(entries)
    logits = session.step(entries)
    for e in entries:
        session.end(e.request)
    return logits


# ---------------------------------------------------------------------- what a pass cannot do without
def _params(case):
    """(parameters of all layers, width, vocabulary, bytes per value)."""
    c = MODELS[case["model"]]
    size = 4 if case["dtype"] == "float32" else 2
    if "vocab_size" in c:
        W, D, H, G, F = c["hidden_size"], c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"], c["intermediate_size"]
        return c["num_hidden_layers"] * (2 * H * D * W + 2 * G * D * W + 3 * F * W), W, c["vocab_size"], size
    W, total = c["width"], 0
    for layer in c["layers"]:
        m, ff = layer["mixer"], layer["mlp"]["ff"]
        total += (3 if c["architecture"] == "Binupel" else 2) * ff * W
        if layer["type"] == "mamba1":
            total += 3 * m["inner"] * W + (m["dt_rank"] + 2 * m["state"]) * m["inner"] + m["dt_rank"] * m["inner"]
        elif layer["type"] == "rglru":
            total += 3 * W * W + 2 * W * W // m["blocks"]
        elif layer["type"] == "attention":
            total += 2 * m["heads"] * m["dim"] * W + m["kv_heads"] * m["dim"] * W
        elif layer["type"] == "mamba2":
            inner = m["heads"] * m["vdim"]
            total += (2 * inner + 2 * m["groups"] * m["state"] + m["heads"]) * W + inner * W
        else:
            total += (m["q_rank"] + m["kv_rank"] + m["rot_dim"]) * W + m["q_rank"] * m["heads"] * (m["dim"] + m["rot_dim"])
            total += 2 * m["kv_rank"] * m["heads"] * m["dim"] + m["heads"] * m["vdim"] * W
    return total, W, c["vocab"], size


def work(case):
    params, W, vocab, size = _params(case)
    rows = _sequences(case)
    new = sum(n for _, n in rows)
    wanted = sum(len(_wanted(case, n)) for _, n in rows)
    c = MODELS[case["model"]]
    # per layer kind: values a token keeps in the cache, flops per (query, key), state values per request, flops per state value and token
    per_token = per_pair = state = scan = 0
    for layer in (c["layers"] if "layers" in c else [{"type": "qwen3"}] * c["num_hidden_layers"]):
        m = layer.get("mixer")
        if layer["type"] == "qwen3":
            per_token += 2 * c["num_key_value_heads"] * c["head_dim"]
            per_pair += 4 * c["num_attention_heads"] * c["head_dim"]
        elif layer["type"] == "attention":
            per_token += 2 * m["kv_heads"] * m["dim"]
            per_pair += 4 * m["heads"] * m["dim"]
        elif layer["type"] == "latent_attention":
            per_token += m["kv_rank"] + m["rot_dim"]
            per_pair += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif layer["type"] == "mamba1":
            state, scan = state + m["inner"] * m["state"], scan + 6 * m["inner"] * m["state"]
        elif layer["type"] == "mamba2":
            values = m["heads"] * m["vdim"] * m["state"]
            state, scan = state + values, scan + 5 * values
        else:
            state, scan = state + m["width"], scan + 4 * m["width"]
    pairs = sum(n * b + n * (n + 1) // 2 for b, n in rows)
    carried = sum((8 if b else 4) for b, _ in rows) * state  # float32, read where a request goes on, and written
    return {"bytes": size * (params + vocab * W) + size * per_token * sum(b + n for b, n in rows) + carried + 4 * wanted * vocab,
            "flops": 2 * params * new + 2 * vocab * W * wanted + per_pair * pairs + scan * new}


def tolerance(case):
    # Measured against 64 bits: the bfloat16 steps are 0.006 to 0.016 off (rounding of activations between the
    # products, layer after layer), the float32 steps 7e-7 to 1.7e-6; sums in another order differ by as much.
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.03, "max": 0.3}


# ---------------------------------------------------------------------- the same in 64 bits, in plain torch
class _Weights:
    """The tensors that ``random_weights=seed`` stands for: each drawn on the GPU by a generator of its own, seeded
    from the seed and its name; matrices in the dtype of the run, vectors in float32."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype = int(seed), getattr(torch, dtype)
        self.g = torch.Generator(device="cuda")

    def _raw(self, name, shape, dtype, mean, std):
        digest = hashlib.sha256(f"{self.seed}:{name}".encode()).digest()
        self.g.manual_seed(int.from_bytes(digest[:8], "little") & ((1 << 63) - 1))
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=self.g)

    def mat(self, name, *shape):
        return self._raw(name, shape, self.dtype, 0.0, 0.02).double()

    def vec(self, name, *shape):
        return self._raw(name, shape, torch.float32, 0.0, 0.02).double()

    def one(self, name, *shape):
        return self._raw(name, shape, torch.float32, 1.0, 0.1).double()

    def eye(self, name, n):
        return (self._raw(name, (n, n), torch.float32, 0.0, 0.1) + torch.eye(n, device="cuda")).double()


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, pos, freq, magnitude=1.0):
    """x [..., T, heads, 2 half]: value i is paired with i + half."""
    a = pos.double()[:, None] * freq
    cos, sin = (a.cos() * magnitude)[:, None, :], (a.sin() * magnitude)[:, None, :]
    u, v = x.chunk(2, dim=-1)
    return torch.cat([u * cos - v * sin, v * cos + u * sin], dim=-1)


def _causal(q, k, v, scale, weigh):
    """q [T, H, D], k, v [T, G, D]: a kv head serves H / G query heads; ``weigh`` makes weights of the scores."""
    T, H, D = q.shape
    G = k.shape[1]
    later = torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1)
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    for g in range(G):
        heads = slice(g * (H // G), (g + 1) * (H // G))
        s = torch.einsum("thd,nd->htn", q[:, heads], k[:, g]) * scale
        out[:, heads] = torch.einsum("htn,nd->thd", weigh(s, later, heads), v[:, g])
    return out


def _softmax(s, later, heads):
    return s.masked_fill_(later, -math.inf).softmax(-1)


def _exact_qwen3(c, w, ids, wanted):
    eps, D, H, G = c["rms_norm_eps"], c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"]
    W, F, V = c["hidden_size"], c["intermediate_size"], c["vocab_size"]
    lens = [len(s) for s in ids]
    # the inverse frequencies are float32 numbers by the model's definition
    freq = (1.0 / (c["rope_theta"] ** (torch.arange(0, D, 2, dtype=torch.float32) / D))).double().cuda()
    embed = w.mat("model.embed_tokens.weight", V, W)
    x = embed[torch.tensor([t for s in ids for t in s], device="cuda")]
    if not c["tie_word_embeddings"]:
        del embed
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w.one(p + "input_layernorm.weight", W)
        q = (h @ w.mat(p + "self_attn.q_proj.weight", H * D, W).t()).view(-1, H, D)
        k = (h @ w.mat(p + "self_attn.k_proj.weight", G * D, W).t()).view(-1, G, D)
        v = (h @ w.mat(p + "self_attn.v_proj.weight", G * D, W).t()).view(-1, G, D)
        q = _rms(q, eps) * w.one(p + "self_attn.q_norm.weight", D)
        k = _rms(k, eps) * w.one(p + "self_attn.k_norm.weight", D)
        parts = []
        for q1, k1, v1 in zip(q.split(lens), k.split(lens), v.split(lens)):
            pos = torch.arange(q1.shape[0], device="cuda")
            parts.append(_causal(_rotate(q1, pos, freq), _rotate(k1, pos, freq), v1, D ** -0.5, _softmax).reshape(-1, H * D))
        x = x + torch.cat(parts) @ w.mat(p + "self_attn.o_proj.weight", W, H * D).t()
        del q, k, v, parts
        h = _rms(x, eps) * w.one(p + "post_attention_layernorm.weight", W)
        gate, up = w.mat(p + "mlp.gate_proj.weight", F, W), w.mat(p + "mlp.up_proj.weight", F, W)
        down = w.mat(p + "mlp.down_proj.weight", W, F)
        for a, b in zip(x.split(8192), h.split(8192)):
            a += (torch.nn.functional.silu(b @ gate.t()) * (b @ up.t())) @ down.t()
    rows = [sum(lens[:i]) + r for i, want in enumerate(wanted) for r in want]
    h = _rms(x[rows], eps) * w.one("model.norm.weight", W)
    return h @ (embed if c["tie_word_embeddings"] else w.mat("lm_head.weight", V, W)).t()


def _conv(x, taps, bias):
    """x [B, T, C], taps [C, K]: the last tap meets the current token."""
    K = taps.shape[1]
    full = torch.cat([x.new_zeros(x.shape[0], K - 1, x.shape[2]), x], dim=1)
    return sum(full[:, j:j + x.shape[1]] * taps[:, j] for j in range(K)) + bias


def _walk(a, b):
    """S_t = a_t S_{t-1} + b_t over the second axis, from zero: all S_t."""
    out, S = torch.empty_like(b), torch.zeros_like(b[:, 0])
    for t in range(a.shape[1]):
        S = torch.addcmul(b[:, t], a[:, t], S)
        out[:, t] = S
    return out


def _padded(ids):
    longest = max(len(s) for s in ids)
    return torch.tensor([s + [0] * (longest - len(s)) for s in ids], device="cuda")


def _exact_binupel(c, w, ids, wanted):
    eps, W, V, alpha = c["norm"]["eps"], c["width"], c["vocab"], c["postln_alpha"]
    x = w.mat("embed", V, W)[_padded(ids)]  # [B, T, W]; what is computed behind a request's end is never looked at
    B, T = x.shape[:2]
    for i, layer in enumerate(c["layers"]):
        p, m, F = f"l{i}.mix.", layer["mixer"], layer["mlp"]["ff"]
        before = torch.cat([x.new_zeros(B, 1, W), x[:, :-1]], dim=1)
        h = x + (before - x) * w.vec(f"l{i}.shift", W)
        if layer["type"] == "mamba1":
            I, N, R = m["inner"], m["state"], m["dt_rank"]
            u, z = (h @ w.mat(p + "in", 2 * I, W).t()).chunk(2, dim=-1)
            u = torch.nn.functional.silu(_conv(u, w.vec(p + "conv", I, m["conv"]), w.vec(p + "conv.b", I)))
            low = u @ w.mat(p + "x", R + 2 * N, I).t()
            step = torch.nn.functional.softplus(low[..., :R] @ w.mat(p + "dt", I, R).t() + w.vec(p + "dt.b", I), threshold=40)
            A, D = -w.vec(p + "A_log", I, N).exp(), w.one(p + "D", I)
            y, S = torch.empty_like(u), x.new_zeros(B, I, N)
            for t0 in range(0, T, 64):
                at = slice(t0, min(T, t0 + 64))
                a = (step[:, at, :, None] * A).exp()
                b = (step[:, at] * u[:, at])[..., None] * low[:, at, None, R:R + N]
                b[:, 0] += a[:, 0] * S
                a[:, 0] = 0
                states = _walk(a, b)
                S = states[:, -1]
                y[:, at] = torch.einsum("btin,btn->bti", states, low[:, at, R + N:])
            mixed = ((y + D * u) * torch.nn.functional.silu(z)) @ w.mat(p + "o", W, I).t()
        elif layer["type"] == "rglru":
            C, n = m["width"], m["blocks"]
            y = torch.nn.functional.gelu(h @ w.mat(p + "y", C, W).t() + w.vec(p + "y.b", C), approximate="tanh")
            u = _conv(h @ w.mat(p + "x", C, W).t() + w.vec(p + "x.b", C), w.vec(p + "conv", C, m["conv"]), w.vec(p + "conv.b", C))
            parts = u.view(B, T, n, C // n)
            gates = [torch.sigmoid(torch.einsum("btnc,ndc->btnd", parts, w.mat(p + g, n, C // n, C // n))
                                   + w.vec(p + g + ".b", n, C // n)).reshape(B, T, C) for g in ("ra", "ri")]
            a = (-8.0 * gates[0] * torch.nn.functional.softplus(w.one(p + "lam", C), threshold=40)).exp()
            mixed = (_walk(a, (1.0 - a * a).sqrt() * gates[1] * u) * y) @ w.mat(p + "o", W, C).t()
        else:
            H, G, D = m["heads"], m["kv_heads"], m["dim"]
            q = _rms((h @ w.mat(p + "q", H * D, W).t()).view(B, T, H, D), eps) * w.one(p + "q.norm", D)
            k = (h @ w.mat(p + "k", G * D, W).t()).view(B, T, G, D)
            kn = _rms(k, eps) * w.one(p + "k.norm", D)
            pos = torch.arange(T, device="cuda").double()
            q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1.0) / m["q_temp"]["every"]) + 1.0))[:, None, None]
            bias, gate = w.vec(p + "pb", H), torch.sigmoid(h @ w.mat(p + "g", H, W).t())
            weigh = lambda s, later, heads: torch.sigmoid(s + bias[heads, None, None]).masked_fill_(later, 0.0)  # noqa: E731
            out = torch.stack([_causal(q[b], kn[b], k[b], m["scale"], weigh) for b in range(B)])
            mixed = (out * gate[..., None]).reshape(B, T, H * D) @ w.mat(p + "o", W, H * D).t()
        x = _rms(alpha * x + mixed, eps) * w.one(f"l{i}.norm1", W)
        p = f"l{i}.mlp."
        ff = (torch.relu(x @ w.mat(p + "gate", F, W).t()) * (x @ w.mat(p + "up", F, W).t())) @ w.mat(p + "down", W, F).t()
        x = _rms(alpha * x + ff, eps) * w.one(f"l{i}.norm2", W)
    rows = torch.stack([x[b, r] for b, want in enumerate(wanted) for r in want])
    return (_rms(rows, eps) * w.one("final.norm", W)) @ w.mat("head", V, W).t()


def _stretched(rot):
    """Frequencies per pair and the factor on sines and cosines: slow pairs slowed, fast ones kept, a ramp between."""
    dims, base, s = rot["dims"], rot["base"], rot["scaling"]
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / dims)
    pair = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return (f / s["factor"] * ramp + f * (1.0 - ramp)).cuda(), 0.1 * math.log(s["factor"]) + 1.0


def _state_space(x, Bm, Cm, step, rate):
    """x [B, T, H, P], Bm, Cm [B, T, H, N], step [B, T, H]: the recurrence S = exp(-rate step) S + step B x^T, y = S^T C,
    64 tokens at a time as products."""
    B, T, H, P = x.shape
    S, y = x.new_zeros(B, H, Bm.shape[3], P), torch.empty_like(x)
    for t0 in range(0, T, 64):
        at = slice(t0, min(T, t0 + 64))
        d = (-rate * step[:, at]).cumsum(1).transpose(1, 2)  # [B, H, t]
        n = d.shape[2]
        decay = (d[..., :, None] - d[..., None, :]).masked_fill(torch.ones(n, n, dtype=torch.bool, device=x.device).triu(1), -math.inf).exp()
        sx = step[:, at, :, None] * x[:, at]
        m = torch.einsum("bthn,bshn->bhts", Cm[:, at], Bm[:, at]) * decay
        y[:, at] = torch.einsum("bhts,bshp->bthp", m, sx)
        y[:, at] += torch.einsum("bthn,bhnp->bthp", Cm[:, at], S) * d.exp().transpose(1, 2)[..., None]
        last = (d[..., -1:] - d).exp().transpose(1, 2)[..., None]
        S = d[..., -1].exp()[..., None, None] * S + torch.einsum("bthn,bthp->bhnp", Bm[:, at] * last, sx)
    return y


def _exact_bikadra(c, w, ids, wanted):
    eps, W, V, streams = c["norm"]["eps"], c["width"], c["vocab"], c["streams"]
    embed = w.mat("embed", V, W)
    x = (embed[_padded(ids)] * c["embedding"]["scale"])[None].repeat(streams, 1, 1, 1)  # [S, B, T, W]
    B, T = x.shape[1:3]

    def around(x, name, norm, inner):
        u = torch.einsum("s,sbtw->btw", w.one(name + "in", streams), x)
        y = inner(_rms(u, eps) * w.one(norm, W))
        return torch.einsum("sr,sbtw->rbtw", w.eye(name + "mix", streams), x) + w.one(name + "out", streams)[:, None, None, None] * y

    for i, layer in enumerate(c["layers"]):
        p, m, F = f"l{i}.mix.", layer["mixer"], layer["mlp"]["ff"]

        def mixer(h):
            if layer["type"] == "mamba2":
                H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
                inner, C = H * P, H * P + 2 * G * N
                proj = h @ w.mat(p + "in", inner + C + H, W).t()
                z, xbc, dt = proj.split([inner, C, H], dim=-1)
                xbc = torch.nn.functional.silu(_conv(xbc, w.vec(p + "conv", C, m["conv"]), w.vec(p + "conv.b", C)))
                u, Bm, Cm = xbc.split([inner, G * N, G * N], dim=-1)
                u = u.reshape(B, T, H, P)
                Bm, Cm = (v.reshape(B, T, G, N).repeat_interleave(H // G, dim=2) for v in (Bm, Cm))
                step = torch.nn.functional.softplus(dt + w.vec(p + "dt_bias", H), threshold=40)
                y = torch.cat([_state_space(u[b:b + 1], Bm[b:b + 1], Cm[b:b + 1], step[b:b + 1], w.vec(p + "A_log", H).exp())
                               for b in range(B)]) + w.one(p + "D", H)[:, None] * u
                y = y.reshape(B, T, inner) * torch.nn.functional.silu(z)
                y = _rms(y.view(B, T, m["norm_groups"], -1), eps).reshape(B, T, inner) * w.one(p + "norm", inner)
                return y @ w.mat(p + "o", W, inner).t()
            H, dn, dr, dv, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            freq, magnitude = _stretched(m["rot"])
            pos = torch.arange(T, device="cuda")
            cq = _rms(h @ w.mat(p + "dq", m["q_rank"], W).t(), eps) * w.one(p + "dq.norm", m["q_rank"])
            q = (cq @ w.mat(p + "uq", H * (dn + dr), m["q_rank"]).t()).view(B, T, H, dn + dr)
            down = h @ w.mat(p + "dkv", rank + dr, W).t()
            latent = _rms(down[..., :rank], eps) * w.one(p + "dkv.norm", rank)
            k = (latent @ w.mat(p + "uk", H * dn, rank).t()).view(B, T, H, dn)
            v = (latent @ w.mat(p + "uv", H * dv, rank).t()).view(B, T, H, dv)
            out = []
            for b in range(B):
                k_rot = _rotate(down[b, :, None, rank:], pos, freq, magnitude).expand(T, H, dr)
                q1 = torch.cat([q[b, ..., :dn], _rotate(q[b, ..., dn:], pos, freq, magnitude)], dim=-1)
                out.append(_causal(q1, torch.cat([k[b], k_rot], dim=-1), v[b], m["scale"], _softmax))
            gate = torch.sigmoid(h @ w.mat(p + "g", H, W).t())
            return (torch.stack(out) * gate[..., None]).reshape(B, T, H * dv) @ w.mat(p + "o", W, H * dv).t()

        x = around(x, f"l{i}.hc1.", f"l{i}.norm1", mixer)
        p2 = f"l{i}.mlp."
        x = around(x, f"l{i}.hc2.", f"l{i}.norm2", lambda h: torch.nn.functional.gelu(
            h @ w.mat(p2 + "up", F, W).t(), approximate="tanh") @ w.mat(p2 + "down", W, F).t())
    rows = torch.stack([x[:, b, r].sum(0) for b, want in enumerate(wanted) for r in want])
    logits = (_rms(rows, eps) * w.one("final.norm", W)) @ embed.t()
    return c["logit_softcap"] * torch.tanh(logits / c["logit_softcap"])


@torch.inference_mode()
def exact(case, seed):
    c, w, ids = MODELS[case["model"]], _Weights(seed, case["dtype"]), _ids(case, seed)
    wanted = [[b + r for r in _wanted(case, n)] for b, n in _sequences(case)]
    forward = {"binupel": _exact_binupel, "bikadra": _exact_bikadra}.get(case["model"], _exact_qwen3)
    return forward(c, w, ids, wanted)
