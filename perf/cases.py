"""The work that this engine is measured by: what its users have it do, from a lone decoded token to a step of
eight long prompts.

A pass goes through ``Engine``: its step function on given token ids (the way of ``bin/trace_run`` and of the timed loops
of ``bench.py``), which returns 32-bit logits, or ``Engine.generate``, which returns tokens.  A program that serves
requests keeps its engine for days, so ``prepare`` hands over an engine that has run steps of these shapes before, with
the requests' earlier tokens in its cache; what a pass appends is forgotten at the start of the next one.  Weights are
seeded random ones, a checkpoint in the temporary folder like that of ``bench.py``; a seed gives other tokens.

Architectures: GPT-2 at the sizes of the presets, and of the six others Kemuzen and Dedunex, at the sizes at which
``bench.py --compare-designs`` puts them side by side.  The other four route rows to experts; in bfloat16 two correct
implementations choose differently where a router's choice is a close call, so their logits cannot be held together.
"""
import json
import math
import os
import struct

import numpy as np
import torch

import nanoinfer_b200 as nb
from nanoinfer_b200 import bench_support as bs
from nanoinfer_b200.cli import _preset_path
from nanoinfer_b200.engine import StepItem

VOCAB = 50257
WEIGHTS_SEED = 1234
#: largest step of the listed and drawn cases, rows
MOST_ROWS = 8000


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # a chat with one user: latency and the number of launches count
        dict(name="small decode 1", kind="decode", model="gpt2-small", batch=1, context=64, steps=8),
        # the headline of bench.py: eight requests near the end of the context
        dict(name="small decode 8", kind="decode", model="gpt2-small", batch=8, context=999, steps=8),
        # a busy server: many requests, all of different age, an odd number of them
        dict(name="medium decode 61 ragged", kind="decode", model="gpt2-medium", batch=61, context=1001, ragged=True, steps=4),
        # the largest model, prompts of 512 tokens and on
        dict(name="xl decode 8", kind="decode", model="gpt2-xl", batch=8, context=640, steps=4),
        # a long context: a step is mostly keys and values
        dict(name="small decode 8 far", kind="decode", model="gpt2-small", positions=8192, batch=8, context=8150, steps=4),
        # a question of a few lines, until its first token
        dict(name="small prompt 77", kind="prompt", model="gpt2-small", prompts=1, length=77),
        # the prefill workload of bench.py, 2,048 rows in a step
        dict(name="small prompt 2x1024", kind="prompt", model="gpt2-small", prompts=2, length=1024),
        # documents through the largest model, the most rows in a step; not a multiple of any tile
        dict(name="xl prompt 8x1003", kind="prompt", model="gpt2-xl", prompts=8, length=1003),
        # continuous batching: decoded tokens beside portions of two prompts, one of which was begun before
        dict(name="medium mixed 24+2x317", kind="mixed", model="gpt2-medium", batch=24, context=600, prompts=2, length=317),
        # the true 32-bit path from prompts to sampled tokens, through scheduler and sampler
        dict(name="small generate f32", kind="generate", model="gpt2-small", dtype="float32", batch=4, length=53, tokens=16,
             temperature=0.8),
        # another architecture, a request's life: its prompt (recurrences, windows), then its tokens
        dict(name="kemuzen 952+8", kind="request", model="kemuzen", batch=1, length=952, tokens=8),
        # the same, decoding above all: eight requests of a chat
        dict(name="dedunex 8x119+24", kind="request", model="dedunex", batch=8, length=119, tokens=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "generate", "request", "request"])
    gpt2 = rng.choice(["gpt2-small", "gpt2-small", "gpt2-medium", "gpt2-xl"])
    if kind == "decode":
        if rng.random() < 0.25:
            return dict(kind=kind, model="gpt2-small", positions=8192, batch=_log(rng, 1, 16), context=_log(rng, 1100, 8180),
                        ragged=rng.random() < 0.5, steps=rng.randint(2, 6))
        return dict(kind=kind, model=gpt2, batch=_log(rng, 1, 64), context=_log(rng, 24, 1010), ragged=rng.random() < 0.5,
                    steps=rng.randint(2, 10))
    if kind == "prompt":
        length = _log(rng, 9, 1024)
        return dict(kind=kind, model=gpt2, prompts=max(1, min(_log(rng, 1, 8), MOST_ROWS // length)), length=length,
                    ragged=rng.random() < 0.5)
    if kind == "mixed":
        return dict(kind=kind, model=gpt2, batch=_log(rng, 1, 48), context=_log(rng, 40, 1000), prompts=rng.randint(1, 3),
                    length=_log(rng, 17, 500))
    if kind == "generate":
        return dict(kind=kind, model="gpt2-small", dtype="float32", batch=_log(rng, 1, 12), length=_log(rng, 8, 200),
                    tokens=rng.randint(4, 24), temperature=rng.choice([0.0, 0.8]))
    return dict(kind=kind, model=rng.choice(["kemuzen", "dedunex"]), batch=_log(rng, 1, 16), length=_log(rng, 24, 980),
                tokens=_log(rng, 2, 32))


# --------------------------------------------------------------------------- models
def _raw_config(case):
    if case["model"] == "kemuzen":
        return bs.kemuzen_like(768, 4, VOCAB)
    if case["model"] == "dedunex":
        return bs.dedunex_like(768, 4, VOCAB)
    with open(_preset_path(case["model"])) as fh:
        raw = json.load(fh)
    if case.get("positions"):
        raw["n_positions"] = case["positions"]
    return raw


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _folder(case):
    return bs.folder_of(_raw_config(case), WEIGHTS_SEED, _dtype(case))


# --------------------------------------------------------------------------- what a pass is made of
def _lengths(n, longest, ragged):
    """``n`` lengths, all the longest or spread between a quarter of it and it, in no order."""
    if not ragged or n == 1:
        return [longest] * n
    order = sorted(range(n), key=lambda i: (i * 37 + 11) % 101)
    return [max(1, round(longest * (0.25 + 0.75 * (k + 1) / n))) for k in order]


def _shape(case):
    """([(tokens kept before the pass, tokens fed in it)], [step: [(request, its first fed token, how many)]])"""
    kind = case["kind"]
    if kind == "decode":
        kept = _lengths(case["batch"], case["context"], case.get("ragged"))
        return [(n, case["steps"]) for n in kept], [[(i, s, 1) for i in range(len(kept))] for s in range(case["steps"])]
    if kind == "prompt":
        fed = _lengths(case["prompts"], case["length"], case.get("ragged"))
        return [(0, n) for n in fed], [[(i, 0, n) for i, n in enumerate(fed)]]
    if kind == "mixed":
        reqs = [(n, 1) for n in _lengths(case["batch"], case["context"], True)]
        reqs += [(0 if i == 0 else case["length"], case["length"]) for i in range(case["prompts"])]
        return reqs, [[(i, 0, fed) for i, (_, fed) in enumerate(reqs)]]
    reqs = [(0, case["length"] + case["tokens"])] * case["batch"]
    steps, per = [], max(1, MOST_ROWS // case["length"])
    for a in range(0, case["batch"], per):
        steps.append([(i, 0, case["length"]) for i in range(a, min(case["batch"], a + per))])
    steps += [[(i, case["length"] + s, 1) for i in range(case["batch"])] for s in range(case["tokens"])]
    return reqs, steps


def _tokens(case, seed):
    """Every request's token ids, kept and fed, from the seed."""
    g = torch.Generator().manual_seed(seed * 7919 + 13)
    return [torch.randint(0, VOCAB, (kept + fed,), generator=g).tolist() for kept, fed in _shape(case)[0]]


def _prompts(case, seed):
    g = torch.Generator().manual_seed(seed * 7919 + 13)
    return [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in _lengths(case["batch"], case["length"], True)]


class _State:
    """An engine, its requests and the tokens that the next passes feed them."""

    def __init__(self, case):
        self.case = case
        self.generates = case["kind"] == "generate"
        if self.generates:
            n, most, rows = case["batch"], case["length"] + case["tokens"], 2048
        else:
            reqs, steps = _shape(case)
            n, most = len(reqs), max(kept + fed for kept, fed in reqs)
            rows = max(2048, max(sum(k for _, _, k in s) for s in steps))
        self.eng = nb.Engine(_folder(case), dtype=_dtype(case), max_tokens=n * (most + 64), max_batch=n, max_rows=rows)

    def keep(self, tokens):
        """Fill the requests with the tokens that they hold before a pass."""
        runner, cache = self.eng.runner, self.eng.cache
        self.reqs = []
        for (kept, _), toks in zip(_shape(self.case)[0], tokens):
            r = cache.open_request() if kept else None
            for a in range(0, kept, runner.max_rows):
                runner.step([StepItem(r, toks[a:min(kept, a + runner.max_rows)])])
            self.reqs.append(r)

    def feed(self, tokens):
        reqs, steps = _shape(self.case)
        self.kept = [kept for kept, _ in reqs]
        self.steps = [[(i, tokens[i][self.kept[i] + a:self.kept[i] + a + k], k - 1) for i, a, k in s] for s in steps]

    def forget(self):
        for r in self.reqs:
            if r is not None:
                self.eng.cache.close_request(r)

    def run(self):
        if self.generates:
            return self.eng.generate(self.prompts, self.params)
        runner, cache = self.eng.runner, self.eng.cache
        live = []
        for r, kept in zip(self.reqs, self.kept):
            if r is None:
                live.append(cache.open_request())
            else:
                cache.truncate(r, kept)
                live.append(r)
        out = []
        for step in self.steps:
            logits = runner.step([StepItem(live[i], toks, [last]) for i, toks, last in step])
            out.append(logits.clone() if len(self.steps) > 1 else logits)   # (valid until the next step)
        for r, mine in zip(live, self.reqs):
            if mine is None:
                cache.close_request(r)
        return out


def prepare(case, seed):
    st = _State(case)
    if st.generates:
        st.params = [nb.SamplingParams(max_new_tokens=case["tokens"], temperature=case["temperature"], top_k=40,
                                       seed=1000 * seed + i) for i in range(case["batch"])]
        st.prompts = _prompts(case, seed + 500009)
        st.run()
        st.run()
        st.prompts = _prompts(case, seed)
        return st
    # (a server has met steps of these shapes before; the fourth is captured at the latest)
    other = _tokens(case, seed + 500009)
    st.keep(other)
    st.feed(other)
    for _ in range(4):
        st.run()
    st.forget()
    mine = _tokens(case, seed)
    st.keep(mine)
    st.feed(mine)
    return st


def run(state):
    return state.run()


# --------------------------------------------------------------------------- what a pass cannot do without
def _stored(case):
    """name -> (shape, bytes) of the checkpoint's tensors."""
    path = os.path.join(_folder(case), "model.safetensors")
    with open(path, "rb") as fh:
        head = json.loads(fh.read(struct.unpack("<Q", fh.read(8))[0]))
    return {k: (v["shape"], v["data_offsets"][1] - v["data_offsets"][0]) for k, v in head.items() if k != "__metadata__"}


def work(case):
    """Per step: every weight read once (of the token and position tables the head's only), the visible cached keys and
    values read once, the new ones and the logits written; two operations a matrix element and row, four a visible key,
    head and value of a head."""
    raw, stored = _raw_config(case), _stored(case)
    size = 4 if case.get("dtype") == "float32" else 2
    if case["model"].startswith("gpt2"):
        c, layers = raw["n_embd"], raw["n_layer"]
        matrix = 12 * c * c * layers
        head = VOCAB * c
        tables = raw["n_positions"] * c * size
        kv_layers = [(0, 2 * c, c)] * layers                     # (window, values kept a position, heads * head size)
        recurrent = 0
    else:
        tables = sum(b for k, (_, b) in stored.items() if k == "side.embed")
        matrix = sum(s[0] * s[1] for k, (s, _) in stored.items() if len(s) == 2 and k.startswith("l") and "conv" not in k)
        head = VOCAB * 768
        tables += stored["embed"][1] if "head" in stored else 0
        if case["model"] == "kemuzen":
            kv_layers = [(512, 2 * 3 * 64, 768), (512, 2 * 3 * 64, 768), (512, 0, 768)]   # (the last reads the one before)
            recurrent = 2 * 12 * 64 * 64
        else:
            kv_layers = [(0, 256 + 32, 768), (512, 3 * 256, 1152), (512, 3 * 256, 1152)]
            recurrent = 768
    weights = sum(b for _, b in stored.values()) - tables
    if case["kind"] == "generate":
        reqs = [(0, n + case["tokens"] - 1) for n in _lengths(case["batch"], case["length"], True)]
        steps = [[(i, 0, fed - case["tokens"] + 1) for i, (_, fed) in enumerate(reqs)]]
        steps += [[(i, fed - case["tokens"] + 1 + s, 1) for i, (_, fed) in enumerate(reqs)] for s in range(case["tokens"] - 1)]
    else:
        reqs, steps = _shape(case)
    total_bytes = total_flops = 0.0
    for step in steps:
        rows = sum(k for _, _, k in step)
        total_bytes += weights + len(step) * VOCAB * 4 + rows * 4
        total_flops += 2.0 * matrix * rows + 2.0 * head * len(step) + 6.0 * recurrent * rows
        for i, a, k in step:
            p0 = reqs[i][0] + a
            for window, kept, dims in kv_layers:
                seen = np.arange(p0 + 1, p0 + k + 1)
                if window:
                    seen = np.minimum(seen, window)
                before = min(p0, window) if window else p0
                total_bytes += (before + k) * kept * size
                total_flops += 4.0 * dims * float(seen.sum())
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if case["kind"] == "generate":
        return {"rel": 0.0, "differ": 0.01}    # a token that falls on the border between two
    # bfloat16 weights, activations and cached keys: 0.0027 to 0.0079 off the 64-bit formulas below, and two runs up to
    # 0.0047 from one another (largest difference 0.023)
    return {"rel": 0.02, "max": 0.1}


# --------------------------------------------------------------------------- the same in 64 bits, plain torch
def _weights64(case):
    """The checkpoint's tensors, in 64 bits on the GPU."""
    path = os.path.join(_folder(case), "model.safetensors")
    kinds = {"BF16": torch.bfloat16, "F32": torch.float32, "I32": torch.int32}
    out = {}
    with open(path, "rb") as fh:
        n = struct.unpack("<Q", fh.read(8))[0]
        head = json.loads(fh.read(n))
        for name, v in head.items():
            if name == "__metadata__":
                continue
            a, b = v["data_offsets"]
            fh.seek(8 + n + a)
            t = torch.frombuffer(bytearray(fh.read(b - a)), dtype=kinds[v["dtype"]]).view(v["shape"])
            out[name] = t.cuda().to(torch.float64)
    return out


def _attend(q, k, v, scale, window=0, keep_first=0, slopes=None, cap=0.0):
    """Causal attention of one sequence: q [n, H, d], k [n, G, d], v [n, G, dv] -> [n, H, dv]."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    kk = k.transpose(0, 1).repeat_interleave(H // G, 0)
    vv = v.transpose(0, 1).repeat_interleave(H // G, 0)
    rows = max(1, (1 << 28) // (H * n))
    j = torch.arange(n, device=q.device)[None, :]
    for a in range(0, n, rows):
        i = torch.arange(a, min(n, a + rows), device=q.device)[:, None]
        s = torch.matmul(q[a:a + rows].transpose(0, 1), kk.transpose(1, 2)) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[:, None, None] * (i - j)
        seen = j <= i
        if window:
            seen = seen & ((i - j < window) | (j < keep_first))
        s = s.masked_fill(~seen, -math.inf)
        out[a:a + rows] = torch.matmul(torch.softmax(s, -1), vv).transpose(0, 1)
    return out


def _layer_norm(x, w, b, eps):
    m = x.mean(-1, keepdim=True)
    return (x - m) / torch.sqrt(((x - m) ** 2).mean(-1, keepdim=True) + eps) * w + b


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _silu(z):
    return z * torch.sigmoid(z)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _gpt2(cfg, w, seqs, wanted):
    """Logits at the wanted positions of every sequence."""
    H, eps = cfg["n_head"], cfg["layer_norm_epsilon"]
    c = cfg["n_embd"]
    x = torch.cat([w["wte.weight"][s] + w["wpe.weight"][:len(s)] for s in seqs])
    bounds = np.cumsum([0] + [len(s) for s in seqs])
    for l in range(cfg["n_layer"]):
        p = "h.%d." % l
        qkv = _layer_norm(x, w[p + "ln_1.weight"], w[p + "ln_1.bias"], eps) @ w[p + "attn.c_attn.weight"] + w[p + "attn.c_attn.bias"]
        q, k, v = (t.reshape(-1, H, c // H) for t in qkv.split(c, 1))
        att = torch.cat([_attend(q[a:b], k[a:b], v[a:b], (c // H) ** -0.5) for a, b in zip(bounds, bounds[1:])]).reshape(-1, c)
        x = x + att @ w[p + "attn.c_proj.weight"] + w[p + "attn.c_proj.bias"]
        h = _layer_norm(x, w[p + "ln_2.weight"], w[p + "ln_2.bias"], eps)
        x = x + _gelu(h @ w[p + "mlp.c_fc.weight"] + w[p + "mlp.c_fc.bias"]) @ w[p + "mlp.c_proj.weight"] + w[p + "mlp.c_proj.bias"]
    rows = torch.cat([x[a + t] for a, t in zip(bounds, wanted)])
    logits = _layer_norm(rows, w["ln_f.weight"], w["ln_f.bias"], eps) @ w["wte.weight"].T
    return logits.split([len(t) for t in wanted])


def _conv(x, taps, bias=0.0):
    """Causal convolution over time, channel by channel; the last tap is the current token's."""
    n, t = x.shape[0], taps.shape[1]
    xx = torch.cat([x.new_zeros(t - 1, x.shape[1]), x])
    return sum(taps[:, j] * xx[j:j + n] for j in range(t)) + bias


def _kemuzen_delta(h, w, p, m, eps):
    n, H, d = h.shape[0], m["heads"], m["dim"]
    q, k, v = (_silu(_conv(h @ w[p + t].T, w[p + t + ".conv"])).view(n, H, -1) for t in "qkv")
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(h @ w[p + "b"].T)
    decay = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
    S, out = h.new_zeros(H, d, m["vdim"]), torch.empty_like(v)
    for t in range(n):
        S = S * decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    out = _rms(out, eps) * w[p + "norm"] * _silu(h @ w[p + "g"].T).view(n, H, -1)
    return out.reshape(n, -1) @ w[p + "o"].T


def _kemuzen_scan(h, w, p, m, eps):
    n, H, dv, N = h.shape[0], m["heads"], m["vdim"], m["state"]
    inner = H * dv
    u = h @ w[p + "in"].T
    z, xbc, dt = u[:, :inner], u[:, inner:2 * inner + 2 * N], u[:, 2 * inner + 2 * N:]
    xbc = _silu(_conv(xbc, w[p + "conv"], w[p + "conv.b"]))
    x, B, C = xbc[:, :inner].view(n, H, dv), xbc[:, inner:inner + N], xbc[:, inner + N:]
    dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"])
    keep = torch.exp(-torch.exp(w[p + "A_log"]) * dt)
    S, y = h.new_zeros(H, N, dv), torch.empty_like(x)
    for t in range(n):
        S = S * keep[t, :, None, None] + B[t, None, :, None] * (dt[t, :, None] * x[t])[:, None, :]
        y[t] = torch.einsum("hnv,n->hv", S, C[t]) + w[p + "D"][:, None] * x[t]
    return (_rms(y.reshape(n, inner) * _silu(z), eps) * w[p + "norm"]) @ w[p + "o"].T


def _kemuzen(cfg, w, seqs, wanted):
    """Gated delta rule, capped and windowed attention that keeps the first tokens, attention beside Mamba-2."""
    eps, width, side = cfg["norm"]["eps"], cfg["width"], cfg["token_side"]["dim"]
    out = []
    for seq, want in zip(seqs, wanted):
        n, tok = len(seq), torch.as_tensor(seq, device="cuda")
        pos = torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
        ang = pos * 10000.0 ** (-2.0 * torch.arange(width // 2, device="cuda", dtype=torch.float64) / width)
        x = w["embed"][tok] * cfg["embedding"]["scale"] + torch.stack([ang.sin(), ang.cos()], -1).view(n, width)
        kv = {}
        for i, layer in enumerate(cfg["layers"]):
            m, p = layer["mixer"], "l%d.mix." % i
            if layer["type"] == "delta":
                y = _kemuzen_delta(x, w, p, m, eps)
            elif layer["type"] == "attention":
                q = _rms((x @ w[p + "q"].T + w[p + "q.b"]).view(n, m["heads"], -1), eps) * w[p + "q.norm"]
                if m.get("kv_from") is None:
                    kv[i] = (_rms((x @ w[p + "k"].T + w[p + "k.b"]).view(n, m["kv_heads"], -1), eps) * w[p + "k.norm"],
                             (x @ w[p + "v"].T + w[p + "v.b"]).view(n, m["kv_heads"], -1))
                k, v = kv[i if m.get("kv_from") is None else m["kv_from"]]
                y = _attend(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], cap=m["softcap"])
                y = y.reshape(n, -1) @ w[p + "o"].T + w[p + "o.b"]
            else:
                a, lp = m["left"], p + "left."
                H = a["heads"]
                q = _rms((x @ w[lp + "q"].T).view(n, H, -1), eps) * w[lp + "q.norm"]
                k = _rms((x @ w[lp + "k"].T).view(n, a["kv_heads"], -1), eps) * w[lp + "k.norm"]
                v = (x @ w[lp + "v"].T).view(n, a["kv_heads"], -1)
                slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, device="cuda", dtype=torch.float64) / H)
                y = _attend(q, k, v, a["scale"], a["mask"]["size"], slopes=slopes) * torch.sigmoid(x @ w[lp + "g"].T)[:, :, None]
                y = y.reshape(n, -1) @ w[lp + "o"].T * m["left_scale"]
                y = y + m["right_scale"] * _kemuzen_scan(x, w, p + "right.", m["right"], eps)
            x = x + _rms(y, eps) * (1.0 + w["l%d.norm1" % i])
            p = "l%d.mlp." % i
            y = (_silu(x @ w[p + "gate"].T) * (x @ w[p + "up"].T)) @ w[p + "down"].T
            x = x + _rms(y, eps) * (1.0 + w["l%d.norm2" % i])
            p = "l%d.side." % i
            y = (_gelu(x @ w[p + "gate"].T) * w["side.embed"][tok][:, i * side:(i + 1) * side]) @ w[p + "proj"].T
            x = x + _rms(y, eps) * w[p + "norm"]
        logits = (_rms(x[want], eps) * (1.0 + w["final.norm"])) @ w["embed"].T
        out.append(cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"]))
    return out


def _frequencies(rot):
    dims, base, sc = rot["dims"], rot["base"], rot.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not sc:
        return f, 1.0
    at = [dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base)) for turns in (sc["fast"], sc["slow"])]
    lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [fi / sc["factor"] * r + fi * (1.0 - r) for fi, r in zip(f, ramp)], 0.1 * math.log(sc["factor"]) + 1.0


def _rotate(x, rot):
    """x [n, heads, d]: value i of the first ``dims`` turns with value i + dims / 2."""
    dims = rot["dims"]
    f, amp = _frequencies(rot)
    ang = torch.arange(x.shape[0], device=x.device, dtype=x.dtype)[:, None] * torch.tensor(f, device=x.device, dtype=x.dtype)
    c, s = (ang.cos() * amp)[:, None], (ang.sin() * amp)[:, None]
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _dedunex(cfg, w, seqs, wanted):
    """Differential attention, attention through a latent, the minimal gated recurrent unit, a grouped norm."""
    eps, groups = cfg["norm"]["eps"], cfg["norm"]["groups"]

    def norm(x, weight):
        return _rms(x.view(x.shape[0], groups, -1), eps).reshape(x.shape) * weight

    out = []
    for seq, want in zip(seqs, wanted):
        n = len(seq)
        x = norm(w["embed"][torch.as_tensor(seq, device="cuda")], w["embed.norm"])
        for i, layer in enumerate(cfg["layers"]):
            if i == cfg["loop"]["start"]:
                x = x + w["loop.step"][0]
            m, p = layer["mixer"], "l%d.mix." % i
            h = norm(x, w["l%d.norm1" % i])
            if layer["type"] == "attention":
                q = _rotate(_rms((h @ w[p + "q"].T + w[p + "q.b"]).view(n, 2 * m["heads"], -1), eps) * w[p + "q.norm"], m["rot"])
                k = _rotate(_rms((h @ w[p + "k"].T + w[p + "k.b"]).view(n, 2 * m["kv_heads"], -1), eps) * w[p + "k.norm"], m["rot"])
                v = (h @ w[p + "v"].T + w[p + "v.b"]).view(n, m["kv_heads"], -1)
                lam = torch.exp((w[p + "lq1"] * w[p + "lk1"]).sum()) - torch.exp((w[p + "lq2"] * w[p + "lk2"]).sum()) + m["diff"]
                one, two = (_attend(q[:, t::2], k[:, t::2], v, m["scale"], m["mask"]["size"], cap=m["softcap"]) for t in (0, 1))
                y = (_rms(one - lam * two, eps) * (1.0 - m["diff"])).reshape(n, -1) @ w[p + "o"].T
            elif layer["type"] == "latent_attention":
                H, d, R = m["heads"], m["dim"], m["kv_rank"]
                q = ((_rms(h @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T).view(n, H, -1)
                kv = h @ w[p + "dkv"].T
                c = _rms(kv[:, :R], eps) * w[p + "dkv.norm"]
                kr = _rotate(kv[:, None, R:], m["rot"]).expand(n, H, -1)
                k = torch.cat([(c @ w[p + "uk"].T).view(n, H, d), kr], -1)
                q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"])], -1)
                y = _attend(q, k, (c @ w[p + "uv"].T).view(n, H, -1), m["scale"]) * torch.sigmoid(h @ w[p + "g"].T)[:, :, None]
                y = y.reshape(n, -1) @ w[p + "o"].T
            else:
                z = torch.sigmoid(h @ w[p + "z"].T + w[p + "z.b"])
                u = h @ w[p + "x"].T + w[p + "x.b"]
                cand = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
                S, y = torch.zeros_like(z[0]), torch.empty_like(z)
                for t in range(n):
                    S = (1.0 - z[t]) * S + z[t] * cand[t]
                    y[t] = S
                y = (y * _silu(h @ w[p + "g"].T)) @ w[p + "o"].T
            p = "l%d.mlp." % i
            x = x + y + (_gelu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T
        out.append(norm(x[want], w["final.norm"]) @ w["head"].T)
    return out


def exact(case, seed):
    """The logits of ``run`` from whole sequences, without a cache; None for generated tokens."""
    if case["kind"] == "generate":
        return None
    reqs, steps = _shape(case)
    tokens = _tokens(case, seed)
    wanted = [[] for _ in reqs]
    places = []
    for step in steps:
        places.append([(i, len(wanted[i])) for i, _, _ in step])
        for i, a, k in step:
            wanted[i].append(reqs[i][0] + a + k - 1)
    with open(os.path.join(_folder(case), "config.json")) as fh:
        cfg = json.load(fh)
    model = {"kemuzen": _kemuzen, "dedunex": _dedunex}.get(case["model"], _gpt2)
    with torch.no_grad():
        logits = model(cfg, _weights64(case), tokens, wanted)
    return [torch.stack([logits[i][at] for i, at in step]) for step in places]
