"""Work that a program has the engine do, as cases to time and to compare: steps of Engine.step over models in a folder.

A case is a model (`family`, `width`, `heads`, `inner`, `vocab`, `layers`, `dtype`, and for GPT-2 its `positions`) and one
step of it (`work`):

  prompt   `requests` new prompts of `shortest` to `longest` tokens in one step, logits wanted at four places of each
  decode   one token of each of `requests` running requests, whose contexts are `shortest` to `longest` tokens long
  mixed    the same beside a portion of `chunk` tokens of a new prompt

Few layers stand for a model's many: a layer's kernels, launches and tolerance show best where few of them follow one
another.  Two cases are whole models.  The model folder is written from the seed (safetensors in the case's type) and read
with load_model, as a program reads its weights.  Sizes are those of configs/*.json, of the two tiny models the tests
use, and of the layers bench.py compares the other designs at.
"""
from __future__ import annotations

import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

from sandyrt_b200.config.base import config_from_normalised
from sandyrt_b200.engine.step import Engine, StepEntry
from sandyrt_b200.models.model import build_model, load_model

ROOM = 256          # tokens a running request may still add to its context before another takes its place

TINY_A = dict(family="gpt2", width=64, heads=4, inner=256, vocab=512, positions=128, layers=2)
SMALL = dict(family="gpt2", width=768, heads=12, inner=3072, vocab=50257, positions=1024)
MEDIUM = dict(family="gpt2", width=1024, heads=16, inner=4096, vocab=50257, positions=1024)
XL = dict(family="gpt2", width=1600, heads=25, inner=6400, vocab=50257, positions=1024)
# bench.py --hybrid / --latent: heads of 64, an inner size that gives the gated feed-forward as many parameters
PANUPEL = dict(family="panupel", width=768, heads=12, inner=2048, vocab=50257, positions=0, layers=2)
SOVEZEN = dict(family="sovezen", width=768, heads=12, inner=2048, vocab=50257, positions=0, layers=4)


def _case(name, model, dtype, work, requests, shortest, longest, chunk=0, **more):
    return dict(model, **more, name=name, dtype=dtype, work=work, requests=requests, shortest=shortest, longest=longest, chunk=chunk)


def listed():
    return [
        # the smallest call there is in earnest: a test or a first try with three short prompts
        _case("gpt2_tiny_prompts_fp32", TINY_A, "float32", "prompt", 3, 5, 33),
        # one user waiting for the next token: a whole model, latency and launches
        _case("gpt2_small_decode_1", SMALL, "bfloat16", "decode", 1, 384, 384, layers=12),
        # a server's decode step with many requests of different ages
        _case("gpt2_small_decode_64", SMALL, "bfloat16", "decode", 64, 64, 448, layers=4),
        # two prompts that fill the context, the whole model
        _case("gpt2_small_prompts_2x1024", SMALL, "bfloat16", "prompt", 2, 1024, 1024, layers=12),
        # continuous batching: a new prompt's portion beside the tokens of running requests
        _case("gpt2_medium_mixed", MEDIUM, "bfloat16", "mixed", 32, 100, 700, chunk=480, layers=4),
        # ragged prompts admitted together, the widest layers
        _case("gpt2_xl_prompts_8", XL, "bfloat16", "prompt", 8, 64, 447, layers=2),
        # decode of the widest layers, where weights are the traffic
        _case("gpt2_xl_decode_16", XL, "bfloat16", "decode", 16, 65, 512, layers=2),
        # the 32-bit path: a few requests, and prompts that fill the context
        _case("gpt2_small_decode_8_fp32", SMALL, "float32", "decode", 8, 128, 512, layers=4),
        _case("gpt2_small_prompts_2x1024_fp32", SMALL, "float32", "prompt", 2, 1024, 1024, layers=4),
        # delta rule and matrix memory beside attention: long prompts, and a few requests' tokens
        _case("panupel_prompts_2x1024", PANUPEL, "bfloat16", "prompt", 2, 1024, 1024),
        _case("panupel_decode_8", PANUPEL, "bfloat16", "decode", 8, 128, 512),
        # attention over a latent and routed experts, in 32 bits, where rounding does not change who is routed where
        _case("sovezen_prompts_4_fp32", SOVEZEN, "float32", "prompt", 4, 100, 412),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        family = rng.choice(["gpt2"] * 7 + ["panupel"] * 2 + ["sovezen"])
        dtype = "float32" if family == "sovezen" else rng.choice(["bfloat16", "bfloat16", "float32"])
        if family == "gpt2" and rng.random() < 0.15:        # small heads and odd inner sizes
            size = rng.choice([16, 32])
            heads = rng.randint(2, 6)
            width, inner = size * heads, 32 * rng.randint(4, 16)
            vocab = rng.randint(300, 2000)
        else:
            heads = rng.choice([3, 6, 12, 18, 24]) if family != "gpt2" else rng.randint(4, 25)
            width, vocab = 64 * heads, rng.choice([1000, 50257])
            inner = 4 * width if family == "gpt2" else 64 * round(width * 8 / 3 / 64)
        work = rng.choice(["prompt", "decode", "mixed"])
        shortest = _log_int(rng, 5, 512)
        case = dict(family=family, width=width, heads=heads, inner=inner, vocab=vocab, positions=1024 if family == "gpt2" else 0,
                    layers={"panupel": 2, "sovezen": 4}.get(family) or rng.randint(1, 4), dtype=dtype, work=work,
                    requests=_log_int(rng, 1, 8 if work == "prompt" else 64), shortest=shortest,
                    longest=min(rng.randint(shortest, 2 * shortest), 760), chunk=_log_int(rng, 16, 700) if work == "mixed" else 0)
        tokens = sum(_lengths(case)) if work == "prompt" else case["requests"] + case["chunk"]
        if tokens <= 2048 and _flops(case) <= (1e11 if dtype == "float32" else 3e11):
            return case


# ---- the model of a case -----------------------------------------------------------------------------------
def _config(case):
    """The case's config.json."""
    if case["family"] == "gpt2":
        return {"architectures": ["GPT2LMHeadModel"], "model_type": "gpt2", "n_layer": case["layers"], "n_embd": case["width"],
                "n_head": case["heads"], "n_positions": case["positions"], "vocab_size": case["vocab"], "n_inner": case["inner"],
                "layer_norm_epsilon": 1e-5, "activation_function": "gelu_new"}
    heads, ff = case["heads"], case["inner"]
    if case["family"] == "panupel":
        kv = heads // 3
        delta = {"type": "delta", "mixer": {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 64, "conv": 4},
                 "mlp": {"kind": "dense", "ff": ff}}
        # the parallel layer's heads are split between attention and the matrix memory
        left, right = (heads // 2, heads // 4) if heads % 2 == 0 and heads >= 6 else (heads - 1, 1)
        groups = max(kv // 2, 1) if left % max(kv // 2, 1) == 0 else 1
        par = {"type": "parallel", "mlp": {"kind": "dense", "ff": ff},
               "mixer": {"left": {"heads": left, "kv_heads": groups, "dim": 64, "vdim": 64, "scale": 0.125,
                                  "rot": {"dims": 64, "base": 10000.0}},
                         "right": {"heads": right, "dim": 64, "vdim": 128, "gate_cap": 12.0}, "left_scale": 1.0, "right_scale": 1.0}}
        return {"architecture": "Panupel", "vocab": case["vocab"], "width": case["width"], "norm": {"eps": 1e-6}, "residual_mult": 1.0,
                "layers": [delta if i % 2 == 0 else par for i in range(case["layers"])]}
    rot = {"type": "latent_attention", "mixer": {"heads": heads, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 96,
                                                 "scale": 96 ** -0.5, "rot": {"dims": 32, "base": 10000.0}}}
    lat = {"type": "latent_attention_2", "mixer": {"heads": heads, "dim": 64, "vdim": 64, "kv_rank": 128,
                                                   "q_rank": case["width"] // 2, "scale": 0.125}}
    dense = {"kind": "dense", "ff": ff}
    moe = {"kind": "moe", "expert": {"ff": ff // 2}, "router": {"experts": 16, "top": 2}}
    order = [(rot, dense), (lat, moe), (lat, dense), (rot, moe)]
    return {"architecture": "Sovezen", "vocab": case["vocab"], "width": case["width"], "norm": {"eps": 1e-6}, "logit_scale": 1.0,
            "layers": [{**order[i % 4][0], "mlp": order[i % 4][1]} for i in range(case["layers"])]}


def _requests(case):
    return build_model(config_from_normalised(_config(case))).tensor_requests()


def _weights(case, seed):
    """The model's tensors by name, on the GPU, in the type in which the file stores them."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)
    store = getattr(torch, case["dtype"])
    out = {}
    for name, r in sorted(_requests(case).items()):
        t = torch.randn(r.shape, generator=gen, device="cuda")
        if name.endswith(".A_log"):                 # decay rates of 1 to 16 ...
            t = torch.rand(r.shape, generator=gen, device="cuda") * math.log(16.0)
        elif name.endswith(".dt_bias"):             # ... times steps of 0.001 to 0.1: states remember tens to thousands of tokens
            dt = torch.exp(torch.rand(r.shape, generator=gen, device="cuda") * math.log(100.0) + math.log(1e-3))
            t = torch.log(torch.expm1(dt))
        elif name.endswith(".f.b"):                 # forget gates open
            t = 3.0 + 3.0 * torch.rand(r.shape, generator=gen, device="cuda")
        elif name.endswith(".conv"):
            t = t * 0.5
        elif name.endswith(".sink"):
            pass
        elif r.init == "gamma":
            t = 1.0 + 0.02 * t
        else:
            t = t * (0.01 if r.init == "bias" else 0.02)
        out[name] = t.to(torch.float32 if r.keep_32bit else store)
    return out


def _write_folder(folder, config, tensors):
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(config, f)
    names, header, at = list(tensors), {}, 0
    for n in names:
        t = tensors[n]
        size = t.numel() * t.element_size()
        header[n] = {"dtype": "F32" if t.dtype == torch.float32 else "BF16", "shape": list(t.shape), "data_offsets": [at, at + size]}
        at += size
    head = json.dumps(header).encode()
    head += b" " * (-len(head) % 8)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(head)))
        f.write(head)
        for n in names:
            f.write(memoryview(tensors[n].contiguous().reshape(-1).view(torch.uint8).cpu().numpy()))


def _lengths(case):
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    return [lo + (hi - lo) * i // (n - 1) for i in range(n)] if n > 1 else [hi]


def _wanted(n):
    """Four places of a prompt, its last among them."""
    return sorted({n // 4, n // 2, 3 * n // 4, n - 1})


def _room(case):
    return min(ROOM, case["positions"] - case["longest"]) if case["positions"] else ROOM


def _tokens(case, seed):
    """The prompts, the tokens that running requests add one after another, and the portion of a new prompt."""
    rng = np.random.default_rng(int(seed))
    ids = lambda n: rng.integers(0, case["vocab"], size=n).tolist()
    prompts = [ids(n) for n in _lengths(case)]
    return prompts, [ids(case["requests"]) for _ in range(_room(case))], ids(case["chunk"])


class _State:
    pass


def prepare(case, seed):
    s = _State()
    with tempfile.TemporaryDirectory(dir="/dev/shm" if os.path.isdir("/dev/shm") else None) as folder:
        _write_folder(folder, _config(case), _weights(case, seed))
        model = load_model(folder, dtype=getattr(torch, case["dtype"]))
    s.work = case["work"]
    s.prompts, s.nexts, s.chunk = _tokens(case, seed)
    held = sum(len(p) + (0 if s.work == "prompt" else ROOM) + 16 for p in s.prompts) + len(s.chunk) + 64
    s.engine = Engine(model, max_tokens=held, max_requests=max(case["requests"] + 1, 2), max_step_tokens=4096)
    s.at = 0
    if s.work != "prompt":
        _fill(s)
    return s


def _fill(s):
    """New requests with the contexts of the case."""
    batch, n = [], 0
    for i, p in enumerate(s.prompts):
        if s.at:
            s.engine.release(i)
        if batch and n + len(p) > 2048:
            s.engine.step(batch)
            batch, n = [], 0
        batch.append(StepEntry(i, p, []))
        n += len(p)
    s.engine.step(batch)
    s.at = 0


def run(s):
    if s.work == "prompt":
        logits = s.engine.step([StepEntry(i, p, _wanted(len(p))) for i, p in enumerate(s.prompts)])
        for i in range(len(s.prompts)):
            s.engine.release(i)
        return logits
    if s.at == len(s.nexts):
        _fill(s)                    # the requests have ended; others take their place
    entries = [StepEntry(i, [t], [0]) for i, t in enumerate(s.nexts[s.at])]
    s.at += 1
    if s.work == "decode":
        return s.engine.step(entries)
    logits = s.engine.step(entries + [StepEntry("new", s.chunk, [len(s.chunk) - 1])])
    s.engine.release("new")
    return logits


# ---- what a pass cannot do without ------------------------------------------------------------------------
def _pass(case):
    """(tokens run, pairs of a token and a token it attends to, tokens read from the cache, rows of logits)"""
    lens = _lengths(case)
    if case["work"] == "prompt":
        return sum(lens), sum(n * (n + 1) // 2 for n in lens), 0, sum(len(_wanted(n)) for n in lens)
    c = case["chunk"]
    return len(lens) + c, sum(n + 1 for n in lens) + c * (c + 1) // 2, sum(lens), len(lens) + (1 if c else 0)


def _counted(case):
    """(weights read, weights a token is multiplied with, elements a cached token has, state elements a request has, flops a
    pair takes, flops of the recurrences a token takes), over the layers"""
    w, h, ff, n = case["width"], case["heads"], case["inner"], case["layers"]
    if case["family"] == "gpt2":
        p = n * (4 * w * w + 2 * w * ff)
        return p, p, n * 2 * w, 0, n * 4 * w, 0
    weights = active = row = state = pair = rec = 0
    for spec in _config(case)["layers"]:
        m = spec["mixer"]
        if spec["type"] == "delta":
            p = w * (2 * m["kv_heads"] * 64 + 3 * h * 64)
            state += h * 64 * 64 + 3 * (2 * m["kv_heads"] + h) * 64
            rec += 6 * h * 64 * 64
        elif spec["type"] == "parallel":
            a, b = m["left"], m["right"]
            p = w * (2 * a["heads"] + 2 * a["kv_heads"]) * 64 + w * b["heads"] * (2 * 64 + 3 * 128)
            row += 2 * a["kv_heads"] * 64
            state += b["heads"] * (64 * 128 + 64 + 1)
            pair += 4 * a["heads"] * 64
            rec += 5 * b["heads"] * 64 * 128
        else:
            r, q = m["kv_rank"], m.get("q_rank")
            width = r + m.get("rot_dim", 0)
            p = w * width + 2 * h * 64 * r + h * 64 * w + (q * (w + h * 64) if q else w * h * (64 + m["rot_dim"]))
            row += width
            pair += 2 * h * (width + r)
        mlp = spec["mlp"]
        every, used = (3 * w * ff, 3 * w * ff) if mlp["kind"] == "dense" else (16 * w * ff + 16 * w, 2 * w * ff + 16 * w)
        weights, active = weights + p + every, active + p + used
    return weights, active, row, state, pair, rec


def _flops(case):
    tokens, pairs, _, rows = _pass(case)
    _, active, _, _, pair, rec = _counted(case)
    return 2.0 * tokens * active + pairs * pair + tokens * rec + 2.0 * rows * case["width"] * case["vocab"]


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    tokens, _, cached, rows = _pass(case)
    weights, _, row, state, _, _ = _counted(case)
    moved = size * (weights + case["vocab"] * case["width"] + row * (tokens + cached)) + 4 * rows * case["vocab"]
    moved += 4 * state * case["requests"] * (1 if case["work"] == "prompt" else 2)
    return {"bytes": float(moved), "flops": float(_flops(case))}


def tolerance(case):
    # About four times what the path shows against 64 bits: 2e-6 in 32 bits, 4.6e-3 in 16, where a model of 12 layers and one
    # of a single layer differ little; the other design's norms behind every sublayer bring a sublayer's rounding to the
    # stream's full size, and its layers show 1.4e-2.
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 3e-2 if case["family"] == "panupel" else 2e-2}


# ---- the same in 64 bits ----------------------------------------------------------------------------------
def _linear(x, w):
    return x @ w.t()


def _rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _causal(q, k, v, scale, sink=None):
    """q [T, H, n], k [T, G, n], v [T, G, e] -> [T, H, e]; exp(sink) joins the softmax's denominator."""
    T, H, _ = q.shape
    k, v = (t.repeat_interleave(H // t.shape[1], dim=1) for t in (k, v))
    s = torch.einsum("ihn,jhn->hij", q, k) * scale
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1), -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.view(H, 1, 1).expand(H, T, 1)], dim=-1)
    p = torch.softmax(s, dim=-1)[..., :T]
    return torch.einsum("hij,jhe->ihe", p, v)


def _angles(T, dims, base, device):
    f = float(base) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=device) / dims)
    a = torch.arange(T, dtype=torch.float64, device=device)[:, None] * f
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _rotate_halves(x, dims, base):
    c, s = _angles(x.shape[0], dims, base, x.device)
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], dim=-1)


def _rotate_pairs(x, dims, base):
    c, s = _angles(x.shape[0], dims, base, x.device)
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2), x[..., dims:]], dim=-1)


def _gpt2(case, w, ids):
    H, T = case["heads"], len(ids)
    norm = lambda x, n: torch.nn.functional.layer_norm(x, x.shape[-1:], w[n + ".weight"], w[n + ".bias"], 1e-5)
    conv = lambda x, n: x @ w[n + ".weight"] + w[n + ".bias"]
    x = w["wte.weight"][ids] + w["wpe.weight"][:T]
    for i in range(case["layers"]):
        p = f"h.{i}."
        q, k, v = (t.view(T, H, -1) for t in conv(norm(x, p + "ln_1"), p + "attn.c_attn").chunk(3, dim=-1))
        x = x + conv(_causal(q, k, v, q.shape[-1] ** -0.5).reshape(T, -1), p + "attn.c_proj")
        u = conv(norm(x, p + "ln_2"), p + "mlp.c_fc")
        u = 0.5 * u * (1 + torch.tanh(math.sqrt(2 / math.pi) * (u + 0.044715 * u ** 3)))
        x = x + conv(u, p + "mlp.c_proj")
    return norm(x, "ln_f"), w["wte.weight"]


def _delta(m, w, p, h, eps):
    H, G, T = m["heads"], m["kv_heads"], h.shape[0]
    silu = torch.nn.functional.silu

    def conv(n, heads):
        taps = w[p + n + ".conv"]
        x = torch.cat([torch.zeros(taps.shape[1] - 1, taps.shape[0], dtype=h.dtype, device=h.device), _linear(h, w[p + n])])
        return silu(sum(x[j:j + T] * taps[:, j] for j in range(taps.shape[1]))).view(T, heads, 64)
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q = (unit(conv("q", G)) / 8.0).repeat_interleave(H // G, dim=1)
    k = unit(conv("k", G)).repeat_interleave(H // G, dim=1)
    v = conv("v", H)
    beta = torch.sigmoid(_linear(h, w[p + "b"]))
    decay = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(_linear(h, w[p + "a"]) + w[p + "dt_bias"]))
    S, out = torch.zeros(H, 64, 64, dtype=h.dtype, device=h.device), []
    for t in range(T):
        S = S * decay[t].view(H, 1, 1)
        u = beta[t].view(H, 1) * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
        S = S + k[t].unsqueeze(2) * u.unsqueeze(1)
        out.append(torch.einsum("hde,hd->he", S, q[t]))
    o = _rms(torch.stack(out), w[p + "norm"], eps).reshape(T, -1) * silu(_linear(h, w[p + "g"]))
    return _linear(o, w[p + "o"])


def _matrix_memory(m, w, p, h, eps):
    H, cap, T = m["heads"], m["gate_cap"], h.shape[0]
    q, k, v = (_linear(h, w[p + n]).view(T, H, -1) for n in ("q", "k", "v"))
    q = q / 8.0
    gate = lambda n: cap * torch.tanh((_linear(h, w[p + n]) + w[p + n + ".b"]) / cap)
    log_i, log_f = gate("i"), torch.nn.functional.logsigmoid(gate("f"))
    S = torch.zeros(H, 64, v.shape[-1], dtype=h.dtype, device=h.device)
    n, top, out = S[:, :, 0], S[:, 0, 0], []
    for t in range(T):
        new = torch.maximum(log_f[t] + top, log_i[t])
        a, b, top = torch.exp(log_f[t] + top - new).unsqueeze(1), torch.exp(log_i[t] - new).unsqueeze(1), new
        S = a.unsqueeze(2) * S + (b * k[t]).unsqueeze(2) * v[t].unsqueeze(1)
        n = a * n + b * k[t]
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out.append(torch.einsum("hde,hd->he", S, q[t]) / den.unsqueeze(1))
    o = _rms(torch.stack(out), None, eps).reshape(T, -1) * w[p + "norm"] * torch.sigmoid(_linear(h, w[p + "g"]))
    return _linear(o, w[p + "o"])


def _left(m, w, p, h, eps):
    T = h.shape[0]
    q = _rms(_linear(h, w[p + "q"]), w[p + "q.norm"], eps).view(T, m["heads"], 64)
    k = _rms(_linear(h, w[p + "k"]), w[p + "k.norm"], eps).view(T, m["kv_heads"], 64)
    v = _linear(h, w[p + "v"]).view(T, m["kv_heads"], 64)
    q, k = (_rotate_halves(t, m["rot"]["dims"], m["rot"]["base"]) for t in (q, k))
    o = _causal(q, k, v, m["scale"], w[p + "sink"]) * torch.sigmoid(_linear(h, w[p + "g"])).unsqueeze(2)
    return _linear(o.reshape(T, -1), w[p + "o"])


def _gated(w, p, h):
    return _linear(torch.nn.functional.silu(_linear(h, w[p + "gate"])) * _linear(h, w[p + "up"]), w[p + "down"])


def _panupel(case, w, ids):
    c = _config(case)
    eps = c["norm"]["eps"]
    x = w["embed"][ids]
    for i, spec in enumerate(c["layers"]):
        p, m = f"l{i}.", spec["mixer"]
        h = _rms(x, w[p + "norm1"], eps)
        if spec["type"] == "delta":
            y = _delta(m, w, p + "mix.", h, eps)
        else:
            y = _left(m["left"], w, p + "mix.left.", h, eps) + _matrix_memory(m["right"], w, p + "mix.right.", h, eps)
        x = x + _rms(y, w[p + "norm1b"], eps)
        x = x + _rms(_gated(w, p + "mlp.", _rms(x, w[p + "norm2"], eps)), w[p + "norm2b"], eps)
    return _rms(x, w["final.norm"], eps), w["head"]


def _latent(spec, w, p, h, eps):
    m, T, H = spec["mixer"], h.shape[0], spec["mixer"]["heads"]
    down, r = _linear(h, w[p + "dkv"]), m["kv_rank"]
    latent = _rms(down[:, :r], w[p + "dkv.norm"], eps)
    k, v = _linear(latent, w[p + "uk"]).view(T, H, 64), _linear(latent, w[p + "uv"]).view(T, H, 64)
    if spec["type"] == "latent_attention_2":
        q = _linear(_rms(_linear(h, w[p + "dq"]), w[p + "dq.norm"], eps), w[p + "uq"]).view(T, H, 64)
        o = _causal(q, k, v, m["scale"])
    else:
        q = _linear(h, w[p + "q"]).view(T, H, -1)
        turn = lambda x: _rotate_pairs(x, m["rot"]["dims"], m["rot"]["base"])
        q = torch.cat([q[..., :64], turn(q[..., 64:])], dim=-1)
        k = torch.cat([k, turn(down[:, r:].unsqueeze(1)).expand(T, H, -1)], dim=-1)
        o = _causal(q, k, v, m["scale"], w[p + "sink"])
    return _linear(o.reshape(T, -1), w[p + "o"])


def _routed(mlp, w, p, h):
    z = _linear(h, w[p + "router"]) + w[p + "router.b"]
    top, who = z.topk(mlp["router"]["top"], dim=-1)
    weight, out = torch.softmax(top, dim=-1), torch.zeros_like(h)
    for e in range(mlp["router"]["experts"]):
        rows, place = (who == e).nonzero(as_tuple=True)
        y = _linear(torch.relu(_linear(h[rows], w[p + f"e{e}.up"])) ** 2, w[p + f"e{e}.down"])
        out.index_add_(0, rows, weight[rows, place].unsqueeze(1) * y)
    return out


def _sovezen(case, w, ids):
    c = _config(case)
    eps = c["norm"]["eps"]
    x = w["embed"][ids]
    for i, spec in enumerate(c["layers"]):
        p, mlp = f"l{i}.", spec["mlp"]
        h = _rms(x, w[p + "norm1"], eps)
        f = _gated(w, p + "mlp.", h) if mlp["kind"] == "dense" else _routed(mlp, w, p + "mlp.", h)
        x = x + _latent(spec, w, p + "mix.", h, eps) * w[p + "ls1"] + f * w[p + "ls2"]
    return _rms(x, w["final.norm"], eps), w["embed"]


def exact(case, seed):
    w = {n: t.to(torch.float64) for n, t in _weights(case, seed).items()}
    prompts, nexts, chunk = _tokens(case, seed)
    if case["work"] == "prompt":
        asked = [(p, _wanted(len(p))) for p in prompts]
    else:
        asked = [(p + [t], [len(p)]) for p, t in zip(prompts, nexts[0])] + ([(chunk, [len(chunk) - 1])] if chunk else [])
    forward = {"gpt2": _gpt2, "panupel": _panupel, "sovezen": _sovezen}[case["family"]]
    rows, head = [], None
    for ids, want in asked:
        x, head = forward(case, w, torch.tensor(ids, device="cuda"))
        rows.append(x[want])
    return _linear(torch.cat(rows), head)
