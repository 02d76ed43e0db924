"""Kernel micro-benchmarks: one kernel alone, inside a CUDA graph, on inputs larger than L2.

    python -m sandyrt_b200.csrc.microbench decode-attention [--heads 12] [--head-dim 64] [--page-size 16]
    python -m sandyrt_b200.csrc.microbench gemm [--rows 2048] [--width 768] [--inner 3072] [--layers 48] [--k-sweep]
    python -m sandyrt_b200.csrc.microbench prefill-attention [--heads 12] [--page-size 16] [--shape 2x1024+0 ...]
    python -m sandyrt_b200.csrc.microbench grouped [--tokens 2048 8] [--experts 16] [--top 2] [--width 1536] [--inner 2048]
    python -m sandyrt_b200.csrc.microbench gemm-f32 [--rows 1 8 24 2048] [--shape 2304x768 ...]
    python -m sandyrt_b200.csrc.microbench attention-f32 [--heads 12] [--head-dim 64] [--shape 2x1024+0 ...]
    python -m sandyrt_b200.csrc.microbench mixed-attention [--heads 16] [--context 400] [--portions 1x480] [--singles 8 16 32]
    python -m sandyrt_b200.csrc.microbench recurrences [--lengths 1024 1024] [--heads 12]

decode-attention: the register kernel and the bulk-copy kernel of single-token attention on
several (tokens, context) shapes.  Each timing replays a graph of one launch per distinct cache
(enough caches to exceed L2), so neither the host's launch cost nor a warm L2 is in the number;
bytes are the keys and values a launch must read.

prefill-attention: the mma.sync kernel and the tcgen05 kernel of prompt attention (heads of 64)
on shapes given as REQUESTSxNEW+CACHED, with the requests' pages one after another in the cache
and scattered; FLOP are those of the causal part (4 * head * keys seen, per query and head).
"""
from __future__ import annotations

import argparse
import sys

import torch

from . import ops


def _time_graph(fn, layers: int, reps: int = 3) -> float:
    """Microseconds per call of fn(l), l = 0..layers-1, replayed from a CUDA graph."""
    for l in range(layers):
        fn(l)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        fn(0)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            for l in range(layers):
                fn(l)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        graph.replay()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) * 1e3 / (reps * layers)


def decode_attention(a) -> int:
    dev = torch.device("cuda:0")
    H, D, PS = a.heads, a.head_dim, a.page_size
    print("tokens context  kernel    splits       us     GB/s")
    shapes = [tuple(int(v) for v in sh.split("x")) for sh in a.shape]
    for T, ctx in shapes:
        blocks = -(-ctx // PS)
        pages = T * blocks
        bytes_per_launch = T * ctx * H * D * 2 * 2
        layers = min(48, max(2, int(400e6 // bytes_per_launch) + 1))
        arena = torch.randn(layers, pages, 2, H, PS, D, device=dev, dtype=torch.bfloat16)
        table = torch.randperm(pages, device=dev).to(torch.int32).view(T, blocks).contiguous()
        q = torch.randn(T, H * D, device=dev, dtype=torch.bfloat16)
        seq = torch.arange(T, device=dev, dtype=torch.int32)
        pos = torch.full((T,), ctx - 1, device=dev, dtype=torch.int32)
        out = torch.empty_like(q)
        splits = min(ops.decode_splits(T, H, blocks * PS), ops.CLUSTER_MAX_SPLITS)
        kernels = [("register", dict(bulk=False)), ("bulk", dict(bulk=True))]
        if D == 64:
            kernels.append(("mma.sync", dict(mma=True)))
        for name, which in kernels:
            def go(l, which=which):
                ops.decode_attention(q, arena[l, :, 0], arena[l, :, 1], table, seq, pos, out, n_heads=H,
                                     scale=D ** -0.5, num_splits=splits, cluster=True, **which)
            us = _time_graph(go, layers)
            print(f"{T:6d} {ctx:7d}  {name:8s} {splits:6d} {us:8.2f} {bytes_per_launch / us / 1e3:8.0f}", flush=True)
        ops.check_kernel_status(dev)
        del arena
    return 0


def gemm(a) -> int:
    """The tcgen05 product at the shapes of a prompt step, every tile choice; activations and
    weights of --layers distinct layers (48 by default: 170 to 230 MB of weights per shape, more
    than L2 holds, so the weights come from memory as they do in a model)."""
    dev = torch.device("cuda:0")
    M = a.rows
    shapes = [("q/k/v", 3 * a.width, a.width, None, False), ("out-projection", a.width, a.width, None, True),
              ("up-projection", a.inner, a.width, "gelu_new", False), ("down-projection", a.width, a.inner, None, True)]
    print(f"rows {M}; us per launch (TFLOP/s) by tile width; negative: one tile per CTA; 2000+: two CTAs a tile")
    layers = a.layers
    for name, N, K, act, res in shapes:
        # inputs are a kernel's output in a model and sit in L2; four of them take turns here
        x4 = [torch.randn(M, K, device=dev, dtype=torch.bfloat16) for _ in range(4)]
        xs = [x4[l % 4] for l in range(layers)]
        ws = [torch.randn(N, K, device=dev, dtype=torch.bfloat16) * 0.05 for _ in range(layers)]
        bias = torch.randn(N, device=dev, dtype=torch.bfloat16)
        # the residual products add into the float32 stream in place, as the blocks do
        out = torch.zeros(M, N, device=dev, dtype=torch.float32 if res else torch.bfloat16)
        resid = out if res else None
        line = f"{name:16s} {M}x{N}x{K}:"
        for tile in ops.GEMM_VARIANTS:
            def go(l, tile=tile):
                ops.gemm_tc(xs[l], ws[l], bias, out, act=act, residual=resid, tile_n=tile)
            us = _time_graph(go, layers)
            line += f"  {tile:5d}: {us:6.1f} ({2.0 * M * N * K / us / 1e6:5.0f})"
        if M <= ops.SKINNY_MAX_ROWS:
            def go_skinny(l):
                ops.gemm_skinny(xs[l], ws[l], bias, out, act=act, residual=resid)
            line += f"  skinny: {_time_graph(go_skinny, layers):6.1f}"

            def go_small(l):
                ops.gemm_small(xs[l], ws[l], bias, out, act=act, residual=resid)
            line += f"  small ({ops.gemm_small_splits(N, K)} splits): {_time_graph(go_small, layers):6.1f}"
        # the library's product with its bias alone (no activation, no residual, bfloat16 out): the yardstick
        lib_out = torch.empty(M, N, device=dev, dtype=torch.bfloat16)

        def go_lib(l):
            torch.addmm(bias, xs[l], ws[l].t(), out=lib_out)
        us = _time_graph(go_lib, layers)
        line += f"  cuBLAS: {us:6.1f} ({2.0 * M * N * K / us / 1e6:5.0f})"
        print(line, flush=True)
        ops.check_kernel_status(dev)
    if a.k_sweep:
        # the q/k/v output size at several K, no bias: what does not move with K is launch,
        # set-up and write-back; the slope is the main loop's rate
        N = 3 * a.width
        print(f"K sweep at {M}x{N}, no bias, bfloat16 out: us (TFLOP/s)")
        for K in (64, 256, 768, 1536, 3072):
            x4 = [torch.randn(M, K, device=dev, dtype=torch.bfloat16) for _ in range(4)]
            xs = [x4[l % 4] for l in range(layers)]
            ws = [torch.randn(N, K, device=dev, dtype=torch.bfloat16) * 0.05 for _ in range(layers)]
            out = torch.empty(M, N, device=dev, dtype=torch.bfloat16)
            line = f"K {K:5d}:"
            for tile in (128, ops.PAIR_TILE + 256):
                def go(l, tile=tile):
                    ops.gemm_tc(xs[l], ws[l], None, out, tile_n=tile)
                us = _time_graph(go, layers)
                line += f"  {tile:5d}: {us:6.1f} ({2.0 * M * N * K / us / 1e6:5.0f})"
            print(line, flush=True)
    return 0


def prefill_attention(a) -> int:
    import math

    dev = "cuda:0"
    H, D, ps = a.heads, 64, a.page_size
    print(f"prefill attention, {H} heads of {D}, pages of {ps}; us per launch and TFLOP/s of the causal part")
    for shape in a.shape:
        reqs, rest = shape.split("x")
        new, cached = rest.split("+")
        n_seqs, q_len, before = int(reqs), int(new), int(cached)
        L = before + q_len
        nb = -(-L // ps)
        num_pages = n_seqs * nb + 1
        g = torch.Generator(device=dev).manual_seed(0)
        arena = torch.randn(num_pages, 2, H, ps, D, device=dev, generator=g).to(torch.bfloat16)
        kc, vc = arena[:, 0], arena[:, 1]
        T = n_seqs * q_len
        q = torch.randn(T, H * D, device=dev, generator=g).to(torch.bfloat16)
        q_start = torch.arange(0, T + 1, q_len, dtype=torch.int32, device=dev)
        kv_before = torch.full((n_seqs,), before, dtype=torch.int32, device=dev)
        flops = 4.0 * n_seqs * H * D * sum(before + i + 1 for i in range(q_len))
        tables = {"runs": torch.arange(n_seqs * nb, device=dev, dtype=torch.int32).view(n_seqs, nb).contiguous(),
                  "scattered": torch.randperm(num_pages - 1, device=dev, generator=g).to(torch.int32)[:n_seqs * nb]
                  .view(n_seqs, nb).contiguous()}
        outs = {}
        for pages, table in tables.items():
            for name, tc in (("mma.sync", False), ("tcgen05", True)):
                out = torch.zeros_like(q)

                def go(l, table=table, tc=tc, out=out):
                    ops.prefill_attention(q, kc, vc, table, q_start, kv_before, out, n_heads=H, max_q_len=q_len,
                                          scale=1 / math.sqrt(D), tc=tc)
                us = _time_graph(go, a.launches)
                ops.check_kernel_status(dev)
                outs[name] = out.float()
                print(f"  {shape:>12} pages {pages:>9} {name:>8}: {us:7.1f} us  {flops / us / 1e6:6.0f} TFLOP/s", flush=True)
            print(f"  {'':>12} largest difference between the two kernels: "
                  f"{(outs['tcgen05'] - outs['mma.sync']).abs().max().item():.4f}")
    return 0


def grouped(a) -> int:
    """The products with one matrix per expert and per head, alone: an expert's up-projection (rows gathered by the
    routing, relu squared) and down-projection on `layers` distinct sets of weights, and the two per-head products of
    attention over a latent.  Bytes: the matrices that are read at least once plus the rows in and out."""
    dev = torch.device("cuda:0")
    E, top, W, F, L = a.experts, a.top, a.width, a.inner, a.layers
    g = torch.Generator(device="cpu").manual_seed(0)
    ups = [(torch.randn(E * F, W, generator=g) * W ** -0.5).to(torch.bfloat16).to(dev) for _ in range(L)]
    downs = [(torch.randn(E * W, F, generator=g) * F ** -0.5).to(torch.bfloat16).to(dev) for _ in range(L)]
    for T in a.tokens:
        h = torch.randn(T, W, generator=g).to(torch.bfloat16).to(dev)
        r = ops.moe_route(torch.randn(T, E, generator=g).to(dev), None, top)
        inner = torch.empty(T * top, F, dtype=torch.bfloat16, device=dev)
        rows = torch.empty(T * top, W, dtype=torch.float32, device=dev)
        used = min(E, T * top)
        for name, fn, byts in (
                ("up", lambda l: ops.expert_product(r, h, ups[l], inner, gather=True, act="relu_squared"), used * F * W * 2 + T * top * (W + F) * 2),
                ("down", lambda l: ops.expert_product(r, inner, downs[l], rows, gather=False), used * F * W * 2 + T * top * (2 * F + 4 * W))):
            us = _time_graph(fn, L)
            print(f"expert {name:4s} T={T:5d} E={E} top={top} {W}x{F}: {us:8.1f} us  {2.0 * T * top * W * F / us / 1e6:7.1f} TFLOP/s  {byts / us / 1e3:7.0f} GB/s")
        sorted_rows = torch.empty(T * top, W, dtype=torch.bfloat16, device=dev)
        ops.moe_gather(r, h, sorted_rows)
        for name, fn in (("up", lambda l: ops.expert_product_tc(r, sorted_rows, ups[l], inner, act="relu_squared")),
                         ("down", lambda l: ops.expert_product_tc(r, inner, downs[l], rows))):
            us = _time_graph(fn, L)
            print(f"expert {name:4s} T={T:5d} tcgen05: {us:8.1f} us  {2.0 * T * top * W * F / us / 1e6:7.1f} TFLOP/s")
        us = _time_graph(lambda l: ops.moe_gather(r, h, sorted_rows), 1)
        print(f"expert rows gathered T={T:5d}: {us:8.1f} us")
        H, d, c, pad = a.heads, 64, 96, 128
        q = torch.randn(T, H * (d + 32), generator=g).to(torch.bfloat16).to(dev)
        uk = [(torch.randn(H * c, d, generator=g) * d ** -0.5).to(torch.bfloat16).to(dev) for _ in range(L)]
        q_abs = torch.empty(T, H * pad, dtype=torch.bfloat16, device=dev)
        us = _time_graph(lambda l: ops.head_product(q, uk[l], q_abs, n_groups=H, a_gcols=d + 32, o_gcols=pad), L)
        print(f"head   q->latent T={T:5d} H={H} {c}x{d}: {us:8.1f} us  {2.0 * T * H * c * d / us / 1e6:7.1f} TFLOP/s  {(T * H * (d + c) * 2 + H * c * d * 2) / us / 1e3:7.0f} GB/s")
    return 0


def gemm_f32(a) -> int:
    """The float32 product on the fma units and on the tensor cores beside the general kernel, on distinct weights that together exceed L2."""
    dev = torch.device("cuda:0")
    for M in a.rows:
        for shape in a.shape:
            N, K = (int(v) for v in shape.split("x"))
            x, out = torch.randn(M, K, device=dev), torch.empty(M, N, device=dev)
            ws = [torch.randn(N, K, device=dev) for _ in range(max(1, min(24, 300_000_000 // (4 * N * K))))]
            us = [_time_graph(lambda l: ops.gemm_f32(x, ws[l], None, out), len(ws)),
                  _time_graph(lambda l: ops.gemm_simt(x, ws[l], None, out, w_out_in=True), len(ws)),
                  _time_graph(lambda l: ops.gemm_f32_tc(x, ws[l], None, out), len(ws))]
            print(f"{M:5d} rows {N:6d} x {K:5d}: {us[0]:8.1f} us  {4e-3 * N * K / us[0]:6.0f} GB/s  {2e-6 * M * N * K / us[0]:5.1f} TFLOP/s"
                  f"   general kernel {us[1]:8.1f} us   tensor cores {us[2]:8.1f} us", flush=True)
    return 0


def _cache(dev, H, D, ps, seqs, dtype):
    """Queries and cache of requests (tokens before, new tokens); the table's width as the engine has it, in steps of 8 pages."""
    g = torch.Generator(device=dev).manual_seed(0)
    blocks = [-(-(b + n) // ps) for b, n in seqs]
    table = torch.full((len(seqs), -(-max(blocks) // 8) * 8), -1, dtype=torch.int32)
    at = 0
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    kc, vc = (torch.randn(at, H, ps, D, generator=g, device=dev).to(dtype) for _ in range(2))
    T = sum(n for _, n in seqs)
    q = torch.randn(T, H * D, generator=g, device=dev).to(dtype)
    start = torch.tensor([0] + [n for _, n in seqs]).cumsum(0).to(torch.int32).to(dev)
    before = torch.tensor([b for b, _ in seqs], dtype=torch.int32, device=dev)
    seq = torch.repeat_interleave(torch.arange(len(seqs)), torch.tensor([n for _, n in seqs])).to(torch.int32).to(dev)
    pos = torch.cat([torch.arange(b, b + n) for b, n in seqs]).to(torch.int32).to(dev)
    return q, kc, vc, table.to(dev), start, before, seq, pos


def attention_f32(a) -> int:
    """Prompt portions in float32: the general kernel and the prompt kernels on the fma units and on the tensor cores."""
    for shape in a.shape:
        reqs, rest = shape.split("x")
        new, cached = (int(v) for v in rest.split("+"))
        q, kc, vc, table, start, before, seq, pos = _cache("cuda:0", a.heads, a.head_dim, a.page_size, [(cached, new)] * int(reqs), torch.float32)
        out, kw = torch.empty_like(q), dict(n_heads=a.heads, scale=a.head_dim ** -0.5)
        general = _time_graph(lambda l: ops.paged_attention(q, kc, vc, table, seq, pos, out, **kw), 10)
        tiles = _time_graph(lambda l: ops.prefill_attention_f32(q, kc, vc, table, start, before, out, max_q_len=new, **kw), 10)
        line = f"{a.heads} heads of {a.head_dim}, {shape:>10}: general {general:8.1f} us  prompt kernel {tiles:8.1f} us"
        if a.head_dim > 32:
            tc = _time_graph(lambda l: ops.prefill_attention_f32(q, kc, vc, table, start, before, out, max_q_len=new, tc=True, **kw), 10)
            line += f"  tensor cores {tc:8.1f} us"
        print(line, flush=True)
    return 0


def mixed_attention(a) -> int:
    """Single tokens beside portions, bfloat16, heads of 64: one launch over everything and two."""
    reqs, new = (int(v) for v in a.portions.split("x"))
    for n in a.singles:
        spread = a.context // 2
        seqs = [(a.context - spread // 2 + spread * i // max(n - 1, 1), 1) for i in range(n)] + [(0, new)] * reqs
        q, kc, vc, table, start, before, _, _ = _cache("cuda:0", a.heads, 64, 16, seqs, torch.bfloat16)
        out, keys = torch.empty_like(q), table.shape[1] * 16
        kw = dict(n_heads=a.heads, max_q_len=new, scale=0.125)
        one = _time_graph(lambda l: ops.prefill_attention(q, kc, vc, table, start, before, out, **kw), 10)
        splits = min(8, ops.decode_splits(n, a.heads, keys))
        two = _time_graph(lambda l: ops.mixed_attention(q, kc, vc, table, start, before, out, num_splits=splits, **kw), 10)
        print(f"{a.heads} heads, {n:3d} tokens behind about {a.context} beside {a.portions}: one launch {one:6.1f} us  two {two:6.1f} us  "
              f"(taken: {'two' if ops.singles_apart(n, a.heads, keys) else 'one'})", flush=True)
    return 0


def recurrences(a) -> int:
    """Delta rule (heads of 64) and matrix memory (a quarter of the heads, 64 x 128) over prompts: chunks walked one by one and side by
    side; and the delta rule's errors against 64 bits in the 2-norm (read-outs, state), from an empty state."""
    dev = torch.device("cuda:0")
    H, T, d = a.heads, sum(a.lengths), 64
    g = torch.Generator(device=dev).manual_seed(0)
    rand = lambda *shape: torch.randn(*shape, generator=g, device=dev)
    start = torch.tensor([0] + a.lengths).cumsum(0).to(torch.int32).to(dev)
    slots = torch.arange(len(a.lengths), dtype=torch.int32, device=dev)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k, v = unit(rand(T, H, d)) / 8, unit(torch.nn.functional.silu(rand(T, H, d))), rand(T, H, d)
    bg = torch.cat([torch.rand(T, H, generator=g, device=dev), -0.1 * torch.rand(T, H, generator=g, device=dev)], 1)
    qkv = torch.cat([x.reshape(T, -1) for x in (q, k, v)], 1)
    want, S = torch.empty(T, H, d, dtype=torch.float64, device=dev), None
    states = []
    for t in range(T):
        if t in start.tolist():
            S = torch.zeros(H, d, d, dtype=torch.float64, device=dev)
        S = S * torch.exp(bg[t, H:].double()).view(H, 1, 1)
        u = bg[t, :H].double().view(H, 1) * (v[t].double() - torch.einsum("hed,hd->he", S, k[t].double()))
        S = S + u.unsqueeze(2) * k[t].double().unsqueeze(1)
        want[t] = torch.einsum("hed,hd->he", S, q[t].double())
        if t + 1 in start.tolist():
            states.append(S)
    off = lambda x, y: ((x.double() - y).norm() / y.norm()).item()
    kw = dict(long_from=8, max_q_len=max(a.lengths))
    for form in ("walk", "chunks"):
        state, out = torch.zeros(len(a.lengths), H * d * d, device=dev), torch.empty(T, H * d, device=dev)
        go = lambda l: ops.delta_scan(qkv, bg, state, start, slots, out, n_heads=H, n_qk_heads=H, qk_dim=d, v_dim=d, form=form, **kw)
        go(0)
        errors = off(out.view(T, H, d), want), off(state.view(-1, H, d, d), torch.stack(states))
        print(f"delta rule, {H} heads, {a.lengths}, {form:6s}: {_time_graph(go, 10):8.1f} us  errors {errors[0]:.1e} {errors[1]:.1e}", flush=True)
    H = max(1, H // 4)
    proj, gates = rand(T, H * (2 * d + 128)).to(torch.bfloat16), rand(T, 2 * H)
    bias = torch.cat([torch.zeros(H), torch.full((H,), 4.0)]).to(dev)
    for form in ("walk", "chunks"):
        state, out = torch.zeros(len(a.lengths), H * (128 * d + 8 * d + 8), device=dev), torch.empty(T, H * 128, device=dev)
        go = lambda l: ops.mlstm_scan(proj, 0, H * d, 2 * H * d, gates, bias, state, start, slots, out, cap=12.0, q_scale=0.125, n_heads=H,
                                      qk_dim=d, v_dim=128, form=form, **kw)
        print(f"matrix memory, {H} heads, {a.lengths}, {form:6s}: {_time_graph(go, 10):8.1f} us", flush=True)
    return 0


def main(argv=None) -> int:
    ap = argparse.ArgumentParser(prog="sandyrt_b200.csrc.microbench")
    sub = ap.add_subparsers(dest="cmd", required=True)
    d = sub.add_parser("decode-attention")
    d.add_argument("--heads", type=int, default=12)
    d.add_argument("--head-dim", type=int, default=64)
    d.add_argument("--page-size", type=int, default=16)
    d.add_argument("--shape", nargs="+", default=["64x384", "64x1024", "256x384", "8x384", "8x1024", "1x1024"],
                   help="tokens x context")
    d.set_defaults(fn=decode_attention)
    g = sub.add_parser("gemm")
    g.add_argument("--rows", type=int, default=2048)
    g.add_argument("--width", type=int, default=768)
    g.add_argument("--inner", type=int, default=3072)
    g.add_argument("--k-sweep", action="store_true", help="also time the q/k/v output size at several K")
    g.add_argument("--layers", type=int, default=48, help="distinct weights and inputs per shape")
    g.set_defaults(fn=gemm)
    pa = sub.add_parser("prefill-attention")
    pa.add_argument("--heads", type=int, default=12)
    pa.add_argument("--page-size", type=int, default=16)
    pa.add_argument("--launches", type=int, default=20, help="launches per timed graph")
    pa.add_argument("--shape", nargs="+", default=["2x1024+0", "8x256+0", "4x512+512", "16x128+0", "2x2048+0", "1x8192+0"],
                    help="REQUESTSxNEW+CACHED")
    pa.set_defaults(fn=prefill_attention)
    gr = sub.add_parser("grouped")
    gr.add_argument("--tokens", type=int, nargs="+", default=[2048, 8])
    gr.add_argument("--experts", type=int, default=16)
    gr.add_argument("--top", type=int, default=2)
    gr.add_argument("--width", type=int, default=1536)
    gr.add_argument("--inner", type=int, default=2048)
    gr.add_argument("--heads", type=int, default=24)
    gr.add_argument("--layers", type=int, default=4, help="distinct sets of weights (together larger than L2)")
    gr.set_defaults(fn=grouped)
    gf = sub.add_parser("gemm-f32")
    gf.add_argument("--rows", type=int, nargs="+", default=[1, 8, 24, 2048])
    gf.add_argument("--shape", nargs="+", default=["2304x768", "768x768", "3072x768", "768x3072", "50257x768"], help="outputs x inputs")
    gf.set_defaults(fn=gemm_f32)
    af = sub.add_parser("attention-f32")
    af.add_argument("--heads", type=int, default=12)
    af.add_argument("--head-dim", type=int, default=64)
    af.add_argument("--page-size", type=int, default=16)
    af.add_argument("--shape", nargs="+", default=["2x1024+0", "1x16+0", "1x32+0", "1x48+0", "1x64+0", "8x16+0", "1x16+100"], help="REQUESTSxNEW+CACHED")
    af.set_defaults(fn=attention_f32)
    mx = sub.add_parser("mixed-attention")
    mx.add_argument("--heads", type=int, default=16)
    mx.add_argument("--context", type=int, default=400)
    mx.add_argument("--portions", default="1x480", help="PORTIONSxTOKENS")
    mx.add_argument("--singles", type=int, nargs="+", default=[4, 8, 16, 32])
    mx.set_defaults(fn=mixed_attention)
    rc = sub.add_parser("recurrences")
    rc.add_argument("--lengths", type=int, nargs="+", default=[1024, 1024])
    rc.add_argument("--heads", type=int, default=12)
    rc.set_defaults(fn=recurrences)
    a = ap.parse_args(argv)
    return a.fn(a)


if __name__ == "__main__":
    sys.exit(main())
