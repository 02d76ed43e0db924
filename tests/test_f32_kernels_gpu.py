"""The float32 kernels alone, at the edges of their tiles and splits, against torch in 64 bits."""
import functools
import types

import numpy as np
import pytest
import torch

from test_kernels_gpu import DEV, _paged_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,splits", [(0, 1), (1, 1), (2, 1), (2, 8), (3, 1), (3, 2), (4, 1), (4, 4), (4, 8)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (2, 7, 132), (4, 129, 128), (8, 768, 768), (9, 50, 12), (24, 1000, 260), (25, 64, 516),
                                   (64, 128, 1024), (65, 130, 36), (130, 257, 640)])
def test_gemm_f32(M, N, K, form, splits):
    """Every kernel and split at sizes that are no multiple of a tile, a step of k or the rows of a block; pitches wider
    than the rows; the residual is the output itself."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(M * 1000 + N + K)
    a = torch.randn(M, K + 4, generator=g).to(DEV)[:, :K]
    w = torch.randn(N, K + 8, generator=g).to(DEV)[:, :K]
    bias, x0 = torch.randn(N, generator=g).to(DEV), torch.randn(M, N + 3, generator=g).to(DEV)
    want = a.double() @ w.double().t() + bias.double()
    # a sum of K products of size |a| |w|, each rounded, any order: K * 2^-24 of the sum of the sizes; 4 for the write-back
    bound = (K + 4) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t() + bias.double().abs() + x0[:, :N].double().abs())
    wide = x0.clone()
    x = wide[:, :N]
    ops.gemm_f32(a, w, bias, x, residual=x, form=form, splits=splits)
    assert bool(((x.double() - want - x0[:, :N].double()).abs() <= bound).all())
    assert torch.equal(wide[:, N:], x0[:, N:])
    out = torch.full((M, N), float("nan"), device=DEV)
    ops.gemm_f32(a, w, bias, out, act="gelu_new", form=form, splits=splits)
    gelu = torch.nn.functional.gelu(want, approximate="tanh")
    assert bool(((out.double() - gelu).abs() <= 2 * bound + 1e-6 * (1 + want.abs())).all())     # the slope stays below 1.13


@pytest.mark.parametrize("form,splits", [(0, 1), (1, 1), (4, 1), (4, 2)])
@pytest.mark.parametrize("M,N,K", [(1, 5, 4), (2, 9, 132), (4, 40, 132), (8, 33, 1600), (9, 33, 260)])
def test_gemm_f32_infinity_at_the_end_of_a_row(M, N, K, form, splits):
    """An infinite activation among the last four k: plus or minus infinity by the weight's sign, nothing for the other rows."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    finite = torch.empty(M, N, device=DEV)
    ops.gemm_f32(a, w, None, finite, form=form, splits=splits)
    for at in (K - 4, K - 1):
        b = a.clone()
        b[M - 1, at] = float("inf")
        out = torch.full((M, N), float("nan"), device=DEV)
        ops.gemm_f32(b, w, None, out, form=form, splits=splits)
        assert torch.equal(out[M - 1], torch.sign(w[:, at]) * float("inf"))
        assert torch.equal(out[:M - 1], finite[:M - 1])


def test_gemm_f32_refuses_what_it_cannot_load():
    from sandyrt_b200.csrc import ops

    a, w, out = torch.zeros(3, 6, device=DEV), torch.zeros(5, 6, device=DEV), torch.zeros(3, 5, device=DEV)
    with pytest.raises(ops.UnsupportedShape):
        ops.gemm_f32(a, w, None, out)                                       # K is no multiple of 4
    with pytest.raises(ops.UnsupportedShape):
        ops.gemm_f32(torch.zeros(25, device=DEV)[1:].view(3, 8)[:, :4], w[:, :4].contiguous(), None, out)   # not on 16 bytes


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (15, 17, 20), (16, 16, 64), (57, 192, 64), (33, 50, 252), (130, 65, 256)])
def test_gemm_f32_short(M, N, K):
    """Remainders of the 16 x 16 tiles, a k that is no multiple of the four warps' share, the longest one; and that a longer is refused."""
    from sandyrt_b200.csrc import ops

    test_gemm_f32(M, N, K, 5, 1)
    test_gemm_f32_infinity_at_the_end_of_a_row(M, N, K, 5, 1)
    with pytest.raises(ops.UnsupportedShape):
        ops.gemm_f32(torch.zeros(2, 260, device=DEV), torch.zeros(3, 260, device=DEV), None, torch.zeros(2, 3, device=DEV), form=5)


@pytest.mark.parametrize("tile,parts", [(0, 0), (64, 1), (64, 8), (96, 1), (96, 4), (128, 1), (128, 2), (128, 8)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (33, 50, 12), (127, 97, 516), (129, 130, 576), (260, 257, 1028)])
@pytest.mark.parametrize("size", [1.0, 2.0 ** -110, 2.0 ** 100])
def test_gemm_f32_on_tensor_cores(M, N, K, tile, parts, size):
    """Tiles, parts and chunks of k with remainders; pitches wider than the rows; the residual is the output itself; an infinite
    activation; very small activations with weights too large to be split (every sum is formed again in float arithmetic), and the reverse,
    which can be split."""
    from sandyrt_b200.csrc import ops

    if parts > (K + 63) // 64:
        pytest.skip("fewer chunks of k than parts")
    g = torch.Generator().manual_seed(M * 1000 + N + K)
    a = (torch.randn(M, K + 4, generator=g) * size).to(DEV)[:, :K]
    w = (torch.randn(N, K + 8, generator=g) / size).to(DEV)[:, :K]
    bias, x0 = torch.randn(N, generator=g).to(DEV), torch.randn(M, N + 3, generator=g).to(DEV)
    want = a.double() @ w.double().t() + bias.double()
    # of a product 2^-24 is left out with the three smallest products of pieces; sixteen products at a time are added with at
    # most 2^-22 of their sizes lost to rounding towards zero: less than K * 2^-24 from K = 4 on; 4 for the write-back
    bound = (K + 4) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t() + bias.double().abs() + x0[:, :N].double().abs())
    wide = x0.clone()
    x = wide[:, :N]
    ops.gemm_f32_tc(a, w, bias, x, residual=x, tile=tile, parts=parts)
    assert bool(((x.double() - want - x0[:, :N].double()).abs() <= bound).all())
    assert torch.equal(wide[:, N:], x0[:, N:])
    finite, out = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm_f32_tc(a, w, None, finite, tile=tile, parts=parts)
    b = a.clone()
    b[M - 1, K - 1] = float("inf")
    ops.gemm_f32_tc(b, w, None, out, tile=tile, parts=parts)
    assert torch.equal(out[M - 1], torch.sign(w[:, K - 1]) * float("inf"))
    assert torch.equal(out[:M - 1], finite[:M - 1])
    assert int(ops.kernel_status(a.device).item()) == 0


# What a product of two floats may be off by: the three products of pieces that are left out reach 2^-24 of it together, and the
# tensor core's last addition takes up to 2^-23 towards zero (the ones before it are of 2^-8 of the size).
ONE_PRODUCT = 2.0 ** -24 + 2.0 ** -23 + 2.0 ** -30

TILES = [(0, 0), (64, 1), (64, 8), (96, 1), (96, 4), (128, 1), (128, 2), (128, 8)]


@pytest.mark.parametrize("tile,parts", TILES)
@pytest.mark.parametrize("M,N,K", [(130, 97, 516), (257, 130, 1028)])
@pytest.mark.parametrize("size_a,size_w", [(0, 0), (-118, 40), (40, -118), (-100, 100)])
def test_gemm_f32_on_tensor_cores_keeps_24_bits(M, N, K, tile, parts, size_a, size_w):
    """Rows with one number each, at every place of every chunk: an output is one product, whose six products of pieces show: without
    any of them it is off by 2^-20 to 2^-8 of its size in one place or another.  Sizes (powers of two) whose last pieces would lie below
    a bfloat16's range were they not scaled; all of them can be split, so no sum is formed again in float arithmetic."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(M + N + K)
    number, w = (1.0 + torch.rand(M, generator=g)) * 2.0 ** size_a, (1.0 + torch.rand(N, K, generator=g)) * 2.0 ** size_w
    at = torch.arange(M) * 37 % K
    a = torch.zeros(M, K)
    a[torch.arange(M), at] = number * torch.where(torch.arange(M) % 2 == 0, 1.0, -1.0)
    want = a[torch.arange(M), at].double()[:, None] * w[:, at].t().double()
    out = torch.empty(M, N, device=DEV)
    ops.gemm_f32_tc(a.to(DEV), w.to(DEV), None, out, tile=tile, parts=parts)
    assert bool(((out.double().cpu() - want).abs() <= ONE_PRODUCT * want.abs()).all())


@pytest.mark.parametrize("tile,parts", TILES)
@pytest.mark.parametrize("M,N,K", [(129, 130, 576), (260, 257, 1028), (64, 96, 3072)])
@pytest.mark.parametrize("sign", ["both", "one operand", "none"])
def test_gemm_f32_on_tensor_cores_error(M, N, K, tile, parts, sign):
    """The whole error (2-norm) over many chunks.  Sums of one sign: four additions of a chunk's own size lose up to 2^-23 of a quarter,
    a half, three quarters and all of it, which is 2.5 * 2^-23 at the most and half of that on average, and the chunks are added with
    float roundings.  Centred ones shrink as their partial sums do: four times half of 2^-23 of a chunk, whose size is sqrt(64 / K) of the
    sum's, once for every chunk.  Three products of pieces less cost 4e-6."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    a, w = a.abs() if sign != "both" else a, w.abs() if sign == "none" else w
    want = a.double() @ w.double().t()
    out = torch.empty(M, N, device=DEV)
    ops.gemm_f32_tc(a, w, None, out, tile=tile, parts=parts)
    assert float((out.double() - want).norm() / want.norm()) < 2.0 * 2.0 ** -23


def _milliseconds(call):
    """The fastest of five calls."""
    times = []
    for _ in range(5):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        call()
        end.record()
        end.synchronize()
        times.append(begin.elapsed_time(end))
    return min(times)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_gemm_f32_on_tensor_cores_is_not_slow_on_what_is_not_finite(bad):
    """A NaN in a row of a is found once (2.7 times as long as finite rows; 35 with every sum formed again by itself); infinities have
    every sum formed again, which is not timed."""
    from sandyrt_b200.csrc import ops

    a, w, out = torch.randn(2048, 768, device=DEV), torch.randn(2304, 768, device=DEV), torch.empty(2048, 2304, device=DEV)
    finite = _milliseconds(lambda: ops.gemm_f32_tc(a, w, None, out))
    a[:, 5] = bad
    time = _milliseconds(lambda: ops.gemm_f32_tc(a, w, None, out))
    assert bad == bad or time < 10 * finite
    assert torch.isnan(out).all() if bad != bad else torch.equal(out, (torch.sign(w[:, 5]) * bad).expand_as(out))
    a, w, out = a[:130, :516].contiguous(), w[:99, :516].contiguous(), torch.empty(130, 99, device=DEV)
    a[::3, 5] = float("nan")                                # rows of NaN between rows of infinities (or of NaN), columns no multiple of 4
    ops.gemm_f32_tc(a, w, None, out)
    assert torch.isnan(out[::3]).all()
    if bad == bad:
        assert torch.equal(out[1::3], (torch.sign(w[:, 5]) * bad).expand_as(out[1::3]))


# ---- attention of prompt portions ---------------------------------------------------------------------------------
def _both(case, H, kw):
    """The prompt kernel's output and the general kernel's, which reads one (token, head) pair at a time."""
    from sandyrt_b200.csrc import ops

    lens = [n for _, n in case["seqs"]]
    q_start = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device=DEV)
    kv_before = torch.tensor([b for b, _ in case["seqs"]], dtype=torch.int32, device=DEV)
    got = torch.full(case["q"].shape, float("nan"), device=DEV)
    want = torch.full(case["q"].shape, float("nan"), device=DEV)
    ops.prefill_attention_f32(case["q"], case["kc"], case["vc"], case["table"], q_start, kv_before, got, n_heads=H,
                              max_q_len=max(lens), **kw)
    ops.paged_attention(case["q"], case["kc"], case["vc"], case["table"], case["tok_seq"], case["tok_pos"], want, n_heads=H, **kw)
    ops.check_kernel_status(DEV)
    return got, want


RULES = [{}, {"window": 70}, {"window": 1}, {"window": 90, "keep_first": 70}, {"window": 30, "keep_first": 3, "gates": True},
         {"softcap": 3.0, "chunk": 50}, {"softcap": 20.0, "bias": 40, "sink": True}, {"sink": True, "out_gate": True, "gates": True}]


@pytest.mark.parametrize("rules", RULES)
@pytest.mark.parametrize("H,Hkv,D,page_size", [(3, 3, 64, 16), (4, 2, 16, 8), (2, 1, 128, 32), (3, 1, 80, 4), (2, 2, 48, 1)])
def test_prompt_attention_f32(H, Hkv, D, page_size, rules):
    """Portions at tile edges (63, 64, 65 tokens), from position 0 and from the middle, single tokens beside them; every
    rule.  A sum of at most 330 weighted values of size 3, weights that add up to at most 1, against the same in another
    order: 330 * 2^-24 of the weights twice (exponentials and sums) and of the values, 3 * 3 * 2e-5 = 1.8e-4 at the worst,
    a tenth of it allowed."""
    g = torch.Generator().manual_seed(D + page_size)
    seqs = [(0, 130), (40, 1), (17, 64), (0, 1), (63, 65), (0, 63), (199, 130)]
    case = _paged_case(torch.float32, H, Hkv, D, page_size, seqs, seed=D + H)
    T = case["q"].shape[0]
    kw = {k: v for k, v in rules.items() if k in ("window", "keep_first", "softcap", "chunk")}
    kw["scale"] = 0.8 / D ** 0.5
    if rules.get("sink"):
        kw["sink"] = torch.randn(H, generator=g).to(DEV)
    if rules.get("out_gate"):
        kw["out_gate"] = torch.rand(T, H, generator=g).to(DEV)
    if rules.get("bias"):
        kw["dist_bias"] = torch.randn(H, rules["bias"], generator=g).to(DEV)
    if rules.get("gates"):
        kw["elem_gate"] = torch.randn(T, H * (D - 5) + 9, generator=g).to(DEV)[:, 2:2 + H * (D - 5)]
    got, want = _both(case, H, kw)
    assert not torch.isnan(got).any()
    assert (got - want).abs().max().item() < 2e-5
    # queries whose rows do not start on 16-byte boundaries
    wide = torch.zeros(T, case["q"].shape[1] + 3, device=DEV)
    wide[:, 1:-2] = case["q"]
    odd, _ = _both({**case, "q": wide[:, 1:-2]}, H, kw)
    assert torch.equal(odd, got)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_value_that_is_not_finite_reaches_only_the_queries_that_see_it(D, bad):
    """Token 70's value: the queries before it share its tile of keys."""
    case = _paged_case(torch.float32, 2, 2, D, 16, [(0, 100), (0, 70)], seed=3)
    page = int(case["table"][0, 70 // 16])
    case["vc"][page, :, 70 % 16] = bad
    got, want = _both(case, 2, {"scale": 0.1})
    assert torch.isfinite(got[:70]).all() and torch.isfinite(got[100:]).all() and not torch.isfinite(got[70:100]).any()
    assert (got[:70] - want[:70]).abs().max().item() < 2e-5 and (got[100:] - want[100:]).abs().max().item() < 2e-5


def _formula(case, H, scale, window, sink):
    """[T, H * D] in 64 bits, request by request; a hidden key has no part in a query's sums, whatever it holds."""
    rows = []
    for s, (before, n) in enumerate(case["seqs"]):
        k, v, q = (case[name][s].double() for name in ("dense_k", "dense_v", "qs"))
        for i in range(n):
            lo, hi = max(0, before + i + 1 - window) if window else 0, before + i + 1
            z = torch.einsum("jhd,hd->hj", k[lo:hi], q[i]) * scale
            if sink is not None:
                z = torch.cat([z, sink.double().cpu().view(H, 1)], 1)
            p = torch.softmax(z, 1)[:, :hi - lo]
            rows.append(torch.einsum("hj,jhd->hd", p, v[lo:hi]).reshape(-1))
    return torch.stack(rows)


@pytest.mark.parametrize("D", [16, 64, 128])
@pytest.mark.parametrize("window", [0, 90])
@pytest.mark.parametrize("with_sink", [False, True])
@pytest.mark.parametrize("bad", ["key", "key and value", "query", "score of minus infinity", "score of minus infinity and value"])
def test_a_token_that_is_not_finite_reaches_every_query_that_sees_it(D, window, with_sink, bad):
    """Token 70 of 200: its tile of keys is at the edge for the queries of its own tile and a whole one for those behind it.
    A NaN score is a NaN in the softmax, and a seen key whose score is minus infinity still brings 0 times its value; what
    the formula leaves finite stays so."""
    H, at = 2, 70
    case = _paged_case(torch.float32, H, H, D, 16, [(0, 200), (0, 70)], seed=3)
    page = int(case["table"][0, at // 16])
    if "minus" in bad:                                      # queries above zero, a key of -inf
        case["q"] = case["q"].abs()
        case["qs"] = [q.abs() for q in case["qs"]]
    for name, cache, dense, x in (("query", None, None, None), ("key", "kc", "dense_k", float("nan")),
                                  ("minus", "kc", "dense_k", -float("inf")), ("value", "vc", "dense_v", float("inf" if "minus" in bad else "nan"))):
        if name in bad and cache:
            case[cache][page, :, at % 16] = x
            case[dense][0][at] = x
    if bad == "query":
        case["q"][at] = float("nan")
        case["qs"][0][at] = float("nan")
    sink = torch.tensor([0.5, -1.0], device=DEV) if with_sink else None
    got, general = _both(case, H, {"scale": 0.1, "window": window, "sink": sink})
    want = _formula(case, H, 0.1, window, sink)
    assert torch.isnan(want).any() == (bad != "score of minus infinity")
    assert torch.equal(torch.isnan(got).cpu(), torch.isnan(want))
    fine = ~torch.isnan(want)
    assert (got.double().cpu() - want)[fine].abs().max().item() < 2e-5      # the bound of test_prompt_attention_f32
    if bad != "key":                                        # (the general kernel gives a NaN score no weight)
        assert torch.equal(torch.isnan(got), torch.isnan(general))


@pytest.fixture
def on_tensor_cores(monkeypatch):
    from sandyrt_b200.csrc import ops

    monkeypatch.setattr(ops, "prefill_attention_f32", functools.partial(ops.prefill_attention_f32, tc=True))


@pytest.mark.parametrize("rules", RULES)
@pytest.mark.parametrize("H,Hkv,D,page_size", [(3, 3, 64, 16), (4, 2, 48, 8), (2, 1, 128, 32), (3, 1, 80, 4), (2, 2, 64, 1)])
def test_prompt_attention_f32_on_tensor_cores(on_tensor_cores, H, Hkv, D, page_size, rules):
    test_prompt_attention_f32(H, Hkv, D, page_size, rules)


@pytest.mark.parametrize("D", [64, 128])
def test_tokens_that_are_not_finite_on_tensor_cores(on_tensor_cores, D):
    """A tile that holds one is formed with float arithmetic: the same queries as before, and no others."""
    for bad in (float("nan"), float("inf")):
        test_a_value_that_is_not_finite_reaches_only_the_queries_that_see_it(D, bad)
    for bad in ("key", "key and value", "query", "score of minus infinity", "score of minus infinity and value"):
        for window, with_sink in ((0, False), (90, True)):
            test_a_token_that_is_not_finite_reaches_every_query_that_sees_it(D, window, with_sink, bad)


@pytest.mark.parametrize("bad", ["a query", "queries", "keys", "values"])
def test_prompt_attention_f32_on_tensor_cores_is_not_slow_on_nan(bad):
    """Only what holds a NaN leaves the tensor cores: one query's scores, or a key's, are known without a sum, a value's part is added by
    itself (whole tiles in float arithmetic took 15 to 40 times as long as finite ones)."""
    from sandyrt_b200.csrc import ops

    case = _paged_case(torch.float32, 12, 12, 64, 16, [(0, 512)], seed=1)
    q_start, kv_before = torch.tensor([0, 512], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.empty_like(case["q"])
    run = lambda: ops.prefill_attention_f32(case["q"], case["kc"], case["vc"], case["table"], q_start, kv_before, out, n_heads=12,
                                            max_q_len=512, scale=0.1, tc=True)
    finite = _milliseconds(run)
    {"a query": case["q"][300], "queries": case["q"], "keys": case["kc"], "values": case["vc"]}[bad].fill_(float("nan"))
    assert _milliseconds(run) < 10 * finite
    assert torch.isnan(out).all() if bad != "a query" else torch.isnan(out).any(1).sum() == 1


@pytest.mark.parametrize("D,splits", [(64, 1), (64, 3), (128, 1), (128, 8)])
@pytest.mark.parametrize("window,bad", [(0, None), (50, None), (0, "key"), (0, "query")])
def test_single_tokens_beside_portions_on_the_decode_kernel(D, splits, window, bad):
    """Requests of one token (the first of a context among them) beside portions; a NaN key or query is one in every row that sees it."""
    from sandyrt_b200.csrc import ops

    seqs = [(0, 1), (40, 1), (0, 70), (199, 1), (330, 1), (64, 65), (17, 1)]
    case = _paged_case(torch.float32, 4, 2, D, 16, seqs, seed=D)
    if bad == "key":
        case["kc"][int(case["table"][4, 200 // 16]), :, 200 % 16] = float("nan")
    if bad == "query":
        case["q"][1 + 1 + 70] = float("nan")                # the token behind 199
    sink = torch.tensor([0.5, -1.0, 0.0, 2.0], device=DEV)
    q_start = torch.tensor([0] + list(np.cumsum([n for _, n in seqs])), dtype=torch.int32, device=DEV)
    kv_before = torch.tensor([b for b, _ in seqs], dtype=torch.int32, device=DEV)
    outs = [torch.full(case["q"].shape, 7.0, device=DEV) for _ in range(2)]
    for out, kw in zip(outs, ({}, {"tc": True, "single_splits": splits})):
        ops.prefill_attention_f32(case["q"], case["kc"], case["vc"], case["table"], q_start, kv_before, out, n_heads=4, max_q_len=70, scale=0.1,
                                  window=window, sink=sink, **kw)
    ops.check_kernel_status(DEV)
    want, got = outs
    assert torch.isnan(want).any() == (bad is not None) and torch.equal(torch.isnan(got), torch.isnan(want))
    fine = ~torch.isnan(want)
    assert (got - want)[fine].abs().max().item() < 2e-5         # the bound of test_prompt_attention_f32


@pytest.mark.parametrize("D,splits", [(64, 1), (64, 3), (128, 8)])
@pytest.mark.parametrize("with_sink", [False, True])
def test_single_tokens_whose_scores_are_all_minus_infinity(D, splits, with_sink):
    """A row ends the same beside many single tokens as beside few: 0 / 0 of the formula without a sink, 0 with one."""
    from sandyrt_b200.csrc import ops

    seqs = [(40, 1), (0, 70), (330, 1), (0, 1)]
    case = _paged_case(torch.float32, 4, 2, D, 16, seqs, seed=D)
    for row, request in ((0, 0), (72, 3)):                  # queries above zero, every key of their requests -inf
        case["q"][row] = case["q"][row].abs()
        pages = case["table"][request]
        case["kc"][pages[pages >= 0].long()] = -float("inf")
    sink = torch.tensor([0.5, -1.0, 0.0, 2.0], device=DEV) if with_sink else None
    q_start = torch.tensor([0] + list(np.cumsum([n for _, n in seqs])), dtype=torch.int32, device=DEV)
    kv_before = torch.tensor([b for b, _ in seqs], dtype=torch.int32, device=DEV)
    outs = []
    for kw in ({}, {"tc": True}, {"tc": True, "single_splits": splits}):
        outs.append(torch.full(case["q"].shape, 7.0, device=DEV))
        ops.prefill_attention_f32(case["q"], case["kc"], case["vc"], case["table"], q_start, kv_before, outs[-1], n_heads=4, max_q_len=70,
                                  scale=0.1, sink=sink, **kw)
    ops.check_kernel_status(DEV)
    for got in outs:
        for row in (0, 72):
            assert torch.isnan(got[row]).all() if sink is None else (got[row] == 0.0).all()
        assert torch.isfinite(got[1:72]).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("size", [2.0 ** -100, 2.0 ** 45])
def test_prompt_attention_f32_sizes_on_tensor_cores(on_tensor_cores, D, size):
    """Small keys and values, and ones too large to be split."""
    case = _paged_case(torch.float32, 2, 2, D, 16, [(0, 130), (63, 65)], seed=D)
    case["kc"] *= size
    case["vc"] *= size
    got, want = _both(case, 2, {"scale": 0.8 / D ** 0.5 / size})
    assert (got - want).abs().max().item() < 2e-5 * size        # the bound of test_prompt_attention_f32


@pytest.mark.parametrize("D", [64, 80, 128])
def test_prompt_attention_f32_on_tensor_cores_keeps_24_bits(on_tensor_cores, D):
    """A query that sees one key has that key's value, every bit of it: its weight is 1, and a value is the sum of its pieces.  With all
    keys: scores of up to 4 may be off by ONE_PRODUCT of the products they add up (sizes of about their own), an exponential by 2^-22, and
    so may the weights' sum; the 2-norm stays below a quarter of what the worst of them add up to, 2^-19.  Scores without their last pieces
    are off by 2^-17."""
    case = _paged_case(torch.float32, 4, 2, D, 16, [(0, 130), (63, 65), (200, 70)], seed=D)
    got, _ = _both(case, 4, {"scale": 1.0, "window": 1})
    own = torch.cat([v[before:].repeat_interleave(2, 1).reshape(n, -1) for (before, n), v in zip(case["seqs"], case["dense_v"])])
    assert torch.equal(got.cpu(), own)
    case["dense_k"], case["dense_v"] = ([x.repeat_interleave(2, 1) for x in case[name]] for name in ("dense_k", "dense_v"))
    got, _ = _both(case, 4, {"scale": D ** -0.5})
    want = _formula(case, 4, D ** -0.5, 0, None)
    assert float((got.double().cpu() - want).norm() / want.norm()) < 2.0 ** -21


@pytest.mark.parametrize("D", [64, 128])
def test_prompt_attention_f32_of_very_small_keys_on_tensor_cores(on_tensor_cores, D):
    """Keys and values of 2^-120, whose last pieces would lie below a bfloat16's range were they not scaled, under queries that make ordinary
    scores of them."""
    case = _paged_case(torch.float32, 2, 2, D, 16, [(0, 130), (63, 65)], seed=D)
    case["kc"] *= 2.0 ** -120
    case["vc"] *= 2.0 ** -120
    case["q"] *= 2.0 ** 35
    got, _ = _both(case, 2, {"scale": 2.0 ** 85 / D ** 0.5})
    want = _formula(case, 2, D ** -0.5, 0, None)
    assert float((got.double().cpu() * 2.0 ** 120 - want).norm() / want.norm()) < 2.0 ** -21


@pytest.mark.parametrize("rules", RULES)
@pytest.mark.parametrize("D", [64, 80, 128])
def test_values_too_large_to_be_split_under_every_rule(on_tensor_cores, D, rules):
    """Some entries of some values at 2^100: their part is added by itself, with the weights that the rules give their keys."""
    case = _paged_case(torch.float32, 2, 2, D, 16, [(0, 130), (40, 1), (63, 65), (199, 70)], seed=D)
    g = torch.Generator().manual_seed(D)
    for s, pages, slots in _keys_of(case):
        some = torch.rand(len(pages), 1, 1, generator=g) < 0.2
        case["vc"][pages, :, slots] *= torch.where(some & (torch.rand(1, 2, D, generator=g) < 0.3), 2.0 ** 100, 1.0).to(DEV)
    kw = {k: v for k, v in rules.items() if k in ("window", "keep_first", "softcap", "chunk")}
    kw["scale"] = 0.8 / D ** 0.5
    if rules.get("sink"):
        kw["sink"] = torch.randn(2, generator=g).to(DEV)
    if rules.get("bias"):
        kw["dist_bias"] = torch.randn(2, rules["bias"], generator=g).to(DEV)
    got, want = _both(case, 2, kw)
    small = want.abs() < 2.0 ** 60
    assert small.any() and not small.all()
    assert (got - want)[~small].abs().max().item() < 2e-5 * 2.0 ** 100          # the bound of test_prompt_attention_f32
    assert (got - want)[small].abs().max().item() < 2e-5


def _keys_of(case):
    """(request, its context's pages and slots) of a _paged_case."""
    for s, (before, n) in enumerate(case["seqs"]):
        at = torch.arange(before + n, device=DEV)
        yield s, case["table"][s, at // 16].long(), at % 16


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("top", [1e8, 3e9, -3e9, 1e10, -1e30])
def test_large_scores_on_tensor_cores(on_tensor_cores, D, top):
    """Scores so far apart that a row is the value of its largest one: its weight is exactly 1, and 24 bits of the value are kept."""
    case = _paged_case(torch.float32, 2, 2, D, 16, [(0, 150), (90, 70)], seed=D)
    g = torch.Generator().manual_seed(D)
    case["q"].fill_(1.0)
    best = []
    for s, pages, slots in _keys_of(case):
        before, n = case["seqs"][s]
        size = 1.0 + torch.randperm(before + n, generator=g).to(DEV) / (before + n)         # at least a 300th apart
        case["kc"][pages, :, slots] = size[:, None, None]
        best += [case["vc"][pages, :, slots][(size * np.sign(top))[:before + i + 1].argmax()].reshape(-1) for i in range(n)]
    got, general = _both(case, 2, {"scale": top / D})
    want = torch.stack(best)
    assert (got - want).abs().max().item() <= 2.0 ** -22 * want.abs().max().item()
    assert (general - want).abs().max().item() <= 2.0 ** -22 * want.abs().max().item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("low", [-1e9, -1e30, -3.4028234663852886e38])
def test_a_bias_that_hides_far_keys_on_tensor_cores(on_tensor_cores, D, low):
    """A bias of very low values is a window; whole tiles have it in front of the keys that count."""
    from sandyrt_b200.csrc import ops

    case = _paged_case(torch.float32, 2, 2, D, 16, [(0, 200), (90, 70)], seed=D)
    bias = torch.zeros(2, 300, device=DEV)
    bias[:, 40:] = low
    got, _ = _both(case, 2, {"scale": 0.8 / D ** 0.5, "dist_bias": bias})
    want = torch.empty_like(got)
    ops.paged_attention(case["q"], case["kc"], case["vc"], case["table"], case["tok_seq"], case["tok_pos"], want, n_heads=2,
                        scale=0.8 / D ** 0.5, window=40)
    assert (got - want).abs().max().item() < 2e-5               # the bound of test_prompt_attention_f32


@pytest.mark.parametrize("name", ["A", "C"])
def test_float32_portions_on_both_sides_of_the_rule(model_dirs, plain_models, name):
    """Heads of 16 and 48: prompts of 32 to 100 tokens (48 is the last that the general kernel keeps) and portions behind a context,
    alone and together; the same step again is a replay."""
    from sandyrt_b200.engine.step import Engine, StepEntry
    from sandyrt_b200.models.model import load_model
    from test_replay_gpu import _close

    plain = plain_models(name, "f32")
    eng = Engine(load_model(model_dirs[name], device="cuda:0", dtype=torch.float32), max_tokens=512, max_requests=8)
    eng.cache.device_caches.poison()
    ids = np.random.default_rng(4).integers(0, 512, size=100).tolist()

    def step(parts):
        out = eng.step([StepEntry(r, ids[a:b], list(range(b - a))) for r, a, b in parts]).cpu().numpy()
        at = 0
        for r, a, b in parts:
            _close(out[at:at + b - a], plain.logits(ids[:b])[a:], "float32", f"{name} {parts}")
            at += b - a

    for n in (32, 48, 49, 64, 100):
        for _ in range(3):
            step([("r", 0, n)])
            eng.release("r")
    step([("a", 0, 31), ("b", 0, 5), ("c", 0, 17)])
    for b in range(31, 63, 4):                          # portions of four tokens, from 35 keys to 63
        step([("a", b, b + 4)])
    for n in (5, 9, 13, 17, 21, 25, 29, 33):
        step([("b", n, n + 4), ("c", 12 + n, 16 + n)])
    assert eng.graph_replays >= 4


# ---- one small matrix per group of rows or columns ---------------------------------------------------------------------
@pytest.mark.parametrize("sizes,N,K", [([1, 0, 2, 1], 33, 132), ([3, 3, 3], 4, 4), ([64, 65, 0, 127, 1], 130, 100), ([200], 64, 64), ([5, 9], 1000, 768)])
def test_expert_product_f32(sizes, N, K):
    """Few rows a group and many, tile edges, empty groups, gathered rows; K that is no multiple of a step."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(N + K)
    n, G = sum(sizes), len(sizes)
    a, w = torch.randn(n, K, generator=g), torch.randn(G, N, K, generator=g)
    rows = torch.randperm(n, generator=g).to(torch.int32)
    start = torch.tensor([0] + list(np.cumsum(sizes)), dtype=torch.int32)
    out = torch.full((n, N), float("nan"), device=DEV)
    r = types.SimpleNamespace(n_experts=G, n_tokens=n, top=1, group_start=start.to(DEV), entry_of_slot=rows.to(DEV))
    ops.expert_product(r, a.to(DEV), w.view(G * N, K).to(DEV), out, gather=True, act="relu_squared")
    src = a[rows.long()].double()
    which = torch.repeat_interleave(torch.arange(G), torch.tensor(sizes))
    z = torch.einsum("sk,snk->sn", src, w[which].double())
    size = torch.einsum("sk,snk->sn", src.abs(), w[which].double().abs())
    off = (K + 2) * 2.0 ** -24 * size                       # of a sum of K products in any order; its square moves by 2 |z| off
    want = torch.relu(z) ** 2
    assert bool(((out.double().cpu() - want).abs() <= 2 * torch.relu(z) * off + off ** 2 + 2.0 ** -23 * want).all())


@pytest.mark.parametrize("sizes", [[1, 0, 2, 1], [64, 65, 0, 127]])
@pytest.mark.parametrize("K", [4, 132, 260])
def test_expert_product_f32_infinity_at_the_end_of_a_row(sizes, K):
    """As in the dense products, for groups of few rows and of many."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(K)
    n, G, N = sum(sizes), len(sizes), 40
    a, w = torch.randn(n, K, generator=g), torch.randn(G, N, K, generator=g)
    start = torch.tensor([0] + list(np.cumsum(sizes)), dtype=torch.int32)
    r = types.SimpleNamespace(n_experts=G, n_tokens=n, top=1, group_start=start.to(DEV), entry_of_slot=torch.arange(n, dtype=torch.int32).to(DEV))
    a[n - 1, K - 2] = float("inf")
    out = torch.full((n, N), float("nan"), device=DEV)
    ops.expert_product(r, a.to(DEV), w.view(G * N, K).to(DEV), out, gather=True)
    last = max(i for i, size in enumerate(sizes) if size)
    assert torch.equal(out[n - 1].cpu(), torch.sign(w[last, :, K - 2]) * float("inf"))
    assert torch.isfinite(out[:n - 1]).all()


@pytest.mark.parametrize("sizes,N,K", [([1, 0, 2, 1], 33, 132), ([128, 129, 0, 127, 1], 130, 576), ([300], 64, 64), ([5, 9], 1000, 768)])
def test_expert_product_f32_on_tensor_cores(sizes, N, K):
    """Tiles that begin and end inside a's rows, empty groups, columns behind N that are the next expert's; an infinite activation stays
    its own row's; rows behind the last group are not written."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(N + K)
    n, G = sum(sizes), len(sizes)
    a, w = torch.randn(n + 3, K, generator=g), torch.randn(G, N, K, generator=g)
    a[n:] = float("nan")
    start = torch.tensor([0] + list(np.cumsum(sizes)), dtype=torch.int32)
    r = types.SimpleNamespace(n_experts=G, n_tokens=n + 3, top=1, group_start=start.to(DEV))
    out = torch.full((n + 3, N), 7.0, device=DEV)
    ops.expert_product_f32_tc(r, a.to(DEV), w.view(G * N, K).to(DEV), out, act="relu_squared")
    which = torch.repeat_interleave(torch.arange(G), torch.tensor(sizes))
    z = torch.einsum("sk,snk->sn", a[:n].double(), w[which].double())
    off = (K + 2) * 2.0 ** -24 * torch.einsum("sk,snk->sn", a[:n].double().abs(), w[which].double().abs())
    want = torch.relu(z) ** 2
    assert bool(((out[:n].double().cpu() - want).abs() <= 2 * torch.relu(z) * off + off ** 2 + 2.0 ** -23 * want).all())
    assert bool((out[n:] == 7.0).all())
    finite, again = torch.empty(n + 3, N, device=DEV), torch.empty(n + 3, N, device=DEV)
    ops.expert_product_f32_tc(r, a.to(DEV), w.view(G * N, K).to(DEV), finite)
    a[n - 1, K - 1] = float("inf")
    ops.expert_product_f32_tc(r, a.to(DEV), w.view(G * N, K).to(DEV), again)
    assert torch.equal(again[n - 1].cpu(), torch.sign(w[which[n - 1], :, K - 1]) * float("inf"))
    assert torch.equal(again[:n - 1], finite[:n - 1])
    assert int(ops.kernel_status(out.device).item()) == 0


@pytest.mark.parametrize("sizes,N,K", [([128, 129, 0, 127, 1], 130, 576), ([300], 64, 516), ([5, 9], 1000, 768)])
def test_expert_product_f32_on_tensor_cores_keeps_24_bits(sizes, N, K):
    """As test_gemm_f32_on_tensor_cores_keeps_24_bits, a matrix per expert."""
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(N + K)
    n, G = sum(sizes), len(sizes)
    at = torch.arange(n) * 37 % K
    a, w = torch.zeros(n, K), 1.0 + torch.rand(G, N, K, generator=g)
    a[torch.arange(n), at] = 1.0 + torch.rand(n, generator=g)
    start = torch.tensor([0] + list(np.cumsum(sizes)), dtype=torch.int32)
    r = types.SimpleNamespace(n_experts=G, n_tokens=n, top=1, group_start=start.to(DEV))
    out = torch.empty(n, N, device=DEV)
    ops.expert_product_f32_tc(r, a.to(DEV), w.view(G * N, K).to(DEV), out)
    which = torch.repeat_interleave(torch.arange(G), torch.tensor(sizes))
    want = a[torch.arange(n), at].double()[:, None] * w[which, :, at].double()
    assert bool(((out.double().cpu() - want).abs() <= ONE_PRODUCT * want.abs()).all())


@pytest.mark.parametrize("T", [1, 4, 5, 64, 65, 150])
def test_head_product_f32(T):
    from sandyrt_b200.csrc import ops

    g = torch.Generator().manual_seed(T)
    a, w = torch.randn(T, 3 * 100 + 4, generator=g), torch.randn(3, 40, 96, generator=g)
    out = torch.full((T, 3 * 48), 7.0, device=DEV)
    ops.head_product(a.to(DEV), w.view(120, 96).to(DEV), out, n_groups=3, a_gcols=100, o_gcols=48)
    for h in range(3):
        want = a[:, h * 100:h * 100 + 96].double() @ w[h].double().t()
        bound = 97 * 2.0 ** -24 * (a[:, h * 100:h * 100 + 96].double().abs() @ w[h].double().abs().t())
        assert bool(((out[:, h * 48:h * 48 + 40].double().cpu() - want).abs() <= bound).all())
        assert bool((out[:, h * 48 + 40:(h + 1) * 48] == 7.0).all())
