"""Attention of a step that holds single tokens beside portions, in two launches, against the formula in 64 bits."""
import numpy as np
import pytest
import torch

from test_kernels_gpu import ATT_TOL, DEV, _paged_case
from test_linear_kernels_gpu import _gate, _want

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hkv,page_size,window,keep,splits", [(4, 2, 16, 0, 0, 1), (3, 3, 8, 0, 0, 3), (12, 4, 16, 0, 0, 8), (2, 1, 32, 60, 0, 2),
                                                                (6, 2, 16, 100, 19, 4)])
@pytest.mark.parametrize("seqs", [[(699, 1), (0, 130), (0, 1), (63, 1), (300, 64), (64, 1), (5, 2)], [(0, 2)], [(40, 3), (100, 70)]])
def test_portions_and_single_tokens(H, Hkv, page_size, window, keep, splits, seqs):
    """Single tokens in front of, between and behind portions; portions alone (the second launch then leaves every row alone)."""
    from sandyrt_b200.csrc import ops

    case = _paged_case(torch.bfloat16, H, Hkv, 64, page_size, seqs, seed=H + window)
    lens = [n for _, n in seqs]
    q_start = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device=DEV)
    kv_before = torch.tensor([b for b, _ in seqs], dtype=torch.int32, device=DEV)
    gate = _gate(case, H, 59, seed=H) if keep else None
    sink = torch.zeros(H, device=DEV) if keep else None
    out = torch.full_like(case["q"], float("nan"))
    ops.mixed_attention(case["q"], case["kc"], case["vc"], case["table"], q_start, kv_before, out, n_heads=H, max_q_len=max(lens), scale=0.1,
                        window=window, keep_first=keep, elem_gate=gate, sink=sink, num_splits=splits)
    ops.check_kernel_status(DEV)
    want = _want(case, H, Hkv, 0.1, window, keep, bool(keep), None if gate is None else gate.double().cpu(), 59)
    assert (out.double().cpu() - want).abs().max().item() < ATT_TOL[torch.bfloat16] * 1.5


# ---- through the engine -----------------------------------------------------------------------------------------
HEADS, WIDTH, LAYERS, VOCAB = 16, 1024, 2, 301


@pytest.fixture(scope="module")
def wide(tmp_path_factory):
    from conftest import make_model_dir
    from plain_gpt2 import PlainGPT2

    folder = make_model_dir(dict(architectures=["GPT2LMHeadModel"], model_type="gpt2", n_layer=LAYERS, n_embd=WIDTH, n_head=HEADS, n_inner=512,
                                 vocab_size=VOCAB, n_positions=512, layer_norm_epsilon=1e-5, activation_function="gelu_new"),
                            str(tmp_path_factory.mktemp("mixed") / "model"), seed=8)
    return folder, PlainGPT2(folder, "bf16")


class _Running:
    """An engine and what its requests have been fed."""

    def __init__(self, wide, contexts, seed, dtype=torch.bfloat16):
        from sandyrt_b200.engine.step import Engine
        from sandyrt_b200.models.model import load_model

        self.plain = wide[1]
        self.eng = Engine(load_model(wide[0], device="cuda:0", dtype=dtype), max_tokens=8192, max_requests=48)
        # two layers of bfloat16 roundings in another order: 5e-3 of the row; of float32 ones: 1e-6; a row that no launch wrote is off by
        # its size
        self.tol = 2e-2 if dtype == torch.bfloat16 else 1e-5
        self.eng.cache.device_caches.poison()
        self.rng = np.random.default_rng(seed)
        self.fed = {}
        for r, n in enumerate(contexts):
            self.step([(r, n)], check=False)

    def step(self, portions, check=True):
        """portions: (request, tokens) in the step's order; every request's last row against the plain model's."""
        from sandyrt_b200.engine.step import StepEntry

        entries = []
        for r, n in portions:
            ids = self.rng.integers(0, VOCAB, size=n).tolist()
            self.fed[r] = self.fed.get(r, []) + ids
            entries.append(StepEntry(r, ids, [n - 1]))
        got = self.eng.step(entries).cpu().double().numpy()
        if check:
            for (r, n), row in zip(portions, got):
                want = self.plain.logits(self.fed[r], [len(self.fed[r]) - 1])[0].astype(np.float64)
                assert np.linalg.norm(row - want) < self.tol * np.linalg.norm(want), (r, n, portions)
        return self.eng.last_launches


def _contexts(n):
    return [3 + 7 * i % 61 for i in range(n - 1)] + [150]           # one behind a table of more than 128 keys


@pytest.mark.parametrize("singles", [15, 16, 20, 33])
def test_engine_steps_of_single_tokens_beside_a_portion(wide, singles):
    """Below and from 256 (token, head) pairs on; the same counts with the portion first, last and in the middle, so that one
    recording serves requests that have changed places."""
    run = _Running(wide, _contexts(singles), seed=singles)
    launches, replays = [], run.eng.graph_replays
    for step, at in enumerate((singles, 0, singles // 2, 1)):
        portions = [(r, 1) for r in range(singles)]
        portions.insert(at, (f"new {step}", 37))
        launches.append(run.step(portions))
        run.eng.release(f"new {step}")
    assert run.eng.graph_replays - replays == 3 and len(set(launches)) == 1
    alone = _Running(wide, [3], seed=1)
    one = alone.step([(0, 1), ("new", 37)])
    assert launches[0] - one == (LAYERS if singles >= 16 else 0)


def test_engine_step_without_single_tokens_takes_no_second_launch(wide):
    """Ragged prompts whose counts would allow for many single tokens, beside prompts with as many tokens and no room for one."""
    run = _Running(wide, [2], seed=5)
    launches = []
    for lengths in ([270] + [20] * 24, [30] * 25):
        for time in range(2):                               # (a product's first step at a new size tries its kernels)
            requests = [f"{time} {i}" for i in range(25)]
            n = run.step(list(zip(requests, lengths)))
            for r in requests:
                run.eng.release(r)
                del run.fed[r]
        launches.append(n)
    assert launches[0] == launches[1]


def test_engine_recording_is_not_shared_by_steps_with_and_without_single_tokens(wide):
    """Equal tokens, requests and longest portion: sixteen single tokens beside two portions, then portions alone."""
    run = _Running(wide, [150] + [4] * 17, seed=6)
    for _ in range(2):
        run.step([(r, 1) for r in range(16)] + [(16, 40), (17, 24)])
    for _ in range(2):
        run.step([(0, 40)] + [(r, 2) for r in range(1, 7)] + [(r, 3) for r in range(7, 13)] + [(r, 2) for r in range(13, 18)])
    for _ in range(2):
        run.step([(r, 1) for r in range(2, 18)] + [(1, 24), (0, 40)])


# ---- the same in float32 ------------------------------------------------------------------------------------------
@pytest.fixture(scope="module")
def models32(tmp_path_factory):
    """16 heads of 64, which the decode kernel has a form for, and 16 of 48, which it has none for."""
    from conftest import make_model_dir
    from plain_gpt2 import PlainGPT2

    out = {}
    for size in (64, 48):
        folder = make_model_dir(dict(architectures=["GPT2LMHeadModel"], model_type="gpt2", n_layer=LAYERS, n_embd=HEADS * size, n_head=HEADS,
                                     n_inner=256, vocab_size=VOCAB, n_positions=1024, layer_norm_epsilon=1e-5, activation_function="gelu_new"),
                                str(tmp_path_factory.mktemp("mixed32") / "model"), seed=8)
        out[size] = (folder, PlainGPT2(folder, "f32"))
    return out


def _attention_classes(run, portions):
    """The classes of attention launches in a step that is not a recorded one."""
    from sandyrt_b200 import core

    core.call("global", None, "profile_kernels", enable=True)
    try:
        run.step(portions)
    finally:
        rows = core.call("global", None, "profile_kernels", enable=False)
    return {r["class"] for r in rows if r["class"].startswith("attention")}


# Heads of 64 leave the prompt kernel behind a table of more than 128 keys from 150 (token, head) pairs on; what cannot leave it stays on the
# tensor cores up to a round of blocks on 148 SMs, up to two behind 256 keys and more.
@pytest.mark.parametrize("size,singles,longest,apart,kernel", [
    (64, 9, 150, False, "tcgen05"), (64, 10, 150, True, "tcgen05"), (64, 15, 150, True, "tcgen05"), (64, 16, 150, True, "tcgen05"),
    (64, 33, 150, True, "tcgen05"), (64, 16, 820, True, "tcgen05"), (64, 9, 60, False, "tcgen05"), (64, 10, 60, False, "fma"),
    (48, 9, 60, False, "tcgen05"), (48, 10, 60, False, "fma"), (48, 18, 150, False, "tcgen05"), (48, 19, 150, False, "fma"),
    (48, 33, 820, False, "fma")])
def test_engine_steps_of_single_tokens_beside_a_portion_in_float32(models32, size, singles, longest, apart, kernel):
    run = _Running(models32[size], _contexts(singles)[:-1] + [longest], seed=singles, dtype=torch.float32)
    launches, replays = [], run.eng.graph_replays
    for step, at in enumerate((singles, 0, singles // 2, 1)):
        portions = [(r, 1) for r in range(singles)]
        portions.insert(at, (f"new {step}", 37))
        if step == 0:
            want = "attention, prompt (float32, tcgen05)" if kernel == "tcgen05" else "attention, prompt (float32)"
            assert _attention_classes(run, portions) == {want}
        else:
            run.step(portions)
        launches.append(run.eng.last_launches)
        run.eng.release(f"new {step}")
    assert run.eng.graph_replays - replays >= 2 and len(set(launches)) == 1
    alone = _Running(models32[size], [3], seed=1, dtype=torch.float32)
    one = alone.step([(0, 1), ("new", 37)])
    assert launches[0] - one == (LAYERS if apart else 0)


def test_engine_recording_in_float32_is_not_shared_by_steps_with_and_without_single_tokens(models32):
    """Equal tokens, requests and longest portion: sixteen single tokens beside two portions, then portions alone."""
    run = _Running(models32[64], [150] + [4] * 17, seed=6, dtype=torch.float32)
    for _ in range(2):
        run.step([(r, 1) for r in range(16)] + [(16, 40), (17, 24)])
    for _ in range(2):
        run.step([(0, 40)] + [(r, 2) for r in range(1, 7)] + [(r, 3) for r in range(7, 13)] + [(r, 2) for r in range(13, 18)])
    for _ in range(2):
        run.step([(r, 1) for r in range(2, 18)] + [(1, 24), (0, 40)])
