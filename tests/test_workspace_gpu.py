"""A device with no room left: steps that ran without the recurrences' scratch for whole prompts still run."""
import contextlib
import gc

import numpy as np
import pytest
import torch

from panupel_models import delta, make_weights, rel_error, write_model, _config

pytestmark = pytest.mark.gpu

# 24 heads: a step of two prompts of 1,024 tokens asks for 65 MB of scratch, more than is left
CONFIG = _config(97, 64, [delta(24, 2, 64, 64, 4, ff=96)])
LEFT = 24 << 20


@pytest.fixture(scope="module")
def folder(tmp_path_factory):
    return write_model(CONFIG, make_weights(CONFIG, seed=5), str(tmp_path_factory.mktemp("workspace") / "model"))


def _engine(folder):
    from sandyrt_b200.engine.step import Engine
    from sandyrt_b200.models.model import load_model

    return Engine(load_model(folder, device="cuda:0", dtype=torch.float32), max_tokens=4096, max_requests=64, max_step_tokens=4096)


def _step(eng, n, length, seed=1):
    from sandyrt_b200.engine.step import StepEntry

    rng = np.random.default_rng(seed)
    out = eng.step([StepEntry(i, rng.integers(0, 97, size=length).tolist(), [length - 1]) for i in range(n)]).cpu().numpy().copy()
    for i in range(n):
        eng.release(i)
    return out


@contextlib.contextmanager
def _full_device():
    """All but LEFT of the device's memory is taken meanwhile."""
    gc.collect()
    torch.cuda.empty_cache()
    held = [torch.empty(torch.cuda.mem_get_info()[0] - LEFT, dtype=torch.uint8, device="cuda:0")]
    try:
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def test_no_room_for_the_scratch(folder):
    want = _step(_engine(folder), 2, 1024)
    eng = _engine(folder)
    _step(eng, 32, 64)                      # as many tokens, in portions that take no scratch: every other buffer has its size
    with _full_device():
        got = [_step(eng, 2, 1024) for _ in range(3)]       # eager, recorded, replayed
    assert eng.graph_replays == 2
    assert all(np.array_equal(got[0], g) for g in got) and rel_error(got[0], want) < 2e-4


def test_scratch_makes_room_for_what_a_step_cannot_do_without(folder):
    want = _step(_engine(folder), 48, 64)
    eng = _engine(folder)
    first = _step(eng, 2, 1024)
    with _full_device():
        got = _step(eng, 48, 64)            # half as many tokens again: every buffer grows
        again = _step(eng, 2, 1024)
    assert rel_error(got, want) < 2e-4 and rel_error(again, first) < 2e-4
