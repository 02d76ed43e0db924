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
