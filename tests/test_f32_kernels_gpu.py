"""The float32 kernels alone, at the edges of their tiles and splits, against torch in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


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


def test_gemm_f32_refuses_what_it_cannot_load():
    from sandyrt_b200.csrc import ops

    a, w, out = torch.zeros(3, 6, device=DEV), torch.zeros(5, 6, device=DEV), torch.zeros(3, 5, device=DEV)
    with pytest.raises(ops.UnsupportedShape):
        ops.gemm_f32(a, w, None, out)                                       # K is no multiple of 4
    with pytest.raises(ops.UnsupportedShape):
        ops.gemm_f32(torch.zeros(25, device=DEV)[1:].view(3, 8)[:, :4], w[:, :4].contiguous(), None, out)   # not on 16 bytes
