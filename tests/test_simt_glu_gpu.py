"""The 32-bit gated product in one launch gives the bits of the product followed by the activation."""
import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


# one wave (one launch) at the edges of a tile of rows, of k and of the ring; then a wave and a CTA, and k, rows and starts that are no whole pieces
# (two launches)
@pytest.mark.parametrize("M,f,K,lead", [(1, 16, 4, 0), (3, 512, 192, 0), (16, 1184, 64, 0), (17, 1184, 68, 0), (33, 496, 512, 0), (16, 2368, 516, 0),
                                        (16, 2384, 516, 0), (17, 1200, 64, 0), (300, 512, 64, 0), (5, 64, 30, 0), (5, 64, 64, 1)])
@pytest.mark.parametrize("act", [ops.GLU_SILU, ops.GLU_GELU_TANH, ops.GLU_CLAMPED])
def test_one_launch_as_two(M, f, K, lead, act):
    g = torch.Generator(device="cuda").manual_seed(M + f + K)
    x = torch.randn(M * K + lead, generator=g, device="cuda")[lead:].view(M, K)
    w = torch.randn((2 * f, K), generator=g, device="cuda") * K ** -0.5
    opts = dict(limit=1.5, slope=1.7) if act == ops.GLU_CLAMPED else {}
    gu = torch.empty((M, 2 * f), device="cuda")
    want, got = torch.empty((M, f), device="cuda"), torch.full((M, f), float("nan"), device="cuda")
    ops.gemm_simt(gu, x, w)
    ops.glu_act(want, gu, act, interleaved=True, **opts)
    ops.gemm_swiglu(got, x, w, act=act, **opts)
    assert torch.equal(got, want)
