"""The 32-bit product's two tile shapes give the same bits for the same row, whatever else is in the batch, and both hold to float64."""
import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(4800, 36), (4672, 64), (4801, 130), (9500, 200), (4736, 33)])
@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
def test_rows_do_not_depend_on_the_tile(N, K, wdt):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randn((130, K), generator=g, device="cuda")
    w = torch.randn((N, K), generator=g, device="cuda").to(wdt)
    whole = torch.empty((130, N), device="cuda")
    ops.gemm_simt(whole, a, w)                                 # 64 x 64 tiles
    for lo, hi in ((0, 1), (1, 17), (17, 50), (113, 130)):     # 16 x 32 tiles
        part = torch.empty((hi - lo, N), device="cuda")
        ops.gemm_simt(part, a[lo:hi], w)
        assert torch.equal(part, whole[lo:hi])
    narrow = torch.empty((130, 95), device="cuda")
    ops.gemm_simt(narrow, a, w[:95])
    assert torch.equal(narrow, whole[:, :95])
    want = a.double() @ w.double().T
    # K products of order one added one by one: each addition off by half an ulp of a sum of order sqrt(K)
    assert float((whole - want).abs().max()) <= K * K ** 0.5 * 4 * 2.0 ** -24


def test_weights_that_the_launch_in_front_writes():
    """A matrix that the launch ahead of the product writes (one wave of tiles, whose ring would hold its first ones): what that launch left."""
    g = torch.Generator(device="cuda").manual_seed(4)
    a, left, right = (torch.randn(s, generator=g, device="cuda") for s in ((16, 1024), (3, 4096, 64), (1024, 64)))
    w, out = torch.zeros(4096, 1024, device="cuda"), torch.empty(3, 16, 4096, device="cuda")
    for i in range(3):
        ops.gemm_simt(w, left[i], right)
        ops.gemm_simt(out[i], a, w)
    for i in range(3):
        want = torch.empty(16, 4096, device="cuda")
        ops.gemm_simt(w, left[i], right)
        torch.cuda.synchronize()
        ops.gemm_simt(want, a, w, settled=True)
        torch.cuda.synchronize()
        assert torch.equal(out[i], want)
