"""The passes ahead of differential and latent attention over portions (vector accesses, several warps a token) against the steps of up to 32 tokens,
which take the general kernels: at most one rounding of the stored type apart, and seldom; and, with the sums in their order, the same bits."""
from types import SimpleNamespace

import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def setup(T, page, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    i32 = dict(dtype=torch.int32, device="cuda")
    pages = -(-T // page)
    bt = torch.randperm(pages, generator=g, device="cuda").to(torch.int32)[None].contiguous()
    return (lambda *s: torch.randn(s, generator=g, device="cuda")), bt, torch.arange(T, **i32), torch.zeros(T, **i32), pages


def parts(T):
    return [(a, min(a + 30, T)) for a in range(0, T, 30)]


def close(got, want):
    d = (got.float() - want.float()).abs()
    assert bool((d <= 2.0 ** -7 * want.float().abs() + 1e-6).all()) and float((d > 0).float().mean()) < 0.01


@pytest.mark.parametrize("n,dv,rot", [(32, 4, 0), (32, 36, 32), (64, 128, 64), (64, 64, 16), (128, 20, 96)])
@pytest.mark.parametrize("H,G,normed,bias", [(2, 1, True, True), (5, 5, False, False), (6, 2, True, False)])
def test_differential(n, dv, rot, H, G, normed, bias):
    T, page = 75, 16
    rnd, bt, pos, seg, pages = setup(T, page, n + dv + H)
    proj = rnd(T, (H + G) * 2 * n + G * dv)
    b, qw, kw = rnd(proj.shape[1]) if bias else None, rnd(n) if normed else None, rnd(n) if normed else None
    cs = rnd(60, rot // 2, 2).reshape(60, rot).contiguous() if rot else None   # (positions beyond the table take its last row)
    table = cs.view(60, rot // 2, 2).contiguous() if rot else None

    def run(cuts):
        q, cache = torch.full((T, H * 2 * n), float("nan"), device="cuda", dtype=BF16), torch.zeros(pages, page, G * (2 * n + dv), device="cuda", dtype=BF16)
        for a, e in cuts:
            ctx = SimpleNamespace(tok_pos=pos[a:e], tok_seg=seg[a:e])
            ops.diff_prepare(q[a:e], proj[a:e], b, qw, kw, 1e-5, table, ctx, bt, cache, H, G, n, dv, rot, page)
        return q, cache

    for got, want in zip(run([(0, T)]), run(parts(T))):
        close(got, want)


@pytest.mark.parametrize("rank,dr,rot,dn", [(8, 8, 8, 2), (256, 64, 64, 128), (512, 64, 32, 64), (1024, 72, 70, 6), (520, 8, 0, 128)])
def test_latent(rank, dr, rot, dn):
    T, page, H = 75, 16, 7
    rnd, bt, pos, seg, pages = setup(T, page, rank + dr)
    width = H * (dn + dr)
    kv_off = -(-width // 8) * 8
    source, w = rnd(T, -(-(kv_off + rank + dr) // 8) * 8).to(BF16), rnd(rank)
    table = rnd(60, rot // 2, 2) if rot else None

    def run(cuts):
        proj, cache = source.clone(), torch.zeros(pages, page, rank + dr, device="cuda", dtype=BF16)
        for a, e in cuts:
            ctx = SimpleNamespace(tok_pos=pos[a:e], tok_seg=seg[a:e])
            ops.latent_prepare(proj[a:e], proj[a:e, :width], kv_off, cache, w, 1e-5, table, ctx, bt, H, dn, dr, rank, rot, page)
        return proj, cache

    for got, want in zip(run([(0, T)]), run(parts(T))):
        close(got, want)


@pytest.mark.parametrize("n,dv,rot", [(32, 36, 32), (64, 128, 64), (128, 20, 96)])
def test_a_token_of_differential_attention_does_not_depend_on_its_step(n, dv, rot):
    T, page, H, G = 170, 16, 4, 2
    rnd, bt, pos, seg, pages = setup(T, page, n)
    proj, b, w = rnd(T, (H + G) * 2 * n + G * dv), rnd((H + G) * 2 * n + G * dv), rnd(n)
    table = rnd(T, rot // 2, 2)

    def run(cuts):
        q, cache = torch.empty(T, H * 2 * n, device="cuda", dtype=BF16), torch.zeros(pages, page, G * (2 * n + dv), device="cuda", dtype=BF16)
        for a, e in cuts:
            ctx = SimpleNamespace(tok_pos=pos[a:e], tok_seg=seg[a:e])
            ops.diff_prepare(q[a:e], proj[a:e], b, w, w, 1e-5, table, ctx, bt, cache, H, G, n, dv, rot, page)
        return q, cache

    assert all(torch.equal(x, y) for x, y in zip(run([(0, T)]), run(parts(T))))


@pytest.mark.parametrize("rank,dr,rot,dn", [(8, 8, 8, 2), (256, 64, 64, 128), (512, 64, 32, 64), (1024, 72, 70, 6)])
def test_a_token_of_latent_attention_does_not_depend_on_its_step(rank, dr, rot, dn):
    T, page, H = 170, 16, 7
    rnd, bt, pos, seg, pages = setup(T, page, rank)
    width = H * (dn + dr)
    kv_off = -(-width // 8) * 8
    source, w, table = rnd(T, -(-(kv_off + rank + dr) // 8) * 8).to(BF16), rnd(rank), rnd(T, rot // 2, 2)

    def run(cuts):
        proj, cache = source.clone(), torch.zeros(pages, page, rank + dr, device="cuda", dtype=BF16)
        for a, e in cuts:
            ctx = SimpleNamespace(tok_pos=pos[a:e], tok_seg=seg[a:e])
            ops.latent_prepare(proj[a:e], proj[a:e, :width], kv_off, cache, w, 1e-5, table, ctx, bt, H, dn, dr, rank, rot, page)
        return proj, cache

    assert all(torch.equal(x, y) for x, y in zip(run([(0, T)]), run(parts(T))))
