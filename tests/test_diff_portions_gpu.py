"""Differential attention of portions on the tcgen05 kernel against float64 over the same cache rows: portions that end inside, at and
behind a tile of 128 queries or keys, windows whose edges fall anywhere, grouped and ungrouped heads, pages out of order, behind single
tokens; and weights whose 24 bits are needed (large values that cancel)."""
from types import SimpleNamespace

import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu
N, DV = 64, 128


def context(lens, past):
    i32 = dict(dtype=torch.int32, device="cuda")
    return SimpleNamespace(num_segments=len(lens), num_tokens=sum(lens), max_q_len=max(lens), max_ctx_len=max(a + b for a, b in zip(lens, past)),
                           seg_len=list(lens), seg_start_pos=list(past), captured=False,
                           seg_q_start=torch.tensor([0] + lens, **i32).cumsum(0).to(torch.int32), seg_pos0=torch.tensor(past, **i32))


def run(lens, past, window, H, G, cache, table, q, lam, page=16):
    ctx = context(lens, past)
    out = torch.full((sum(lens), H * DV), float("nan"), device="cuda", dtype=torch.bfloat16)
    first = next(i for i, n in enumerate(lens) if n > 1)
    ops.diff_attention(out, q, cache, ctx, table, H, G, N, DV, page, window, 0.125, lam, 1e-5, 0.8)
    assert ops.diff_attention_rows(out, q, cache, ctx, table, first, H, G, N, DV, page, window, 0.125, lam, 1e-5, 0.8)
    ops.check_kernel_errors()
    return out


def want(lens, past, window, H, G, cache, table, q, lam):
    rows_out, at = [], 0
    for s, (n, p) in enumerate(zip(lens, past)):
        rows = cache[table[s].long()].reshape(-1, G * (2 * N + DV))[: p + n].double()
        qs = q[at: at + n].double().view(n, H, 2, N)
        i, j = torch.arange(p, p + n, device="cuda")[:, None], torch.arange(p + n, device="cuda")[None, :]
        hidden = (j > i) | ((i - j >= window) if window else False)
        heads = []
        for h in range(H):
            g = h // (H // G)
            v = rows[:, G * 2 * N + g * DV: G * 2 * N + (g + 1) * DV]
            a = [torch.softmax((qs[:, h, m] @ rows[:, (2 * g + m) * N:(2 * g + m + 1) * N].T * 0.125).masked_fill(hidden, float("-inf")), dim=1) @ v
                 for m in (0, 1)]
            d = a[0] - lam * a[1]
            heads.append(d / torch.sqrt((d * d).mean(-1, keepdim=True) + 1e-5) * 0.8)
        rows_out.append(torch.cat(heads, dim=1))
        at += n
    return torch.cat(rows_out)


@pytest.mark.parametrize("lens,past,window,H,G", [([64], [0], 0, 2, 2), ([127, 128, 129], [0, 1, 300], 0, 4, 2), ([1, 1, 200], [40, 700, 60], 64, 4, 1),
                                                  ([300, 5], [128, 90], 100, 2, 1), ([256], [500], 1, 2, 2), ([130], [1000], 1024, 4, 4)])
def test_portions_against_float64(lens, past, window, H, G):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + window)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    blocks = -(-max(a + b for a, b in zip(lens, past)) // 16)
    table = torch.randperm(len(lens) * blocks, generator=g, device="cuda").to(torch.int32).view(len(lens), blocks)
    cache = rnd(len(lens) * blocks + 1, 16, G * (2 * N + DV))
    q = rnd(sum(lens), H * 2 * N + 8)[:, : H * 2 * N]
    got, ref = run(lens, past, window, H, G, cache, table, q, 0.3).double(), want(lens, past, window, H, G, cache, table, q, 0.3)
    # the output's rounding alone (2^-9 a value, some 2^-9.8 in the root mean square): everything ahead of it is 32-bit
    assert float((got - ref).norm() / ref.norm()) < 2.5e-3


def test_all_bits_of_the_weights_enter():
    """Values of +-1000 in equal shares under nearly equal weights: what is left of the difference is some 1e-3 of a value, so weights of 8 or
    16 bits would show at full size."""
    g = torch.Generator(device="cuda").manual_seed(5)
    lens, past, H, G = [192], [64], 2, 1
    table = torch.arange(16, dtype=torch.int32, device="cuda").view(1, 16)
    cache = torch.randn((17, 16, G * (2 * N + DV)), generator=g, device="cuda") * 0.05
    sign = torch.where(torch.arange(17 * 16, device="cuda") % 2 == 0, 1000.0, -1000.0).view(17, 16, 1)
    cache[..., 2 * N:] = sign + torch.randn((17, 16, DV), generator=g, device="cuda").round()
    cache = cache.to(torch.bfloat16)
    q = (torch.randn((192, H * 2 * N), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    got, ref = run(lens, past, 0, H, G, cache, table, q, 0.7).double(), want(lens, past, 0, H, G, cache, table, q, 0.7)
    assert float((got - ref).norm() / ref.norm()) < 6e-3


@pytest.mark.parametrize("lens,past,window", [([100], [37], 0), ([128], [0], 0), ([1, 200, 90], [20, 130, 900], 100), ([300], [1000], 64), ([70, 65], [3, 15], 1)])
def test_rows_that_nobody_sees_may_hold_anything(lens, past, window):
    """Rows behind a request's last token, and ahead of its first token's window, belong to whoever had the page before: infinities and NaN
    there leave every output as it is."""
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    H, G = 4, 2
    blocks = -(-max(a + b for a, b in zip(lens, past)) // 16) + 1
    table = torch.randperm(len(lens) * blocks, generator=g, device="cuda").to(torch.int32).view(len(lens), blocks)
    cache = torch.randn((len(lens) * blocks, 16, G * (2 * N + DV)), generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn((sum(lens), H * 2 * N), generator=g, device="cuda").to(torch.bfloat16)
    clean = run(lens, past, window, H, G, cache, table, q, 0.3)
    for s, (n, p) in enumerate(zip(lens, past)):
        rows = cache[table[s].long()].reshape(blocks * 16, -1)
        first = max(0, p + 1 - window) if window else 0
        for part in (rows[p + n:], rows[:first]):
            part[0::2] = float("inf")
            part[1::2] = float("nan")
        cache[table[s].long()] = rows.view(blocks, 16, -1)
    assert bool(torch.isfinite(clean).all())
    assert torch.equal(run(lens, past, window, H, G, cache, table, q, 0.3), clean)


@pytest.mark.parametrize("lens,past,window,first", [([1, 1, 200], [40, 700, 60], 64, 2), ([1, 20, 33, 200, 9], [5, 300, 0, 90, 40], 0, 3),
                                                    ([20, 300], [900, 0], 100, 1), ([64, 3, 3, 3], [0, 9, 9, 9], 0, 4), ([40, 63], [0, 0], 0, 2)])
def test_a_step_is_shared_by_the_kernels(monkeypatch, lens, past, window, first):
    """One call over single tokens, short segments and portions: each kernel takes its segments, and no row is left out."""
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    H, G = 4, 2
    blocks = -(-max(a + b for a, b in zip(lens, past)) // 16)
    table = torch.randperm(len(lens) * blocks, generator=g, device="cuda").to(torch.int32).view(len(lens), blocks)
    cache = torch.randn((len(lens) * blocks, 16, G * (2 * N + DV)), generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn((sum(lens), H * 2 * N), generator=g, device="cuda").to(torch.bfloat16)
    taken = []
    inner = ops.diff_attention_rows
    monkeypatch.setattr(ops, "diff_attention_rows", lambda *a: taken.append(a[5]) or inner(*a))
    monkeypatch.setattr(ops, "DIFF_ROWS_WORK", 0)
    ctx = context(lens, past)
    out = torch.full((sum(lens), H * DV), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.diff_attention(out, q, cache, ctx, table, H, G, N, DV, 16, window, 0.125, 0.3, 1e-5, 0.8)
    ops.check_kernel_errors()
    assert taken == ([first] if first < len(lens) else [])
    ref = want(lens, past, window, H, G, cache, table, q, 0.3)
    assert float((out.double() - ref).norm() / ref.norm()) < 2.5e-3


def test_without_room_for_the_rows(monkeypatch):
    """No room for the float32 rows on the device: the kernel that needs none takes the portions too."""
    lens, past, H, G = [1, 200], [40, 60], 4, 2
    g = torch.Generator(device="cuda").manual_seed(3)
    table = torch.arange(2 * 17, dtype=torch.int32, device="cuda").view(2, 17)
    cache = torch.randn((2 * 17, 16, G * (2 * N + DV)), generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn((sum(lens), H * 2 * N), generator=g, device="cuda").to(torch.bfloat16)
    monkeypatch.setattr(ops, "DIFF_ROWS_WORK", 0)
    monkeypatch.setattr(ops, "_room", lambda *a: None)
    out = torch.full((sum(lens), H * DV), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.diff_attention(out, q, cache, context(lens, past), table, H, G, N, DV, 16, 0, 0.125, 0.3, 1e-5, 0.8)
    ref = want(lens, past, 0, H, G, cache, table, q, 0.3)
    assert float((out.double() - ref).norm() / ref.norm()) < 2.5e-3
