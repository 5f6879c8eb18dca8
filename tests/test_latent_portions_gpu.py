"""Latent attention of portions whose keys and values are formed per head, against float64 over the same cache rows: portions that end
inside, at and behind a tile of 128 queries or keys, far into their requests, behind single tokens and before them, with and without
window and gate, pages out of order; and which segments take that path."""
from types import SimpleNamespace

import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu
H, DN, DR, DV = 3, 128, 64, 128


def context(lens, past):
    i32 = dict(dtype=torch.int32, device="cuda")
    return SimpleNamespace(num_segments=len(lens), num_tokens=sum(lens), max_q_len=max(lens), max_ctx_len=max(a + b for a, b in zip(lens, past)),
                           seg_len=list(lens), seg_start_pos=list(past), captured=False,
                           seg_q_start=torch.tensor([0] + lens, **i32).cumsum(0).to(torch.int32), seg_pos0=torch.tensor(past, **i32),
                           tok_pos=torch.cat([torch.arange(p, p + n, **i32) for n, p in zip(lens, past)]),
                           tok_seg=torch.repeat_interleave(torch.arange(len(lens), **i32), torch.tensor(lens, device="cuda")).to(torch.int32))


@pytest.mark.parametrize("lens,past,window,gated,rank", [
    ([32], [0], 0, True, 64), ([127, 128, 129], [0, 1, 300], 0, False, 128), ([1, 1, 200], [40, 700, 60], 0, True, 64),
    ([260, 1, 33], [128, 90, 511], 0, True, 64), ([140, 64], [500, 130], 100, False, 64), ([300], [255], 128, True, 512), ([40, 31], [3, 9], 1, True, 64)])
def test_portions_against_float64(lens, past, window, gated, rank):
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    T, page, S = sum(lens), 16, len(lens)
    ctx = context(lens, past)
    blocks = -(-ctx.max_ctx_len // page)
    table = torch.randperm(S * blocks, generator=g, device="cuda").to(torch.int32).view(S, blocks)
    cache = rnd(S * blocks + 1, page, rank + DR)
    proj = rnd(T, H * (DN + DR) + 8)
    q = proj[:, : H * (DN + DR)]
    gate = rnd(T, H * DV) if gated else None
    wuk, wuv = rnd(H * DN, rank).mul_(rank ** -0.5), rnd(H * DV, rank).mul_(rank ** -0.5)
    up = torch.cat([wuk, wuv])
    out = torch.full((T, H * DV), float("nan"), device="cuda", dtype=torch.bfloat16)
    scale = (DN + DR) ** -0.5
    packed = (ops.pack_weight(up), up.shape[0])
    ops.latent_attention(out, q, gate, cache, wuk, wuv, ctx, table, H, DN, DR, DV, rank, page, window, scale,
                         wuk_t=wuk.view(H, DN, rank).transpose(1, 2).contiguous(), kv_up=packed)
    left = ops.latent_attention_expanded(out, q, gate, cache, packed, ctx, table, H, DN, DR, DV, rank, page, window, scale)
    ops.check_kernel_errors()
    assert left == next(i for i, n in enumerate(lens) if n >= ops.LATENT_EXPAND_FROM)
    at = 0
    for s, (n, p) in enumerate(zip(lens, past)):
        rows = cache[table[s].long()].reshape(-1, rank + DR)[: p + n].double()
        c, kr = rows[:, :rank], rows[:, rank:]
        qs = q[at: at + n].double().view(n, H, DN + DR)
        i, j = torch.arange(p, p + n, device="cuda")[:, None], torch.arange(p + n, device="cuda")[None, :]
        hidden = (j > i) | ((i - j >= window) if window else False)
        for h in range(H):
            k, v = c @ wuk[h * DN:(h + 1) * DN].double().T, c @ wuv[h * DV:(h + 1) * DV].double().T
            sc = (qs[:, h, :DN] @ k.T + qs[:, h, DN:] @ kr.T) * scale
            want = torch.softmax(sc.masked_fill(hidden, float("-inf")), dim=1) @ v
            if gated:
                want = want * torch.sigmoid(gate[at: at + n, h * DV:(h + 1) * DV].double())
            got = out[at: at + n, h * DV:(h + 1) * DV].double()
            # keys and values rounded to bfloat16 (2^-9 of each: scores of order one move by some 2^-9, weights with them), weights and
            # output rounded once more
            assert float((got - want).norm() / want.norm()) < 8e-3, (s, h)
        at += n


def test_what_stays_with_the_latents():
    ctx = context([1, 5, 31], [9, 0, 4])
    args = (torch.empty(37, H * DV, device="cuda", dtype=torch.bfloat16), torch.empty(37, H * (DN + DR), device="cuda", dtype=torch.bfloat16), None,
            torch.empty(9, 16, 64 + DR, device="cuda", dtype=torch.bfloat16), (None, H * (DN + DV)))
    table = torch.zeros(3, 3, device="cuda", dtype=torch.int32)
    assert ops.latent_attention_expanded(*args, ctx, table, H, DN, DR, DV, 64, 16, 0, 1.0) == 3           # short segments
    ctx.seg_len = [1, 5, 1 << 21]
    assert ops.latent_attention_expanded(*args, ctx, table, H, DN, DR, DV, 64, 16, 0, 1.0) == 3           # rows beyond the room for them


@pytest.mark.parametrize("lens,past,window", [([40], [200], 0), ([140], [500], 100), ([64, 33], [130, 1000], 50), ([40], [300], 1)])
def test_rows_that_nobody_sees_may_hold_anything(lens, past, window):
    """Rows behind a request's last token, and ahead of its first token's window, belong to whoever had the page before."""
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    T, rank, ctx = sum(lens), 64, context(lens, past)
    blocks = -(-ctx.max_ctx_len // 16) + 1
    table = torch.randperm(len(lens) * blocks, generator=g, device="cuda").to(torch.int32).view(len(lens), blocks)
    cache, q, up = rnd(len(lens) * blocks, 16, rank + DR), rnd(T, H * (DN + DR)), rnd(H * (DN + DV), rank).mul_(rank ** -0.5)
    packed = (ops.pack_weight(up), up.shape[0])

    def run():
        out = torch.full((T, H * DV), float("nan"), device="cuda", dtype=torch.bfloat16)
        assert ops.latent_attention_expanded(out, q, None, cache, packed, ctx, table, H, DN, DR, DV, rank, 16, window, (DN + DR) ** -0.5) == 0
        ops.check_kernel_errors()
        return out

    clean = run()
    for s, (n, p) in enumerate(zip(lens, past)):
        rows = cache[table[s].long()].reshape(blocks * 16, -1)
        for part in (rows[p + n:], rows[: max(0, p + 1 - window) if window else 0]):
            part[0::2], part[1::2] = float("inf"), float("nan")
        cache[table[s].long()] = rows.view(blocks, 16, -1)
    assert bool(torch.isfinite(clean).all())
    assert torch.equal(run(), clean)


def mixed(lens, past, rank=64, seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    ctx, T = context(lens, past), sum(lens)
    blocks = -(-ctx.max_ctx_len // 16)
    table = torch.randperm(len(lens) * blocks, generator=g, device="cuda").to(torch.int32).view(len(lens), blocks)
    cache, q, gate = rnd(len(lens) * blocks, 16, rank + DR), rnd(T, H * (DN + DR)), rnd(T, H * DV)
    wuk, wuv = rnd(H * DN, rank).mul_(rank ** -0.5), rnd(H * DV, rank).mul_(rank ** -0.5)
    up = torch.cat([wuk, wuv])
    args = (q, gate, cache, wuk, wuv, ctx, table, H, DN, DR, DV, rank, 16, 0, (DN + DR) ** -0.5)

    def call(kv_up=True):
        out = torch.full((T, H * DV), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.latent_attention(out, *args, wuk_t=wuk.view(H, DN, rank).transpose(1, 2).contiguous(),
                             kv_up=(ops.pack_weight(up), up.shape[0]) if kv_up else None)
        ops.check_kernel_errors()
        return out.float()
    return call


def test_without_room_for_the_rows(monkeypatch):
    """No room for the rows on the device, at any of the three allocations: the kernels over the latents take the whole step, bit for bit."""
    call = mixed([1, 200], [40, 60])
    want = call(kv_up=False)
    monkeypatch.setattr(ops, "LATENT_EXPAND_WORK", 0)
    monkeypatch.setattr(ops, "latent_expand_pays", lambda *a: True)
    inner = ops._room
    for fits in (0, 1, 2):
        left = [fits]

        def room(*a):
            left[0] -= 1
            return inner(*a) if left[0] >= 0 else None
        monkeypatch.setattr(ops, "_room", room)
        assert torch.equal(call(), want)
        assert left[0] == -1


@pytest.mark.parametrize("lens,past,lead", [([1, 1, 200], [40, 700, 60], 2), ([1, 5, 40, 9], [30, 0, 17, 50], 2), ([130], [2500], 0), ([31, 64], [9, 1200], 1)])
def test_a_step_is_shared_by_the_kernels(monkeypatch, lens, past, lead):
    """One call over single tokens and portions: the segments ahead of the first portion stay with the kernels over the latents, and no row is
    left out."""
    call = mixed(lens, past)
    want = call(kv_up=False)
    taken = []
    inner = ops.latent_attention_expanded
    monkeypatch.setattr(ops, "latent_attention_expanded", lambda *a: taken.append(inner(*a)) or taken[-1])
    monkeypatch.setattr(ops, "LATENT_EXPAND_WORK", 0)
    monkeypatch.setattr(ops, "latent_expand_pays", lambda *a: True)
    got = call()
    assert taken == [lead]
    n = sum(lens[:lead])
    # other slices of keys ahead, keys and values rounded per head behind: a few bfloat16 roundings either way
    for a, b in ((got[:n], want[:n]), (got[n:], want[n:])):
        assert a.numel() == 0 or float((a - b).norm() / b.norm()) < 1.2e-2


def test_a_layer_with_a_single_token_ahead_of_a_portion(monkeypatch):
    """The mixer at the sizes of this path, which packs both matrices at load: a step that holds one request's next token and another's
    first portion, against float64."""
    import deganex_helpers as dh
    import plain_deganex as plain
    from qorvix_b200.engine.batch import BatchBuilder
    from test_deganex_gpu import close, mixer_setup, rnd
    layer = dh.attn(heads=3, dim=128, rot_dim=64, vdim=128, kv_rank=64, scale=192 ** -0.5)
    part, cache, w = mixer_setup(layer, torch.bfloat16, sharp=3.0)
    assert part.kv_up is not None
    taken = []
    inner = ops.latent_attention_expanded
    monkeypatch.setattr(ops, "latent_attention_expanded", lambda *a: taken.append(inner(*a)) or taken[-1])
    monkeypatch.setattr(ops, "LATENT_EXPAND_WORK", 0)
    monkeypatch.setattr(ops, "latent_expand_pays", lambda *a: True)
    builder, at = BatchBuilder("cuda"), {"a": 0, "b": 0}
    xs = {r: rnd(95, 72, seed=s).to(torch.bfloat16).float() for r, s in (("a", 3), ("b", 4))}
    want = {r: plain.latent_attention(xs[r].double(), w, layer["mixer"], 2e-5) for r in xs}
    for step in ([("a", 40)], [("a", 1), ("b", 60)], [("a", 1), ("b", 1)], [("a", 3), ("b", 34)]):
        segs, tables = [], {g: [] for g in cache.paged_groups()}
        for r, n in step:
            if not cache.has(r):
                cache.admit(r)
            assert cache.reserve(r, n)
            segs.append(dict(tokens=[0] * n, pos0=at[r], slot=cache.slot(r), want=[], first=at[r] == 0))
            for g in tables:
                tables[g].append(cache.block_table(r, g))
        ctx = builder.build(segs, tables, cache.scratch_page)
        x = torch.cat([xs[r][at[r]: at[r] + n] for r, n in step]).to(torch.bfloat16).to("cuda")
        got = part.forward(x, ctx, cache.layer_view(0)).float()
        close(got, torch.cat([want[r][at[r]: at[r] + n] for r, n in step]), torch.bfloat16, str(step), loose=2.0)
        for r, n in step:
            cache.commit(r, n)
            at[r] += n
    assert taken == [0, 1, 1]
