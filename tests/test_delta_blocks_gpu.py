"""The delta rule as a step takes it (sixteen tokens at a time from the first portion on that pays for it, others token by token) against
float64 token by token, over every size of lane groups, segments that end anywhere in a block, strong and weak decays; and no further off
than the token-by-token kernel."""
from types import SimpleNamespace

import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


def context(lens):
    S = len(lens)
    i32 = dict(dtype=torch.int32, device="cuda")
    return SimpleNamespace(num_segments=S, num_tokens=sum(lens), max_q_len=max(lens), seg_len=list(lens), seg_slot=torch.arange(S, **i32).flip(0).contiguous(),
                           seg_q_start=torch.tensor([0] + lens, **i32).cumsum(0).to(torch.int32),
                           tok_seg=torch.repeat_interleave(torch.arange(S, **i32), torch.tensor(lens, device="cuda")).to(torch.int32))


@pytest.mark.parametrize("dk,dv,H,G,lens,rate", [(12, 20, 2, 1, [4, 1, 5], 0.1), (32, 128, 2, 2, [17, 3], 2.0), (64, 24, 4, 2, [33, 2, 16], 0.02),
                                                 (128, 40, 2, 1, [70, 6, 1], 0.3), (128, 128, 2, 2, [300], 0.01), (256, 24, 2, 1, [9, 40], 6.0)])
def test_blocks_against_float64(dk, dv, H, G, lens, rate):
    g = torch.Generator(device="cuda").manual_seed(dk * 3 + dv)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, ctx = sum(lens), context(lens)
    conv = rnd(T, 2 * G * dk + H * dv)
    q, k, v = conv[:, : G * dk], conv[:, G * dk: 2 * G * dk], conv[:, 2 * G * dk:]
    b = rnd(T, H + 3)[:, :H]
    decay = torch.exp(-rate * torch.rand((T, H * dk), generator=g, device="cuda") * 2)
    scale, eps = dk ** -0.5, 1e-6
    floats = ops.channel_scan_state_floats(H, dk, dv)
    start = torch.zeros(len(lens), floats, device="cuda")

    def single(state, out):
        qh = torch.empty((T, H * dk), device="cuda")
        kb, ug = torch.empty_like(qh), torch.empty_like(qh)
        ops.delta_operands(qh, kb, ug, q, k, b, decay, H, G, dk, eps, scale)
        ops.channel_scan(out, qh, kb, v, decay, kb, ug, 1.0, state, ctx, H, dk, dv)

    single(start, torch.empty((T, H * dv), device="cuda"))               # a state that earlier tokens left
    outs, states = [], []
    for blocks in (True, False):
        state, out = start.clone(), torch.full((T, H * dv), float("nan"), device="cuda")
        if blocks:
            assert ops.channel_delta(out, q, k, v, b, decay, state, ctx, H, G, dk, dv, eps, scale)
        else:
            single(state, out)
        outs.append(out.double())
        states.append(state.double())
    lpc = 1 if dk <= 16 else 2 if dk <= 32 else 4 if dk <= 64 else 8 if dk <= 128 else 16
    cpt = 32 // lpc
    tiles = -(-dv // cpt)
    # [head][tile][row of the lane][lane = column * lpc + rows' group] -> S [dk, dv]
    matrix = lambda st, s, h: (st[s].view(H, tiles, 16, cpt, lpc)[h].permute(3, 1, 0, 2).reshape(lpc * 16, tiles * cpt)[:dk, :dv])
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + eps)
    err, norm, at = torch.zeros(2, 2, dtype=torch.float64), torch.zeros(2, dtype=torch.float64), 0
    for s, n in enumerate(lens):
        slot = len(lens) - 1 - s
        for h in range(H):
            c = h // (H // G)
            rows = slice(at, at + n)
            qs, ks = unit(q[rows, c * dk:(c + 1) * dk].double()) * scale, unit(k[rows, c * dk:(c + 1) * dk].double())
            vs, gs, beta = v[rows, h * dv:(h + 1) * dv].double(), decay[rows, h * dk:(h + 1) * dk].double(), torch.sigmoid(b[rows, h].double())
            S, ys = matrix(start.double(), slot, h), []
            for t in range(n):
                S = gs[t][:, None] * S
                S = S + torch.outer(ks[t], beta[t] * (vs[t] - ks[t] @ S))
                ys.append(qs[t] @ S)
            ys = torch.stack(ys)
            norm += torch.stack([(ys ** 2).sum(), (S ** 2).sum()]).cpu()
            for i in range(2):
                err[i] += torch.stack([((outs[i][rows, h * dv:(h + 1) * dv] - ys) ** 2).sum(), ((matrix(states[i], slot, h) - S) ** 2).sum()]).cpu()
        at += n
    rel = (err / norm).sqrt()
    # sums of up to 256 float32 products: some 1e-7; sixteen tokens at a time may not be further off than one at a time
    assert bool((rel[0] <= torch.maximum(1.2 * rel[1], torch.full((2,), 2.5e-7, dtype=torch.float64))).all()), rel.tolist()


@pytest.mark.parametrize("dk,dv,lens", [(128, 40, [1, 1, 3, 40, 2]), (68, 24, [15, 16]), (256, 24, [1, 70]), (64, 24, [1, 40]), (128, 128, [1, 15, 2])])
def test_short_segments_ahead_keep_their_kernel(dk, dv, lens):
    """Segments ahead of the first portion are the token-by-token kernel's, bit for bit; the portions behind them agree to rounding."""
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    H, G, T, ctx = 2, 1, sum(lens), context(lens)
    q, k, v, b = rnd(T, G * dk), rnd(T, G * dk), rnd(T, H * dv), rnd(T, H)
    decay = torch.exp(-torch.rand((T, H * dk), generator=g, device="cuda"))
    start = rnd(len(lens), ops.channel_scan_state_floats(H, dk, dv)) * 0.1
    results = []
    for blocks in (True, False):
        state, out = start.clone(), torch.full((T, H * dv), float("nan"), device="cuda")
        assert ops.channel_delta(out, q, k, v, b, decay, state, ctx, H, G, dk, dv, 1e-6, dk ** -0.5, blocks=blocks)
        results.append((out, state))
    (out, state), (ref, ref_state) = results
    lead = ops.delta_lead(lens, dk)
    n = sum(lens[:lead])
    slots = ctx.seg_slot.long()
    assert torch.equal(out[:n], ref[:n]) and torch.equal(state[slots[:lead]], ref_state[slots[:lead]])
    # float32 sums of up to 256 products in two orders, some 1e-7 each
    assert float((out - ref).norm() / ref.norm()) < 2e-6 and float((state - ref_state).norm() / ref_state.norm()) < 2e-6
    qh = torch.empty((T, H * dk), device="cuda")
    kb, ug = torch.empty_like(qh), torch.empty_like(qh)
    ops.delta_operands(qh, kb, ug, q, k, b, decay, H, G, dk, 1e-6, dk ** -0.5)
    state, alone = start.clone(), torch.empty_like(ref)
    ops.channel_scan(alone, qh, kb, v, decay, kb, ug, 1.0, state, ctx, H, dk, dv)
    assert torch.equal(alone, ref) and torch.equal(state, ref_state)


def test_without_room_for_the_blocks(monkeypatch):
    """No room for the blocks' operands on the device: token by token."""
    lens, H, dk, dv = [1, 40], 2, 128, 40
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, ctx = sum(lens), context(lens)
    q, k, v, b, decay = rnd(T, dk), rnd(T, dk), rnd(T, H * dv), rnd(T, H), torch.exp(-rnd(T, H * dk).abs())
    results = []
    for blocks in (False, True):
        state, out = torch.zeros(2, ops.channel_scan_state_floats(H, dk, dv), device="cuda"), torch.empty((T, H * dv), device="cuda")
        if blocks:
            monkeypatch.setattr(ops, "_room", lambda *a: None)
        ops.channel_delta(out, q, k, v, b, decay, state, ctx, H, 1, dk, dv, 1e-6, dk ** -0.5, blocks=blocks)
        results.append((out, state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
