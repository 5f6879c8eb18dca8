"""The gated recurrence over long portions (the chunks' outputs side by side, from 896, 1,024 or 2,048 tokens on; shorter ones go one chunk after the
other) at the edges of its chunks, key blocks and column blocks, by the same measures as the shorter portions' kernel; a workspace that holds a part of the chunks; no room for one."""
import pytest
import torch

import test_scan_chunks_gpu as chunks
from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dk,dv,H,qg,lens,shift", [(8, 8, 2, 1, [640], 0.0), (72, 40, 2, 2, [703, 1, 640], 2.0), (128, 272, 1, 1, [705, 20], -3.0),
                                                   (256, 512, 1, 1, [1027], 3.0)])
def test_long_portions_against_float64(dk, dv, H, qg, lens, shift):
    chunks.test_chunks_against_float64(ops.SCAN_GATED_MAX, dk, dv, H, qg, lens, shift)


@pytest.mark.parametrize("dk,dv,H,qg,lens,shift", [(8, 8, 2, 1, [1024], 0.0), (72, 40, 2, 2, [1087, 1, 1024], 2.0), (128, 272, 1, 1, [1089, 20], -3.0),
                                                   (256, 512, 2, 1, [900, 896], 3.0), (136, 72, 2, 1, [1500], 1.0)])
def test_edges_against_token_by_token(dk, dv, H, qg, lens, shift):
    """At the edges of chunks, key blocks and column blocks: the median row and the states within 2e-6 of token by token, whose rows are off float64 by
    some 7e-7 in the median, as the chunks' are by 5e-7 (a row with a small n . q is off by more in either)."""
    assert min(n for n in lens if n > 64) >= ops.scan_parallel_from(ops.SCAN_GATED_MAX, H, dk, dv)
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, S = sum(lens), len(lens)
    q, k, v = (rnd(T, n).to(torch.bfloat16) for n in (H // qg * dk, H // qg * dk, H * dv))
    g1, g2, p1, p2 = rnd(T, H) * 2, rnd(T, H) * 2 + shift, rnd(H), rnd(H)
    results = []
    for chunked in (False, True):
        state = torch.zeros(S, ops.linear_scan_state_floats(ops.SCAN_GATED_MAX, H, dk, dv), device="cuda")
        out, before = torch.full((T, H * dv), float("nan"), device="cuda"), ops.launch_count()
        ops.linear_scan(ops.SCAN_GATED_MAX, out, q, k, v, g1, g2, p1, p2, None, 6.0, dk ** -0.5, state, chunks.context(lens, chunked), H, dk, dv, q_group=qg)
        results.append((out.double().view(T * H, dv), state.double()))
        assert ops.launch_count() - before >= (3 if chunked else 1)
    (tokens, tokens_state), (got, state) = results
    rows = (got - tokens).norm(dim=1) / tokens.norm(dim=1)
    assert float(rows.median()) < 2e-6 and bool(torch.isfinite(got).all()) and float((state - tokens_state).norm() / tokens_state.norm()) < 2e-6



@pytest.mark.parametrize("dk,dv,lens", [(64, 136, [640, 40]), (256, 16, [16, 700]), (64, 136, [2048, 40]), (256, 16, [16, 1084])])
@pytest.mark.parametrize("what", ["value", "gate"])
def test_what_is_not_finite_reaches_no_earlier_token(dk, dv, lens, what):
    chunks.test_what_is_not_finite_reaches_no_earlier_token(ops.SCAN_GATED_MAX, dk, dv, lens, what)


@pytest.mark.parametrize("lens", [[1, 1, 639, 640], [700, 3, 641], [1, 1, 1023, 1024], [1084, 3, 1025]])
def test_a_segment_does_not_depend_on_its_neighbours(lens):
    chunks.test_a_segment_does_not_depend_on_its_neighbours(ops.SCAN_GATED_MAX, lens)


@pytest.mark.parametrize("lens", [[704, 640, 650, 900], [1088, 1024, 1034, 1284]])
def test_a_part_of_the_chunks_at_a_time_and_no_room(monkeypatch, lens):
    """Four segments whose chunks' states are more than the workspace may hold take several launches, each from where the last one ended;
    without a workspace the shorter portions' kernel takes them.  Against token by token, whose rows are off float64 by some 7e-7 in the median,
    as the chunks' are by 5e-7 (few rows, with a small n . q, by more): the median row and the states within 2e-6."""
    H, dk, dv = 8, 256, 512
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T = sum(lens)
    q, k, v = (rnd(T, H * n).to(torch.bfloat16) for n in (dk, dk, dv))
    g1, g2, p1, p2 = rnd(T, H), rnd(T, H) + 2, rnd(H), rnd(H)
    need = ops._lib("recurrent").qv_linear_scan_workspace_bytes(ops.SCAN_GATED_MAX, 4, max(lens), H, dk, dv)
    assert need < -(-max(lens) // 64) * 4 * H * dk * dv * 4     # less than the longest one's chunks' states, four times

    def run(chunked):
        state = torch.zeros(4, ops.linear_scan_state_floats(ops.SCAN_GATED_MAX, H, dk, dv), device="cuda")
        out = torch.full((T, H * dv), float("nan"), device="cuda")
        ops.linear_scan(ops.SCAN_GATED_MAX, out, q, k, v, g1, g2, p1, p2, None, 6.0, dk ** -0.5, state, chunks.context(lens, chunked), H, dk, dv)
        return out.double(), state.double()

    tokens, parts = run(False), run(True)
    monkeypatch.setattr(ops, "_room", lambda *a: None)
    one = run(True)
    for got in (parts, one):
        rows = (got[0] - tokens[0]).norm(dim=1) / tokens[0].norm(dim=1)
        assert float(rows.median()) < 2e-6 and bool(torch.isfinite(rows).all())
        assert float((got[1] - tokens[1]).norm() / tokens[1].norm()) < 2e-6


@pytest.mark.parametrize("lens", [[32] * 15 + [1100], [1700, 20, 1400, 1024, 40, 1200, 1600]])
def test_a_segment_among_many_does_not_depend_on_them(lens):
    """One long segment beside many short ones, and five whose chunks' states take several rounds of launches: every segment's outputs and
    state are, bit for bit, those of a step that holds it alone; short neighbours add no rounds."""
    H, dk, dv, S, T = 4, 256, 512, len(lens), sum(lens)
    g = torch.Generator(device="cuda").manual_seed(S)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    q, k, v = (rnd(T, H * n).to(torch.bfloat16) for n in (dk, dk, dv))
    g1, g2, p1, p2 = rnd(T, H), rnd(T, H) + 2, rnd(H), rnd(H)
    start = rnd(S, ops.linear_scan_state_floats(ops.SCAN_GATED_MAX, H, dk, dv)) * 0.1

    def run(rows, state, lens):
        out = torch.full((rows.stop - rows.start, H * dv), float("nan"), device="cuda")
        before = ops.launch_count()
        ops.linear_scan(ops.SCAN_GATED_MAX, out, q[rows], k[rows], v[rows], g1[rows], g2[rows], p1, p2, None, 6.0, dk ** -0.5, state, chunks.context(lens),
                        H, dk, dv)
        return out, ops.launch_count() - before

    state, at = start.clone(), 0
    whole, launches = run(slice(0, T), state, lens)
    assert launches == (4 if S == 16 else 7)                    # (three a round, and the kernel that takes the short ones)
    for s, n in enumerate(lens):
        slot = S - 1 - s
        one = start[slot: slot + 1].clone()
        alone, launches = run(slice(at, at + n), one, [n])
        assert launches == (3 if n >= 1024 else 1)
        assert torch.equal(alone, whole[at: at + n]) and torch.equal(one[0], state[slot]), s
        at += n


def test_an_infinite_value_ahead_of_a_later_round():
    """An infinite value in the first of two rounds of launches, whose block of columns then goes token by token: tokens ahead of it, other columns
    and the normaliser stay what they are, through the second round too (float32 sums of up to 64 products in another order: 2e-5)."""
    H, dk, dv, lens = 8, 256, 512, [1700, 1500]
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T = sum(lens)
    q, k, v = (rnd(T, H * n).to(torch.bfloat16) for n in (dk, dk, dv))
    g1, g2, p1, p2 = rnd(T, H), rnd(T, H) + 2, rnd(H), rnd(H)

    def run():
        state = torch.zeros(2, ops.linear_scan_state_floats(ops.SCAN_GATED_MAX, H, dk, dv), device="cuda")
        out, before = torch.full((T, H * dv), float("nan"), device="cuda"), ops.launch_count()
        ops.linear_scan(ops.SCAN_GATED_MAX, out, q, k, v, g1, g2, p1, p2, None, 6.0, dk ** -0.5, state, chunks.context(lens), H, dk, dv)
        assert ops.launch_count() - before == 6
        return out, state.view(2, H, dv // 16, dk * 16 + dk + 1)[:, :, :, dk * 16:]        # n and m of every value tile

    (clean, clean_n), at = run(), 133
    assert bool(torch.isfinite(clean).all())
    v[at, 3] = float("inf")
    got, n = run()
    others, scale = torch.arange(H * dv, device="cuda") != 3, clean.abs().max()
    assert bool(((got[:, others] - clean[:, others]).abs() <= 2e-5 * scale).all()) and bool(((got[:at] - clean[:at]).abs() <= 2e-5 * scale).all())
    assert torch.equal(got[1700:], clean[1700:]) and not bool(torch.isfinite(got[at:1700, 3]).any())
    assert float((n - clean_n).norm() / clean_n.norm()) < 2e-6
