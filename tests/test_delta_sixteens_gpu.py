"""The delta rule sixteen tokens at a time at the edges of its blocks, key slices and column tiles, by the measures of the other sizes; and what
a value that is not finite reaches."""
import pytest
import torch

import test_delta_blocks_gpu as blocks
from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dk,dv,H,G,lens,rate", [(4, 1, 2, 1, [256, 17, 1], 0.1), (20, 17, 2, 2, [257, 32, 33], 1.0), (68, 16, 2, 1, [47, 15, 48], 0.05),
                                                 (132, 33, 1, 1, [49, 16], 0.2)])
def test_edges_of_blocks_against_float64(dk, dv, H, G, lens, rate):
    blocks.test_blocks_against_float64(dk, dv, H, G, lens, rate)


@pytest.mark.parametrize("dk,dv", [(72, 24), (128, 40)])
def test_an_infinite_value_reaches_no_earlier_token_and_no_other_column(dk, dv):
    g = torch.Generator(device="cuda").manual_seed(dk)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    lens, H = [37, 50], 2
    T, ctx = sum(lens), blocks.context(lens)
    q, k, v, b, decay = rnd(T, dk), rnd(T, dk), rnd(T, H * dv), rnd(T, H), torch.exp(-rnd(T, H * dk).abs())

    def run():
        state, out = torch.zeros(2, ops.channel_scan_state_floats(H, dk, dv), device="cuda"), torch.full((T, H * dv), float("nan"), device="cuda")
        ops.channel_delta(out, q, k, v, b, decay, state, ctx, H, 1, dk, dv, 1e-6, dk ** -0.5)
        return out

    clean = run()
    at = 37 + 21                                                # inside the second segment's second block
    v[at, 3] = float("inf")
    got = run()
    others = torch.arange(H * dv, device="cuda") != 3
    assert bool(torch.isfinite(clean).all()) and torch.equal(got[:at], clean[:at]) and torch.equal(got[:, others], clean[:, others])
    assert not bool(torch.isfinite(got[at:, 3]).any())


def test_a_part_of_the_blocks_at_a_time():
    """Four portions whose blocks' operands are more than the workspace may hold take two rounds of launches, the second from where the first
    one ended; against token by token, float32 sums of up to 256 products in two orders, some 1e-7 each."""
    H, dk, dv, lens = 16, 256, 256, [640, 600, 20, 477]
    g = torch.Generator(device="cuda").manual_seed(9)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, ctx = sum(lens), blocks.context(lens)
    need = ops._lib("channel_scan").qv_channel_delta_workspace_floats
    assert need(0, 4, 640, H, dk, dv) < 40 * need(0, 4, 16, H, dk, dv)
    q, k, v, b, decay = rnd(T, dk), rnd(T, dk), rnd(T, H * dv), rnd(T, H), torch.exp(-0.2 * rnd(T, H * dk).abs())
    results = []
    for sixteens in (True, False):
        state, out = torch.zeros(4, ops.channel_scan_state_floats(H, dk, dv), device="cuda"), torch.full((T, H * dv), float("nan"), device="cuda")
        ops.channel_delta(out, q, k, v, b, decay, state, ctx, H, 1, dk, dv, 1e-6, dk ** -0.5, blocks=sixteens)
        results.append((out, state))
    for x, y in zip(*results):
        assert float((x - y).norm() / y.norm()) < 2e-6


@pytest.mark.parametrize("lens,dk,launches", [([32] * 15 + [600], 128, 2), ([1000, 600, 33, 900], 256, 4)])
def test_a_segment_among_others_does_not_depend_on_them(lens, dk, launches):
    """One long portion beside many short ones (all blocks in one round of launches), and portions whose blocks take two: every segment's outputs
    and state are, bit for bit, those of a step that holds it alone."""
    H, dv, T, S = 16, dk, sum(lens), len(lens)
    g = torch.Generator(device="cuda").manual_seed(dk)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    q, k, v, b, decay = rnd(T, dk), rnd(T, dk), rnd(T, H * dv), rnd(T, H), torch.exp(-0.2 * rnd(T, H * dk).abs())
    start = rnd(S, ops.channel_scan_state_floats(H, dk, dv)) * 0.1

    def run(rows, state, lens):
        out, before = torch.full((rows.stop - rows.start, H * dv), float("nan"), device="cuda"), ops.launch_count()
        ops.channel_delta(out, q[rows], k[rows], v[rows], b[rows], decay[rows], state, blocks.context(lens), H, 1, dk, dv, 1e-6, dk ** -0.5)
        return out, ops.launch_count() - before

    state, at = start.clone(), 0
    whole, count = run(slice(0, T), state, lens)
    assert count == launches
    for s, n in enumerate(lens):
        slot = S - 1 - s
        one = start[slot: slot + 1].clone()
        alone, count = run(slice(at, at + n), one, [n])
        assert count == 2 and torch.equal(alone, whole[at: at + n]) and torch.equal(one[0], state[slot]), s
        at += n


def test_an_infinite_value_ahead_of_a_later_round():
    """An infinite value in the first of two rounds of launches: earlier tokens and other columns keep their bits through both."""
    lens, H, dk, dv = [1200, 1100], 16, 256, 256
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, ctx = sum(lens), blocks.context(lens)
    q, k, v, b, decay = rnd(T, dk), rnd(T, dk), rnd(T, H * dv), rnd(T, H), torch.exp(-0.2 * rnd(T, H * dk).abs())

    def run():
        state, out = torch.zeros(2, ops.channel_scan_state_floats(H, dk, dv), device="cuda"), torch.full((T, H * dv), float("nan"), device="cuda")
        before = ops.launch_count()
        ops.channel_delta(out, q, k, v, b, decay, state, ctx, H, 1, dk, dv, 1e-6, dk ** -0.5)
        assert ops.launch_count() - before == 4
        return out

    clean, at = run(), 133
    v[at, 3] = float("inf")
    got = run()
    others = torch.arange(H * dv, device="cuda") != 3
    assert bool(torch.isfinite(clean).all()) and torch.equal(got[:, others], clean[:, others])
    assert torch.equal(got[:at], clean[:at]) and torch.equal(got[1200:], clean[1200:]) and not bool(torch.isfinite(got[at:1200, 3]).any())
