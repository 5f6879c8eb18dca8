"""The recurrences over portions (chunks of 64 tokens on the tensor cores) against float64 token by token, at the edges of chunks and of the
kernel's sizes, beside short segments that the token-by-token kernel takes; and no further off than that kernel is."""
from types import SimpleNamespace

import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu
F64 = torch.float64


def context(lens, chunked=True):
    S = len(lens)
    qs = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    return SimpleNamespace(num_segments=S, num_tokens=sum(lens), max_q_len=max(lens) if chunked else 1, seg_len=list(lens), seg_q_start=qs,
                           seg_slot=torch.arange(S, dtype=torch.int32, device="cuda").flip(0).contiguous())


def plain(kind, q, k, v, g1, g2, p1, p2, p3, cap, scale, S, n, m):
    """One head in float64: q, k [T, dk], v [T, dv], state S [dk, dv], n [dk], m."""
    ys = []
    for t in range(q.shape[0]):
        if kind == ops.SCAN_GATED_MAX:
            li = cap * torch.tanh((g1[t] + p1) / cap)
            lf = torch.nn.functional.logsigmoid(cap * torch.tanh((g2[t] + p2) / cap))
            new = torch.maximum(lf + m, li)
            a, b, m = torch.exp(lf + m - new), torch.exp(li - new), new
        else:
            dt = torch.nn.functional.softplus(g1[t] + p1)
            a, b = torch.exp(-torch.exp(p2) * dt), dt
        S = a * S + b * torch.outer(k[t], v[t])
        n = a * n + b * k[t]
        y = scale * (q[t] @ S)
        if kind == ops.SCAN_GATED_MAX:
            y = y / (torch.maximum((scale * (n @ q[t])).abs(), torch.exp(-m)) + 1e-6)
        else:
            y = y + p3 * v[t]
        ys.append(y)
    return torch.stack(ys), S, n, m


@pytest.mark.parametrize("kind", [ops.SCAN_GATED_MAX, ops.SCAN_DECAY])
@pytest.mark.parametrize("dk,dv,H,qg,lens,shift", [(8, 8, 2, 1, [16, 1, 65], 0.0), (64, 40, 3, 1, [63, 15, 64], 2.0), (72, 24, 2, 2, [130, 2, 17], -3.0),
                                                   (128, 64, 2, 1, [200, 128], 4.0), (136, 48, 1, 1, [127, 16], 0.0), (256, 16, 2, 1, [129, 1, 33], 3.0)])
def test_chunks_against_float64(kind, dk, dv, H, qg, lens, shift):
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, cap, scale = sum(lens), 6.0, dk ** -0.5
    width = (H // qg) * dk
    both = rnd(T, 2 * width).to(torch.bfloat16)                # q and k as columns of one product
    q, k, v = both[:, :width], both[:, width:], rnd(T, H * dv).to(torch.bfloat16)
    g1, g2 = rnd(T, H) * 2 - (2.0 if kind == ops.SCAN_DECAY else 0.0), rnd(T, H) * 2 + shift
    p1, p2, p3 = rnd(H), rnd(H), rnd(H)
    floats = ops.linear_scan_state_floats(kind, H, dk, dv)
    start = torch.zeros(len(lens), floats, device="cuda")
    gated = kind == ops.SCAN_GATED_MAX
    args = lambda out, state, ctx: ops.linear_scan(kind, out, q, k, v, g1, g2 if gated else None, p1, p2 if True else None, None if gated else p3, cap,
                                                   scale, state, ctx, H, dk, dv, q_group=qg)
    # a state that earlier tokens left: the same tokens once, token by token
    args(torch.empty(T, H * dv, device="cuda"), start, context(lens, chunked=False))
    outs, states = [], []
    for chunked in (True, False):
        state, out = start.clone(), torch.full((T, H * dv), float("nan"), device="cuda")
        args(out, state, context(lens, chunked))
        outs.append(out.double())
        states.append(state)
    vt = 16 if 128 < dk <= 256 else 32
    tiles = -(-dv // vt)
    def state_of(state, s, h):
        per = dk * vt + (dk + 1 if gated else 0)
        block = state[s].view(H, tiles, per)[h].double()
        S = block[:, : dk * vt].reshape(tiles, dk, vt).permute(1, 0, 2).reshape(dk, tiles * vt)[:, :dv]
        return S, block[0, dk * vt: dk * vt + dk] if gated else torch.zeros(dk, dtype=F64, device="cuda"), block[0, -1] if gated else None
    def normalisers(state, s, h):                               # n of every value tile, and m
        block = state[s].view(H, tiles, dk * vt + dk + 1)[h].double()
        return block[:, dk * vt: dk * vt + dk], block[:, -1]
    errors = torch.zeros(2, 2, dtype=F64)
    norms = torch.zeros(2, dtype=F64)
    at = 0
    for s, n_tok in enumerate(lens):
        slot = len(lens) - 1 - s
        for h in range(H):
            rows, kh = slice(at, at + n_tok), slice((h // qg) * dk, (h // qg) * dk + dk)
            S0, n0, m0 = state_of(start, slot, h)
            y, S1, n1, m1 = plain(kind, q[rows, kh].double(), k[rows, kh].double(), v[rows, h * dv:(h + 1) * dv].double(), g1[rows, h].double(),
                                g2[rows, h].double(), p1[h].double(), p2[h].double(), p3[h].double(), cap, scale, S0, n0, m0)
            norms += torch.stack([(y ** 2).sum(), (S1 ** 2).sum()]).cpu()
            for i in range(2):
                errors[i] += torch.stack([((outs[i][rows, h * dv:(h + 1) * dv] - y) ** 2).sum(), ((state_of(states[i], slot, h)[0] - S1) ** 2).sum()]).cpu()
                if gated:                                       # float32 sums and a float32 running maximum, in every tile's own copy
                    n, m = normalisers(states[i], slot, h)
                    assert float((n - n1).norm() / (n1.norm() * tiles ** 0.5)) < 2e-6 and float((m - m1).abs().max()) < 2e-6 * (1 + abs(float(m1)))
        at += n_tok
    rel = (errors / norms).sqrt()
    # a float32 sum of some 64 to 256 products that cancel: a few 1e-7; the chunks may not be further off than token by token
    assert bool((rel[0] <= torch.maximum(1.2 * rel[1], torch.full((2,), 3e-7, dtype=F64))).all()), rel.tolist()


@pytest.mark.parametrize("kind", [ops.SCAN_GATED_MAX, ops.SCAN_DECAY])
@pytest.mark.parametrize("dk,dv,lens", [(64, 40, [63, 140]), (128, 64, [200]), (256, 16, [16, 129])])
@pytest.mark.parametrize("what", ["value", "gate"])
def test_what_is_not_finite_reaches_no_earlier_token(kind, dk, dv, lens, what):
    """An infinite value (in one column), or a gate that is NaN, at one token a segment: the tokens ahead of it keep their outputs, and an
    infinite value leaves the other columns of later tokens finite."""
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, H = sum(lens), 2
    q, k, v = (rnd(T, H * n).to(torch.bfloat16) for n in (dk, dk, dv))
    g1, g2, p1, p2, p3 = rnd(T, H), rnd(T, H) + 2, rnd(H), rnd(H), rnd(H)
    gated = kind == ops.SCAN_GATED_MAX

    def run():
        state = torch.zeros(len(lens), ops.linear_scan_state_floats(kind, H, dk, dv), device="cuda")
        out = torch.full((T, H * dv), float("nan"), device="cuda")
        ops.linear_scan(kind, out, q, k, v, g1, g2 if gated else None, p1, p2, None if gated else p3, 6.0, dk ** -0.5, state, context(lens), H, dk, dv)
        return out

    clean, at, spots = run(), 0, []
    assert bool(torch.isfinite(clean).all())
    for n in lens:
        spots.append((at, at + 2 * (n // 4) + 1, at + n))      # an odd token inside a chunk
        at += n
    for _, t, _ in spots:
        if what == "value":
            v[t, 3] = float("inf")
        else:
            g1[t] = float("nan")
    got = run()
    for first, t, end in spots:
        scale = clean[first:end].abs().max()
        # chunks with such a value sum W v in another order: float32 sums of up to 64 products
        assert bool(((got[first:t] - clean[first:t]).abs() <= 2e-5 * scale).all())
        assert not bool(torch.isfinite(got[t, 3]))
        if what == "value":
            others = torch.arange(H * dv, device="cuda") != 3
            assert bool(((got[first:end] - clean[first:end])[:, others].abs() <= 2e-5 * scale).all())


def test_the_length_from_which_segments_go_in_chunks():
    assert ops._lib("recurrent").qv_linear_scan_chunk_from() == ops.SCAN_CHUNK_FROM
    rest = lambda lens: ops._scan_rest(SimpleNamespace(seg_len=lens, max_q_len=max(lens)))
    assert rest([1, 1, 15]) == (0, 15, 0) and rest([1, 1, 16]) == (2, 16, 16) and rest([1, 40, 3, 16]) == (1, 40, 3) and rest([16]) == (0, 16, 16)


@pytest.mark.parametrize("kind", [ops.SCAN_GATED_MAX, ops.SCAN_DECAY])
@pytest.mark.parametrize("lens", [[1, 1, 1, 40], [3, 15, 16], [1, 70, 2, 33], [64, 1]])
def test_a_segment_does_not_depend_on_its_neighbours(kind, lens):
    """Single tokens ahead of portions, short segments between and behind them: every segment's outputs and state are, bit for bit, those
    of a step that holds it alone."""
    g = torch.Generator(device="cuda").manual_seed(len(lens))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, H, dk, dv, S = sum(lens), 2, 64, 40, len(lens)
    q, k, v = (rnd(T, H * n).to(torch.bfloat16) for n in (dk, dk, dv))
    g1, g2, p1, p2, p3 = rnd(T, H), rnd(T, H) + 2, rnd(H), rnd(H), rnd(H)
    gated = kind == ops.SCAN_GATED_MAX
    start = rnd(S, ops.linear_scan_state_floats(kind, H, dk, dv)) * 0.1

    def run(rows, state, ctx):
        out = torch.full((rows.stop - rows.start, H * dv), float("nan"), device="cuda")
        ops.linear_scan(kind, out, q[rows], k[rows], v[rows], g1[rows], g2[rows] if gated else None, p1, p2, None if gated else p3, 6.0, dk ** -0.5,
                        state, ctx, H, dk, dv)
        return out

    state = start.clone()
    whole, at = run(slice(0, T), state, context(lens)), 0
    for s, n in enumerate(lens):
        slot = S - 1 - s
        one = start[slot: slot + 1].clone()
        assert torch.equal(run(slice(at, at + n), one, context([n])), whole[at: at + n]), s
        assert torch.equal(one[0], state[slot]), s
        at += n
