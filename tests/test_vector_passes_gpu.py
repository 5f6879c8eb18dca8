"""The passes behind the recurrences and ahead of the experts at the sizes where their kernels change: gates of many tokens, norms of long and
short parts, grouping over more experts than a block has threads."""
import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


def rnd(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


@pytest.mark.parametrize("R,N", [(16, 70), (64, 128), (24, 40), (7, 65)])
@pytest.mark.parametrize("T", [255, 256, 271])
def test_gates_of_many_tokens(T, R, N):
    """From 256 tokens on 16 tokens a CTA, four entries of a row a read where the rank is a multiple of 16: the same sums as eight
    tokens at a time, bit for bit, and close to float64."""
    wide = rnd(T, R + 4, seed=T)
    x1, w2t, bias, rate = wide[:, 4:], rnd(R, N, seed=1), rnd(N, seed=2), rnd(N, seed=3).abs()
    for kind in (ops.GATE_LINEAR, ops.GATE_EXP_NEG_SOFTPLUS):
        for pre_tanh in (False, True):
            run = lambda x: (lambda o: (ops.channel_gates(o, x, w2t, bias, pre_tanh, kind, 0.0, rate=rate), o)[1])(torch.empty(x.shape[0], N, device="cuda"))
            got = run(x1)
            assert torch.equal(got, torch.cat([run(x1[a: a + 40]) for a in range(0, T, 40)]))
            x = x1.double().tanh() if pre_tanh else x1.double()
            z = x @ w2t.double() + bias.double()
            want = z if kind == ops.GATE_LINEAR else torch.exp(-rate.double() * torch.nn.functional.softplus(z))
            # R float32 products of order one: some sqrt(R) * 2^-24 a sum, and as much again from tanh and softplus
            assert float((got.double() - want).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("part,groups", [(2044, 2), (2052, 1), (4096, 1), (4100, 1), (4100, 2), (8192, 1), (8196, 1), (37, 3)])
@pytest.mark.parametrize("gate_first", [False, True])
def test_norm_in_equal_parts(part, groups, gate_first, dtype):
    W, T = part * groups, 5
    y, gate, w = rnd(T, W, seed=part), rnd(T, W, seed=1).to(dtype), rnd(W, seed=2)
    out = torch.empty(T, W, device="cuda", dtype=dtype)
    ops.gated_group_norm(out, y, gate, w, groups, 1e-5, gate_first)
    z, v = gate.double(), y.double()
    if gate_first:
        v = v * z * torch.sigmoid(z)
    p = v.view(T, groups, part)
    n = (p / torch.sqrt((p * p).mean(-1, keepdim=True) + 1e-5)).view(T, W) * w.double()
    want = n if gate_first else n * torch.sigmoid(z)
    bound = (1e-5 if dtype == torch.float32 else 2.0 ** -8) * want.abs() + 1e-6        # a few float32 roundings, then the output's own
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dv", [128, 132, 256, 260, 512, 516, 30])
@pytest.mark.parametrize("kind", [ops.HEAD_GATE_SIGMOID, ops.HEAD_GATE_SILU])
def test_norm_of_heads(dv, kind, dtype):
    H, T = 3, 6
    y, gate, w = rnd(T, H * dv, seed=dv), rnd(T, H * dv + 4, seed=1)[:, : H * dv], rnd(H * dv, seed=2)
    out = torch.empty(T, H * dv, device="cuda", dtype=dtype)
    ops.head_norm_gate(out, y, gate, w, H, 1e-5, kind, 0.7)
    p, z = y.double().view(T, H, dv), gate.double()
    n = (p / torch.sqrt((p * p).mean(-1, keepdim=True) + 1e-5)).reshape(T, H * dv) * w.double()
    want = n * torch.sigmoid(z) * (z if kind == ops.HEAD_GATE_SILU else 1.0) * 0.7
    bound = (1e-5 if dtype == torch.float32 else 2.0 ** -8) * want.abs() + 1e-6
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("T,top,E", [(40, 3, 1024), (40, 3, 1025), (300, 4, 2000), (70, 2, 5000), (13000, 1, 3), (6200, 2, 1500)])
@pytest.mark.parametrize("tile_rows", [32, 64])
def test_grouping(T, top, E, tile_rows):
    """More experts than the block has threads, more choices than its threads keep in registers, identity experts among them."""
    g = torch.Generator(device="cuda").manual_seed(T + E)
    idx = torch.randint(0, E + 2, (T, top), generator=g, device="cuda", dtype=torch.int32)
    R = T * top
    row_token, slot_row, scratch = (torch.full((R,), -7, device="cuda", dtype=torch.int32) for _ in range(3))
    tiles = torch.full((3 * ops.moe_max_tiles(R, E, tile_rows),), -7, device="cuda", dtype=torch.int32)
    ops.moe_group(row_token, slot_row, tiles, idx, scratch, E, tile_rows)
    flat, slot = idx.reshape(-1).cpu(), slot_row.cpu()
    real = flat < E
    n = int(real.sum())
    assert bool((slot[~real] == -1).all()) and torch.equal(torch.sort(slot[real]).values, torch.arange(n, dtype=torch.int32))
    assert torch.equal(row_token.cpu()[slot[real].long()], (torch.arange(R) // top).int()[real])
    counts = torch.bincount(flat[real].long(), minlength=E)
    rows = [(e, int(first) + r, min(tile_rows, int(c) - r)) for e, (c, first) in enumerate(zip(counts, counts.cumsum(0) - counts))
            for r in range(0, int(c), tile_rows)]
    table = tiles.view(-1, 3).cpu().tolist()
    assert [tuple(t) for t in table[: len(rows)]] == rows and all(t[0] == -1 for t in table[len(rows):])
    start = counts.cumsum(0) - counts
    assert bool((flat[real].long() == torch.searchsorted(start + counts, slot[real].long(), right=True)).all())     # a row lies with its expert
