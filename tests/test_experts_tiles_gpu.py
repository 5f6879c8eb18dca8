"""The experts' tensor-core products at the edges of their tiles: numbers of tokens around the sizes where the narrow operand or the tile
table changes, features and inner sizes that are no multiples of a tile, an expert with more rows than a tile and experts without any."""
import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


def grouped(idx, experts, tile_rows):
    T, top = idx.shape
    R = T * top
    ints = torch.empty(3 * R + 3 * ops.moe_max_tiles(R, experts, tile_rows), device="cuda", dtype=torch.int32)
    row_token, slot_row, scratch, tiles = ints[:R], ints[R: 2 * R], ints[2 * R: 3 * R], ints[3 * R:]
    ops.moe_group(row_token, slot_row, tiles, idx, scratch, experts, tile_rows)
    return row_token, slot_row, tiles


@pytest.mark.parametrize("T,E,top,K,N", [(1, 3, 1, 8, 8), (16, 5, 2, 72, 40), (17, 4, 3, 64, 136), (32, 9, 2, 200, 64), (33, 9, 2, 200, 72),
                                         (70, 3, 1, 128, 200), (300, 4, 2, 136, 72), (2200, 6, 6, 64, 128)])
@pytest.mark.parametrize("up", [1, 2, 0])
def test_products_at_tile_edges(T, E, top, K, N, up):
    g = torch.Generator(device="cuda").manual_seed(T * 7 + up)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    # (all choices of the first half of the tokens go to the first experts: more rows there than a tile holds, and fewer elsewhere)
    idx = torch.argsort(torch.rand((T, E), generator=g, device="cuda"), dim=1)[:, :top].to(torch.int32)
    idx[: T // 2] = torch.arange(top, device="cuda", dtype=torch.int32)
    idx = idx.contiguous()
    tile_rows = ops.moe_tile_rows(True, T, T * top, E)
    row_token, slot_row, tiles = grouped(idx, E, tile_rows)
    R = T * top
    w1, w2 = (rnd(E, N, K).mul_(K ** -0.5).to(torch.bfloat16) for _ in range(2))
    x = rnd(T, K).to(torch.bfloat16) if up else rnd(R, K).to(torch.bfloat16)
    out = torch.empty((R, N), device="cuda", dtype=torch.bfloat16 if up else torch.float32)
    ops.moe_experts_tc(up, out, x, ops.moe_pack_experts(w1), ops.moe_pack_experts(w2) if up == 1 else None, row_token, tiles, tile_rows=tile_rows)
    ops.check_kernel_errors()
    flat = slot_row.long()
    assert torch.equal(torch.sort(flat).values, torch.arange(R, device="cuda"))             # every choice has a row of its own
    e = idx.reshape(-1).long()
    src = x.double()[torch.arange(T, device="cuda").repeat_interleave(top)] if up else x.double()[flat]
    a = torch.einsum("rnk,rk->rn", w1.double()[e], src) if R * N * K < 3e7 else torch.cat(
        [(w1.double()[int(e[i])] @ src[i])[None] for i in range(0, R, 97)])
    b = torch.einsum("rnk,rk->rn", w2.double()[e], src) if R * N * K < 3e7 else torch.cat(
        [(w2.double()[int(e[i])] @ src[i])[None] for i in range(0, R, 97)])
    want = a * torch.sigmoid(a) * b if up == 1 else torch.relu(a) ** 2 if up == 2 else a
    got = out.double()[flat]
    if got.shape != want.shape:
        got = got[::97]
    # K float32 products of order 1/sqrt(K): an absolute error of some K^0.5 * 2^-24, twice that behind a product of two; bfloat16 rounding
    bound = 2e-5 * (1 + want.abs()) + (2.0 ** -8 * want.abs() if up else 0.0)
    assert bool(((got - want).abs() <= bound).all()), float((got - want).abs().max())


@pytest.mark.parametrize("T", [33, 64, 65, 128, 129])
def test_the_tokens_themselves_as_the_narrow_operand(T):
    """Up to 64 tokens the up product reads the tokens where they lie: the same bits as from rows in grouped order, with an expert that has
    all tokens and one that has none."""
    E, top, K, N = 5, 2, 72, 72
    g = torch.Generator(device="cuda").manual_seed(T)
    idx = torch.stack([torch.zeros(T, device="cuda"), torch.randint(1, E - 1, (T,), generator=g, device="cuda")], dim=1).to(torch.int32).contiguous()
    w = ops.moe_pack_experts(torch.randn((E, N, K), generator=g, device="cuda").to(torch.bfloat16))
    x = torch.randn((T, K + 8), generator=g, device="cuda").to(torch.bfloat16)[:, :K]
    rows = []
    for tile_rows in (ops.moe_tile_rows(True, T, T * top, E), 32):          # (a table of 32 rows a tile: 33 tokens and more are gathered)
        row_token, slot_row, tiles = grouped(idx, E, tile_rows)
        out = torch.empty((T * top, N), device="cuda", dtype=torch.bfloat16)
        ops.moe_experts_tc(2, out, x, w, None, row_token, tiles, tile_rows=tile_rows)
        ops.check_kernel_errors()
        rows.append(out[slot_row.long()])
    assert T > ops.MOE_DIRECT or ops.moe_tile_rows(True, T, T * top, E) >= T
    assert torch.equal(rows[0], rows[1])
