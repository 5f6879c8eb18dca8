"""The router's logits for many tokens, rows of it and tokens in groups, at the edges of the groups."""
import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


def rnd(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


@pytest.mark.parametrize("E", [6, 31, 39, 64, 71, 72, 130, 256])
@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("d", [64, 264, 2048])
def test_router_of_many_tokens(E, gate, d):
    """Rows and tokens in groups: the choices, weights and gates of short steps, bit for bit."""
    x, w = (rnd(301, d, seed=d) * 0.5).to(torch.bfloat16), (rnd(E + 1, d, seed=E) * d ** -0.5 * 4).to(torch.bfloat16)
    wg = w[E:].contiguous() if gate else None

    def route(rows):
        n = rows.shape[0]
        idx, wts = torch.empty(n, 4, device="cuda", dtype=torch.int32), torch.empty(n, 4, device="cuda")
        out = torch.empty(n, device="cuda") if gate else None
        ops.moe_route(idx, wts, out, rows, w[:E].contiguous(), wg)
        return [idx, wts] + ([out] if gate else [])

    for whole, *parts in zip(route(x), route(x[:200]), route(x[200:])):
        assert torch.equal(whole, torch.cat(parts))
