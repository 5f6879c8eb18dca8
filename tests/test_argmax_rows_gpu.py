"""The argmax of long rows (a cluster of CTAs a row) at the edges of its parts: the first of the largest, as for short rows."""
import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [16384, 16385, 16390, 32771, 128256])
@pytest.mark.parametrize("shift", [0, 1])
def test_first_of_the_largest(V, shift):
    g = torch.Generator(device="cuda").manual_seed(V)
    wide = torch.randn(9, V + 3, generator=g, device="cuda")
    rows = wide[:, shift: shift + V]
    part = -(-(-(-V // 8)) // 4) * 4
    for r, at in enumerate((0, V - 1, part - 1, part, V // 4 * 4 - 1)):
        rows[r, at] = 100.0
        if r == 2:
            rows[r, part] = 100.0                               # a tie over the border of two parts
    rows[5] = float("-inf")
    rows[6] = float("nan")
    rows[7, :100] = float("nan")
    want = [0, V - 1, part - 1, part, V // 4 * 4 - 1, 0, 0] + [100 + int(rows[7, 100:].cpu().argmax()), int(rows[8].cpu().argmax())]
    out = torch.full((9,), -1, device="cuda", dtype=torch.int32)
    ops.argmax(out, rows)
    assert out.tolist() == want
