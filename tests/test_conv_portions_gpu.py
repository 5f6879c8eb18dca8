"""The short convolution over portions, four channels a thread, against a channel a thread (which an odd address of the state asks for): the same
bits, outputs and state, with segments shorter than the filter's reach beside longer ones."""
from types import SimpleNamespace

import pytest
import torch

from qorvix_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("channels", [4, 132, 516])
@pytest.mark.parametrize("types", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
def test_four_channels_a_thread(taps, channels, types):
    lens = [1, 16, 2, 3, 17, 33, 1]
    g = torch.Generator(device="cuda").manual_seed(taps * 1000 + channels)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, S, size = sum(lens), len(lens), (taps - 1) * channels
    ctx = SimpleNamespace(num_segments=S, max_q_len=max(lens), seg_slot=torch.arange(S, dtype=torch.int32, device="cuda").flip(0).contiguous(),
                          seg_q_start=torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32))
    x = rnd(T, channels + 8).to(types[0])[:, 8:]
    w, bias = rnd(channels, taps), rnd(channels)
    wide = rnd(S, size + 4)
    for act, add, b in ((True, False, bias), (False, True, None)):
        results = []
        for shift in (0, 1):
            state = torch.zeros(S, size + 4, device="cuda")
            state[:, shift: shift + size] = wide[:, :size]
            out = torch.full((T, channels), float("nan"), device="cuda", dtype=types[1])
            ops.conv_state(out, x, w, b, state[:, shift: shift + size], ctx, act=act, add_input=add)
            results.append((out, state[:, shift: shift + size].clone()))
        assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
