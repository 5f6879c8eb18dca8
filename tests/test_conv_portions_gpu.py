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


def plain(x, w, bias, tail, lens, act, add):
    """The convolution in float64: outputs, and each segment's last inputs."""
    taps, at, ys, tails = w.shape[1], 0, [], []
    for s, n in enumerate(lens):
        seq = torch.cat([tail[s].double(), x[at: at + n].double()])
        y = sum(seq[i: i + n] * w[:, i].double() for i in range(taps))
        if bias is not None:
            y = y + bias.double()
        if act:
            y = y / (1 + torch.exp(-y))
        ys.append(y + x[at: at + n].double() if add else y)
        tails.append(seq[seq.shape[0] - (taps - 1):])
        at += n
    return torch.cat(ys), torch.stack(tails)


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("types", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("lens", [[1, 16, 2, 3, 17, 33, 1], [1, 2, 1]])
def test_against_float64(taps, types, lens):
    """Outputs over sums from -90 to 90 and the state, over portions and in steps of short ones; float32 outputs within a few roundings of the
    sum and of the function's argument, bfloat16 ones within one more rounding of theirs (numbers of 8 bits: half an ulp is at most 2^-8 of the value)."""
    channels, T, S = 132, sum(lens), len(lens)
    g = torch.Generator(device="cuda").manual_seed(taps)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    ctx = SimpleNamespace(num_segments=S, max_q_len=max(lens), seg_slot=torch.arange(S, dtype=torch.int32, device="cuda"),
                          seg_q_start=torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32))
    x, w, bias = rnd(T, channels).to(types[0]), rnd(channels, taps), torch.linspace(-90, 90, channels, device="cuda")
    start = rnd(S, taps - 1, channels).to(types[0]).float()
    for act, add, b in ((True, False, bias), (False, True, None), (True, True, None)):
        state, out = torch.zeros(S, max(4, (taps - 1) * channels), device="cuda"), torch.full((T, channels), float("nan"), device="cuda", dtype=types[1])
        state[:, : (taps - 1) * channels] = start.reshape(S, -1)
        ops.conv_state(out, x, w, b, state, ctx, act=act, add_input=add)
        want, tails = plain(x, w, b, start, lens, act, add)
        assert torch.equal(state[:, : (taps - 1) * channels], tails.reshape(S, -1).float())
        # the sum: taps + 1 float32 roundings of numbers up to 90 + |x| |w| sums; SiLU passes an error of its argument on by at most 1.1 where
        # its result is large and relatively by the error itself where it is small (90 x 2^-24 a rounding), and adds a few ulp of its own
        err = (out.double() - want).abs()
        size = want.abs() + (x.double().abs() if add else 0)
        bound = (taps + 8) * 2.0 ** -24 * (100 * size + 1e-30) if act else (taps + 2) * 2.0 ** -24 * (size + 20)
        if types[1] == torch.bfloat16:
            bound = bound + want.abs() * 2.0 ** -8 * 1.01 + 1e-38
        assert bool((err <= bound).all()), float((err / bound).max())


def test_silu_rounded_to_bfloat16_is_the_accurate_one():
    """Arguments of -90 to 90 through a filter that passes its input: the bfloat16 next to float64's SiLU but for what lies within float32's error of
    the middle of two, also where 1 + exp(-x) is above 2^126 (a quotient of the fast functions is zero there); zero or about as small
    where exp(-x) is no float32 number any more, below -88.7."""
    x = torch.cat([torch.linspace(-90, 90, 32768), torch.linspace(-88.3, -86, 8192)]).reshape(40, 1024).cuda()
    w = torch.zeros(1024, 2, device="cuda")
    w[:, 1] = 1
    for lens in ([40], [1] * 40):
        S = len(lens)
        ctx = SimpleNamespace(num_segments=S, max_q_len=max(lens), seg_slot=torch.arange(S, dtype=torch.int32, device="cuda"),
                              seg_q_start=torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32))
        out = torch.empty(40, 1024, device="cuda", dtype=torch.bfloat16)
        ops.conv_state(out, x, w, None, torch.zeros(S, 1024, device="cuda"), ctx)
        want = x.double() / (1 + torch.exp(-x.double()))
        normal = (want.abs() >= 2.0 ** -126) & (x > -88.7)
        assert bool(((out.double() - want).abs()[~normal] <= 2.0 ** -119).all())           # (88.7 exp(-88.7) is 2^-121.5)
        assert bool(((out.double() - want).abs() <= want.abs() * (2.0 ** -8 + 1e-5) + 2.0 ** -133)[normal].all())
        assert float((out.double() != want.to(torch.bfloat16).double())[normal].double().mean()) < 1e-3
