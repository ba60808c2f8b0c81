"""The residual convolution through runs of tokens and token by token: the same bits, with requests that begin and end inside a run and states of their own."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200.ops import recurrent

pytestmark = pytest.mark.gpu


def _conv(x, weight, state, counts):
    starts = torch.tensor([0] + counts, dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    rows = torch.repeat_interleave(torch.arange(len(counts), dtype=torch.int32), torch.tensor(counts)).cuda()
    slots = torch.arange(len(counts), dtype=torch.int32).flip(0).contiguous().cuda()
    return recurrent.residual_conv(x, weight, state, 0, slots, rows, starts)


@pytest.mark.parametrize("taps", range(1, 9))
@pytest.mark.parametrize("counts", [[1, 3, 8, 13, 7, 1, 1, 600], [5, 300, 9, 1, 2], [1] * 7 + [900]])
def test_runs(taps, counts):
    g = torch.Generator("cuda").manual_seed(taps)
    tokens, channels = sum(counts), 1608
    channels = channels if taps > 3 else 8192  # past the line where runs begin
    x = torch.randn(tokens, channels, device="cuda", generator=g).to(torch.bfloat16)
    weight, state = torch.randn(channels, taps, device="cuda", generator=g), torch.randn(len(counts), max(1, (taps - 1) * channels), device="cuda", generator=g)
    got = _conv(x, weight, state, counts)
    first = 0
    for r, n in enumerate(counts):  # each request by itself, at most seven tokens of it: steps of single tokens
        own = state[len(counts) - 1 - r : len(counts) - r].contiguous()
        few = min(n, 7)
        assert torch.equal(got[first : first + few], _conv(x[first : first + few].contiguous(), weight, own, [few]))
        before = torch.cat([own[0, : (taps - 1) * channels].view(taps - 1, channels).double(), x[first : first + n].double()])
        want = x[first : first + n].double() + sum(weight[:, j].double() * before[j : j + n] for j in range(taps))
        size = x[first : first + n].double().abs() + sum(weight[:, j].double().abs() * before[j : j + n].abs() for j in range(taps))
        # taps + 1 sums in float, one rounding to bfloat16
        assert ((got[first : first + n].double() - want).abs() <= 2.0 ** -8 * want.abs() + (taps + 1) * 2.0 ** -23 * size).all()
        first += n
