"""Experts' products on pairs of SMs: runs of one, two and three row tiles, experts without rows, widths that are no whole tiles, against 64 bits."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200 import ops
from hyperion_b200.ops import gemm, moe

pytestmark = pytest.mark.gpu


def _case(counts, k, n, seed):
    """Tokens with one choice each, ``counts`` of them for each expert, in a shuffled order."""
    g = torch.Generator().manual_seed(seed)
    chosen = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    chosen = chosen[torch.randperm(len(chosen), generator=g)].view(-1, 1).cuda()
    x = torch.randn(len(chosen), k, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(len(counts), n, k, generator=g) * k ** -0.5).to(torch.bfloat16).cuda()
    where = moe.plan(chosen, None, len(counts))
    return chosen.view(-1).long(), x, w, where, moe.gather(x, where)


def _close(got, want, magnitude, k):
    """One rounding to bfloat16, and k products added up in float: at most k * 2^-23 (sums cut off) of the sum of their sizes, times two for what an activation makes of it."""
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2 * k * 2.0 ** -23 * magnitude + 1e-30).all()


# runs of whole pairs, of an odd tile, of a row more than a tile or a pair, none at all; one expert alone; k and n past whole tiles
@pytest.mark.parametrize("counts,k,n", [((256, 128, 129, 0, 257, 1), 64, 256), ((0, 384, 0, 511), 200, 1032), ((300,), 72, 512), ((1, 255, 640), 1024, 1024)])
@pytest.mark.parametrize("activation", [None, "relu_squared", "gelu_erf", "gelu_tanh"])
def test_pairs(counts, k, n, activation):
    chosen, x, w, where, rows = _case(counts, k, n, k + n)
    assert moe.takes_pairs(w, where)
    got = (moe.grouped_gelu if activation in moe.GELUS else moe.grouped_linear)(rows, w, where, activation)[where.slot_of.long()]
    z = torch.stack([w[e].double() @ r.double() for e, r in zip(chosen, x)])
    magnitude = torch.stack([w[e].double().abs() @ r.double().abs() for e, r in zip(chosen, x)])
    if activation == "relu_squared":
        want, magnitude = z.clamp(min=0) ** 2, magnitude * (1 + 2 * z.abs())
    elif activation is not None:
        want = torch.nn.functional.gelu(z, approximate="tanh" if activation == "gelu_tanh" else "none")
    else:
        want = z
    _close(got, want, magnitude, k)


@pytest.mark.parametrize("counts,k,inter", [((129, 0, 400), 136, 128), ((512, 1), 64, 384)])
def test_swiglu_in_the_epilogue(counts, k, inter):
    chosen, x, w, where, rows = _case(counts, k, 2 * inter, k)
    got = moe.grouped_swiglu(rows, torch.stack([gemm.interleave_gate_up(m[:inter], m[inter:]) for m in w]), where, gemm.SWIGLU_BLOCK)[where.slot_of.long()]
    z = torch.stack([w[e].double() @ r.double() for e, r in zip(chosen, x)])
    size = torch.stack([w[e].double().abs() @ r.double().abs() for e, r in zip(chosen, x)])
    gate, up = z.chunk(2, -1)
    _close(got, gate * torch.sigmoid(gate) * up, size[:, :inter] * up.abs() + size[:, inter:] * gate.abs(), 2 * k)
    plain = ops.swiglu(moe.grouped_linear(rows, w, where))[where.slot_of.long()]  # three roundings where the epilogue has one
    assert ((got.double() - plain.double()).abs() <= 2.0 ** -6 * (plain.double().abs() + up.abs() * 2.0 ** -2 + 2.0 ** -8)).all()


def test_few_pairs_per_expert_keep_single_tiles():
    _, _, w, where, _ = _case((100, 60, 30), 64, 256, 0)
    assert not moe.takes_pairs(w, where)
