"""The experts' plan over lists of every length that is told apart: kept in registers, with a second round behind them; skewed choices, experts without rows and choices beyond the experts."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200.ops import moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,top,experts", [(1, 1, 1), (5, 2, 40), (1024, 8, 7), (8192, 1, 16), (8193, 1, 16), (2731, 3, 3), (10000, 2, 64), (5000, 4, 300), (20001, 1, 1)])
@pytest.mark.parametrize("choices", ["even", "one_expert", "skewed", "beyond"])
@pytest.mark.parametrize("weighted", [False, True])
def test_plan(tokens, top, experts, choices, weighted):
    g = torch.Generator("cuda").manual_seed(tokens + experts)
    chosen = torch.randint(0, experts, (tokens, top), device="cuda", generator=g)
    if choices == "one_expert":
        chosen[:] = experts - 1
    elif choices == "skewed":  # most to the first, some experts without any
        chosen = (chosen.float() * torch.rand(chosen.shape, device="cuda", generator=g) ** 4).long()
    elif choices == "beyond":
        chosen[torch.rand(chosen.shape, device="cuda", generator=g) < 0.3] = experts + 2
    chosen = chosen.to(torch.int32)
    weights = torch.rand(tokens, top, device="cuda", generator=g) if weighted else None
    where = moe.plan(chosen, weights, experts)
    flat, slots = chosen.view(-1).long(), where.slot_of.view(-1).long()
    taken = flat < experts
    assert (slots[~taken] == -1).all()
    used = slots[taken]
    assert used.unique().numel() == used.numel() and (used >= 0).all() and (used < where.capacity).all()
    token = torch.arange(tokens, device="cuda").repeat_interleave(top)
    want_token = torch.full((where.capacity,), -1, device="cuda", dtype=torch.long)
    want_token[used] = token[taken]
    assert torch.equal(where.slot_token.long(), want_token)
    want_weight = torch.zeros(where.capacity, device="cuda")
    want_weight[used] = weights.view(-1)[taken] if weighted else 1.0
    assert torch.equal(where.slot_weight, want_weight)
    # whole tiles per expert, in the experts' order, their real rows first
    counts = torch.bincount(flat[taken], minlength=experts).tolist()
    tiles = [(e, min(moe.PAD, n - first)) for e, n in enumerate(counts) for first in range(0, n, moe.PAD)]
    rest = where.capacity // moe.PAD - len(tiles)
    assert where.tile_expert.tolist() == [e for e, _ in tiles] + [-1] * rest
    assert where.tile_rows.tolist() == [r for _, r in tiles] + [0] * rest
    tile_of = torch.tensor([e for e, _ in tiles] + [-1] * rest, device="cuda")
    assert torch.equal(tile_of[used // moe.PAD], flat[taken])
    rows = torch.tensor([r for _, r in tiles] + [0] * rest, device="cuda")
    assert (used % moe.PAD < rows[used // moe.PAD]).all()
