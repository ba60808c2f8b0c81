"""Prompts cut into tiles of half the rows: which steps are, and that every row's result is the same bits."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from hyperion_b200.ops import attention
from hyperion_b200.ops.native import sm_count

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,page,window", [(4, 4, 128, 16, 0), (8, 2, 128, 64, 100), (7, 1, 64, 8, 0), (6, 2, 128, 32, -128)])
@pytest.mark.parametrize("counts,first", [((5,), (0,)), ((255, 256, 257), (0, 3, 0)), ((130, 600), (200, 0))])
def test_same_bits(heads, kv_heads, dim, page, window, counts, first):
    rows = SimpleNamespace(counts=np.array(counts, np.int32))
    g = torch.Generator("cuda").manual_seed(sum(counts))
    total, width = sum(counts), -(-max(a + n for a, n in zip(first, counts)) // page)
    cache = torch.randn(len(counts) * width, 2, kv_heads, page, dim, device="cuda", generator=g).to(torch.bfloat16)
    table = torch.arange(len(counts) * width, dtype=torch.int32, device="cuda").view(len(counts), width)
    q = torch.randn(total, heads * dim, device="cuda", generator=g).to(torch.bfloat16)
    token_row = torch.repeat_interleave(torch.arange(len(counts), dtype=torch.int32), torch.tensor(counts)).to(torch.int32).cuda()
    positions = torch.cat([torch.arange(a, a + n, dtype=torch.int32) for a, n in zip(first, counts)]).cuda()
    per_tile = attention.tile_tokens(heads, kv_heads, attention.TC_TILE_ROWS)
    outs = []
    for most in (0.0, 1e9):
        tiles, _ = attention.plan_prompts(rows, per_tile, kv_heads, most)
        assert (tiles[1::3] * (heads // kv_heads) <= (128 if most else 256)).all() and tiles[1::3].sum() == total
        out = torch.zeros_like(q)
        attention.attention_tiles(q, heads, cache, table, token_row, positions, torch.from_numpy(tiles.copy()).cuda(), len(tiles) // 3, dim ** -0.5, window, out,
                                  tile_size=attention.TC_TILE_ROWS)
        outs.append(out)
    assert torch.equal(*outs) and outs[0].abs().amax(1).min() > 0


def test_rule():
    sms = sm_count()
    for tiles, blocks in ((sms // 8, 4), (sms // 8 + 1, 4), (sms // 2, 1), (sms // 2 + 1, 1)):
        planned, _ = attention.plan_prompts(SimpleNamespace(counts=np.array([64 * tiles], np.int32)), 64, blocks)
        assert len(planned) // 3 == (2 * tiles if 2 * tiles * blocks <= sms else tiles)
    whole, _ = attention.plan_prompts(SimpleNamespace(counts=np.array([40], np.int32)), 1, 1)  # a head group of more than 128 rows a token has no halves
    assert len(whole) // 3 == 40
