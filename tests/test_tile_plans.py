"""Layers whose heads form groups of one size but in other numbers: each finds the tiles that the rule for its own blocks gives, whichever layer planned first."""
from types import SimpleNamespace

import numpy as np
import pytest

from hyperion_b200.ops import attention
from hyperion_b200.parts.attention import GroupedQueryAttention


class Packer:
    def __init__(self):
        self._items = []

    def add(self, name, values, shape=None):
        self._items.append((name, np.asarray(values)))


@pytest.mark.parametrize("order", [1, -1])
@pytest.mark.parametrize("counts", [[1000], [300, 3, 700]])
def test_every_number_of_blocks_has_its_own_tiles(order, counts, monkeypatch):
    monkeypatch.setattr(attention, "sm_count", lambda *a: 148)
    shapes = [(28, 4, 128), (224, 32, 128), (7, 1, 128)][::order]  # groups of seven
    planners = {}
    for heads, kv_heads, dim in shapes:
        planners.update(GroupedQueryAttention.plans_for(heads, kv_heads, dim))
    planners.update(GroupedQueryAttention.plans_for(14, 2, 128, lambda page_size: 256))  # a kernel of its own, which takes its tiles whole
    rows, packer, host = SimpleNamespace(counts=np.array(counts, np.int32)), Packer(), {"page_size": 16}
    for plan in planners.values():
        plan(rows, packer, host)
    placed = dict(packer._items)
    for heads, kv_heads, dim in shapes:
        size = attention.tile_rows(dim, 16)
        tokens, blocks = attention.tile_tokens(heads, kv_heads, size), attention.tile_blocks(heads, kv_heads, size)
        assert size == attention.TC_TILE_ROWS and blocks == kv_heads
        want, _ = attention.plan_prompts(rows, tokens, blocks)
        key = attention.tiles_key(tokens, blocks)
        assert np.array_equal(placed[key], want) and host[key] == len(want) // 3
    whole, _ = attention.plan(rows, 36)
    assert np.array_equal(placed[attention.tiles_key(36, 0)], whole)
    few, many = (len(placed[attention.tiles_key(36, b)]) for b in (1, 32))
    assert few > many == len(whole)  # halved where the SMs allow it, and only there


def test_other_kernels_tiles_do_not_count_blocks():
    assert attention.tile_blocks(32, 8, attention.TILE_ROWS) == 0 and attention.tile_blocks(512, 1, attention.TC_TILE_ROWS) == 2
