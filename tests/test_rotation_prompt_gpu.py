"""Rotation with the write to the cache at a prompt's sizes: the bits of the two separate steps, and tokens without a place or a page left out and reported."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q_heads,kv_heads,dim", [(7, 1, 64), (4, 2, 128), (3, 3, 80)])
@pytest.mark.parametrize("tokens", [1027, 511])
@pytest.mark.parametrize("bad", [False, True])
def test_prompt(q_heads, kv_heads, dim, tokens, bad):
    g = torch.Generator("cuda").manual_seed(tokens + dim)
    page, positions = 16, torch.arange(tokens, dtype=torch.int32, device="cuda")
    table = torch.randperm(-(-tokens // page), device="cuda", generator=g).to(torch.int32).view(1, -1)
    angles = torch.rand(2048, dim // 2, device="cuda", generator=g) * 6
    rope = torch.stack([angles.cos(), angles.sin()], -1).contiguous()
    x = torch.randn(tokens, (q_heads + 2 * kv_heads) * dim, device="cuda", generator=g).to(torch.bfloat16)
    cache = torch.zeros(table.shape[1], 2, kv_heads, page, dim, dtype=torch.bfloat16, device="cuda")
    rows = torch.zeros(tokens, dtype=torch.int32, device="cuda")
    left_out = torch.zeros(tokens, dtype=torch.bool, device="cuda")
    one, two, cache_two = x.clone(), x.clone(), cache.clone()
    ops.rope_(two, q_heads + kv_heads, dim, positions, rope)
    if bad:  # among their neighbours: a position past the table, and a page that is not there
        positions[[2, 401]] = 2048
        table[0, 20] = -1
        left_out[[2, 401]] = True
        left_out[20 * page : 21 * page] = True
        keep = ~left_out
        ops.kv_store(two[keep].contiguous(), q_heads * dim, (q_heads + kv_heads) * dim, cache_two, table, rows[keep], positions[keep])
    else:
        ops.kv_store(two, q_heads * dim, (q_heads + kv_heads) * dim, cache_two, table, rows, positions)
    ops.rope_kv_store_(one, q_heads, kv_heads, dim, positions, rope, cache, table, rows)
    device = torch.device("cuda:0")
    if bad:
        with pytest.raises(ops.KernelError, match="(?i)position|page"):
            ops.raise_on_status(device)
    ops.raise_on_status(device)
    rotated = torch.arange(tokens, device="cuda") != -1
    rotated[[2, 401]] = not bad
    scale = 2.0 ** -8  # one rounding, of a product and a sum in one step or two
    assert (one[rotated, : q_heads * dim].float() - two[rotated, : q_heads * dim].float()).abs().max() <= scale * 4
    assert torch.equal(cache == 0, cache_two == 0)
    assert (cache.float() - cache_two.float()).abs().max() <= scale * 8
    assert torch.equal(cache[:, 1], cache_two[:, 1])  # values pass as they are
