"""Matrices, weights, positions and row lists that a kernel of this package has just written, and that let the next kernel start early: who reads them waits for them."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200 import ops
from hyperion_b200.ops import moe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _random(*shape, seed=0, dtype=BF):
    return torch.randn(*shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed)).to(dtype)


def _late_integers(seed, tokens=2048, count=64):
    """[tokens] int32 below ``count``, as the tail of a long kernel whose successor may start before it has finished."""
    return moe.route(_random(tokens, 1024, seed=seed), _random(count, 1024, seed=seed + 1, dtype=torch.float32), 1)[0].view(-1)


def _twice(call, make, seeds):
    """``call`` of what ``make`` has just launched, and of the same once everything stands."""
    for seed in seeds:
        made = make(seed)
        got = call(made)
        torch.cuda.synchronize()
        assert torch.equal(got, call(made.clone())), seed


@pytest.mark.parametrize("n,k", [(2048, 2048), (896, 896), (9728, 896)])
@pytest.mark.parametrize("form", ["plain", "pieces", "gated"])
def test_a_matrix(n, k, form):
    x = _random(4, k)

    def call(w):
        if form == "gated":
            return ops.gated_linear(x, w, None)
        y = ops.linear(x, w, may_leave_partials=form == "pieces")
        return y if isinstance(y, torch.Tensor) else y.partials
    if k < 2048 or form == "gated":  # the split product, which may take the others, fetches its matrix early by its own contract
        _twice(call, lambda seed: ops.gelu_tanh(_random(n, k, seed=seed)), range(8))


def test_positions():
    frequencies = torch.rand(32, device="cuda")

    def in_place(positions):
        x = _random(2048, 4 * 128, seed=7)
        ops.heads_prepare_(x, 4, 0, 128, 128, positions, inv_freq=frequencies, rot_dims=64)
        return x

    def wide(positions):
        x, q, k = _random(2048, 8 * 128, seed=7, dtype=torch.float32), torch.empty(2048, 512, device="cuda", dtype=BF), torch.empty(2048, 512, device="cuda", dtype=BF)
        ops.heads_prepare_wide(x, 0, 512, 512, 4, 4, 128, 128, positions, q_out=q, k_out=k, inv_freq=frequencies, rot_dims=64)
        return torch.cat([q, k])

    def expanded(positions):
        q, kv, part = _random(2048, 2 * 192, seed=7), _random(2048, 2 * 256, seed=8), _random(2048, 64, seed=9)
        pages, table = torch.empty(1, 2, 2, 64, 192, device="cuda", dtype=BF), torch.zeros(1, 1, device="cuda", dtype=torch.int32)
        ops.latent_expand_(q, kv, part, 2, 128, 128, frequencies, 64, positions, torch.zeros(2048, device="cuda", dtype=torch.int32), table, pages)
        return q
    for call in (in_place, wide, expanded):
        call(torch.zeros(2048, device="cuda", dtype=torch.int32))
        _twice(call, _late_integers, range(0, 12, 2))
    ops.raise_on_status(torch.device("cuda:0"))


def test_a_norm_s_weight_and_rows():
    y = _random(64, 2048, seed=1)

    def add(weight):
        h = torch.zeros(64, 2048, device="cuda")
        ops.rmsnorm_add(h, y, weight[0], 1e-6)
        return h
    _twice(add, lambda seed: ops.gelu_tanh(_random(4096, 2048, seed=seed, dtype=torch.float32)), range(6))
    h, ones = _random(64, 2048, seed=2, dtype=torch.float32), torch.ones(2048, device="cuda")
    _twice(lambda rows: ops.norm_add_norm(h, y, ones, 1e-6, None, ones, 1e-6, BF, rows=rows[-16:]), _late_integers, range(0, 12, 2))
