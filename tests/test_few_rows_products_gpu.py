"""Products of steps that bring every expert a few rows, against 64 bits."""
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from hyperion_b200.ops import moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("activation", [None, "relu_squared"])
@pytest.mark.parametrize("streams", [True, False])
@pytest.mark.parametrize("tokens,top,experts,n,k", [
    (4, 2, 4, 128, 64), (8, 1, 4, 16, 32),          # the least that takes the kernel: two rows per expert; one warp's columns
    (17, 2, 5, 130, 40), (20, 2, 4, 259, 1000),     # columns and k that end inside a warp's and a piece's
    (9, 1, 1, 64, 8), (33, 1, 1, 48, 264),          # nine rows of one expert, thirty-three: several passes over a tile
    (64, 2, 16, 300, 2056),                         # the most pairs
    (3, 2, 16, 96, 520), (7, 2, 8, 33, 24),         # fewer: the other kernel
    (16, 1, 1, 24, 6400),                           # rows too long for sixteen in shared memory
])
def test_few_rows_per_expert(tokens, top, experts, n, k, streams, activation, monkeypatch):
    monkeypatch.setattr(moe, "SOME_COLUMNS", 0)  # the kernel takes any, the dispatch gives it the longer ones
    g = torch.Generator("cuda").manual_seed(tokens * 1000 + k)
    x = torch.randn(tokens, k, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(experts, n, k, device="cuda", generator=g) / k**0.5).to(torch.bfloat16)
    chosen = torch.stack([torch.randperm(experts, device="cuda", generator=g)[:top] for _ in range(tokens)]).to(torch.int32)
    where = moe.plan(chosen, None, experts, streams)
    assert where.streams == streams
    rows = x if streams else moe.gather(x, where)
    slots = where.slot_of.view(tokens, top).long()
    got = moe.grouped_linear(rows, w, where, activation)[slots].double()
    per_choice = w.double()[chosen.long()]
    want = torch.einsum("tk,tjnk->tjn", x.double(), per_choice)
    # every one of k exact products is added once in float (half a unit per addition, a whole one where sixteen are cut off), and the result is rounded to bfloat16
    room = torch.einsum("tk,tjnk->tjn", x.double().abs(), per_choice.abs()) * k * 2.0**-23
    if activation:
        want, room = want.clamp(min=0).square(), 2 * want.abs() * room + room.square()
    assert ((got - want).abs() <= room + want.abs() * 2.0**-8 + 1e-30).all()


@pytest.mark.parametrize("tokens,k", [(64, 1536), (64, 2048), (64, 4096), (9, 7176)])
def test_sums_are_as_close_as_without_tensor_cores(tokens, k, monkeypatch):
    """Every product stands beside its negative somewhere else in the row, so the sums are exactly zero and the results nothing but the sums' roundings (which the result's own rounding to
    bfloat16 would hide).  Over a thousand columns and more the tensor cores' are not larger than the float units'."""
    experts, n, top = 4, 1024, 1
    g = torch.Generator("cuda").manual_seed(k)
    half = torch.randn(tokens, k // 2, device="cuda", generator=g).to(torch.bfloat16)
    weights = (torch.randn(experts, n, k // 2, device="cuda", generator=g) / k**0.5).to(torch.bfloat16)
    places = torch.randperm(k, device="cuda", generator=g)
    x, w = torch.cat([half, -half], 1)[:, places].contiguous(), torch.cat([weights, weights], 2)[..., places].contiguous()
    where = moe.plan((torch.arange(tokens, device="cuda", dtype=torch.int32) % experts).view(tokens, top), None, experts, True)
    assert k > moe.SOME_COLUMNS
    far = []
    for rows_per_expert in (0, 1 << 20):  # all steps through the tensor cores, none
        monkeypatch.setattr(moe, "SOME_ROWS", rows_per_expert)
        got = moe.grouped_linear(x, w, where)[where.slot_of.view(tokens, top).long()].double()
        far.append(float(got.square().mean().sqrt()))
    assert 0 < far[0] <= far[1], far


@pytest.mark.parametrize("rows_per_expert", [0, 1 << 20])  # all steps through the tensor cores, none
def test_threads_with_rows_of_different_lengths(rows_per_expert, monkeypatch):
    """Rows of 4,096 and of 6,400 entries take different amounts of shared memory; two threads that launch both kinds at once must not take each other's allowance away."""
    monkeypatch.setattr(moe, "SOME_ROWS", rows_per_expert)

    def products(k, seed):
        g = torch.Generator("cuda").manual_seed(seed)
        x, w = torch.randn(16, k, device="cuda", generator=g).to(torch.bfloat16), (torch.randn(2, 64, k, device="cuda", generator=g) / k**0.5).to(torch.bfloat16)
        where = moe.plan((torch.arange(16, device="cuda", dtype=torch.int32) % 2).view(16, 1), None, 2, True)
        want = moe.grouped_linear(x, w, where)[where.slot_of.long()]
        torch.cuda.synchronize()
        return all(torch.equal(moe.grouped_linear(x, w, where)[where.slot_of.long()], want) for _ in range(150))

    with ThreadPoolExecutor(2) as pool:
        assert all(pool.map(products, (4096, 6400), (1, 2)))
