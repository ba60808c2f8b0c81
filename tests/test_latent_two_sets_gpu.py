"""Two sets of 32 rows on one key tile: the same numbers as one set."""
import pytest
import torch

from hyperion_b200.ops import attention as fast


@pytest.mark.gpu
@pytest.mark.parametrize("heads,record,value,page", [(16, 576, 512, 32), (5, 320, 256, 16), (7, 64, 56, 8), (32, 128, 64, 16)])
@pytest.mark.parametrize("with_sink", [False, True])
def test_two_sets_equal_one(heads, record, value, page, with_sink):
    """Requests of 1 to 70 tokens behind 0 to 300 cached ones: sets that end inside the block, sets without a row, keys split over blocks.
    Both forms take a score and a result from the same sums in the same order, so the results are equal bit by bit (one set against
    64 bits is tested elsewhere)."""
    g = torch.Generator().manual_seed(record)
    counts, firsts = [1, 70, 3, 13, 17], [300, 0, 129, 63, 64]
    blocks = [-(-(f + c) // page) for c, f in zip(counts, firsts)]
    order = torch.randperm(sum(blocks) + 3, generator=g).to(torch.int32)
    table, at = torch.full((len(counts), max(blocks)), -1, dtype=torch.int32), 0
    for row, n in enumerate(blocks):
        table[row, :n] = order[at : at + n]
        at += n
    cache = torch.randn(len(order), 1, page, record, generator=g).to(torch.bfloat16).cuda()
    query = torch.randn(sum(counts), heads * record, generator=g).to(torch.bfloat16).cuda()
    starts = torch.tensor([0, *torch.tensor(counts).cumsum(0).tolist()], dtype=torch.int32).cuda()
    positions = torch.cat([torch.arange(c, dtype=torch.int32) + f for c, f in zip(counts, firsts)]).cuda()
    sinks = torch.randn(heads, generator=g).cuda() if with_sink else None
    for splits in (1, 3, 7):
        one, two = (fast.attention_latent(query, heads, record, value, cache, table.cuda(), starts, positions, len(counts), max(counts),
                                          max(c + f for c, f in zip(counts, firsts)), record**-0.5, sinks=sinks, shape=(rows, splits)) for rows in (1, 2))
        assert torch.equal(one, two), splits


@pytest.mark.parametrize("asked,shape", [
    ((1, 2048, 16, 2048, 576, 2048), (2, 1)),
    ((1, 2048, 16, 2048, 592, 2048), (1, 1)),  # no room for two sets
    ((1, 2048, 16, 2048, 560, 2048), (1, 1)),  # records of no whole 128 bytes
    ((1, 600, 16, 600, 576, 600), (1, 1)),     # too few blocks of 64 rows
    ((8, 1, 16, 2048, 576, 8), (0, 16)),       # decoded tokens
    ((1000, 1, 16, 2048, 576, 1000), (0, 1)),  # many of them: sixteen pairs each
    ((9, 100, 16, 2048, 576, 108), (1, 1)),    # a short prompt beside decoded tokens
    ((8, 1000, 16, 2048, 576, 1007), (2, 1)),  # a long one
])
def test_rule(asked, shape):
    *sizes, record, tokens = asked
    assert fast.choose_latent_shape(*sizes, sms=148, record=record, tokens=tokens) == shape
