"""The recurrences that walk long bfloat16 rows in chunks at float precision (csrc/chunked_float.cu): the plan on the CPU, the kernels against 64-bit arithmetic."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from hyperion_b200.ops import recurrent


def test_the_plan_covers_every_long_row_once():
    assert recurrent.plan_rule_chunks([127, 64, 1]) is None
    for counts in ([128], [1, 300, 15, 16, 64, 65, 2], [2048, 1], [129] * 3):
        chunks, walks, others = recurrent.plan_rule_chunks(counts)
        covered = [t for first, count in zip(chunks[::2], chunks[1::2]) for t in range(first, first + count)]
        starts = [sum(counts[:i]) for i in range(len(counts))]
        long_rows = [i for i, c in enumerate(counts) if c >= recurrent.CHUNKED_RULE_ROWS]
        assert covered == [t for i in long_rows for t in range(starts[i], starts[i] + counts[i])]
        assert all(0 < c <= recurrent.CHUNK for c in chunks[1::2]) and others == (len(long_rows) < len(counts))
        assert walks[2::3] == long_rows and walks[0::3] == [0, *walks[1::3]][: len(long_rows)] and walks[-2] == len(chunks) // 2
        for begun, end, row in zip(walks[::3], walks[1::3], walks[2::3]):
            assert sum(chunks[2 * begun + 1 : 2 * end : 2]) == counts[row]


def test_chunks_go_fewer_at_a_time_where_memory_is_short(monkeypatch):
    """A device with room for so many floats and no more: as many chunks as fit after halving, one at the least, and an error only where one does not fit."""
    piece, empty = 1000, torch.empty

    def short_of(room):
        def allocate(size, **kwargs):
            if size > room:
                raise torch.cuda.OutOfMemoryError(f"{size} of {room}")
            return empty(size, **kwargs)
        return allocate

    for room, span in ((40_000, 40), (39_999, 20), (11_000, 10), (4_999, 3), (1_000, 1)):
        monkeypatch.setattr(torch, "empty", short_of(room))
        got, scratch = recurrent._scratch_of_chunks(40, piece, "cpu")
        assert got == span and scratch.numel() == span * piece
    monkeypatch.setattr(torch, "empty", short_of(999))
    with pytest.raises(torch.cuda.OutOfMemoryError):
        recurrent._scratch_of_chunks(40, piece, "cpu")


def test_steps_take_chunks_where_these_are_faster():
    """Steps as measured on 148 multiprocessors, 16 heads of 128 x 128 (time mixing: 32 of 64): a long row or two alone leave the device to the chunks, many rows at once fill it token by token
    too, and rows of a quarter of a chunk beside a short one are padding."""
    def pay(rule, counts, more=1):
        chunks, walks, _ = recurrent.plan_rule_chunks(counts)
        heads, e = (32, 64) if rule == recurrent.RULE_WKV else (16, 128)
        return recurrent.chunks_pay(rule, len(chunks) // 2, -(-max(counts) // recurrent.CHUNK), sum(chunks[1::2]), more * heads, e, 148)

    for rule in (recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA, recurrent.RULE_RETENTION, recurrent.RULE_WKV):
        delta = rule in (recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA)
        assert all(pay(rule, counts) for counts in ([128], [2048], [600, 700], [300] + [1] * 40, [2048] + [100] * 15, [512] * 4))
        assert [pay(rule, counts) for counts in ([128] * 16, [512] * 8, [128] + [16] * 7)] == [delta] * 3 and not pay(rule, [128] + [16] * 7, more=2)
        assert pay(rule, [1024] * 4, more=2) == (rule != recurrent.RULE_WKV)


@pytest.mark.parametrize("counts", [[1] * 7, [300, 1, 15, 16], [128], [127, 2], [700, 1, 512]])
def test_the_planners_read_rows_as_arrays_and_as_objects(counts):
    """A step's rows come as arrays (the runner's) or as a list of rows: the same plans, of plain integers, and none in a step without a long row."""
    class Packer(dict):
        add = dict.__setitem__

    arrays, objects = SimpleNamespace(counts=np.array(counts, dtype=np.int32)), [SimpleNamespace(count=c) for c in counts]
    for planner in (recurrent.rule_planner, recurrent.chunk_planner, recurrent.segment_planner):
        plan, seen = next(iter(planner(torch.bfloat16).values())), []
        for rows in (arrays, objects):
            packer, host = Packer(), {}
            plan(rows, packer, host)
            seen.append((dict(packer), host))
        assert seen[0] == seen[1] and bool(seen[0][0]) == (max(counts) >= (512 if planner is recurrent.segment_planner else 128))
        assert all(type(value) is int for values in seen[0][0].values() for value in values)


def token_by_token(rule, k, q, v, a, beta, S, bonus):
    out = torch.empty_like(v)
    for t in range(k.shape[0]):
        kv = k[t][:, :, None] * v[t][:, None, :]
        if rule == recurrent.RULE_WKV:
            out[t] = torch.einsum("hde,hd->he", S + bonus[:, :, None] * kv, q[t])
            S = a[t][:, :, None] * S + kv
            continue
        S = S * a[t][:, :, None]
        if beta is not None:
            kv = k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t])))[:, None, :]
        S = S + kv
        out[t] = torch.einsum("hde,hd->he", S, q[t])
    return out, S


# heads, groups, key size, value size: one tile and several, a padded key, a key of one tile row less than the kernel's, strides that allow no 16-byte loads (an odd key size)
SHAPES = [(2, 1, 128, 128), (3, 3, 64, 16), (2, 2, 100, 48), (2, 1, 21, 32)]
COUNTS = [128 + 65, 1, 16, 15, 64, 130, 17]


@pytest.mark.gpu
@pytest.mark.parametrize("steep", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("rule", [recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA, recurrent.RULE_RETENTION, recurrent.RULE_WKV])
def test_rules_in_chunks(rule, shape, steep, monkeypatch):
    """Rows of 1 to 193 tokens (those below the limit are left alone) from states that are not zero, columns of wider matrices, decays from nearly 1 down to 1e-9 a token
    (``steep``: the pairs of a sub-block one by one), scratch for three chunks at a time.

    Both this and the token-by-token scan are sums of float terms: a result's error is some 1e-7 of the norm of what it adds up, several times that where decays are near 1 and a
    state has passed 200 tokens; 3e-6 is six times the largest seen here (5e-7)."""
    heads, groups, n, e = shape
    if rule in (recurrent.RULE_RETENTION, recurrent.RULE_WKV):
        groups = heads
    monkeypatch.setattr(recurrent, "SCRATCH_BYTES", 3 * 4 * heads * (3 * 64 * 136 + 64 * 68 + 64 * e + 256))
    g = torch.Generator().manual_seed(rule * 10 + n)
    tokens, width, n_padded = sum(COUNTS), groups * n, -(-n // 4) * 4
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    x = rnd(tokens, 2 * width + heads * e + 3)
    entries = heads * n if rule in (recurrent.RULE_CHANNEL_DELTA, recurrent.RULE_WKV) else heads
    pre, step = rnd(tokens, entries + 2), rnd(tokens, heads + 1)
    if rule == recurrent.RULE_RETENTION:
        rate, bias = torch.linspace(0.999, 1e-3 if steep else 0.9, heads), None
        a = rate.double()[None, :, None].expand(tokens, heads, n)
    elif rule == recurrent.RULE_WKV:
        rate, bias = torch.rand(entries, generator=g) * (9 if steep else 5) - 6, rnd(entries) * 0.5
        a = torch.exp(-torch.exp(pre[:, :entries].double() + rate.double())).view(tokens, heads, n)
    else:
        rate, bias = torch.linspace(0, 2.7, heads), torch.rand(entries, generator=g) * (4 if steep else 5) - (1 if steep else 7)
        a = torch.exp(-torch.exp(rate.double())[:, None] * torch.nn.functional.softplus(pre[:, :entries].double() + bias.double()).view(tokens, heads, -1)).expand(tokens, heads, n)
    delta = rule in (recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA)
    q_scale = n ** -0.5 if delta else 1.0
    q, k, v = (t.double().view(tokens, h, w) for t, h, w in ((x[:, :width], groups, n), (x[:, width : 2 * width], groups, n), (x[:, 2 * width : 2 * width + heads * e], heads, e)))
    if delta:
        q = q / torch.sqrt(q.pow(2).sum(-1, keepdim=True) + 1e-6) * q_scale
        k = k / torch.sqrt(k.pow(2).sum(-1, keepdim=True) + 1e-6)
    q, k = (t.repeat_interleave(heads // groups, 1) for t in (q, k))
    beta = torch.sigmoid(step[:, :heads].double()) if delta else None
    record = heads * e * n_padded
    begin = rnd(len(COUNTS) + 2, record + 5)
    begin[:, :record].view(-1, heads, e, n_padded)[..., n:] = 0
    slots = torch.tensor([5, 0, 8, 3, 1, 7, 2], dtype=torch.int32)

    table, walks, others = recurrent.plan_rule_chunks(COUNTS)
    assert others
    dev = lambda t: None if t is None else t.cuda()  # noqa: E731
    state, xd = begin.cuda(), x.cuda()
    got = recurrent.chunked_rule(rule, xd[:, width:], xd, xd[:, 2 * width :], dev(pre) if rule != recurrent.RULE_RETENTION else None, 0, dev(step) if delta else None, 0, dev(rate), dev(bias), state, 0,
                                 slots.cuda(), torch.tensor(table, dtype=torch.int32).cuda(), len(table) // 2, torch.tensor(walks, dtype=torch.int32).cuda(), len(walks) // 3, heads, groups, n,
                                 n_padded, e, q_scale).cpu().view(tokens, heads, e)
    at = 0
    for row, count in enumerate(COUNTS):
        here, slot = slice(at, at + count), int(slots[row])
        at += count
        if count < recurrent.CHUNKED_RULE_ROWS:
            assert torch.equal(state[slot].cpu(), begin[slot])
            continue
        S = begin[slot, :record].double().view(heads, e, n_padded)[..., :n].transpose(1, 2)
        want, S = token_by_token(rule, k[here], q[here], v[here], a[here], None if beta is None else beta[here], S, bias.double().view(heads, n) if rule == recurrent.RULE_WKV else None)
        kept = state[slot, :record].cpu().double().view(heads, e, n_padded)
        for name, one, other in (("outputs", got[here].double(), want), ("state", kept[..., :n].transpose(1, 2), S)):
            assert torch.isfinite(one).all() and (one - other).norm() <= 3e-6 * other.norm(), (name, row, float((one - other).norm() / other.norm()))
        assert not kept[..., n:].any() and torch.equal(state[slot, record:].cpu(), begin[slot, record:])


def inputs_for_scan(rule, heads, n, e, tokens, decays, g):
    """Random inputs on the GPU with ``decays`` mostly near 1 (0), around a half (1) or next to nothing (2); the 64-bit vectors of the recurrence beside them."""
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    uniform = lambda size, lo, hi: torch.rand(size, device="cuda", generator=g) * (hi - lo) + lo  # noqa: E731
    x, pre, step = rnd(tokens, heads * (2 * n + e)), rnd(tokens, heads * n if rule in (recurrent.RULE_CHANNEL_DELTA, recurrent.RULE_WKV) else 2 * heads), rnd(tokens, heads)
    delta = rule in (recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA)
    entries, bias, beta = pre.shape[1] if rule != recurrent.RULE_DELTA else heads, None, None
    if rule == recurrent.RULE_RETENTION:
        rate = 1 - torch.linspace(*((5, 10), (2, 5), (0.5, 2))[decays], heads, device="cuda").neg().exp2()
        a = rate.double()[None, :, None].expand(tokens, heads, n)
    elif rule == recurrent.RULE_WKV:
        rate, bias = uniform(entries, *((-6, -1), (-2, 0), (-1, 2))[decays]), rnd(entries) * 0.5
        a = torch.exp(-torch.exp(pre.double() + rate.double())).view(tokens, heads, n)
    else:
        rate, bias, beta = uniform(heads, 0, 2.77), uniform(entries, *((-7, -2.3), (-4, -1), (-1, 3))[decays]), torch.sigmoid(step.double())
        a = torch.exp(-torch.exp(rate.double())[:, None] * torch.nn.functional.softplus(pre[:, :entries].double() + bias.double()).view(tokens, heads, -1)).expand(tokens, heads, n)
        if rule == recurrent.RULE_DELTA:
            pre[:, heads:] = step
    q, k, v = (t.double().reshape(tokens, heads, -1) for t in x.split([heads * n, heads * n, heads * e], 1))
    if delta:
        q, k = (t / torch.sqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q = q * n ** -0.5
    return (x, pre, step, rate, bias), (k, q, v, a, beta, None if rule != recurrent.RULE_WKV else bias.double().view(heads, n))


def both_ways(rule, heads, n, e, tokens, given, begin):
    """(outputs, state) in chunks and token by token."""
    x, pre, step, rate, bias = given
    delta, slots, row_start = rule in (recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA), torch.zeros(1, dtype=torch.int32, device="cuda"), torch.tensor([0, tokens], dtype=torch.int32, device="cuda")
    q, k, v, q_scale = x, x[:, heads * n :], x[:, 2 * heads * n :], n ** -0.5 if delta else 1.0
    table, walks, _ = recurrent.plan_rule_chunks([tokens])
    table, walks = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in (table, walks))
    many, one = begin.clone(), begin.clone()
    got = recurrent.chunked_rule(rule, k, q, v, None if rule == recurrent.RULE_RETENTION else pre, 0, step if delta else None, 0, rate, bias, many, 0, slots, table, table.numel() // 2, walks, 1,
                                 heads, heads, n, n, e, q_scale)
    sizes, at = (heads, heads, n, n, e), (heads * n, 0, 2 * heads * n)
    if rule == recurrent.RULE_DELTA:
        scan = recurrent.state_scan(recurrent.MODE_DELTA, x, *at, pre, 0, heads, rate, bias, None, one, 0, slots, row_start, 1, *sizes, q_scale)
    elif rule == recurrent.RULE_CHANNEL_DELTA:
        scan = recurrent.channel_delta_scan(x, *at, pre, step, 0, rate, bias, one, 0, slots, row_start, 1, *sizes, q_scale)
    elif rule == recurrent.RULE_RETENTION:
        scan = recurrent.state_scan(recurrent.MODE_RETENTION, x, *at, x, 0, 0, rate, rate, None, one, 0, slots, row_start, 1, *sizes)
    else:
        scan = recurrent.wkv_scan(k, q, v, pre, 0, rate, bias, one, 0, slots, row_start, 1, heads, n, n, e)
    return (got, many), (scan, one)


@pytest.mark.gpu
@pytest.mark.parametrize("decays", [0, 1, 2])
@pytest.mark.parametrize("rule", [recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA, recurrent.RULE_RETENTION, recurrent.RULE_WKV])
def test_chunks_are_as_close_to_64_bits_as_the_scan(rule, decays):
    """Both are sums of float terms whose roundings differ; over four draws and three sizes the chunks' distance from 64 bits is not above the scan's.  Single draws differ by 3 % (outputs)
    and 15 % (states, of which under strong decays only the last tokens' rounding is left), so a mean of twelve by 1 % and 5 %: twice that is allowed."""
    ratios = []
    for heads, n, e, tokens in ((8, 128, 128, 128), (8, 64, 64, 333), (4, 96, 48, 700)):
        for seed in range(4):
            g = torch.Generator("cuda").manual_seed(100 * seed + tokens)
            given, exact = inputs_for_scan(rule, heads, n, e, tokens, decays, g)
            begin = torch.randn(1, heads * e * n, device="cuda", generator=g)
            want, S = token_by_token(rule, *exact[:5], begin.double().view(heads, e, n).transpose(1, 2), exact[5])
            far = [((out.double().view_as(want) - want).norm(), (state.double().view(heads, e, n) - S.transpose(1, 2)).norm()) for out, state in both_ways(rule, heads, n, e, tokens, given, begin)]
            ratios.append([float(chunks / scan) for chunks, scan in zip(*far)])
    outputs, states = torch.tensor(ratios).log().mean(0).exp().tolist()
    assert outputs <= 1.02 and states <= 1.1, (outputs, states)


@pytest.mark.gpu
@pytest.mark.parametrize("n, e", [(128, 128), (64, 32), (100, 96)])
@pytest.mark.parametrize("rule", [recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA, recurrent.RULE_RETENTION, recurrent.RULE_WKV])
def test_narrow_and_wide_tiles_of_value_columns_give_the_same_bits(rule, n, e, monkeypatch):
    """Sixteen value columns to a block while such blocks fit the multiprocessors side by side, else thirty-two: a device of one and one of a million multiprocessors."""
    heads, tokens = 3, 150
    g = torch.Generator("cuda").manual_seed(n)
    given, _ = inputs_for_scan(rule, heads, n, e, tokens, 1, g)
    begin = torch.randn(1, heads * e * n, device="cuda", generator=g)
    results = []
    for sms in (1, 10**6):
        monkeypatch.setattr(recurrent, "sm_count", lambda device, sms=sms: sms)
        (out, state), (scan, kept) = both_ways(rule, heads, n, e, tokens, given, begin)
        assert (out - scan).norm() <= 2e-6 * scan.norm() and (state - kept).norm() <= 2e-6 * kept.norm()  # two float computations, 3e-6 from 64 bits at the most together
        results.append((out, state))
    assert all(torch.equal(one, other) for one, other in zip(*results))


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("rule", [recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA, recurrent.RULE_RETENTION, recurrent.RULE_WKV])
def test_earlier_tokens_do_not_see_what_is_not_finite(rule, value):
    """One value, query, key, decay or step of a token in the middle of a block of sixteen in the middle of a chunk: outputs before it are those of the clean inputs, and from it on the same
    ones are finite as in the token-by-token scan, the state's entries too."""
    heads, n, e, tokens, t = 2, 64, 32, 200, 64 + 37
    g = torch.Generator("cuda").manual_seed(rule)
    given, _ = inputs_for_scan(rule, heads, n, e, tokens, 1, g)
    begin = torch.randn(1, heads * e * n, device="cuda", generator=g)
    (clean, _), _ = both_ways(rule, heads, n, e, tokens, given, begin)
    places = [(0, 5), (0, heads * n + 7), (0, 2 * heads * n + e + 3)]  # a query's entry, a key's, a value's
    if rule != recurrent.RULE_RETENTION:
        places.append((1, 1))
    if rule in (recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA):
        places.append((1, heads + 1) if rule == recurrent.RULE_DELTA else (2, 1))
    for which, column in places:
        spoilt = [x.clone() if isinstance(x, torch.Tensor) else x for x in given]
        spoilt[which][t, column] = value
        if rule == recurrent.RULE_DELTA:
            spoilt[2] = spoilt[1][:, heads:].contiguous()
        (got, state), (scan, kept) = both_ways(rule, heads, n, e, tokens, spoilt, begin)
        assert torch.isfinite(got[:t]).all() and (got[:t] - clean[:t]).norm() <= 1e-6 * clean[:t].norm(), (which, column)
        assert torch.equal(torch.isfinite(got), torch.isfinite(scan)) and torch.equal(torch.isfinite(state), torch.isfinite(kept)), (which, column)


@pytest.mark.gpu
@pytest.mark.parametrize("steep", [False, True])
@pytest.mark.parametrize("rule", [recurrent.RULE_DELTA, recurrent.RULE_CHANNEL_DELTA])
def test_delta_rules_give_the_same_bits_again(rule, steep):
    """A chunk's triangular system is put together by all warps and solved by others: 976 chunks of many heads, last chunks of 17, 33 and 64 tokens (fewer pairs to make before the
    solution starts), sub-blocks with and without steep decays, twelve times over; every time the same bits in outputs and states."""
    heads, n, e, counts = 16, 128, 64, [2048 + 17, 1024 + 33, 640]
    tokens, g = sum(counts), torch.Generator("cuda").manual_seed(rule)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    entries = heads * n if rule == recurrent.RULE_CHANNEL_DELTA else heads
    x, pre, step, rate = rnd(tokens, heads * (2 * n + e)), rnd(tokens, entries), rnd(tokens, heads), torch.linspace(0, 2.7, heads, device="cuda")
    bias, begin, slots = rnd(entries) * 0.5 + (2 if steep else -3), rnd(len(counts), heads * e * n), torch.arange(len(counts), dtype=torch.int32, device="cuda")
    table, walks, _ = recurrent.plan_rule_chunks(counts)
    table, walks = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in (table, walks))
    first = None
    for _ in range(12):
        state = begin.clone()
        out = recurrent.chunked_rule(rule, x[:, heads * n :], x, x[:, 2 * heads * n :], pre, 0, step, 0, rate, bias, state, 0, slots, table, table.numel() // 2, walks, len(counts), heads, heads, n, n,
                                     e, n ** -0.5)
        first = first or (out, state)
        assert torch.equal(out, first[0]) and torch.equal(state, first[1]) and torch.isfinite(out).all()


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[1, 130, 15, 16, 1, 65], [200], [3, 128, 1]])
def test_short_rows_beside_chunked_ones(counts):
    """The state-space recurrence in bfloat16-valued chunks with its rows of fewer than 16 tokens left to the token-by-token scan: the same as all rows in the scan, and the chunks touch
    neither the short rows' outputs nor their states."""
    heads, n, e = 3, 24, 40
    tokens, g = sum(counts), torch.Generator().manual_seed(len(counts))
    x = torch.randn(tokens, 2 * n + heads * e, generator=g).to(torch.bfloat16).float().cuda()
    gate = torch.randn(tokens, heads, generator=g).cuda()
    a_log, dt_bias, skip = torch.linspace(-2, 1, heads).cuda(), torch.linspace(-4, 1, heads).cuda(), torch.randn(heads, generator=g).cuda()
    starts = [sum(counts[:i]) for i in range(len(counts) + 1)]
    row_start, slots = (torch.tensor(v, dtype=torch.int32).cuda() for v in (starts, list(range(len(counts)))[::-1]))
    one, many = (torch.randn(len(counts), heads * e * n, generator=torch.Generator().manual_seed(7)).cuda() for _ in range(2))
    begin = many.clone()
    cut = recurrent.plan_chunks(counts)
    chunk_start, chunk_row = (torch.tensor(v, dtype=torch.int32).cuda() for v in cut)
    want = recurrent.state_scan(recurrent.MODE_STATE_SPACE, x, 0, n, 2 * n, gate, 0, 0, a_log, dt_bias, skip, one, 0, slots, row_start, len(counts), heads, 1, n, n, e)
    below = recurrent.CHUNKED_RULE_ROWS
    got = recurrent.chunked_scan(recurrent.KIND_STATE_SPACE, x, x[:, n:], x[:, 2 * n :], gate, 0, 0, many, 0, slots, chunk_start, chunk_row, len(cut[1]), heads, 1, n, n, e, a_log=a_log,
                                 dt_bias=dt_bias, skip=skip, below=below).view(tokens, heads * e)
    for row, count in enumerate(counts):
        assert torch.equal(many[slots[row].long()], begin[slots[row].long()]) == (count < below)
    got = recurrent.state_scan(recurrent.MODE_STATE_SPACE, x, 0, n, 2 * n, gate, 0, 0, a_log, dt_bias, skip, many, 0, slots, row_start, len(counts), heads, 1, n, n, e, below=below, out=got)
    for row, count in enumerate(counts):
        here, slot = slice(starts[row], starts[row + 1]), slots[row].long()
        if count < below:
            assert torch.equal(got[here], want[here]) and torch.equal(many[slot], one[slot])
        else:  # two float computations of the same sums, states and scores as bfloat16 pairs: 2e-5 of the norm
            assert (got[here] - want[here]).norm() <= 2e-5 * want[here].norm() and (many[slot] - one[slot]).norm() <= 2e-5 * one[slot].norm()
