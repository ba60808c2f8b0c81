"""Kernels whose shared memory follows a width, launched by two threads at widths of their own: neither takes the other's allowance away."""
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from hyperion_b200 import ops
from hyperion_b200.ops import moe, recurrent

pytestmark = pytest.mark.gpu


def routes(call, tokens):
    def prepared(hidden, g, dtype):
        x, router = torch.randn(tokens, hidden, device="cuda", generator=g).to(dtype), torch.randn(16, hidden, device="cuda", generator=g)
        return lambda: call(x, router)
    return prepared


def two_norms(hidden, g, dtype):
    h, y, w = (torch.randn(*shape, device="cuda", generator=g) for shape in ((3, hidden), (3, hidden), (hidden,)))
    y = y.to(dtype)

    def call():
        stream = h.clone()
        return stream, ops.norm_add_norm(stream, y, w, 1e-6, None, w, 1e-6, dtype)
    return call


def chunks(n, g, dtype):
    heads, e, tokens = 2, 64, 150
    x, gate = torch.randn(tokens, heads * (2 * n + e), device="cuda", generator=g), -torch.rand(tokens, 2 * heads, device="cuda", generator=g)
    begin, slots = torch.randn(1, heads * e * n, device="cuda", generator=g), torch.zeros(1, dtype=torch.int32, device="cuda")
    starts, rows = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in recurrent.plan_chunks([tokens]))

    def call():
        state = begin.clone()
        return state, recurrent.chunked_scan(recurrent.KIND_GIVEN, x, x[:, heads * n :], x[:, 2 * heads * n :], gate, 0, heads, state, 0, slots, starts, rows, len(rows), heads, heads, n, n, e)
    return call


# widths of which both take more than a block's ordinary 48 KB; four tokens to a block from 512 on
CALLS = {
    "route": (routes(lambda x, r: moe.route(x, r, 2), 3), (13000, 20000)),
    "route_scored": (routes(lambda x, r: moe.route_scored(x, r, None, 2, 1, 1, 1.0), 3), (13000, 20000)),
    "route_softmax": (routes(lambda x, r: moe.route_softmax(x, r, None, 2), 3), (13000, 20000)),
    "route_softmax_by_four": (routes(lambda x, r: moe.route_softmax(x, r, None, 2), 512), (3584, 5120)),
    "norm_add_norm": (two_norms, (13000, 20000)),
    "chunked_scan": (chunks, (128, 256)),
}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", CALLS)
def test_threads_at_widths_of_their_own(name, dtype):
    prepared, widths = CALLS[name]

    def repeated(hidden):
        g = torch.Generator("cuda").manual_seed(hidden)
        call = prepared(hidden, g, dtype)
        want = call()
        torch.cuda.synchronize()
        return all(torch.equal(one, other) for _ in range(150) for one, other in zip(call(), want))

    with ThreadPoolExecutor(2) as pool:
        assert all(pool.map(repeated, widths))
