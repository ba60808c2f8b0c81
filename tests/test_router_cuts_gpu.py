"""The three routers at every cut of their work: the same bits as a token a block, up to steps of thousands of tokens and a block that ends past the last one."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200.ops import moe

pytestmark = pytest.mark.gpu

ROUTERS = {
    "chosen": lambda x, router, extra, top: moe.route(x, router, top),
    "scored": lambda x, router, extra, top: moe.route_scored(x, router, extra, top, 0, 0, 1.5),
    "softmax": lambda x, router, extra, top: moe.route_softmax(x, router, extra, top),
}


@pytest.mark.parametrize("router", sorted(ROUTERS))
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
# on 148 multiprocessors and on fewer: steps that go token by token, by two experts a warp, by four tokens in small and large blocks, by eight; columns that are no multiple of four
@pytest.mark.parametrize("tokens,outputs,hidden,sms", [(150, 18, 260, 148), (301, 64, 256, 148), (597, 12, 256, 148), (1029, 18, 2048, 148), (1187, 18, 512, 148), (2053, 33, 1024, 148),
                                                       (1029, 256, 128, 148), (2049, 8, 512, 148), (300, 4, 7168, 148), (67, 20, 1024, 4), (67, 70, 7168, 4), (33, 5, 99, 2), (35, 24, 99, 2)])
def test_same_bits_as_a_few_tokens_at_a_time(router, dtype, tokens, outputs, hidden, sms, monkeypatch):
    monkeypatch.setattr(moe, "sm_count", lambda device: sms)
    g = torch.Generator("cuda").manual_seed(tokens + outputs)
    x, matrix = torch.randn(tokens, hidden, device="cuda", generator=g).to(dtype), torch.randn(outputs, hidden, device="cuda", generator=g) * hidden ** -0.5
    extra, call = torch.randn(outputs, device="cuda", generator=g) * 0.1, ROUTERS[router]
    top = min(3, outputs)
    chosen, weights = call(x, matrix, extra, top)
    monkeypatch.setattr(moe, "sm_count", lambda device: 1 << 20)  # a token a block
    for first in (0, tokens // 2, tokens - 7):
        some = call(x[first : first + 7], matrix, extra, top)
        assert torch.equal(chosen[first : first + 7], some[0]) and torch.equal(weights[first : first + 7], some[1])
    alone = call(x, matrix, extra, top)
    assert torch.equal(chosen, alone[0]) and torch.equal(weights, alone[1])
    if router == "chosen":  # the choices stand by their logits: `hidden` products added in float
        logits = x.double() @ matrix.double().t()
        room = hidden * 2.0 ** -23 * (x.double().abs() @ matrix.double().abs().t())
        taken = logits.gather(1, chosen.long())
        assert (taken.amin(1) + 2 * room.amax(1) >= logits.topk(top).values[:, -1]).all()
        assert ((weights.double() - taken.sigmoid()).abs() <= room.amax(1, keepdim=True) + 2.0 ** -20).all()
