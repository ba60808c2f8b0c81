"""The float32 product at sizes that have more than three small tiles to an SM on a device of one: both tilings run, and give the same bits."""
import pytest
import torch

from hyperion_b200 import ops
from hyperion_b200.ops import basic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 130, 63), (40, 65, 64)])
@pytest.mark.parametrize("aligned", [True, False])
def test_both_tilings(m, n, k, aligned, monkeypatch):
    """A sum of k products in float, one after another: k rounding errors of at most 2^-24 of the largest partial sum."""
    assert -(-m // 32) * -(-n // 32) > 3
    g = torch.Generator().manual_seed(m + n + k)
    pad = 4 - k % 4 if aligned else 1
    x, w = torch.randn(m, k + pad, generator=g).cuda()[:, :k], torch.randn(n, k, generator=g).cuda()
    results = []
    for sms in (148, 1):
        monkeypatch.setattr(basic, "sm_count", lambda device, sms=sms: sms)
        results.append(ops.sgemm_f32(x, w))
    assert torch.equal(*results)
    assert ((results[0].double() - x.double() @ w.double().t()).abs() <= (k + 1) * 2.0 ** -24 * (x.abs().double() @ w.abs().double().t())).all()
