"""The float32 product's two tile shapes and its copies of four bytes: against 64 bits, and the same bits whatever stands beside a row."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200 import ops
from hyperion_b200.ops import basic

pytestmark = pytest.mark.gpu


# rows, columns, k: edges of the 32 x 32 and of the 64 x 128 tiles, the rows from which large ones are taken, k of a few entries, of whole slices and past them
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 36), (33, 97, 64), (65, 20000, 20), (130, 19000, 48), (394, 9729, 68), (33, 37900, 16)])
@pytest.mark.parametrize("aligned", [True, False])
def test_tiles(m, n, k, aligned):
    """A sum of k products in float, one after another: k rounding errors of at most 2^-24 of the largest partial sum."""
    g = torch.Generator().manual_seed(m + n + k)
    pad = 4 if aligned else 3
    x = torch.randn(m, k + pad, generator=g).cuda()[:, :k] if k % 4 == 0 else torch.randn(m, k, generator=g).cuda()
    w, b = torch.randn(n, k, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    got = ops.sgemm_f32(x, w, b)
    want = x.double() @ w.double().t() + b.double()
    assert ((got.double() - want).abs() <= (k + 1) * 2.0 ** -24 * (x.abs().double() @ w.abs().double().t() + b.abs().double())).all()
    for rows in {1, min(m, 30), min(m, 64)}:  # few rows take the small tiles, whatever the whole took
        assert torch.equal(ops.sgemm_f32(x[:rows], w, b), got[:rows])
    assert torch.equal(ops.sgemm_f32(x, w[: min(n, 40)].contiguous(), b[: min(n, 40)].contiguous()), got[:, : min(n, 40)])


@pytest.mark.parametrize("m,n,k", [(65, 300, 36), (33, 256, 17), (200, 20000, 64)])
def test_the_tile_follows_the_device(m, n, k, monkeypatch):
    """Two large tiles to an SM decide on the tile: on a device of one SM all of these (two such tiles and more) take large ones, on one of a million none does, and the bits are the same."""
    g = torch.Generator().manual_seed(k)
    x, w = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    results = []
    for sms in (1, 10**6):
        monkeypatch.setattr(basic, "sm_count", lambda device, sms=sms: sms)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
            results.append(ops.sgemm_f32(x, w))
            torch.cuda.synchronize()
        names = [event.name for event in profile.events() if "sgemm_kernel" in event.name]
        assert names and all(("64, 128" in name) == (sms == 1) for name in names), names
    assert torch.equal(*results)


@pytest.mark.parametrize("k,large", [(1000, False), (1001, True)])
def test_rows_off_16_bytes_take_large_tiles_earlier(k, large, monkeypatch):
    """128 large tiles on 148 multiprocessors: too few for rows that are copied 16 bytes at a time, enough for rows that go four bytes at a time."""
    x, w = torch.randn(1000, k, device="cuda"), torch.randn(1003, k, device="cuda")
    monkeypatch.setattr(basic, "sm_count", lambda device: 148)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as profile:
        ops.sgemm_f32(x, w)
        torch.cuda.synchronize()
    names = [event.name for event in profile.events() if "sgemm_kernel" in event.name]
    assert names and all(("64, 128" in name) == large for name in names), names
