"""Products of a few rows with a small matrix: tiles that warps and blocks share, parts of k, every epilogue, against 64 bits and whatever the other rows hold."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200 import ops
from hyperion_b200.ops import gemm

pytestmark = pytest.mark.gpu

# one unit and fewer units than warps; more tiles than blocks hold at a time; tiles a warp has to itself beside shared ones; k of several parts
SIZES = [(16, 64), (32, 128), (1152, 896), (896, 4864), (9728, 192), (160, 2048), (4800, 64), (2048, 1088)]


def _operands(m, n, k):
    g = torch.Generator("cuda").manual_seed(m * 10007 + n + k)
    x = torch.randn(m, k + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :k]  # rows that are not dense
    w = (torch.randn(n, k, device="cuda", generator=g) * k ** -0.5).to(torch.bfloat16)
    return x, w, x.double() @ w.double().T, x.double().abs() @ w.double().abs().T


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("n,k", SIZES)
def test_epilogues(m, n, k):
    """k exact products added in float, at most a unit cut off per addition: k * 2^-23 of the sum of their sizes; then one rounding to bfloat16."""
    x, w, want, size = _operands(m, n, k)
    room = k * 2.0 ** -23 * size
    assert gemm.takes_few_rows(x, w)
    bias_h, bias_f = torch.randn(n, device="cuda").to(torch.bfloat16), torch.randn(n, device="cuda")
    got = gemm.few_rows(x, w, bias_f, gemm.FEW_F32)
    assert ((got.double() - want - bias_f.double()).abs() <= room + 2.0 ** -23 * (want.abs() + bias_f.abs())).all()
    got = gemm.few_rows(x, w, bias_h)
    exact = want + bias_h.double()
    assert ((got.double() - exact).abs() <= room + 2.0 ** -8 * exact.abs() + 2.0 ** -23 * size).all()
    left = gemm.few_rows(x, w, bias_h, gemm.FEW_PIECES)
    got = left.tensor() if isinstance(left, gemm.SplitSum) else left
    assert ((got.double() - exact).abs() <= room + 2.0 ** -8 * exact.abs() + 2.0 ** -23 * size).all()


@pytest.mark.parametrize("m", [1, 8, 11])
@pytest.mark.parametrize("inter,k,block", [(16, 64, 16), (4864, 896, 128), (608, 128, 32), (608, 192, 608), (128, 1024, 8)])
def test_swiglu(m, inter, k, block):
    x, w, _, _ = _operands(m, 2 * inter, k)
    assert gemm.takes_few_rows(x, w, block)
    got = gemm.few_rows(x, w, None, gemm.FEW_SWIGLU, block).double()
    want = ops.swiglu(gemm.few_rows(x, w), block=block).double()  # the same roundings in two launches; sums may be shared out among warps another way
    assert ((got - want).abs() <= 2.0 ** -6 * want.abs() + 2.0 ** -9).all()


def test_a_row_does_not_depend_on_the_others():
    x, w, _, _ = _operands(16, 1152, 896)
    other = torch.randn_like(x)
    for m in (8, 16):
        mixed = torch.cat([other[: m - 1], x[:1]])
        assert torch.equal(gemm.few_rows(mixed, w)[m - 1], gemm.few_rows(x[:m], w)[0])


def test_which_products_are_taken():
    x = torch.zeros(16, 2048, device="cuda", dtype=torch.bfloat16)

    def takes(rows, n, k, block=None):
        return gemm.takes_few_rows(torch.empty(rows, k, device="cuda", dtype=torch.bfloat16), torch.empty(n, k, device="cuda", dtype=torch.bfloat16), block)

    assert takes(8, 4096, 2048) and not takes(9, 4096, 2048) and takes(16, 2048, 2048) and not takes(17, 2048, 2048)
    assert not takes(1, 4096, 4096) and not takes(1, 32000, 2048) and takes(8, 16384, 2048, 128) and not takes(8, 16384, 2048, 96)
    assert not takes(1, 40, 64) and not takes(1, 48, 96)
    assert x.shape[0] == gemm.FEW_ROWS
