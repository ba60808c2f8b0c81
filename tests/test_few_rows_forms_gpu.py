"""Small products whose operands are not what the kernel for a few rows reads: they take the library's way, with its results and its refusals."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200 import ops

pytestmark = pytest.mark.gpu


def _operands(m, n, k):
    g = torch.Generator("cuda").manual_seed(m + n + k)
    return torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16), (torch.randn(n, k, device="cuda", generator=g) * k ** -0.5).to(torch.bfloat16)


@pytest.mark.parametrize("k", [64, 2048])  # the library's own, and what the split product would take
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", [lambda b: b[0, :1], lambda b: b, lambda b: b[:1], lambda b: b[:, :1], lambda b: b[0, 0], lambda b: b.t()[:, 0]])
def test_biases_that_broadcast(k, out, form):
    x, w = _operands(3, 32, k)
    bias = form(torch.arange(96, device="cuda").view(3, 32).to(torch.bfloat16))  # whole numbers: no rounding of theirs
    exact = x.double() @ w.double().T + bias.double()
    got = ops.linear(x, w, bias, out).double()
    # a product rounded to bfloat16 before the bias at the most, and the sum rounded once: 2^-8 of each
    assert ((got - exact).abs() <= 2.0 ** -8 * (exact.abs() + (exact - bias.double()).abs()) + k * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)).all()


@pytest.mark.parametrize("k", [64, 2048])
def test_a_bias_of_another_length_is_refused(k):
    x, w = _operands(3, 32, k)
    with pytest.raises(RuntimeError):
        ops.linear(x, w, torch.zeros(31, device="cuda", dtype=torch.bfloat16))


def test_operands_without_rows_columns_or_a_dimension():
    x, w = _operands(3, 32, 64)
    assert torch.equal(ops.linear(x[:0], w), torch.empty(0, 32, device="cuda", dtype=torch.bfloat16))
    assert ops.linear(x, w[:0], may_leave_partials=True).shape == (3, 0)
    assert torch.equal(ops.linear(x, w[0]), torch.nn.functional.linear(x, w[0]))
    assert torch.equal(ops.linear(x[None], w), torch.nn.functional.linear(x[None], w))


def test_gradients_are_kept():
    x, w = _operands(3, 32, 64)
    x.requires_grad_()
    ops.linear(x, w).float().sum().backward()
    assert torch.allclose(x.grad.float(), w.float().sum(0).expand(3, -1), rtol=2.0 ** -7, atol=2.0 ** -7)
    with torch.no_grad():
        assert not ops.linear(x, w).requires_grad
