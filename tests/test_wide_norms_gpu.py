"""The norm on a sublayer's output at a prompt's rows: the same bits as the same rows a few at a time, and within float of 64 bits; split-K pieces up to the most there are."""
import pytest
import torch

from hyperion_b200 import ops
from hyperion_b200.ops import gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [3072, 4104, 8192, 2048])
def test_many_rows(hidden):
    g = torch.Generator("cuda").manual_seed(hidden)
    h, y, w = (torch.randn(*s, device="cuda", generator=g) for s in ((513, hidden), (513, hidden), (hidden,)))
    y = y.to(torch.bfloat16)
    many, few = h.clone(), h[250:260].clone()
    copies = ops.rmsnorm_add(many, y, w, 1e-6, copy_dtype=torch.bfloat16), ops.rmsnorm_add(few, y[250:260].contiguous(), w, 1e-6, copy_dtype=torch.bfloat16)
    assert torch.equal(many[250:260], few) and torch.equal(copies[0][250:260], copies[1])
    d = y.double()
    step = d * (d.square().mean(1, keepdim=True) + 1e-6).rsqrt() * w.double()
    # a sum of `hidden` squares in float, a root, three products and a sum
    assert ((many.double() - h.double() - step).abs() <= (hidden + 8) * 2.0 ** -24 * step.abs() + 2.0 ** -23 * (h.double().abs() + step.abs())).all()


@pytest.mark.parametrize("splits", [1, 7, 8, 11, 12, 16])
@pytest.mark.parametrize("hidden", [896, 5120, 9216])
def test_pieces(splits, hidden):
    """One, two and three groups of eight a thread; pieces up to what a thread asks for at once, and past that."""
    g = torch.Generator("cuda").manual_seed(splits)
    h, pieces, w = (torch.randn(*s, device="cuda", generator=g) for s in ((9, hidden), (splits, 9, hidden), (hidden,)))
    delta = torch.zeros(9, hidden, device="cuda")
    for piece in pieces:  # in their order
        delta = delta + piece
    one, two = h.clone(), h.clone()
    got = ops.add_rmsnorm(one, gemm.SplitSum(pieces, None, torch.bfloat16), w, 1e-6, torch.bfloat16)
    assert torch.equal(got, ops.add_rmsnorm(two, delta.to(torch.bfloat16), w, 1e-6, torch.bfloat16)) and torch.equal(one, two)
