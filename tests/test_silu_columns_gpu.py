"""silu over columns, four at a time and one by one: the same bits, within float of 64 bits."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200.ops import recurrent

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns,tokens", [(256, 512), (256, 511), (512, 300), (260, 600), (258, 600), (4096, 32)])
def test_silu_columns(columns, tokens):
    x = torch.randn(tokens, columns + 12, device="cuda", generator=torch.Generator("cuda").manual_seed(columns))
    many, few = x.clone(), x[:3].clone()
    recurrent.silu_columns_(many, 8, columns)
    recurrent.silu_columns_(few, 8, columns)
    assert torch.equal(many[:3], few) and torch.equal(many[:, :8], x[:, :8]) and torch.equal(many[:, 8 + columns :], x[:, 8 + columns :])
    want = torch.nn.functional.silu(x[:, 8 : 8 + columns].double())
    assert ((many[:, 8 : 8 + columns].double() - want).abs() <= 2.0 ** -20 * want.abs() + 1e-30).all()
