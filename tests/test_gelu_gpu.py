"""GELU over tensors that take sixteen bytes per access and over those that do not, against 64 bits."""
import pytest
import torch

from hyperion_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("count,offset", [(8, 0), (7, 0), (9, 0), (4096, 0), (4096, 1), (4095, 0), (8 * 256 * 16384 + 8, 0), (8, 8)])
def test_gelu(count, offset, dtype):
    g = torch.Generator("cuda").manual_seed(count + offset)
    x = (torch.randn(count + offset, device="cuda", generator=g) * 3).to(dtype)[offset:]
    x[:3] = torch.tensor([0.0, -100.0, 100.0], dtype=dtype)
    z = x.double()
    # one rounding of the result; in float, 1 + erf loses up to a few units of 2^-24 against 1, which z multiplies
    room = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-21
    for got, want in ((ops.gelu_erf(x), torch.nn.functional.gelu(z)), (ops.gelu_tanh(x), torch.nn.functional.gelu(z, approximate="tanh"))):
        assert ((got.double() - want).abs() <= room * want.abs() + z.abs() * 2.0**-21).all()
