"""Gates of values that go back to bfloat16, over the whole range of the type: the reciprocal in them has no special cases of its own."""
import pytest
import torch

from test_gpu_vifelix import _batch, _ops, _run

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _every_value():
    return torch.arange(-32768, 32768, dtype=torch.int32, device=DEV).to(torch.int16).view(torch.bfloat16).view(256, 256)


@pytest.mark.parametrize("kind", ["swiglu", "sigmoid_mul"])
def test_gates_over_all_bfloat16_values(kind):
    z = _every_value()
    one = torch.ones_like(z)
    out = torch.empty_like(z)
    if kind == "swiglu":
        _ops().swiglu(torch.cat([z, one], 1), out)
        want = z.double() / (1 + torch.exp(-z.double()))
    else:
        _run(_ops(), lambda p: p.pointwise("sigmoid_mul", one, z, out), _batch([256], [0]))
        want = 1 / (1 + torch.exp(-z.double()))
    got, smallest = out.double(), 2.0 ** -126
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    number = ~torch.isnan(want) & ~torch.isinf(want)
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    # half a bfloat16 step; the hardware's exponential at -z: 2^-21 and 2^-23 |z| of it; where the 32-bit exponential has left the normal
    # numbers, their smallest times z
    bound = want.abs() * (2.0 ** -8 + 2.0 ** -20 + 2.0 ** -22 * z.double().abs().clamp(max=128)) + smallest * (1 + z.double().abs().clamp(max=2.0 ** 10))
    assert bool(((got - want).abs() <= bound)[number].all())
