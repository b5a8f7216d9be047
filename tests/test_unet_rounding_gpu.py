"""The fused parts of the UNet give the bits of the operations that they stand for."""
import pytest
import torch
import torch.nn.functional as F

from maxdiffusion_b200.models.layers import Conv2d, conv_plus

pytestmark = pytest.mark.gpu


def _cl(*shape, scale=1.0):
  return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)


@pytest.mark.parametrize("shape,co,k,stride", [((2, 32, 8, 8), 40, 3, 1), ((1, 48, 17, 5), 64, 3, 1), ((2, 1280, 8, 8), 1280, 3, 1),
                                               ((1, 64, 40, 24), 320, 3, 1), ((2, 32, 6, 10), 32, 3, 2)])
@pytest.mark.parametrize("grad", [False, True])
def test_a_convolution_and_its_residual(shape, co, k, stride, grad):
  """A residual in the epilogue is added to the rounded result, over whole and cut contractions."""
  torch.manual_seed(1)
  m = Conv2d(shape[1], co, k, stride=stride, padding=k // 2).to("cuda", torch.bfloat16)
  x, res = _cl(*shape), _cl(shape[0], co, shape[2] // stride, shape[3] // stride, scale=30.0)
  with torch.set_grad_enabled(grad):
    assert torch.equal(conv_plus(m, x, res), res + m(x))
    assert torch.equal(conv_plus(m, x, res.contiguous()), res.contiguous() + m(x))
