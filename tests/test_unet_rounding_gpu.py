"""The fused parts of the UNet give the bits of the operations that they stand for."""
import pytest
import torch
import torch.nn.functional as F

from maxdiffusion_b200.models.layers import Conv2d, conv_plus
from maxdiffusion_b200.models.vae import ResnetBlock2D

pytestmark = pytest.mark.gpu


def _cl(*shape, scale=1.0):
  return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)


@pytest.mark.parametrize("shape,co,k,stride", [((2, 32, 8, 8), 40, 3, 1), ((1, 48, 17, 5), 64, 3, 1), ((2, 1280, 8, 8), 1280, 3, 1),
                                               ((1, 64, 40, 24), 320, 3, 1), ((2, 32, 6, 10), 32, 3, 2), ((2, 64, 9, 8), 40, 1, 1)])
@pytest.mark.parametrize("grad", [False, True])
def test_a_convolution_and_its_residual(shape, co, k, stride, grad):
  """A residual in the epilogue is added to the rounded result, over whole and cut contractions."""
  torch.manual_seed(1)
  m = Conv2d(shape[1], co, k, stride=stride, padding=k // 2).to("cuda", torch.bfloat16)
  x, res = _cl(*shape), _cl(shape[0], co, shape[2] // stride, shape[3] // stride, scale=30.0)
  with torch.set_grad_enabled(grad):
    assert torch.equal(conv_plus(m, x, res), res + m(x))
    assert torch.equal(conv_plus(m, x, res.contiguous()), res.contiguous() + m(x))


@pytest.mark.parametrize("linear_proj", [True, False])
@pytest.mark.parametrize("grad", [False, True])
def test_a_transformer_and_its_residual(linear_proj, grad):
  """The output projection's result is rounded before the input is added, as a hook that does nothing leaves it."""
  from maxdiffusion_b200.models.unet_2d_condition import Transformer2DModel

  torch.manual_seed(2)
  m = Transformer2DModel(128, 2, 1, 64, 32, linear_proj).to("cuda", torch.bfloat16)
  x, context = _cl(2, 128, 8, 12, scale=30.0), torch.randn(2, 7, 64, device="cuda").to(torch.bfloat16)
  with torch.set_grad_enabled(grad):
    out = m(x, context)
    seen = []
    m.proj_out.register_forward_hook(lambda mod, args, y: seen.append(y))
    assert torch.equal(m(x, context), out)
  y = seen[0].unflatten(1, (8, 12)).permute(0, 3, 1, 2) if linear_proj else seen[0]
  assert torch.equal(out, y + x)


@pytest.mark.parametrize("cin,cout,size,rows", [(64, 64, (16, 16), 2), (96, 64, (17, 5), 2), (320, 640, (40, 40), 1)])
@pytest.mark.parametrize("grad", [False, True])
def test_a_resnet_block_and_its_time_embedding(cin, cout, size, rows, grad):
  """The embedding is added in bf16 in front of the norm, its projection is the module's own product."""
  torch.manual_seed(3)
  m = ResnetBlock2D(cin, cout, temb_channels=128, eps=1e-5).to("cuda", torch.bfloat16)
  x, temb = _cl(2, cin, *size), torch.randn(rows, 128, device="cuda").to(torch.bfloat16)
  with torch.set_grad_enabled(grad):
    h = m.conv1(m.norm1(x, act=True))
    h = h + F.linear(F.silu(temb), m.time_emb_proj.weight, m.time_emb_proj.bias)[:, :, None, None]
    h = m.conv2(m.norm2(h, act=True))
    assert torch.equal(m(x, temb), (x if m.conv_shortcut is None else m.conv_shortcut(x)) + h)
