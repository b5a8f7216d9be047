"""GroupNorm in one launch gives the bits of the kernels that it stands for."""
import pytest
import torch

from maxdiffusion_b200.ops import conv as C
from maxdiffusion_b200.ops import functional as OF
from maxdiffusion_b200.ops import kernels as K

pytestmark = pytest.mark.gpu

# (N, channels, H, W), groups: vectors of one pixel and of eight, strips of one and of several, few and many channels a group
_THREE = [((2, 64, 8, 8), 32), ((1, 320, 17, 5), 32), ((3, 96, 1, 9), 3), ((2, 320, 32, 32), 32), ((1, 1280, 3, 5), 32), ((2, 1280, 8, 8), 32),
          ((1, 1920, 16, 16), 32), ((2, 16, 2, 1), 8), ((2, 2048, 2, 2), 1), ((1, 320, 5, 5), 1), ((4, 64, 61, 67), 32), ((60, 32, 3, 7), 4)]
_FIRST = [((2, 2560, 8, 8), 32), ((1, 2560, 16, 16), 32), ((2, 2560, 32, 32), 32), ((1, 2560, 31, 33), 32), ((1, 2560, 1, 3), 32),
          ((1, 2560, 5, 3), 32), ((2, 2064, 48, 40), 129), ((1, 3840, 9, 8), 32)]


def _params(channels, dtype):
  return (torch.randn(channels, device="cuda").to(dtype), torch.randn(channels, device="cuda").to(dtype)) if dtype is not None else (None, None)


@pytest.mark.parametrize("act,dtype", [(True, torch.bfloat16), (False, torch.float32), (True, None)])
@pytest.mark.parametrize("shape,groups", _THREE)
def test_bits_of_the_three_launches(shape, groups, act, dtype):
  torch.manual_seed(1)
  N, channels, H, W = shape
  x = (torch.randn(*shape, device="cuda") * 2 + 30).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
  x3 = x.permute(0, 2, 3, 1).reshape(N, H * W, channels)
  for x3 in (x3, (x3 - 30) * 1e-3):
    gamma, beta = _params(channels, dtype)
    want = C.group_norm_cl_fwd(x3, groups, gamma, beta, 1e-5, act)[0]
    got = C.group_norm_cl_group(x3, groups, gamma, beta, 1e-5, act)
    assert torch.equal(got, want)
    with torch.no_grad():
      assert torch.equal(OF.group_norm(x3.view(N, H, W, channels).permute(0, 3, 1, 2), groups, gamma, beta, 1e-5, act).permute(0, 2, 3, 1).reshape(x3.shape), want)


@pytest.mark.parametrize("act,dtype", [(True, torch.bfloat16), (False, torch.float32), (True, None)])
@pytest.mark.parametrize("shape,groups", _FIRST)
def test_bits_of_the_channels_first_kernels(shape, groups, act, dtype):
  torch.manual_seed(2)
  N, channels, H, W = shape
  x = (torch.randn(*shape, device="cuda") * 2 + 30).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
  gamma, beta = _params(channels, dtype)
  for x in (x, (x - 30) * 1e-3):
    want, _ = K.groupnorm_fwd(x.contiguous(), groups, gamma, beta, 1e-5, act)
    got = C.group_norm_cl_group(x.permute(0, 2, 3, 1).reshape(N, H * W, channels), groups, gamma, beta, 1e-5, act)
    assert torch.equal(got.view(N, H, W, channels).permute(0, 3, 1, 2), want)
    with torch.no_grad():
      assert torch.equal(OF.group_norm(x, groups, gamma, beta, 1e-5, act), want)


def test_one_pixel_and_values_that_are_not_finite():
  torch.manual_seed(3)
  x3 = torch.randn(3, 1, 64, device="cuda").to(torch.bfloat16)
  gamma, beta = _params(64, torch.float32)
  want = torch.nn.functional.group_norm(x3.double().transpose(1, 2), 4, gamma.double(), beta.double(), 1e-2).transpose(1, 2)
  got = C.group_norm_cl_group(x3, 4, gamma, beta, 1e-2, False)
  # sixteen values of order one a group: fp32 statistics, one rounding to bf16
  assert ((got.double() - want).abs() <= want.abs() / 256 + 1e-4).all()
  for channels in (64, 2560):  # the values of a group that has one of them are those of the other kernels, the other groups finite
    x3 = torch.randn(2, 16, channels, device="cuda").to(torch.bfloat16)
    x3[0, 3, 5], x3[1, 2, 7] = float("inf"), float("nan")
    got = C.group_norm_cl_group(x3, 32, None, None, 1e-5, True)
    if channels == 64:
      want = C.group_norm_cl_fwd(x3, 32, None, None, 1e-5, True)[0]
    else:
      want = K.groupnorm_fwd(x3.transpose(1, 2).contiguous(), 32, None, None, 1e-5, True)[0].transpose(1, 2)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))
    bad = torch.zeros(2, 32, dtype=torch.bool)
    bad[0, 5 * 32 // channels], bad[1, 7 * 32 // channels] = True, True
    assert torch.equal(got.unflatten(2, (32, -1)).isfinite().all(3).all(1).cpu(), ~bad)
