"""Convolutions of a 1 x 1 image: the same answer with the host extension and without it."""
import pytest
import torch

from maxdiffusion_b200.ops import _lib
from maxdiffusion_b200.ops import functional as OF

pytestmark = pytest.mark.gpu


def test_one_pixel_by_either_route(monkeypatch):
  torch.manual_seed(8)
  w, b = (torch.randn(48, 32, 3, 3, device="cuda") * 0.05).to(torch.bfloat16), torch.randn(48, device="cuda").to(torch.bfloat16)
  plain = torch.randn(2, 32, 1, 1, device="cuda").to(torch.bfloat16)  # strides (32, 1, 1, 1): rows that the kernel cannot address
  dense = torch.empty(2, 32, 1, 1, device="cuda", dtype=torch.bfloat16, memory_format=torch.channels_last).copy_(plain)  # (32, 1, 32, 32)

  def answers():
    with torch.no_grad():
      try:
        first = OF.conv2d(plain, w, b)
      except AssertionError:
        first = None
      return first, OF.conv2d(dense, w, b)

  with_it = answers()
  monkeypatch.setattr(_lib, "_HOST", _lib._NoHostOps())
  without = answers()
  assert (with_it[0] is None) == (without[0] is None)
  assert torch.equal(with_it[1], without[1])
  want = torch.nn.functional.conv2d(dense.double(), w.double(), b.double(), padding=1)
  assert ((with_it[1].double() - want).norm() / want.norm()) < 4e-3  # one rounding to bf16
