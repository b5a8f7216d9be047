"""A quantised layer whose class has another `forward` is not run in parts."""
import pytest
import torch

from maxdiffusion_b200.models.layers import Linear
from maxdiffusion_b200.models.quantizations import Fp8Linear, Int8Linear, is_plain_quantized


@pytest.mark.parametrize("cls", [Fp8Linear, Int8Linear])
def test_a_replaced_forward_of_the_class(cls, monkeypatch):
  m = cls(Linear(16, 16))
  assert is_plain_quantized(m)
  with monkeypatch.context() as mp:
    mp.setattr(cls, "forward", lambda self, x, activation=None: torch.zeros_like(x))
    assert not is_plain_quantized(m)
  assert is_plain_quantized(m)


def test_a_replaced_forward_of_the_base_class(monkeypatch):
  monkeypatch.setattr(Fp8Linear, "forward", lambda self, x, activation=None: torch.zeros_like(x))
  assert not is_plain_quantized(Int8Linear(Linear(16, 16))) and not is_plain_quantized(Fp8Linear(Linear(16, 16)))
