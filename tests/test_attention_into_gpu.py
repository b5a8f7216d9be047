"""Attention stored into a part of a wider buffer, at every kind of head size that the extension takes."""
import pytest
import torch

from maxdiffusion_b200.ops import functional as OF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [8, 40, 64, 72, 80, 120, 128])
@pytest.mark.parametrize("B,S,Skv,H", [(1, 1, 1, 1), (2, 65, 130, 3), (1, 257, 77, 2)])
def test_into_a_wider_buffer(B, S, Skv, H, D):
  torch.manual_seed(9)
  q, k, v = (torch.randn(B, n, H, D, device="cuda").to(torch.bfloat16) for n in (S, Skv, Skv))
  with torch.no_grad():
    want = OF.attention(q, k, v)
    wide = torch.full((B, S, 16 + H * D), 7.0, device="cuda", dtype=torch.bfloat16)
    OF.attention_into(wide[..., 8:8 + H * D].unflatten(-1, (H, D)), q, k, v)
  assert torch.equal(wide[..., 8:8 + H * D], want.flatten(2))
  assert wide[..., :8].eq(7).all() and wide[..., 8 + H * D:].eq(7).all()
