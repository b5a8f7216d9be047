"""A Flux double block without autograd under function transforms, and streams of different types."""
import pytest
import torch

from maxdiffusion_b200.models.flux import transformer_flux as T
from maxdiffusion_b200.ops import functional as OF


def _block():
  torch.manual_seed(0)
  blk = T.FluxDoubleBlock(T.FluxConfig(num_attention_heads=2, attention_head_dim=128))
  rope = lambda n: (torch.randn(n, 64), torch.randn(n, 64))
  return blk, torch.randn(3, 1, 6, 256), torch.randn(3, 1, 4, 256), torch.randn(3, 1, 256), rope(6), rope(4)


def test_vmap_of_a_double_block():
  blk, img, txt, temb, ri, rt = _block()
  with torch.no_grad():
    got = torch.func.vmap(lambda i, t, e: blk(i, t, e, ri, rt))(img, txt, temb)
    for n in range(3):
      for g, w in zip(got, blk(img[n], txt[n], temb[n], ri, rt)):
        torch.testing.assert_close(g[n], w, rtol=1e-4, atol=1e-4)  # fp32 products batched otherwise


@pytest.mark.parametrize("grad", [False, True])
def test_streams_of_two_types_are_promoted(grad):
  a, b = torch.randn(2, 3, 8).to(torch.bfloat16), torch.randn(2, 5, 8)
  with torch.set_grad_enabled(grad):
    for parts in ([a, b], [b, a], [a, a.half()]):
      got = OF.joint_rows(parts)
      assert got.dtype == torch.float32 and torch.equal(got, torch.cat([p.float() for p in parts], dim=1))
