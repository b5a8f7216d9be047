"""Flux's single block with quantised layers: what it allocates on either way."""
import pytest
import torch

from maxdiffusion_b200.models.flux.transformer_flux import FLUX_PRESETS, FluxConfig, FluxSingleBlock
from maxdiffusion_b200.models.quantizations import quantize_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp8", "int8"])
def test_the_wide_buffer_is_allocated_where_it_is_used(mode, monkeypatch):
  torch.manual_seed(6)
  cfg = FluxConfig(**{**FLUX_PRESETS["flux-dev"], "num_attention_heads": 2})
  block = FluxSingleBlock(cfg).to("cuda", torch.bfloat16)
  model = torch.nn.Module()
  model.single_transformer_blocks = torch.nn.ModuleList([block])
  quantize_model(model, mode)
  assert type(block.qkv_mlp).__name__ == ("Fp8Linear" if mode == "fp8" else "Int8Linear")
  wide = block.dim + block.hidden
  seen, empty = [], torch.empty
  monkeypatch.setattr(torch, "empty", lambda *a, **kw: seen.append(tuple(a[0]) if a and not isinstance(a[0], int) else a) or empty(*a, **kw))

  def run(S, grad):
    seen.clear()
    x = torch.randn(1, S, block.dim, device="cuda").to(torch.bfloat16)
    temb = torch.randn(1, block.dim, device="cuda").to(torch.bfloat16)
    rope = (torch.rand(S, 64, device="cuda"), torch.rand(S, 64, device="cuda"))
    with torch.set_grad_enabled(grad):
      assert block(x, temb, rope).shape == x.shape
    return (1, S, wide) in seen

  assert run(64, False)
  assert not run(64, True)  # autograd: one product, torch.cat
  assert not run(60, False)  # rows that the 8-bit product does not take
