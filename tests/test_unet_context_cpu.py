"""Cross-attention of a UNet over a context of one sample."""
import pytest
import torch

from maxdiffusion_b200.models.unet_2d_condition import UNET_PRESETS, UNet2DConditionModel, UNetConfig


@pytest.mark.parametrize("grad", [False, True])
def test_a_context_of_one_sample_broadcasts(grad):
  torch.manual_seed(0)
  cfg = UNetConfig(**UNET_PRESETS["tiny_sd"])
  model = UNet2DConditionModel(cfg)
  x, t, ctx = torch.randn(3, cfg.in_channels, 16, 16), torch.tensor([5.0, 6.0, 7.0]), torch.randn(1, 7, cfg.cross_attention_dim)
  with torch.set_grad_enabled(grad):
    torch.testing.assert_close(model(x, t, ctx), model(x, t, ctx.expand(3, -1, -1)), rtol=1e-5, atol=1e-5)
