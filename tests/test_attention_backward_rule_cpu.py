"""When the attention backward keeps dS: sizes at which both ways were measured, and what it takes where memory is short."""
import pytest
import torch

from maxdiffusion_b200.ops import kernels as K


@pytest.mark.parametrize("B,H,Sq,Skv,n,faster", [
    (1, 12, 4096, 4096, 12, True), (4, 10, 4096, 77, 40, True), (1, 40, 32760, 512, 40, True), (1, 1, 1, 1, 1, True),  # all at once
    (1, 40, 32760, 32760, 4, True), (1, 24, 18000, 18000, 14, True), (1, 12, 28500, 28500, 5, True), (1, 40, 22000, 22000, 4, True),
    (1, 24, 16000, 16000, 4, True), (1, 12, 10000, 10000, 5, False), (1, 40, 22000, 22000, 2, False), (1, 40, 22000, 22000, 1, False),
    (8, 10, 4096, 4096, 10, False), (2, 20, 1024, 1024, 20, False), (1, 40, 32760, 512, 10, False)])
def test_measured_sizes(B, H, Sq, Skv, n, faster):
  assert K._ds_pays(n, B, H, Sq, Skv) == faster


def test_too_few_heads_at_a_time_are_not_asked_for(monkeypatch):
  asked = []
  monkeypatch.setattr(torch, "empty", lambda n, **kw: asked.append(n))
  monkeypatch.setattr(K, "_ds_refused", {})
  monkeypatch.setattr(K, "_ds_stats", lambda device: (0, 0))
  monkeypatch.setattr(K, "_ds_room", lambda device, enough: 4 << 30)  # 3 GB for dS: three heads of 22000^2
  assert K._ds_buffer(1, 40, 22000, 22000, torch.device("cpu")) == (0, None) and asked == []
  monkeypatch.setattr(K, "_ds_room", lambda device, enough: 5 << 30)  # 4 GB: four
  assert K._ds_buffer(1, 40, 22000, 22000, torch.device("cpu"))[0] == 4 and len(asked) == 1
