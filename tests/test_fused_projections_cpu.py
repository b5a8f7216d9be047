"""Projections that run fused with one another (the UNet's q / k / v and GEGLU) are modules all the same: what a user hangs on
one of them takes effect as when it is called."""
import pytest
import torch
import torch.nn.modules.module as nn_module

from maxdiffusion_b200.models import layers, unet_2d_condition as U


def _block():
  torch.manual_seed(0)
  attn, ff = U.Attention(16, 2, 24), U.FeedForward(16)
  return attn, ff, torch.randn(2, 5, 16, requires_grad=True), torch.randn(2, 7, 24)


def _parts(attn, ff):
  return {"to_q": attn.to_q, "to_k": attn.to_k, "to_v": attn.to_v, "to_out": attn.to_out[0], "proj": ff.net[0].proj, "ff_out": ff.net[2]}


_KINDS = {"forward": ("register_forward_hook", lambda note: lambda m, i, o: note()),
          "forward_pre": ("register_forward_pre_hook", lambda note: lambda m, i: note()),
          "backward": ("register_full_backward_hook", lambda note: lambda m, gi, go: note()),
          "backward_pre": ("register_full_backward_pre_hook", lambda note: lambda m, go: note())}


@pytest.mark.parametrize("kind", list(_KINDS))
def test_every_kind_of_hook_fires(kind):
  attn, ff, x, ctx = _block()
  seen = set()
  for name, m in _parts(attn, ff).items():
    register, make = _KINDS[kind]
    getattr(m, register)(make(lambda name=name: seen.add(name)))
  ff(attn(x, ctx)).sum().backward()
  assert seen == set(_parts(attn, ff))


@pytest.mark.parametrize("kind", list(_KINDS))
def test_every_kind_of_global_hook_fires(kind):
  attn, ff, x, ctx = _block()
  parts, seen = _parts(attn, ff), set()
  register = {"forward": nn_module.register_module_forward_hook, "forward_pre": nn_module.register_module_forward_pre_hook,
              "backward": nn_module.register_module_full_backward_hook,
              "backward_pre": nn_module.register_module_full_backward_pre_hook}[kind]
  handle = register(lambda m, *a: seen.update(n for n, p in parts.items() if p is m))
  try:
    ff(attn(x, ctx)).sum().backward()
  finally:
    handle.remove()
  assert seen == set(parts)


def test_a_gradient_changed_by_a_hook_is_changed():
  attn, ff, x, ctx = _block()
  ff(attn(x, ctx)).sum().backward()
  plain = x.grad.clone()
  x.grad = None
  attn.to_q.register_full_backward_hook(lambda m, gi, go: (gi[0] * 0,))
  ff(attn(x, ctx)).sum().backward()
  assert not torch.equal(x.grad, plain)


def test_a_replaced_forward_runs(monkeypatch):
  attn, ff, x, ctx = _block()
  seen, forward = [], layers.Linear.forward
  monkeypatch.setattr(layers.Linear, "forward", lambda self, *a, **k: (seen.append(self), forward(self, *a, **k))[1])
  ff(attn(x, ctx))
  assert {id(m) for m in seen} == {id(m) for m in _parts(attn, ff).values()}


@pytest.mark.parametrize("which", ["to_q", "to_v"])  # a bias of the keys moves all scores of a row alike
@pytest.mark.parametrize("cross", [False, True])
def test_a_bias_put_on_a_projection_is_added(which, cross):
  torch.manual_seed(1)
  attn, x = U.Attention(16, 2), torch.randn(2, 5, 16)
  ctx = torch.randn(2, 7, 16) if cross else None
  getattr(attn, which).bias = torch.nn.Parameter(torch.randn(16))
  src = x if ctx is None else ctx
  q, k, v = (t.unflatten(-1, (2, 8)) for t in (attn.to_q(x), attn.to_k(src), attn.to_v(src)))
  want = attn.to_out[0](U.OF.attention(q, k, v).reshape(2, 5, 16))
  torch.testing.assert_close(attn(x, ctx), want, rtol=1e-6, atol=1e-6)  # the same fp32 products
