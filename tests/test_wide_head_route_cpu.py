"""Which calls of `wide_head_attention` leave PyTorch's operations for the kernels of odd lengths."""
import torch
import torch.autograd.forward_ad as fwAD

from maxdiffusion_b200.ops import conv as C, functional as OF


def test_route(monkeypatch):
  monkeypatch.setattr(C, "use_kernel", lambda t: t.dtype == torch.bfloat16)  # as if on the GPU
  q, k, v = (torch.randn(77, 16).to(torch.bfloat16) for _ in range(3))
  ok = C._odd_head_ok
  assert ok(q, k, v) and ok(q, k, v[:, :8])
  assert not ok(q[:72], k[:72], v[:72]) and not ok(q, k[:50], v[:50]) and not ok(q, k, v[:, :9]) and not ok(q[:, :9], k[:, :9], v)
  assert not ok(q, k, v.float()) and not ok(q, k.float(), v)
  w = v.clone().requires_grad_()
  assert not ok(q, k, w)
  with torch.no_grad():
    assert ok(q, k, w)
    with fwAD.dual_level():
      assert not ok(q, k, v)
    seen = []
    torch.func.vmap(lambda t: (seen.append(ok(q, k, t)), t)[1])(torch.stack([v, v]))
    assert seen == [False]
  OF.set_library_mode(True)
  try:
    assert not ok(q, k, v)
  finally:
    OF.set_library_mode(False)


def test_general_path_on_the_cpu():
  torch.manual_seed(0)
  q, k, v = torch.randn(7, 16), torch.randn(5, 16), torch.randn(5, 24)
  want = ((q.double() @ k.double().t()) * 0.25).softmax(-1) @ v.double()
  torch.testing.assert_close(C.wide_head_attention(q, k, v).double(), want, rtol=1e-5, atol=1e-5)
