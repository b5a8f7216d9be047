"""The CPython extension against the Python wrappers: the same kernels on the same launch shapes, so equal bit for bit, over
the layouts that a caller can hand in (the extension passes on what it does not take)."""
import pytest
import torch

from maxdiffusion_b200.ops import _lib, conv as OC, functional as OF, kernels as K

pytestmark = pytest.mark.gpu


def _both(monkeypatch, fn):
  with torch.no_grad():
    before = _lib.host_ops().launches()
    got = fn()
    used = _lib.host_ops().launches() > before
    with monkeypatch.context() as m:
      m.setattr(_lib, "_HOST", _lib._NoHostOps())
      want = fn()
  assert torch.equal(got, want) and got.shape == want.shape and got.stride() == want.stride() and got.dtype == want.dtype
  return used


def _launches(fn):
  before = _lib.launch_count()
  return fn(), _lib.launch_count() - before


def _randn(*shape):
  return torch.randn(shape, device="cuda").to(torch.bfloat16)


_FORMS = {"dense": lambda: _randn(3, 40, 64), "2d": lambda: _randn(17, 64), "4d": lambda: _randn(2, 3, 5, 64),
          "slice of channels": lambda: _randn(3, 40, 192)[..., 64:128], "part of a sequence": lambda: _randn(3, 50, 64)[:, 5:45],
          "transposed": lambda: _randn(40, 3, 64).transpose(0, 1), "every second row": lambda: _randn(3, 80, 64)[:, ::2],
          "expanded": lambda: _randn(1, 40, 64).expand(3, 40, 64), "one row": lambda: _randn(1, 1, 64),
          "columns apart": lambda: _randn(3, 40, 128)[..., ::2]}
_COPIED = ("transposed", "part of a sequence", "expanded", "columns apart")  # not one pitch: the wrappers copy these


@pytest.mark.parametrize("form", list(_FORMS))
@pytest.mark.parametrize("act", [None, "gelu_tanh", "silu", "residual"])
def test_linear(monkeypatch, form, act):
  torch.manual_seed(0)
  x, w, b = _FORMS[form](), _randn(72, 64), _randn(72)
  res = _randn(*x.shape[:-1], 72) if act == "residual" else None
  used = _both(monkeypatch, lambda: OF.linear(x, w, b, None if res is not None else act, residual=res))
  assert used or form in _COPIED
  _both(monkeypatch, lambda: OF.linear(x, w[::2], None))  # a strided weight
  if res is not None:
    _both(monkeypatch, lambda: OF.linear(x, w, b, residual=res.transpose(0, 1).contiguous().transpose(0, 1)))
    _both(monkeypatch, lambda: OF.linear(x, w, b, residual=res.float()))


@pytest.mark.parametrize("name,cut", [("odd offset", lambda t: t[..., 4:76]), ("odd pitch", lambda t: t[..., :72]), ("misaligned", None),
                                      ("in place", lambda t: t[..., 8:80])])
def test_linear_residual_layouts(monkeypatch, name, cut):
  """A residual that cannot be read 16 bytes at a time where it lies is copied, with and without the extension and autograd."""
  torch.manual_seed(7)
  x, w, b = _randn(3, 40, 64), _randn(72, 64), _randn(72)
  if cut is None:  # dense, but it starts 8 bytes into its storage
    res = _randn(3 * 40 * 72 + 4)[4:].view(3, 40, 72)
  else:
    res = cut(_randn(3, 40, {"odd offset": 80, "odd pitch": 76, "in place": 80}[name]))
  want = OF.linear(x, w, b, residual=res.clone(memory_format=torch.contiguous_format))
  _both(monkeypatch, lambda: OF.linear(x, w, b, residual=res))
  with torch.enable_grad():
    got = OF.linear(x, torch.nn.Parameter(w), b, residual=res)
    assert torch.equal(got, want)


_TALL = {"more than a tile": lambda: _randn(3, 87, 64), "slice of channels, tall": lambda: _randn(3, 87, 192)[..., 64:128],
         "every second row, tall": lambda: _randn(3, 174, 64)[:, ::2]}
_FORMS.update(_TALL)


@pytest.mark.parametrize("form", list(_FORMS))
@pytest.mark.parametrize("N", [8, 136, 320])
def test_geglu_linear(form, N):
  """Against float64; the product is not rounded to bf16 in between, so one rounding (2^-9 of a value) is all."""
  torch.manual_seed(4)
  x, w, b = _FORMS[form](), _randn(2 * N, 64), _randn(2 * N)
  with torch.no_grad():
    for bias in (b, None):
      u = x.double() @ w.double().t() + (0 if bias is None else bias.double())
      want = u[..., :N] * torch.nn.functional.gelu(u[..., N:])
      got, n = _launches(lambda: OF.geglu_linear(x, w, bias))
      assert n == (1 if form in _TALL else 2)  # one kernel from 129 rows on
      assert got.shape == want.shape and (got.double() - want).norm() < 4e-3 * want.norm()
  assert OF.geglu_linear(x, torch.nn.Parameter(w)).requires_grad


@pytest.mark.parametrize("form", list(_FORMS))
@pytest.mark.parametrize("n,N", [(2, 8), (3, 72), (3, 320), (2, 264)])
def test_linear_group(form, n, N):
  torch.manual_seed(5)
  x, ws = _FORMS[form](), [_randn(N, 64) for _ in range(n)]
  with torch.no_grad():
    got, launched = _launches(lambda: OF.linear_group(x, ws))
    assert len(got) == n and launched == (n if form in _COPIED else 1)
    for g, w in zip(got, ws):
      want = x.double() @ w.double().t()
      assert g.shape == want.shape and (g.double() - want).norm() < 4e-3 * want.norm()  # one rounding to bf16
    odd, launched = _launches(lambda: OF.linear_group(x, [ws[0], ws[1][:8]]))
    assert odd[1].shape[-1] == 8 and launched == (1 if N == 8 and form not in _COPIED else 2)
  assert OF.linear_group(x, [torch.nn.Parameter(w) for w in ws])[1].requires_grad


@pytest.mark.parametrize("D", [8, 40, 64, 80, 128])
def test_attention(monkeypatch, D):
  torch.manual_seed(1)
  q, k, v = _randn(2, 70, 3, D), _randn(2, 90, 3, D), _randn(2, 90, 3, D)
  assert _both(monkeypatch, lambda: OF.attention(q, k, v))
  fused = _randn(2, 70, 3, 3, D)
  assert _both(monkeypatch, lambda: OF.attention(fused[:, :, 0], fused[:, :, 1], fused[:, :, 2], scale=0.3))
  _both(monkeypatch, lambda: OF.attention(q.transpose(1, 2).contiguous().transpose(1, 2), [k, k], [v, v]))
  if D in K.FLASH_HEAD_DIMS:
    return  # there the kernel itself refuses strides that TMA cannot take
  one = _randn(1, 70, 1, D)  # keys and values shared by all heads and samples
  shared = one.expand(2, 70, 3, D)
  with torch.no_grad():
    assert torch.equal(OF.attention(q, shared, shared), OF.attention(q, shared.contiguous(), shared.contiguous()))
    assert torch.equal(OF.attention(shared, k, v), OF.attention(shared.contiguous(), k, v))
  wide = _randn(2, 70, 3, D + 4)
  _both(monkeypatch, lambda: OF.attention(wide[..., :D], wide[..., :D], wide[..., :D]))  # copied


def test_norms_and_gates(monkeypatch):
  torch.manual_seed(2)
  for C in (64, 640, 1280, 3072):
    x, g, b = _randn(2, 33, C), _randn(C), _randn(C)
    s = torch.randn(2, 3 * C, device="cuda")
    assert _both(monkeypatch, lambda: OF.layer_norm_mod(x, g, b))
    assert _both(monkeypatch, lambda: OF.layer_norm_mod(x, scale=s[:, :C], shift=s[:, C:2 * C]))
    _both(monkeypatch, lambda: OF.layer_norm_mod(x, scale=s[:, :C].to(torch.bfloat16), shift=s[:, C:2 * C]))
    _both(monkeypatch, lambda: OF.layer_norm_mod(x.transpose(0, 1), g, b))
    assert _both(monkeypatch, lambda: OF.geglu(x))
  qkv, w = _randn(2, 33, 3 * 256), _randn(128)
  cos, sin = torch.randn(33, 64, device="cuda"), torch.randn(33, 64, device="cuda")
  assert _both(monkeypatch, lambda: OF.rms_norm_rope(qkv[..., 256:512], w, cos, sin, heads=2, per_head=True))
  assert _both(monkeypatch, lambda: OF.rms_norm_rope(qkv[..., :256], _randn(256) * 0 + 1, heads=2))
  two = [(qkv[..., :256], w, cos, sin), (_randn(2, 7, 256), w, cos[:7].contiguous(), sin[:7].contiguous())]
  joint = torch.cat([OF.rms_norm_rope(x, w, c, s, heads=2, per_head=True) for x, w, c, s in two], dim=1)
  with torch.no_grad():
    assert torch.equal(OF.joint_norm_rope(two, 2), joint)


@pytest.mark.parametrize("shape", [(2, 64, 8, 8), (1, 320, 17, 5), (3, 96, 1, 9)])
def test_group_norm_and_conv(monkeypatch, shape):
  torch.manual_seed(3)
  C = shape[1]
  x = _randn(*shape).contiguous(memory_format=torch.channels_last)
  g, b, w, cb = _randn(C), _randn(C), _randn(48, C, 3, 3) * 0.05, _randn(48)
  for act in (False, True):
    assert _both(monkeypatch, lambda: OF.group_norm(x, 32, g, b, 1e-5, act))
    assert not _both(monkeypatch, lambda: OF.group_norm(x, 32, g.float(), b.float(), 1e-5, act))
  assert _both(monkeypatch, lambda: OF.conv2d(x, w, cb))
  assert _both(monkeypatch, lambda: OF.conv2d(x.contiguous(), w, None, upsample=True))
  clip, hist = _randn(1, 3, 6, 10, C), _randn(1, 2, 6, 10, C)
  pk = OC.pack_conv3d(_randn(40, C, 3, 3, 3) * 0.05, _randn(40))
  assert _both(monkeypatch, lambda: OC.conv3d_causal(clip, pk, hist))


def test_direct_calls_leave_autograd_alone():
  """Everything that works through the autograd functions still goes through them."""
  x, w = _randn(2, 8, 64), torch.nn.Parameter(_randn(72, 64))
  assert OF.linear(x, w).requires_grad
  with torch.no_grad():
    assert OF._direct(x, w) and not OF._direct(torch.nn.Buffer(x).as_subclass(type("T", (torch.Tensor,), {})))
    import torch.autograd.forward_ad as fwAD
    with fwAD.dual_level():
      assert not OF._direct(x)
    out = []
    torch.func.vmap(lambda t: (out.append(OF._direct(t)), t)[1])(x)
    assert out == [False]
  store = []
  y = OF.checkpoint_block(lambda t: (store.append(OF._direct(t)), OF.linear(t, w))[1], x.requires_grad_())
  y.float().sum().backward()
  assert store == [False, False] and w.grad is not None


def test_fused_calls_without_the_extension(monkeypatch):
  torch.manual_seed(8)
  x, w, b, ws = _randn(3, 87, 64), _randn(272, 64), _randn(272), [_randn(72, 64) for _ in range(3)]
  monkeypatch.setattr(_lib, "_HOST", _lib._NoHostOps())
  with torch.no_grad():
    u = x.double() @ w.double().t() + b.double()
    want = u[..., :136] * torch.nn.functional.gelu(u[..., 136:])
    assert (OF.geglu_linear(x, w, b).double() - want).norm() < 8e-3 * want.norm()  # the product is rounded in between
    for got, m in zip(OF.linear_group(x, ws), ws):
      want = x.double() @ m.double().t()
      assert (got.double() - want).norm() < 4e-3 * want.norm()


@pytest.mark.parametrize("B,rows,heads", [(1, (1, 1), 1), (2, (7, 33), 3), (1, (128, 256), 24), (2, (40,), 2), (1, (5,), 9)])
def test_fused_qkv_and_attention_into(B, rows, heads):
  """One launch for the norm, rotation and joining of q, k, v against one launch per stream and matrix: the same bits; attention
  stored into a part of a wider buffer against a copy of its result."""
  torch.manual_seed(6)
  C, extra = heads * 128, 0 if len(rows) == 2 else 72
  parts = [(_randn(B, s, 3 * C + extra), _randn(128), _randn(128), torch.randn(s, 64, device="cuda"), torch.randn(s, 64, device="cuda"))
           for s in rows]
  one = lambda x, w, c, s: OF.rms_norm_rope(x, w, c, s, heads=heads, per_head=True)
  with torch.no_grad():
    q, k, v = OF.fused_qkv(parts, heads, copy_v=len(rows) == 2)
    assert torch.equal(q, torch.cat([one(x[..., :C], wq, c, s) for x, wq, wk, c, s in parts], dim=1))
    assert torch.equal(k, torch.cat([one(x[..., C:2 * C], wk, c, s) for x, wq, wk, c, s in parts], dim=1))
    assert torch.equal(v, torch.cat([x[..., 2 * C:3 * C].unflatten(-1, (heads, 128)) for x, *_ in parts], dim=1))
    wide = torch.zeros((B, sum(rows), C + 264), device="cuda", dtype=torch.bfloat16)
    OF.attention_into(wide[..., 8:8 + C].unflatten(-1, (heads, 128)), q, k, v)
    assert torch.equal(wide[..., 8:8 + C], OF.attention(q, k, v).flatten(2)) and wide[..., :8].eq(0).all() and wide[..., 8 + C:].eq(0).all()
    off = torch.zeros((B, sum(rows), C + 3), device="cuda", dtype=torch.bfloat16)  # rows of no 16-byte pitch: copied
    OF.attention_into(off[..., 1:1 + C].unflatten(-1, (heads, 128)), q, k, v)
    assert torch.equal(off[..., 1:1 + C], wide[..., 8:8 + C])
  x, wq, wk, c, s = parts[0]
  assert OF.fused_qkv([(x, wq.requires_grad_(), wk, c, s)], heads, copy_v=False) is None  # autograd: the differentiable ops
  with torch.no_grad():
    for bad in ((x.float(), wq, wk, c, s), (x, wq.float(), wk, c, s), (x, wq, wk, c.double(), s), (x[..., 4:], wq, wk, c, s)):
      assert OF.fused_qkv([bad], heads, copy_v=False) is None


@pytest.mark.parametrize("stride,shape", [(1, (2, 32, 8, 8)), (1, (1, 48, 17, 5)), (2, (2, 32, 6, 10)), (1, (3, 32, 1, 9))])
def test_conv2d_nchw_launches_what_conv2d_does(stride, shape):
  """The kept launch arguments against those of `conv2d`: the same bits over several sizes, with and without a residual, and
  again after a change of the weights."""
  torch.manual_seed(7)
  cl = dict(memory_format=torch.channels_last)
  w, b = _randn(40, shape[1], 3, 3) * 0.05, _randn(40)
  with torch.no_grad():
    for pad in (0, 1) if stride == 2 else (1,):
      pk = OC.pack_conv2d(w, b, stride=stride, pad_top_left=pad)
      for B in (shape[0], shape[0] + 1, shape[0]):
        x = _randn(B, *shape[1:]).contiguous(**cl)
        res = _randn(B, 40, shape[2] // stride, shape[3] // stride).contiguous(**cl)
        for r in (None, res):
          rows = None if r is None else r.permute(0, 2, 3, 1)
          got = OC.conv2d_nchw(x, pk, rows)
          assert torch.equal(got.permute(0, 2, 3, 1), OC.conv2d(x.permute(0, 2, 3, 1), pk, residual=rows))
      assert OC.conv2d_nchw(_randn(1, shape[1], 6, 6), pk) is None  # not channels-last
    x = _randn(*shape).contiguous(**cl)
    first = OF.conv2d(x, w, b, stride=stride)
    assert torch.equal(OF.conv2d(x, w.mul_(2), b * 2, stride=stride), (first.float() * 2).to(torch.bfloat16))
