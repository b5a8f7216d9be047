"""Launch shapes of the tensor-core kernels at the edges of their tiles: GEMM tiles of one CTA or a pair, cut contractions
with an epilogue in the fold, convolutions by pairs and in parts. Oracle: float64 PyTorch.

Tolerances: fp32 accumulation of bf16 products and one rounding to bf16 (2^-9 relative to a value) give 1.7e-3 in the
2-norm; 4e-3 leaves room for a second rounding (the residual)."""
import pytest
import torch

from maxdiffusion_b200.ops import conv as C
from maxdiffusion_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _randn(*shape, scale=1.0):
  return (torch.randn(shape, device="cuda") * scale).to(torch.bfloat16)


def _rel(got, want):
  return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("ctas,bn", [(1, 64), (1, 192), (1, 256), (2, 64), (2, 128), (2, 192), (2, 256)])
@pytest.mark.parametrize("M,N,Kd", [(8, 8, 8), (128, 64, 64), (129, 200, 136), (257, 264, 72), (640, 520, 1032)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_tiles(ctas, bn, M, N, Kd, a_mn, b_mn):
  if b_mn and (bn // ctas) % 64:
    pytest.skip("a transposed B needs a multiple of 64 columns per CTA")
  torch.manual_seed(0)
  M -= M % 8 if a_mn else 0
  a, b, bias = _randn(*((Kd, M) if a_mn else (M, Kd))), _randn(*((Kd, N) if b_mn else (N, Kd))), _randn(N)
  want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t()) + bias.double()
  guard = torch.full((M + 2, N), 7.0, device="cuda", dtype=torch.bfloat16)
  K.gemm_force_ctas(ctas)
  K.gemm_force_tile_n(bn)
  try:
    assert K.gemm_plan(M, N, Kd, b_mn, True, 148, bn, ctas)[:2] == (ctas, bn)
    K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, out=guard[1:-1])
  finally:
    K.gemm_force_ctas(0)
    K.gemm_force_tile_n(0)
  assert _rel(guard[1:-1], want) < 4e-3
  assert bool((guard[0] == 7).all()) and bool((guard[-1] == 7).all())


@pytest.mark.parametrize("epi", ["none", "gelu_tanh", "silu", "add_res", "gated_res"])
@pytest.mark.parametrize("M,N,Kd", [(136, 328, 4104), (384, 512, 8192)])
def test_gemm_cut_contraction_with_epilogue(epi, M, N, Kd):
  """Few tiles and a long contraction: the fold kernel applies the epilogue."""
  torch.manual_seed(1)
  a, b, bias, res = _randn(M, Kd), _randn(N, Kd, scale=0.05), _randn(N), _randn(M, N)
  rows = M // 2
  gate = torch.randn((2, N), device="cuda")
  assert K.gemm_plan(M, N, Kd)[2] > 1
  got = K.gemm(a, b, bias=bias, epi=epi, residual=res if "res" in epi else None, gate=gate if epi == "gated_res" else None,
               rows_per_batch=rows if epi == "gated_res" else 0)
  want = a.double() @ b.double().t() + bias.double()
  if epi == "gelu_tanh":
    want = torch.nn.functional.gelu(want, approximate="tanh")
  elif epi == "silu":
    want = torch.nn.functional.silu(want)
  elif epi == "add_res":
    want = want + res.double()
  elif epi == "gated_res":
    want = res.double() + gate.double().repeat_interleave(rows, 0) * want
  assert _rel(got, want) < 4e-3


def test_cut_contraction_takes_a_bias_that_starts_anywhere():
  torch.manual_seed(4)
  a, b, store = _randn(136, 4096), _randn(328, 4096, scale=0.05), _randn(400)
  bias = store[3:331]  # 6 bytes into a 16-byte line
  assert K.gemm_plan(136, 328, 4096)[2] > 1
  assert _rel(K.gemm(a, b, bias=bias), a.double() @ b.double().t() + bias.double()) < 4e-3


@pytest.mark.parametrize("Sq,B,H", [(256 * 37, 2, 2), (300, 7, 23), (1024, 2, 20), (129, 1, 1)])
def test_attention_last_round_of_single_tiles(Sq, B, H):
  """148 whole items, a last round of single tiles, and items whose second tile does not exist."""
  torch.manual_seed(5)
  q, k, v = _randn(B, Sq, H, 64), _randn(B, 200, H, 64), _randn(B, 200, H, 64)
  out, lse = K.flash_fwd(q, [k], [v])
  s = torch.einsum("bshd,bthd->bhst", q.double(), k.double()) / 8.0
  assert _rel(out, torch.einsum("bhst,bthd->bshd", s.softmax(-1), v.double())) < 5e-3  # P is rounded to bf16 too
  assert (lse.double() * 0.6931471805599453 - s.logsumexp(-1)).abs().max() < 1e-4


@pytest.mark.parametrize("plan", [(1, 64, 3), (2, 256, 1), (2, 64, 2), (1, 256, 7), (2, 32, 1)])
@pytest.mark.parametrize("B,H,W,Ci,Co", [(1, 8, 16, 64, 64), (2, 17, 23, 64, 328), (1, 33, 40, 96, 96), (3, 9, 70, 192, 24),
                                         (1, 5, 128, 64, 64), (1, 9, 250, 96, 96), (2, 3, 127, 320, 40)])
def test_conv_launch_shapes(plan, B, H, W, Ci, Co):
  """An odd number of M-tiles (the pair's second half lies outside), ragged edges, parts of the contraction, rows of 128
  positions shared by neighbouring taps."""
  torch.manual_seed(2)
  x, w, b, res = _randn(B, H, W, Ci), _randn(Co, Ci, 3, 3, scale=0.05), _randn(Co), _randn(B, H, W, Co)
  nchw = x.permute(0, 3, 1, 2).double()
  want = torch.nn.functional.conv2d(nchw, w.double(), b.double(), padding=1).permute(0, 2, 3, 1)
  up = torch.nn.functional.conv2d(torch.nn.functional.interpolate(nchw, scale_factor=2, mode="nearest"), w.double(), b.double(),
                                  padding=1).permute(0, 2, 3, 1)
  pk, pu = C.pack_conv2d(w, b), C.pack_upsample_conv2d(w, b)
  blocks = -(-Ci // 64)
  try:  # a part of a contraction has at least one step: (rows of) taps times channel blocks
    C._PLAN = (*plan[:2], min(plan[2], 3 * blocks))
    got, fused = C.conv2d(x, pk), C.conv2d(x, pk, residual=res, silu=True)
    C._PLAN = (*plan[:2], min(plan[2], 2 * blocks))
    got_up = C.upsample2x_conv2d(x, pu)
  finally:
    C._PLAN = None
  assert _rel(got, want) < 4e-3
  assert _rel(fused, torch.nn.functional.silu(want) + res.double()) < 4e-3
  assert _rel(got_up, up) < 6e-3  # the parity weights are sums, rounded to bf16 once more


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk", [(1, 1), (127, 63), (129, 65), (300, 128), (257, 191)])
def test_attention_ragged_tails(D, Sq, Sk):
  torch.manual_seed(3)
  q, k, v = _randn(2, Sq, 3, D), _randn(2, Sk, 3, D), _randn(2, Sk, 3, D)
  out, lse = K.flash_fwd(q, [k], [v])
  s = torch.einsum("bshd,bthd->bhst", q.double(), k.double()) / D ** 0.5
  assert _rel(out, torch.einsum("bhst,bthd->bshd", s.softmax(-1), v.double())) < 5e-3  # P is rounded to bf16 too
  assert (lse.double() * 0.6931471805599453 - s.logsumexp(-1)).abs().max() < 1e-4


@pytest.mark.parametrize("T,D", [(1, 384), (7, 64), (500, 384), (4500, 384), (9001, 16)])
def test_wide_head_attention_of_odd_lengths(T, D):
  """Scores and probabilities stay in 32 bits: the result is the float64 one rounded to bf16 once (2^-9 of a value; 1.7e-3 in
  the 2-norm)."""
  torch.manual_seed(6)
  q, k, v = _randn(T, D, scale=2.0), _randn(T, D), _randn(T, D)
  s = (q.double() @ k.double().t()) * D ** -0.5
  with torch.no_grad():
    assert _rel(C.wide_head_attention(q, k, v), s.softmax(-1) @ v.double()) < 2e-3


@pytest.mark.parametrize("cols,pitch", [(1, 8), (7, 8), (255, 256), (4500, 4504), (9001, 9008), (32767, 32768)])
def test_softmax_in_three_planes(cols, pitch):
  """Against float64, probability by probability: in units of 2^-24 the rounded difference to the maximum costs |v|,
  expf (2 ulp) and the division 5, the additions of the sum one each (cols / 256 + 13) and the third plane's rounding 1."""
  torch.manual_seed(7)
  x = torch.randn(9, pitch, device="cuda") * 8
  x[1, : cols // 2] = -float("inf")  # what an overflowing product of finite values leaves
  x[2, : cols // 2] = -3e38
  x[3, : cols // 2] = -3.4e38
  x[3, cols - 1] = 3.4e38
  x[4, 0] = float("nan")
  x[5, cols - 1] = float("inf")
  x[6] = -float("inf")
  x[:, cols:] = float("nan")  # not read
  got = C.softmax_split(x, cols).view(9, 3, pitch)
  assert not got[:, :, cols:].any()
  p, want = got[:, :, :cols].double().sum(1), x[:, :cols].double().softmax(-1)
  assert torch.equal(p.isnan(), x[:, :cols].softmax(-1).isnan())
  ok = [0, 1, 2, 3, 7, 8]
  v = (x[ok, :cols].double() - x[ok, :cols].double().amax(-1, keepdim=True)).clamp(min=-100)
  bound = (v.abs() + 24 + cols / 256) * 2.0 ** -24 * want[ok] + 2.0 ** -133  # below that bf16 has no values left
  assert ((p[ok] - want[ok]).abs() <= bound).all()


def test_wide_head_attention_forms():
  """Other numbers of keys, other widths of values, fp32 values, misaligned queries and infinite values: as plain PyTorch has it."""
  torch.manual_seed(8)
  T, D = 77, 64
  q, k, v = _randn(T, D), _randn(T, D), _randn(T, D)
  off = torch.empty(T * D + 4, device="cuda", dtype=torch.bfloat16)[4:].view(T, D).copy_(q)
  inf = v.clone()
  inf[3, 5], inf[4, 6], inf[70, 7] = float("inf"), -float("inf"), float("nan")
  with torch.no_grad():
    for a, b, c in ((q, k[:50], v[:50]), (q, k, v[:, :24]), (q, k, v.float()), (off, k, v), (q[:, ::2][:, :16], k[:, :16], v), (q, k, inf)):
      got = C.wide_head_attention(a, b, c)
      want = ((a.double() @ b.double().t()) * a.shape[1] ** -0.5).softmax(-1) @ c.double()
      assert got.shape == want.shape and got.dtype == torch.bfloat16
      bad = ~want.isfinite()
      assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[bad].double().nan_to_num(), want[bad].nan_to_num().to(torch.bfloat16).double().nan_to_num())
      assert _rel(got[~bad], want[~bad]) < 4e-3  # one rounding to bf16


@pytest.mark.parametrize("epi", ["none", "gelu_tanh", "silu", "add_res"])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("direct", [False, True])
def test_a_bias_may_start_anywhere(epi, f32, direct):
  """Every epilogue in one part: fp32 results with an activation or a residual are stored straight from the accumulator."""
  torch.manual_seed(9)
  a, b, store, res = _randn(136, 64), _randn(328, 64, scale=0.1), _randn(400), _randn(136, 328)
  bias = store[3:331]  # 6 bytes into a 16-byte line
  kw = dict(epi=epi, residual=res if epi == "add_res" else None, out_dtype=torch.float32 if f32 else torch.bfloat16)
  K.gemm_epilogue_mode(direct)
  try:
    got, want = K.gemm(a, b, bias=bias, **kw), K.gemm(a, b, bias=bias.clone(), **kw)
  finally:
    K.gemm_epilogue_mode(False)
  assert torch.equal(got, want)
  y = a.double() @ b.double().t() + bias.double()
  y = {"none": lambda: y, "gelu_tanh": lambda: torch.nn.functional.gelu(y, approximate="tanh"),
       "silu": lambda: torch.nn.functional.silu(y), "add_res": lambda: y + res.double()}[epi]()
  assert _rel(got, y) < (1e-3 if f32 else 4e-3)  # the approximate tanh and exponential; one rounding to bf16


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,lens", [(128, [65]), (257, [128]), (300, [192]), (130, [577]), (384, [64, 129, 200])])
def test_attention_when_the_maximum_moves(D, Sq, lens):
  """A block is exponentiated against the running maximum and again when its own is far above it: scores that grow from
  block to block for some rows, stay for others, over tails and segments. Probabilities and the output are rounded to bf16."""
  torch.manual_seed(11)
  q = _randn(2, Sq, 3, D)
  k = [_randn(2, n, 3, D) for n in lens]
  v = [_randn(2, n, 3, D) for n in lens]
  q[:, ::5] *= 0.05  # rows whose maximum hardly moves beside rows whose maximum does
  at = 0
  for x in k:
    x *= (1.0 + (torch.arange(x.shape[1], device="cuda") + at)[None, :, None, None] / 24).to(torch.bfloat16)
    at += x.shape[1]
  kk, vv = torch.cat(k, 1).double().transpose(1, 2), torch.cat(v, 1).double().transpose(1, 2)
  s = q.double().transpose(1, 2) @ kk.transpose(-1, -2) * D ** -0.5
  big = torch.zeros((2, at + max(lens), 3, D), device="cuda", dtype=torch.bfloat16)  # segments of one allocation share strides
  kb, vb = [], []
  for x, y in zip(k, v):
    kb.append(big.clone()[:, :x.shape[1]].copy_(x))
    vb.append(big.clone()[:, :y.shape[1]].copy_(y))
  got, lse = K.flash_fwd(q, kb, vb)
  assert _rel(got.transpose(1, 2), s.softmax(-1) @ vv) < 4e-3
  want = torch.logsumexp(s, -1) / 0.6931471805599453
  # sums of fp32 exponentials in the log2 domain, scores of up to a few hundred
  assert (lse.double() - want).abs().max() < 1e-5 * want.abs().max() + 1e-4


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("M,N,Kd", [(8, 8, 16), (136, 264, 144), (256, 640, 3072)])
def test_gelu_behind_an_8_bit_product(int8, M, N, Kd):
  """GELU in the epilogue is the GELU of the stored product: one rounding of the same value, so at most one unit of bf16 off
  where the two forms of tanh fall on different sides of a tie."""
  torch.manual_seed(12)
  quant = K.quantize_int8 if int8 else K.quantize_fp8
  (aq, sa), (bq, sb), bias = quant(_randn(M, Kd)), quant(_randn(N, Kd, scale=0.05)), _randn(N)
  y = (K.gemm_int8 if int8 else K.gemm_fp8)(aq, sa, bq, sb, bias)
  want = torch.nn.functional.gelu(y.double(), approximate="tanh")
  wide = torch.zeros((M, N + 72), device="cuda", dtype=torch.bfloat16)
  got = K.gemm8(aq, sa, bq, sb, bias, gelu=True, out=wide[:, 64:64 + N])
  assert ((got.double() - want).abs() <= want.abs() / 256 + 1e-6).all() and wide[:, :64].eq(0).all() and wide[:, 64 + N:].eq(0).all()
  assert torch.equal(K.gemm8(aq, sa, bq, sb, bias), y)


@pytest.mark.parametrize("mode", ["fp8", "int8"])
def test_quantised_linear_in_parts(mode):
  from maxdiffusion_b200.models.layers import Linear
  from maxdiffusion_b200.models.quantizations import Fp8Linear, Int8Linear, is_plain_quantized

  torch.manual_seed(13)
  m = (Int8Linear if mode == "int8" else Fp8Linear)(Linear(128, 400).to("cuda", torch.bfloat16))
  x = _randn(2, 12, 128)
  whole = m(x.detach().requires_grad_()).detach()  # through autograd
  with torch.no_grad():
    assert torch.equal(m(x), whole)
    cat = torch.zeros((2, 12, 80 + 160), device="cuda", dtype=torch.bfloat16)
    assert torch.equal(m.split_gelu(x, 240, cat[..., 80:]), whole[..., :240]) and cat[..., :80].eq(0).all()
    assert torch.equal(cat[..., 80:], m(x, "gelu_tanh")[..., 240:])
    assert m.split_gelu(x, 241, cat[..., 81:]) is None and m.split_gelu(x[:, :3, :], 240, cat[:, :3, 80:]) is None
  assert m.split_gelu(x, 240, cat[..., 80:]) is None  # the weight wants a gradient
  assert is_plain_quantized(m)
  m.register_forward_hook(lambda *a: None)
  assert not is_plain_quantized(m)


@pytest.mark.parametrize("shape,groups", [((2, 64, 8, 8), 32), ((1, 320, 17, 5), 32), ((3, 96, 1, 9), 3)])
def test_norm_of_sum_and_conv_with_a_residual(shape, groups):
  """The value per sample and channel enters the fold of GroupNorm's sums, the residual the convolution's epilogue; wrappers,
  hooks and other layouts take the separate additions. Oracle: float64."""
  from maxdiffusion_b200.models.layers import Conv2d, GroupNorm, conv_plus, norm_of_sum

  torch.manual_seed(14)
  N, C, H, W = shape
  cl = dict(memory_format=torch.channels_last)
  x, t = _randn(*shape).contiguous(**cl), _randn(N, C) * 3
  rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
  norm, conv = GroupNorm(groups, C, eps=1e-5).to("cuda", torch.bfloat16), Conv2d(C, 48, 3, padding=1).to("cuda", torch.bfloat16)
  one = Conv2d(C, 48, 1).to("cuda", torch.bfloat16)
  norm.weight.data.normal_(), norm.bias.data.normal_()
  res = _randn(N, 48, H, W).contiguous(**cl)
  F = torch.nn.functional
  with torch.no_grad():
    want = F.silu(F.group_norm(x.double() + t.double()[:, :, None, None], groups, norm.weight.double(), norm.bias.double(), 1e-5))
    assert rel(norm_of_sum(norm, x, t), want) < 4e-3  # one rounding to bf16
    assert rel(norm_of_sum(norm, x, t.t().contiguous().t()), want) < 8e-3  # another stride: x + t is rounded as well
    for m in (conv, one):
      y = F.conv2d(x.double(), m.weight.double(), m.bias.double(), padding=m.padding) + res.double()
      fused = conv_plus(m, x, res)
      assert rel(fused, y) < 4e-3 and fused.shape == y.shape
      assert rel(conv_plus(m, x, res.contiguous()), y) < 6e-3 and rel(conv_plus(m, x, res.float()), y) < 6e-3
      h = m.register_forward_hook(lambda mod, a, out: out * 0)
      assert torch.equal(conv_plus(m, x, res), res)  # a hook on the module sees the convolution alone
      h.remove()
  a, b = x.detach().requires_grad_(), t.detach().requires_grad_()
  norm_of_sum(norm, a, b).float().square().sum().backward()
  a64, b64 = x.double().requires_grad_(), t.double().requires_grad_()
  F.silu(F.group_norm(a64 + b64[:, :, None, None], groups, norm.weight.double(), norm.bias.double(), 1e-5)).square().sum().backward()
  assert rel(a.grad, a64.grad) < 3e-2 and rel(b.grad, b64.grad) < 3e-2  # bf16 gradients of a bf16 sum


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Sq,Skv,H", [(1, 1, 1, 1), (2, 64, 65, 3), (1, 129, 128, 2), (2, 300, 77, 2), (1, 577, 450, 4)])
def test_attention_backward_with_ds_kept(D, B, Sq, Skv, H, monkeypatch):
  """dQ from the dS that the pass over keys wrote, whole and a head at a time, against float64 and against the two passes."""
  torch.manual_seed(15)
  q, k, v, g = _randn(B, Sq, H, D), _randn(B, Skv, 2 * H, D)[:, :, ::2], _randn(B, Skv, H, D), _randn(B, H, Sq, D).transpose(1, 2)
  out, lse = K.flash_fwd(q, [k], [v])
  delta = K.flash_delta(out, g)
  dq, dk, dv = K.flash_bwd(q, g, k, v, lse, delta)
  monkeypatch.setattr(K, "_DS_BYTES", -(-Skv // 128) * -(-Sq // 64) * 16384)
  assert K.flash_ds_chunk(B, H, Sq, Skv) == 1
  assert all(torch.equal(a, b) for a, b in zip(K.flash_bwd(q, g, k, v, lse, delta), (dq, dk, dv)))
  monkeypatch.setattr(K, "_DS_BYTES", 0)  # no room: the two passes
  old = K.flash_bwd(q, g, k, v, lse, delta)
  assert torch.equal(old[1], dk) and torch.equal(old[2], dv) and torch.equal(old[0], K.flash_bwd_dq(q, g, [k], [v], lse, delta))
  qd, kd, vd = (t.double().transpose(1, 2).requires_grad_() for t in (q, k, v))
  y = ((qd @ kd.transpose(-1, -2)) * D ** -0.5).softmax(-1) @ vd
  y.backward(g.double().transpose(1, 2))
  if Skv > 1:  # one key: its probability is 1 and dS is rounding alone
    assert _rel(dq.transpose(1, 2), qd.grad) < 1.05 * _rel(old[0].transpose(1, 2), qd.grad) + 1e-4
    assert _rel(dk.transpose(1, 2), kd.grad) < 2e-2
  assert _rel(dv.transpose(1, 2), vd.grad) < 2e-2


@pytest.mark.parametrize("shape,groups", [((2, 64, 8, 8), 32), ((1, 320, 17, 5), 32), ((3, 96, 1, 9), 3), ((2, 640, 32, 32), 32), ((1, 1280, 31, 33), 32), ((2, 16, 1, 1), 8), ((2, 2560, 8, 8), 32), ((1, 2560, 32, 32), 32)])
@pytest.mark.parametrize("act,affine,shifted", [(True, True, True), (False, False, False)])
def test_group_norm_of_few_pixels(shape, groups, act, affine, shifted):
  """One launch with the group's values in shared memory (2, 4 or 8 channels a load), against float64 and the three launches."""
  from maxdiffusion_b200.ops import functional as OF

  torch.manual_seed(17)
  N, Ch, H, W = shape
  x = (_randn(*shape) * 2 + 30).contiguous(memory_format=torch.channels_last)  # a mean far above the deviation
  gamma, beta = (_randn(Ch), _randn(Ch)) if affine else (None, None)
  t = _randn(N, 2 * Ch)[:, Ch:] if shifted else None
  xs = x.double() + (t.double()[:, :, None, None] if shifted else 0.0)
  want = torch.nn.functional.group_norm(xs, groups, None if gamma is None else gamma.double(), None if beta is None else beta.double(), 1e-5)
  want = torch.nn.functional.silu(want) if act else want
  with torch.no_grad():
    got = OF.group_norm(x, groups, gamma, beta, 1e-5, act, t)
    rows = None if Ch > 2048 else C.group_norm_cl_fwd(x.permute(0, 2, 3, 1).reshape(N, H * W, Ch), groups, gamma, beta, 1e-5, act, t)[0]
  assert got.is_contiguous(memory_format=torch.channels_last)
  assert got.shape == x.shape
  if rows is None:
    assert _rel(got, want) < 4e-3
  elif H * W * Ch // groups > 2:  # two values: the deviation is rounding alone
    three = _rel(rows.view(N, H, W, Ch).permute(0, 3, 1, 2), want)
    assert _rel(got, want) < 4e-3 and _rel(got, want) < three + 1e-4
