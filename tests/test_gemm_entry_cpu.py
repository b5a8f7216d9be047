"""What the GEMM does without a GPU: what its C entry point refuses before it touches one (the pointers are made up and never
read), and products over nothing."""
import pytest
import torch
import torch.nn.functional as F

from maxdiffusion_b200.ops import _lib, kernels as K

ADDR = 1 << 20
NONE, GELU, GATED, SILU, ADD = range(5)


def _call(out=ADDR, residual=0, gate=0, epi=NONE, partial=0, splits=1, ldr=64):
  if not _lib.LIB_PATH.exists():
    pytest.skip("the kernel library is not built")
  return _lib.lib().mdb_gemm_bf16(ADDR, ADDR, out, 0, residual, gate, 128, 64, 64, 64, 64, 64, ldr, 64, 128, 0, 0, epi, 0, 1.0, 1, 64,
                                  splits, partial, 0)


@pytest.mark.parametrize("off", [2, 4, 8])
def test_pointers_that_cannot_be_read_16_bytes_at_a_time_are_refused(off):
  assert _call(out=ADDR + off) == 3006
  assert _call(residual=ADDR + off, epi=ADD) == 3006
  assert _call(residual=ADDR + off, gate=ADDR, epi=GATED) == 3006
  assert _call(residual=ADDR, gate=ADDR + off, epi=GATED) == 3006
  assert _call(partial=ADDR + off, splits=2) == 3006
  assert _call(residual=ADDR, epi=ADD, ldr=68) == 3002


@pytest.mark.parametrize("epi", ["none", "gelu_tanh", "silu", "add_res", "gated_res"])
def test_an_empty_contraction_is_the_epilogue_of_zero(epi):
  bf = lambda *s: torch.randn(s).to(torch.bfloat16)
  a, b, bias, res, gate = bf(6, 0), bf(8, 0), bf(8), bf(6, 8), torch.randn(2, 8)
  kw = dict(residual=res) if epi in ("add_res", "gated_res") else {}
  if epi == "gated_res":
    kw.update(gate=gate, rows_per_batch=3)
  row = bias.float().expand(6, 8)
  want = {"none": lambda: row, "gelu_tanh": lambda: F.gelu(row, approximate="tanh"), "silu": lambda: F.silu(row),
          "add_res": lambda: res + row, "gated_res": lambda: res + gate.repeat_interleave(3, 0) * row}[epi]()
  assert torch.equal(K.gemm(a, b, bias=bias, epi=epi, **kw), want.to(torch.bfloat16))
  if epi == "none":
    assert not K.gemm(a, b, out_dtype=torch.float32).any()
    assert torch.equal(K.gemm(a.t(), b.t(), a_mn=True, b_mn=True, bias=bias), want.to(torch.bfloat16))
  assert K.split_k_for(6, 8, 0) == 1 and K.gemm_plan(6, 8, 0)[2] == 1
  assert K.gemm(bf(0, 16), bf(8, 16)).shape == (0, 8) and K.gemm(bf(6, 16), bf(0, 16)).shape == (6, 0)
