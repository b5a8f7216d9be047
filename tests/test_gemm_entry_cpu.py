"""What the GEMM's C entry point refuses before it touches a GPU. The pointers are made up and never read."""
import ctypes

import pytest

from maxdiffusion_b200.ops import _lib

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
