"""Kernels whose registers are all taken keep nothing in local memory."""
import re

import pytest

from maxdiffusion_b200 import build


@pytest.mark.parametrize("source", ["flash_fwd", "flash_bwd", "gemm_tcgen05", "conv_igemm"])
def test_tensor_core_kernels_do_not_spill(source):
  log = build.OBJ_DIR / f"{source}.ptxas.log"
  if not log.exists():
    pytest.skip("the kernel library was not built here")
  found = re.findall(r"Compiling entry function '(\w+)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads", log.read_text(), re.S)
  assert found and [f for f in found if f[1:] != ("0", "0")] == []
