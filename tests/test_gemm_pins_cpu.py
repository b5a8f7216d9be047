"""Pinned launch shapes of the GEMM (tile search, benchmarks): what cannot be pinned says so, and no product escapes a pin."""
import pytest
import torch

from maxdiffusion_b200.ops import _lib, functional as OF, kernels as K


@pytest.mark.parametrize("tile_n,ctas", [(64, 2), (192, 2)])
def test_a_pair_cannot_split_such_a_tile_of_a_transposed_b(tile_n, ctas):
  with pytest.raises(_lib.KernelError):
    K.gemm_plan(512, 512, 512, True, True, 148, tile_n, ctas)
  assert K.gemm_plan(512, 512, 512, False, True, 148, tile_n, ctas)[:2] == (ctas, tile_n)


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("tile_n", [0, 64, 128, 192, 256])
def test_a_single_pin_is_followed(tile_n, b_mn):
  plan = K.gemm_plan(512, 512, 512, b_mn, True, 148, tile_n, 0)
  assert tile_n in (0, plan[1]) and K.gemm_plan(512, 512, 512, b_mn, True, 148, 0, 2)[0] == 2


@pytest.mark.parametrize("pin", ["tile", "ctas", "epilogue"])
def test_fused_products_give_way_to_a_pin(monkeypatch, pin):
  asked = []

  class Host:
    def __getattr__(self, name):
      return lambda *a: (asked.append(name), NotImplemented)[1]

  monkeypatch.setattr(_lib, "host_ops", Host)
  monkeypatch.setattr(OF, "_direct", lambda *t: True)
  monkeypatch.setattr(OF, "linear", lambda x, w, b=None: x @ w.t())
  monkeypatch.setattr(OF, "geglu", lambda u: u)
  x, w = torch.zeros(2, 16), torch.zeros(16, 16)
  run = lambda: (monkeypatch.setattr(OF, "_fast", lambda t: True), OF.linear_group(x, (w, w)), OF.geglu_linear(x, w))
  run()
  assert asked == ["linear_group", "geglu_linear"]
  monkeypatch.setattr(K, {"tile": "_FORCE_TILE_N", "ctas": "_FORCE_CTAS", "epilogue": "_DIRECT_EPILOGUE"}[pin], 2)
  run()
  assert asked == ["linear_group", "geglu_linear"]


@pytest.mark.parametrize("M,N,Kd,b_mn,avoid", [(7000, 2048, 8192, False, (2, 256)), (640, 640, 16384, True, (2, 256))])
def test_a_nearly_empty_last_round_of_pairs_is_not_preferred(M, N, Kd, b_mn, avoid):
  assert K.gemm_plan(M, N, Kd, b_mn)[:2] != avoid


@pytest.mark.parametrize("M,N,Kd", [(4608, 9216, 3072), (65520, 5120, 5120), (32760, 5120, 13824)])
def test_large_products_run_on_wide_pairs(M, N, Kd):
  assert K.gemm_plan(M, N, Kd) == (2, 256, 1)
