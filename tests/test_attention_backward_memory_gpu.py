"""The attention backward on a GPU whose memory is short, and inside a captured graph: the bits of the plain call."""
import pytest
import torch

from maxdiffusion_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _inputs(B, S, H, D):
  torch.manual_seed(4)
  q, k, v, g = (torch.randn(B, S, H, D, device="cuda").to(torch.bfloat16) for _ in range(4))
  out, lse = K.flash_fwd(q, [k], [v])
  return q, g, k, v, lse, K.flash_delta(out, g)


def test_memory_that_does_not_hold_ds(monkeypatch):
  """The process may take 300 MiB more; the results take 35 and dS of all heads 282: refused once, then what fits."""
  monkeypatch.setattr(K, "_ds_refused", {})
  monkeypatch.setattr(K, "_ds_pays", lambda *a: True)
  args = _inputs(1, 3000, 16, 128)
  want = K.flash_bwd(*args)
  torch.cuda.empty_cache()
  device = torch.device("cuda", torch.cuda.current_device())
  total = torch.cuda.mem_get_info(device)[1]
  torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(device) + (300 << 20)) / total, device)
  try:
    got = K.flash_bwd(*args)
    ooms = torch.cuda.memory_stats(device)["num_ooms"]
    again = [K.flash_bwd(*args) for _ in range(3)]
    assert torch.cuda.memory_stats(device)["num_ooms"] == ooms and K._ds_refused
  finally:
    torch.cuda.set_per_process_memory_fraction(1.0, device)
  for one in (got, *again):
    assert all(torch.equal(a, b) for a, b in zip(one, want))


@pytest.mark.parametrize("most", [1 << 30, 0])
def test_inside_a_captured_graph(monkeypatch, most):
  """With dS in the graph's pool, and without."""
  monkeypatch.setattr(K, "_DS_CAPTURED", most)
  args = _inputs(2, 700, 4, 64)
  want = K.flash_bwd(*args)
  side = torch.cuda.Stream()
  side.wait_stream(torch.cuda.current_stream())
  with torch.cuda.stream(side):
    K.flash_bwd(*args)
  torch.cuda.current_stream().wait_stream(side)
  graph = torch.cuda.CUDAGraph()
  with torch.cuda.graph(graph):
    got = K.flash_bwd(*args)
  for _ in range(2):
    for t in got:
      t.zero_()
    graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_whole_and_in_parts_are_the_same_bits(monkeypatch):
  args = _inputs(2, 577, 4, 128)
  per = -(-577 // 128) * -(-577 // 64) * 16384
  want = (K.flash_bwd_dq(args[0], args[1], [args[2]], [args[3]], args[4], args[5]), *K.flash_bwd_dkv(*args))
  for pairs in (8, 4, 3, 1):
    monkeypatch.setattr(K, "flash_ds_chunk", lambda *a, n=pairs: n)
    monkeypatch.setattr(K, "_ds_pays", lambda *a: True)
    assert all(torch.equal(a, b) for a, b in zip(K.flash_bwd(*args), want))
