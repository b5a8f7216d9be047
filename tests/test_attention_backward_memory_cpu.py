"""What the attention backward does where the memory for dS is short: the allocator and the kernels are stand-ins."""
import pytest
import torch

from maxdiffusion_b200.ops import _lib
from maxdiffusion_b200.ops import kernels as K

H, S = 8, 130
PER = -(-S // 128) * -(-S // 64) * 16384  # dS of a head


@pytest.fixture
def world(monkeypatch):
  """Records requests for memory and launches. `most`: bytes that a request may have; `room`: what `_ds_room` says."""

  class World:
    most, room, retries, asked, launched = 1 << 60, 1 << 60, 0, [], []

  w = World()
  w.asked, w.launched = [], []
  empty = torch.empty

  def limited(*args, **kw):
    t = empty(*args, **kw)
    w.asked.append((str(t.dtype), t.numel() * t.element_size()))
    if t.dtype == torch.uint8 and t.numel() > w.most:
      raise torch.OutOfMemoryError("no memory")
    return t

  monkeypatch.setattr(torch, "empty", limited)
  monkeypatch.setattr(K, "_flash_entry", lambda name, d: lambda *args: w.launched.append(name) or 0)
  monkeypatch.setattr(_lib, "stream", lambda: 0)
  monkeypatch.setattr(K, "_ds_room", lambda device, enough: w.room, raising=False)
  monkeypatch.setattr(K, "_ds_stats", lambda device: (0, w.retries), raising=False)
  monkeypatch.setattr(K, "_ds_pays", lambda *a: True, raising=False)
  monkeypatch.setattr(K, "_ds_refused", {}, raising=False)
  monkeypatch.setattr(K, "_ds_flushed", {}, raising=False)
  return w


def _backward():
  q = torch.zeros(1, S, H, 64, dtype=torch.bfloat16)
  out = K.flash_bwd(q, q, q, q, torch.zeros(1, H, S), torch.zeros(1, H, S))
  assert [t.shape for t in out] == [q.shape] * 3


def _ds(w):
  return [n for dtype, n in w.asked if dtype == "torch.uint8"]


def test_the_results_are_allocated_before_ds(world):
  _backward()
  assert [dtype for dtype, _ in world.asked] == ["torch.bfloat16"] * 3 + ["torch.uint8"]
  assert world.launched == ["mdb_flash_bwd_dkv_ds", "mdb_flash_dq_from_ds"]


def test_a_refusal_is_remembered_until_there_is_more_memory(world):
  world.most, world.room = 0, 100 << 30
  _backward()
  first = len(_ds(world))
  assert first >= 1 and world.launched == ["mdb_flash_bwd_dq", "mdb_flash_bwd_dkv"]
  for _ in range(3):
    _backward()
  assert len(_ds(world)) - first <= 3 and max(_ds(world)[first:], default=0) < max(_ds(world))  # nothing of that size again
  world.most, world.room = 1 << 60, 200 << 30
  _backward()
  assert world.launched[-2:] == ["mdb_flash_bwd_dkv_ds", "mdb_flash_dq_from_ds"]


def test_fewer_heads_before_giving_up(world):
  world.most = 3 * PER
  _backward()
  assert _ds(world)[0] == H * PER and _ds(world)[-1] <= 3 * PER and world.launched.count("mdb_flash_bwd_dkv_ds") > 1
  assert "mdb_flash_bwd_dq" not in world.launched


def test_a_large_buffer_is_asked_for_only_where_the_memory_is(world, monkeypatch):
  monkeypatch.setattr(K, "_DS_TEMPORARY", 0, raising=False)
  world.room = (1 << 30) + PER - 1
  _backward()
  assert _ds(world) == [] and world.launched == ["mdb_flash_bwd_dq", "mdb_flash_bwd_dkv"]


def test_requests_that_make_the_allocator_flush_are_not_repeated(world, monkeypatch):
  monkeypatch.setattr(K, "_DS_TEMPORARY", 0, raising=False)
  world.room = 100 << 30

  def stats(device):  # looked at before a request and after it: it has made the allocator flush
    world.retries += 1
    return 0, world.retries

  monkeypatch.setattr(K, "_ds_stats", stats, raising=False)
  for _ in range(4):
    _backward()
  assert _ds(world)[:2] == [H * PER] * 2 and max(_ds(world)[2:], default=0) < H * PER  # the first may have left a block for the second
