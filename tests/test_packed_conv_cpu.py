"""Packed convolution weights can be saved with the module that keeps them, used or not."""
import copy
import pickle

import pytest
import torch

from maxdiffusion_b200.ops import conv as C


@pytest.mark.parametrize("trip", [lambda p: pickle.loads(pickle.dumps(p)), copy.deepcopy, copy.copy])
def test_round_trip_after_use(trip):
  pk = C.pack_conv2d(torch.randn(16, 16, 3, 3), torch.randn(16))
  arrays, group = pk.tap_arrays(), pk.row_group()
  got = trip(pk)
  assert torch.equal(got.w, pk.w) and got.taps == pk.taps and got.kind == pk.kind and got.row_group() == group == 3
  again = got.tap_arrays()
  assert list(again[0]) == list(arrays[0]) and list(again[1]) == list(arrays[1]) and again[2] == arrays[2]


def test_a_state_without_the_cache():
  pk = C.pack_conv2d(torch.randn(16, 16, 3, 3), None)
  old = C.PackedConv.__new__(C.PackedConv)
  old.__setstate__({k: v for k, v in pk.__dict__.items() if k != "_tap_cache"})  # as files of earlier versions have it
  assert old.row_group() == 3 and len(old.tap_arrays()) == 3
