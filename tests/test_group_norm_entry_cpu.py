"""Which calls the one-launch GroupNorm leaves to the other kernels: nothing is launched, so no GPU is needed."""
from maxdiffusion_b200.ops import _lib
from maxdiffusion_b200.ops import conv as C  # declares the entry point

ADDR = 1 << 20


def _call(N=2, HW=64, channels=1280, groups=32, x=ADDR, y=ADDR):
  return _lib.lib().mdb_gn_cl_group(x, y, N, HW, channels, groups, C._gn_splits(max(N, 1), HW), 1e-5, None, None, 0, None, 0, 1, None)


def test_calls_left_to_other_kernels():
  assert C._GN_ELSEWHERE == 3705
  assert _call(N=65536) == 3705 and _call(N=65536, channels=2560) == 3705  # the grid's second dimension
  assert _call(channels=1280 + 8, groups=56) == 3705  # an odd number of channels a group: 23
  assert _call(x=ADDR + 8) == 3705 and _call(y=ADDR + 8) == 3705
  assert _call(HW=385) == 3705 and _call(N=4, HW=205) == 3705 and _call(N=1, HW=65, channels=128, groups=1) == 3705  # slower: 30, 16, 16 KB
  assert _call(N=9, HW=1) == 3705  # 288 CTAs
  assert _call(HW=4096, channels=2560, groups=1280) == 3705  # channels cut into several sums
  assert _call(HW=2048, channels=2560) == 3705  # more than shared memory holds
  assert _call(groups=33) == 3704 and _call(channels=1284, groups=2) == 3704
  assert _call(N=0) == 0 and _call(HW=0) == 0
