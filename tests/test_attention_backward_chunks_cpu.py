"""How much of dS the attention backward holds at a time."""
from maxdiffusion_b200.ops import kernels as K


def test_ds_chunks():
  per = lambda sq, skv: -(-skv // 128) * -(-sq // 64) * 16384
  assert K.flash_ds_chunk(4, 20, 1024, 1024) == 80  # everything fits
  assert K.flash_ds_chunk(1, 40, 32760, 32760) == 4  # 7 rounds of 148 CTAs for 1024 blocks, where three heads take 6 for 768
  assert K.flash_ds_chunk(1, 40, 75600, 75600) == 0 and K.flash_ds_chunk(1, 2, 8, 0) == 0
  for B, H, sq, skv in ((2, 10, 4096, 77), (2, 24, 9000, 9000), (1, 7, 20000, 20000), (3, 5, 130, 257)):
    for limit in (per(sq, skv) - 1, per(sq, skv), 3 * per(sq, skv), 1 << 40):
      n = K.flash_ds_chunk(B, H, sq, skv, limit)
      assert n * per(sq, skv) <= limit and (n == B * H or n <= H) and (n > 0) == (limit >= per(sq, skv))
