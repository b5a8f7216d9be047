// Convolution as an implicit GEMM on sm_100a (tcgen05 + TMEM + TMA), channels-last, bf16 in / fp32 accumulate.
//
//     Y[pixel, co] = epilogue( sum_{tap, ci} X[pixel + shift(tap), ci] * W[co, tap, ci] )
//
// There is no im2col buffer and no gather pass. The activation tensor is described to TMA as a 5-D array
// (channels innermost) and an M-tile is a BOX of 128 output positions (e.g. 4 rows x 32 columns of one frame).
// The A operand of one (tap, channel block) step is that box fetched at coordinates shifted by the tap's offset:
// positions that fall outside the tensor are filled with zeros by TMA, which is exactly the zero padding of the
// convolution, and the box lands in shared memory as a K-major, 128-byte-swizzled 128 x 64 tile that `tcgen05.mma`
// consumes directly. The weights are a plain K-major matrix [Cout, taps * Cpad]. Everything that distinguishes one
// convolution from another is a table of tap offsets prepared on the host:
//   * 3x3x3 causal conv3d: 27 taps over (t, h, w); a tap that reaches before the chunk's first frame reads the
//     2-frame history ("feature cache") through a second tensor map, or zeros when there is none;
//   * 3x3 / 1x1 conv2d, (3,1,1) time convolution: the same with fewer taps;
//   * stride 2: the input is viewed as [.., H/2, 2, W/2, 2*C], so that a tap becomes (row pair, parity, column pair,
//     parity * C + channel) and the box stays dense;
//   * nearest-2x upsample + 3x3 conv: four output-parity classes, each a 2x2 convolution of the LOW resolution
//     input with pre-summed weights (2.25x fewer FLOPs than up-sampling first), written with stride 2.
// Neighbouring taps along the width read almost the same positions. When a tile is 128 positions of one row (`group` taps
// wide), the row is fetched once with the spare columns of all of them, and tap j's operand starts j rows (128 bytes each)
// further in shared memory: the fetched positions of a 3x3 kernel fall to a third. 96 -> 96 channels at 4 x 480 x 832: 22 KB
// per 192 tensor clocks become 11.7 KB, 943 us become 678 us.
// Roles per CTA (persistent): warp 0 TMA producer, warp 1 TMEM owner + MMA issuer, warps 2..5 epilogue
// (bias, SiLU, residual add, ragged-edge masking). Accumulators are double buffered in TMEM.
//
// What bounds it is the operand feed from L2 (about 57 bytes per clock and SM on every shape): a 128 x 96 tile of one CTA
// needs 28 KB per 192 tensor clocks. So two neighbouring M-tiles are computed by a PAIR of CTAs (`cta_group::2`), each
// fetching its own box of positions and half of the weights, and draining its own 128 accumulator rows.
// A product with too few tiles for the chip (the low-resolution stages of a UNet) is cut along the contraction into
// `splits` work items with fp32 partials, which a second kernel sums in order and finishes (bias, SiLU, residual).
// Channel counts that are not multiples of 64 (96, 192, 320) cost no tensor work: the last channel block is
// fetched with zero fill and only its valid 16-wide K steps are issued.
// The lane that issues the MMAs pays a fixed price per pipeline stage (barrier wait, fence, commit: several hundred
// cycles) besides the price per instruction, and with few output channels (N <= 128) a stage of one 64-channel block
// holds less tensor work than that. Narrow tiles therefore put TWO (tap, channel block) units into a stage.
//
// Replaces the XLA:GPU / cuDNN convolutions behind the reference's `WanCausalConv3d`, `WanResample`,
// `WanResidualBlock` (src/maxdiffusion/models/wan/autoencoder_kl_wan.py:70-147, 245-389, 452-484) and the UNet /
// VAE `nn.Conv` layers (src/maxdiffusion/models/resnet_flax.py:37-186).
#include "host_common.h"

namespace mdb {
namespace conv {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int NUM_THREADS = 192;
constexpr int MAX_STAGES = 6;
constexpr int MAX_TAPS = 36;      // 27 (3x3x3) or 4 classes x 9
constexpr int MAX_CLASSES = 4;
// TMEM columns per accumulator: 256 (two accumulators = all 512 columns, one CTA per SM) for wide tiles, 128 for
// tiles of at most 128 output channels, which run TWO CTAs per SM (256 columns and half the shared memory each).
// A narrow tile holds little tensor work per pipeline stage; two co-resident CTAs overlap one's waits and epilogue with
// the other's products, each tile still accumulated by one thread in a fixed order (bitwise reproducible).

struct Tap {
  int o0;              // added to the channel coordinate (parity * C in the stride-2 view, else 0)
  short o1, o2, o3, o4;  // added to the tile's base coordinates along dims 1..4
  int koff;            // first K index of this tap in the weight matrix
};

// Flags; kEpiRoundFirst: a residual is added to the result as bf16 holds it.
enum Epilogue : int { kEpiNone = 0, kEpiSilu = 1, kEpiRoundFirst = 2 };

struct Params {
  int n_classes;
  int tap_begin[MAX_CLASSES + 1];
  Tap taps[MAX_TAPS];
  int box1, box2, box3;          // tile extents along dims 1..3, product 128
  int ext1, ext2, ext3, ext4;    // output positions along dims 1..4 (per class)
  int C;                         // input channels, multiple of 16
  int N;                         // output channels, multiple of 8
  int BN;                        // tile width: multiple of 16, <= 256
  int stages;
  int ups;                       // (tap group, channel block) units per pipeline stage: 1 or 2
  int group;                     // taps that share a fetched row: 1, 2 or 3 (more than 1 only with boxes of one row)
  int a_bytes;                   // shared memory of a unit's positions: (128 + group - 1) rows, a multiple of 1024
  int acc_cols;                  // TMEM columns per accumulator: 128 or 256
  int alt_dim, alt_shift, has_alt;  // a tap whose coordinate along alt_dim is negative reads the second map at +alt_shift
  long long os1, os2, os3, os4;  // output strides (elements) along dims 1..4
  long long class_off[MAX_CLASSES];
  __nv_bfloat16* out;
  const __nv_bfloat16* bias;      // [N] or nullptr
  const __nv_bfloat16* residual;  // addressed like out, or nullptr
  int epi;
  int tap_step;                   // K index distance of the taps of a group
  int splits;                     // > 1: fp32 partials [splits][class, M-tile, 128 positions][N] instead of the output
  float* partial;
  DeviceStatus* status;
};

struct TileCoord {
  int cls, n_idx, m1, m2, m3, m4;
  int mt;         // M-tile within the class
  bool in_range;  // false: the second half of a pair that covers the class's odd last M-tile
};

// First (tap, channel block) unit of work item `split`: the units are cut into ranges that differ by at most one. A whole
// contraction goes without the divisions here and in `split_of`, which a tile of few steps feels: three taps in time at
// 2 x 240 x 416 x 96 35.9 us with 64-bit divisions, 34.6 so; 3x3 at 256 x 256, 128 -> 8 11.5 / 11.0 us.
__device__ __forceinline__ int unit_cut(int split, int splits, int units) {
  return splits == 1 ? split * units : units * split / splits;  // at most 36 taps of 128 blocks times 64 parts
}
__device__ __forceinline__ int split_of(int work, int splits, int num_tiles) { return splits == 1 ? 0 : work / num_tiles; }

// Epilogue of 8 channels of one output position: bias, SiLU, residual, store. With kEpiRoundFirst the bits are those of a
// convolution whose result is stored and added in a pass of its own.
__device__ __forceinline__ void finish8(float (&x)[8], const Params& p, long long off, int col) {
  if (p.bias) {
    const uint4 bv = *reinterpret_cast<const uint4*>(p.bias + col);
    const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = unpack_bf16x2(bw[j]);
      x[2 * j] += f.x;
      x[2 * j + 1] += f.y;
    }
  }
  if (p.epi & kEpiSilu) {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = x[j] / (1.0f + __expf(-x[j]));
  }
  if (p.residual) {
    if (p.epi & kEpiRoundFirst) {
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = __bfloat162float(__float2bfloat16(x[j]));
    }
    const uint4 rv = *reinterpret_cast<const uint4*>(p.residual + off + col);
    const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = unpack_bf16x2(rw[j]);
      x[2 * j] += f.x;
      x[2 * j + 1] += f.y;
    }
  }
  uint4 ov;
  ov.x = pack_bf16x2(x[0], x[1]);
  ov.y = pack_bf16x2(x[2], x[3]);
  ov.z = pack_bf16x2(x[4], x[5]);
  ov.w = pack_bf16x2(x[6], x[7]);
  *reinterpret_cast<uint4*>(p.out + off + col) = ov;
}

// M-tiles of a class, in coordinates.
__device__ __forceinline__ void decode_m(int mt, const Params& p, int nt1, int nt2, int nt3, TileCoord& c) {
  c.mt = mt;
  c.m1 = (mt % nt1) * p.box1; mt /= nt1;
  c.m2 = (mt % nt2) * p.box2; mt /= nt2;
  c.m3 = (mt % nt3) * p.box3; mt /= nt3;
  c.m4 = mt;  // == ext4 for the tile after the last: its boxes lie outside the tensor and are filled with zeros
}

template <int CG>
__device__ __forceinline__ TileCoord decode_tile(int tile, int rank, const Params& p, int nt1, int nt2, int nt3, int num_mt,
                                                 int num_n) {
  TileCoord c;
  const int num_mp = (num_mt + CG - 1) / CG;
  c.n_idx = tile % num_n; tile /= num_n;
  c.cls = tile / num_mp;
  decode_m((tile - c.cls * num_mp) * CG + rank, p, nt1, nt2, nt3, c);
  c.in_range = c.mt < num_mt;
  return c;
}

// ROWS: taps may share a fetched row. A kernel of its own, because the issuing lane pays for a loop over one tap: 4 x 30 x 52,
// 192 -> 384 39.9 / 37.2 us with the loop / without, 3 x 33 x 57, 96 -> 96 26.0 / 24.6 us.
template <int CG, bool ROWS>
__global__ void __cluster_dims__(CG, 1, 1) __launch_bounds__(NUM_THREADS, 2)
conv_igemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_alt,
                  const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int STAGES = p.stages;
  const int B_BYTES = p.BN / CG * BK * 2;     // this CTA's share of the weights
  const int GROUP = ROWS ? p.group : 1;
  const int UNIT_BYTES = p.a_bytes + GROUP * B_BYTES;  // a multiple of 1024: BN / CG is a multiple of 8
  const int UNIT_TX = (BM + GROUP - 1) * 128 + GROUP * B_BYTES;  // bytes that a unit's copies deliver
  const int STAGE_BYTES = p.ups * UNIT_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full_bar = bars;                          // [MAX_STAGES]; of a pair: only the even CTA's are used
  uint64_t* empty_bar = bars + MAX_STAGES;            // [MAX_STAGES]
  uint64_t* tmem_full = bars + 2 * MAX_STAGES;        // [2]
  uint64_t* tmem_empty = bars + 2 * MAX_STAGES + 2;   // [2]; of a pair: only the even CTA's are used
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nt1 = (p.ext1 + p.box1 - 1) / p.box1;
  const int nt2 = (p.ext2 + p.box2 - 1) / p.box2;
  const int nt3 = (p.ext3 + p.box3 - 1) / p.box3;
  const int num_n = (p.N + p.BN - 1) / p.BN;
  const int num_mt = p.ext4 * nt3 * nt2 * nt1;
  const int num_tiles = p.n_classes * ((num_mt + CG - 1) / CG) * num_n;
  const int num_work = num_tiles * p.splits;
  const int num_kb = (p.C + BK - 1) / BK;
  const int rank = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const int group_id = static_cast<int>(blockIdx.x) / CG, num_groups = static_cast<int>(gridDim.x) / CG;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], CG * 4);  // the epilogue warps (of both CTAs)
    }
    *abort_flag = 0;
    fence_mbar_init();
    prefetch_tensormap(&tmap_x);
    prefetch_tensormap(&tmap_w);
  }
  const int ACC_COLS = p.acc_cols;
  if (warp == 1) {
    if (CG == 2) {
      tmem_alloc_pair(tmem_ptr_smem, 2 * ACC_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_ptr_smem, 2 * ACC_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (CG == 2) cluster_sync();  // the partner's barriers are initialised and its TMEM is allocated
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  allow_successor();
  wait_for_predecessor();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      bool ok = true;
      for (int work = group_id; work < num_work && ok; work += num_groups) {
        const int split = split_of(work, p.splits, num_tiles);
        const TileCoord tc = decode_tile<CG>(work - split * num_tiles, rank, p, nt1, nt2, nt3, num_mt, num_n);
        const int n0 = tc.n_idx * p.BN + rank * (p.BN / CG);
        const int t0 = p.tap_begin[tc.cls];
        const int all_units = (p.tap_begin[tc.cls + 1] - t0) / GROUP * num_kb;
        const int u_begin = unit_cut(split, p.splits, all_units), n_units = unit_cut(split + 1, p.splits, all_units);
        int ti = t0 + u_begin / num_kb * GROUP, kb = u_begin % num_kb;
        Tap tap = p.taps[min(ti, MAX_TAPS - 1)];
        for (int u0 = u_begin; u0 < n_units && ok; u0 += p.ups) {
          const int nu = min(p.ups, n_units - u0);
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag, p.status, 110)) { ok = false; break; }
          // both CTAs' copies complete on the even CTA's barrier, which expects the bytes of both
          if (rank == 0) mbar_expect_tx(&full_bar[stage], CG * nu * UNIT_TX);
          const uint32_t pair_bar = CG == 2 ? cluster_map(&full_bar[stage], 0) : 0u;
          uint8_t* sa = smem + stage * STAGE_BYTES;
          for (int j = 0; j < nu; ++j, sa += UNIT_BYTES) {
            int c1 = tc.m1 + tap.o1, c2 = tc.m2 + tap.o2, c3 = tc.m3 + tap.o3, c4 = tc.m4 + tap.o4;
            const CUtensorMap* map = &tmap_x;
            if (p.has_alt) {
              // a tap that reaches before the first position along alt_dim reads the history tensor instead
              if (p.alt_dim == 3 && c3 < 0) { c3 += p.alt_shift; map = &tmap_alt; }
              else if (p.alt_dim == 2 && c2 < 0) { c2 += p.alt_shift; map = &tmap_alt; }
            }
            if (CG == 2) {
              tma_load_5d_pair(sa, map, pair_bar, tap.o0 + kb * BK, c1, c2, c3, c4);
              for (int g = 0; g < GROUP; ++g)
                tma_load_2d_pair(sa + p.a_bytes + g * B_BYTES, &tmap_w, pair_bar, tap.koff + g * p.tap_step + kb * BK, n0);
            } else {
              tma_load_5d(sa, map, &full_bar[stage], tap.o0 + kb * BK, c1, c2, c3, c4);
              for (int g = 0; g < GROUP; ++g)
                tma_load_2d(sa + p.a_bytes + g * B_BYTES, &tmap_w, &full_bar[stage], tap.koff + g * p.tap_step + kb * BK, n0);
            }
            if (++kb == num_kb) {
              kb = 0;
              ti += GROUP;
              if (ti < p.tap_begin[tc.cls + 1]) tap = p.taps[ti];
            }
          }
          ++issued;
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        // Give the copies already in flight a bounded chance to land before the CTA exits. The odd CTA of a pair has no
        // barrier of its own to look at: it gives its copies a fixed time.
        const int pending = issued < STAGES ? issued : STAGES;
        for (int i = 0; i < pending && rank == 0; ++i) {
          int s = (stage - 1 - i + 2 * STAGES) % STAGES;
          uint32_t ph = (i < stage) ? phase : (phase ^ 1u);
          for (int spin = 0; spin < (1 << 16) && !mbar_try_wait(&full_bar[s], ph); ++spin) {}
        }
        for (int i = 0; i < 100 && CG == 2; ++i) __nanosleep(10000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (of a pair: in the even CTA) ----
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(CG * BM, p.BN, false, false);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int work = group_id; work < num_work && ok; work += num_groups, ++it) {
        const int split = split_of(work, p.splits, num_tiles);
        const int cls = (work - split * num_tiles) / (num_tiles / p.n_classes);
        const int n_taps = (p.tap_begin[cls + 1] - p.tap_begin[cls]) / GROUP;
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1u;
        if (!mbar_wait(&tmem_empty[acc], acc_phase ^ 1u, abort_flag, p.status, 120)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
        uint32_t accumulate = 0;
        const int u_begin = unit_cut(split, p.splits, n_taps * num_kb), n_units = unit_cut(split + 1, p.splits, n_taps * num_kb);
        // this lane is the critical resource of the kernel: no divisions, descriptors advance by addition
        const int last_ksteps = (p.C - (num_kb - 1) * BK + 15) / 16;
        int kb = u_begin % num_kb;
        for (int u0 = u_begin; u0 < n_units; u0 += p.ups) {
          const int nu = min(p.ups, n_units - u0);
          if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, 121)) { ok = false; break; }
          tc_fence_after_sync();
          uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          for (int j = 0; j < nu; ++j, sa += UNIT_BYTES) {
            const bool last = (kb + 1 == num_kb);
            for (int g = 0; g < GROUP; ++g) {
              // the 128-byte swizzle follows the address, so an operand may start at any row of the fetched tile
              const uint64_t da = make_smem_desc(sa + g * 128, 16, 1024);
              const uint64_t db = make_smem_desc(sa + p.a_bytes + g * B_BYTES, 16, 1024);
              // one K step (16 bf16 = 32 bytes) advances the descriptors' address field (units of 16 bytes) by 2
              if (CG == 2) {
                if (!last || last_ksteps == BK / 16) {
                  umma_ss_pair(d_tmem, da, db, idesc, accumulate);
                  umma_ss_pair(d_tmem, da + 2, db + 2, idesc, 1u);
                  umma_ss_pair(d_tmem, da + 4, db + 4, idesc, 1u);
                  umma_ss_pair(d_tmem, da + 6, db + 6, idesc, 1u);
                } else {
                  for (int k = 0; k < last_ksteps; ++k) umma_ss_pair(d_tmem, da + 2 * k, db + 2 * k, idesc, k ? 1u : accumulate);
                }
              } else if (!last || last_ksteps == BK / 16) {
                umma_ss(d_tmem, da, db, idesc, accumulate);
                umma_ss(d_tmem, da + 2, db + 2, idesc, 1u);
                umma_ss(d_tmem, da + 4, db + 4, idesc, 1u);
                umma_ss(d_tmem, da + 6, db + 6, idesc, 1u);
              } else {
                for (int k = 0; k < last_ksteps; ++k) umma_ss(d_tmem, da + 2 * k, db + 2 * k, idesc, k ? 1u : accumulate);
              }
              accumulate = 1u;
            }
            kb = last ? 0 : kb + 1;
          }
          if (CG == 2) umma_commit_pair(&empty_bar[stage]);
          else umma_commit(&empty_bar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok) {
          if (CG == 2) umma_commit_pair(&tmem_full[acc]);
          else umma_commit(&tmem_full[acc]);
        }
      }
    }
  } else {
    // ------------------------------ Epilogue ----------------------------------
    const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 are reachable from this warp
    const int r = quarter * 32 + lane;
    const int r1 = r % p.box1;
    const int r2 = (r / p.box1) % p.box2;
    const int r3 = r / (p.box1 * p.box2);
    int it = 0;
    bool ok = true;
    for (int work = group_id; work < num_work && ok; work += num_groups, ++it) {
      const int split = split_of(work, p.splits, num_tiles);
      const TileCoord tc = decode_tile<CG>(work - split * num_tiles, rank, p, nt1, nt2, nt3, num_mt, num_n);
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1u;
      if (!mbar_wait(&tmem_full[acc], acc_phase, abort_flag, p.status, 130)) { ok = false; break; }
      tc_fence_after_sync();
      const int p1 = tc.m1 + r1, p2 = tc.m2 + r2, p3 = tc.m3 + r3;
      const bool row_ok = tc.in_range && p1 < p.ext1 && p2 < p.ext2 && p3 < p.ext3;
      const long long off = tc.m4 * p.os4 + p3 * p.os3 + p2 * p.os2 + p1 * p.os1 + p.class_off[tc.cls];
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * ACC_COLS;
      const int n0 = tc.n_idx * p.BN;
#pragma unroll 1
      for (int c = 0; c < p.BN / 16; ++c) {
        const int col0 = n0 + c * 16;
        if (col0 >= p.N) break;  // uniform across the CTA
        uint32_t v[16];
        tmem_ld_x16(taddr + c * 16, v);
        tmem_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int col = col0 + h * 8;
            if (col >= p.N) break;
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(v[h * 8 + j]);
            if (p.splits > 1) {
              float* o = p.partial +
                         ((static_cast<long long>(split) * p.n_classes + tc.cls) * num_mt + tc.mt) * BM * p.N +
                         static_cast<long long>(r) * p.N + col;
              *reinterpret_cast<float4*>(o) = make_float4(x[0], x[1], x[2], x[3]);
              *reinterpret_cast<float4*>(o + 4) = make_float4(x[4], x[5], x[6], x[7]);
            } else {
              finish8(x, p, off, col);
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_cluster(cluster_map(&tmem_empty[acc], 0));
        else mbar_arrive(&tmem_empty[acc]);
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (CG == 2) cluster_sync();  // neither CTA leaves while the other's products or arrivals still reach into it
  if (warp == 1) {
    tc_fence_after_sync();
    if (CG == 2) tmem_dealloc_pair(tmem_base, 2 * ACC_COLS);
    else tmem_dealloc(tmem_base, 2 * ACC_COLS);
  }
}

// Sum of the partials of a split contraction, in split order, and the epilogue. One thread per 8 channels of a position.
__global__ void conv_fold_kernel(const __grid_constant__ Params p) {
  allow_successor();
  wait_for_predecessor();
  const int nt1 = (p.ext1 + p.box1 - 1) / p.box1, nt2 = (p.ext2 + p.box2 - 1) / p.box2, nt3 = (p.ext3 + p.box3 - 1) / p.box3;
  const int num_mt = p.ext4 * nt3 * nt2 * nt1;
  const int n_vec = p.N / 8;
  const long long rows = static_cast<long long>(p.n_classes) * num_mt * BM;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < rows * n_vec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long row = i / n_vec;
    const int col = static_cast<int>(i - row * n_vec) * 8;
    const int r = static_cast<int>(row % BM);
    TileCoord tc;
    tc.cls = static_cast<int>(row / BM / num_mt);
    decode_m(static_cast<int>(row / BM % num_mt), p, nt1, nt2, nt3, tc);
    const int p1 = tc.m1 + r % p.box1, p2 = tc.m2 + (r / p.box1) % p.box2, p3 = tc.m3 + r / (p.box1 * p.box2);
    if (p1 >= p.ext1 || p2 >= p.ext2 || p3 >= p.ext3) continue;
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = 0; s < p.splits; ++s) {
      const float4* src = reinterpret_cast<const float4*>(p.partial + (s * rows + row) * p.N + col);
      const float4 a = src[0], b = src[1];
      x[0] += a.x; x[1] += a.y; x[2] += a.z; x[3] += a.w;
      x[4] += b.x; x[5] += b.y; x[6] += b.z; x[7] += b.w;
    }
    finish8(x, p, tc.m4 * p.os4 + p3 * p.os3 + p2 * p.os2 + p1 * p.os1 + p.class_off[tc.cls], col);
  }
}

// Tile width for N output channels: the multiple of `step` (16; 32 for a pair) up to `most` that wastes the fewest padded
// columns, the widest among equals (a wider tile moves fewer operand bytes per FLOP).
static int pick_bn(int N, int most, int step) {
  int best = step;
  long long best_cost = -1;
  for (int bn = step; bn <= most; bn += step) {
    const long long cost = static_cast<long long>((N + bn - 1) / bn) * bn;
    if (best_cost < 0 || cost < best_cost || (cost == best_cost && bn > best)) {
      best = bn;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace conv
}  // namespace mdb

// Tuning overrides for the tile search and the benchmarks (0 = the launcher's own choice): units per stage (1 / 2),
// an upper limit on the pipeline stages, CTAs per SM (1 / 2; 2 only applies to tiles of at most 128 channels).
static int g_tune_ups = 0, g_tune_stages = 0, g_tune_ctas = 0;

extern "C" int mdb_conv_igemm_tune(int ups, int stages, int ctas_per_sm) {
  if (ups < 0 || ups > 2 || stages < 0 || stages > 6 || ctas_per_sm < 0 || ctas_per_sm > 2) return 3609;
  g_tune_ups = ups;
  g_tune_stages = stages;
  g_tune_ctas = ctas_per_sm;
  return 0;
}

// Generic entry point; `ops/conv.py` builds the descriptions for the concrete convolutions.
//   x / x_alt : activation tensor and optional history tensor, both seen as 5-D arrays with `dims` / `alt_dims`
//               (innermost first, dim 0 = channels, contiguous) and element strides `strides` / `alt_strides` of dims 1..4
//   w         : [N, k_total] bf16, row-major (K-major); the K range of tap i starts at taps[i].koff and spans Cpad
//   box       : tile extents along dims 1..3 (product 128);  ext: output positions along dims 1..4
//   taps      : n_taps_total x 6 ints (o0, o1, o2, o3, o4, koff);  tap_begin: n_classes + 1 ints
//   out_strides (dims 1..4, elements), class_off (n_classes): where output position (p1..p4) of a class goes
//   epi: flags of `Epilogue`
//   group: taps that share a fetched row (consecutive in the table, one step along dim 1 apart; box[0] = 128)
//   ctas_per_tile (1 / 2), max_bn (widest tile), splits: the launch shape (`ops/conv.py: conv_plan`); with splits > 1
//   `partial` holds splits * n_classes * M-tiles * 128 * N fp32 values
// All channel counts and strides must keep 16-byte alignment (multiples of 8 elements); C a multiple of 16.
extern "C" int mdb_conv_igemm(const void* x, const void* x_alt, const void* w, void* out, const void* bias,
                              const void* residual, const long long* dims, const long long* strides,
                              const long long* alt_dims, const long long* alt_strides, const int* box, const int* ext,
                              int C, int N, long long k_total, int n_classes, const int* tap_begin, const int* taps,
                              int alt_dim, int alt_shift, const long long* out_strides, const long long* class_off,
                              int epi, int ctas_per_tile, int max_bn, int splits, void* partial, int group,
                              void* stream_ptr) {
  using namespace mdb;
  using namespace mdb::conv;
  if (n_classes < 1 || n_classes > MAX_CLASSES) return 3601;
  const int n_taps = tap_begin[n_classes];
  if (n_taps < 1 || n_taps > MAX_TAPS) return 3602;
  if ((C & 15) || (N & 7) || C <= 0 || N <= 0) return 3603;
  if (box[0] * box[1] * box[2] != BM || box[0] > 256 || box[1] > 256 || box[2] > 256) return 3604;
  for (int i = 0; i < 4; ++i) {
    if (ext[i] <= 0) return 0;  // nothing to compute
    if ((strides[i] & 7) || (out_strides[i] & 7)) return 3605;
  }
  if (k_total & 7) return 3605;
  Params p;
  p.n_classes = n_classes;
  for (int c = 0; c <= MAX_CLASSES; ++c) p.tap_begin[c] = tap_begin[c <= n_classes ? c : n_classes];
  for (int c = 0; c < n_classes; ++c) {
    if (tap_begin[c + 1] <= tap_begin[c]) return 3602;
    p.class_off[c] = class_off[c];
    if (class_off[c] & 7) return 3605;
  }
  for (int i = 0; i < n_taps; ++i) {
    const int* t = taps + 6 * i;
    if (t[0] & 7) return 3606;  // the innermost TMA coordinate must stay 16-byte aligned
    p.taps[i].o0 = t[0];
    p.taps[i].o1 = static_cast<short>(t[1]);
    p.taps[i].o2 = static_cast<short>(t[2]);
    p.taps[i].o3 = static_cast<short>(t[3]);
    p.taps[i].o4 = static_cast<short>(t[4]);
    p.taps[i].koff = t[5];
    if (t[5] & 7) return 3606;
  }
  if (group < 1 || group > 3 || (group > 1 && (box[0] != BM || n_taps % group))) return 3604;
  p.group = group;
  p.tap_step = group > 1 ? taps[6 + 5] - taps[5] : 0;
  for (int c = 0; c < n_classes; ++c) {
    if ((tap_begin[c + 1] - tap_begin[c]) % group) return 3604;
  }
  for (int i = 0; i < n_taps; ++i) {  // a group: the same position but for one step along dim 1 per tap, K ranges in line
    const int *t = taps + 6 * i, *f = taps + 6 * (i - i % group);
    const int g = i % group;
    if (t[0] != f[0] || t[1] != f[1] + g || t[2] != f[2] || t[3] != f[3] || t[4] != f[4] || t[5] != f[5] + g * p.tap_step) return 3604;
  }
  p.a_bytes = ((BM + group - 1) * 128 + 1023) / 1024 * 1024;
  p.box1 = box[0]; p.box2 = box[1]; p.box3 = box[2];
  p.ext1 = ext[0]; p.ext2 = ext[1]; p.ext3 = ext[2]; p.ext4 = ext[3];
  p.C = C; p.N = N;
  const int cg = ctas_per_tile == 2 ? 2 : 1;
  if (max_bn < 16 * cg || max_bn > 256 || splits < 1 || (splits > 1 && partial == nullptr)) return 3608;
  p.BN = pick_bn(N, max_bn, 16 * cg);
  p.splits = splits;
  p.partial = static_cast<float*>(partial);
  for (int c = 0; c < n_classes; ++c) {
    if (splits > (tap_begin[c + 1] - tap_begin[c]) / group * ((C + BK - 1) / BK)) return 3608;  // every split has a unit
  }
  const int unit_bytes = p.a_bytes + group * (p.BN / cg * BK * 2);
  constexpr int kHalfSm = 112 * 1024 - 1024 - 256;
  int ctas_per_sm = p.BN <= 128 && 2 * unit_bytes <= kHalfSm ? 2 : 1;  // two stages each
  if (g_tune_ctas > 0) ctas_per_sm = (g_tune_ctas == 2 && p.BN <= 128 && 2 * unit_bytes <= kHalfSm) ? 2 : 1;
  p.acc_cols = ctas_per_sm == 2 ? 128 : 256;
  const int budget = ctas_per_sm == 2 ? kHalfSm : 226 * 1024 - 1024 - 256;
  p.ups = g_tune_ups > 0 ? g_tune_ups : (ctas_per_sm == 2 ? 1 : (p.BN <= 128 && group == 1 ? 2 : 1));
  if (p.ups < 1 || p.ups > 2) return 3608;
  p.stages = budget / (p.ups * unit_bytes);
  if (g_tune_stages > 0 && g_tune_stages < p.stages) p.stages = g_tune_stages;
  if (p.stages < 2 && p.ups == 2) {  // two units a stage were asked for and do not fit twice
    p.ups = 1;
    p.stages = budget / unit_bytes;
  }
  if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
  if (p.stages < 2) return 3608;
  p.alt_dim = alt_dim; p.alt_shift = alt_shift; p.has_alt = (x_alt != nullptr && alt_dim >= 2 && alt_dim <= 3) ? 1 : 0;
  p.os1 = out_strides[0]; p.os2 = out_strides[1]; p.os3 = out_strides[2]; p.os4 = out_strides[3];
  p.out = static_cast<__nv_bfloat16*>(out);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.epi = epi;
  p.status = status_buffer();

  CUtensorMap tx, talt, tw;
  {
    uint64_t d[5], s[4];
    uint32_t b[5] = {BK, static_cast<uint32_t>(box[0] + group - 1), static_cast<uint32_t>(box[1]), static_cast<uint32_t>(box[2]), 1};
    for (int i = 0; i < 5; ++i) d[i] = static_cast<uint64_t>(dims[i]);
    for (int i = 0; i < 4; ++i) s[i] = static_cast<uint64_t>(strides[i]) * 2;
    int rc = encode_tmap_bf16(&tx, x, 5, d, s, b);
    if (rc) return rc;
    if (p.has_alt) {
      if ((alt_strides[0] | alt_strides[1] | alt_strides[2] | alt_strides[3]) & 7) return 3605;
      for (int i = 0; i < 5; ++i) d[i] = static_cast<uint64_t>(alt_dims[i]);
      for (int i = 0; i < 4; ++i) s[i] = static_cast<uint64_t>(alt_strides[i]) * 2;
      rc = encode_tmap_bf16(&talt, x_alt, 5, d, s, b);
      if (rc) return rc;
    } else {
      talt = tx;
    }
    uint64_t wd[2] = {static_cast<uint64_t>(k_total), static_cast<uint64_t>(N)};
    uint64_t ws[1] = {static_cast<uint64_t>(k_total) * 2};
    uint32_t wb[2] = {BK, static_cast<uint32_t>(p.BN / cg)};
    rc = encode_tmap_bf16(&tw, w, 2, wd, ws, wb);
    if (rc) return rc;
  }
  int smem = p.stages * p.ups * unit_bytes + 1024 + 256;
  // the shared-memory request decides how many CTAs share an SM; it has to agree with the TMEM each one allocates
  if (ctas_per_sm == 1 && smem < 120 * 1024) smem = 120 * 1024;
  if (ctas_per_sm == 2 && smem < 80 * 1024) smem = 80 * 1024;
  static bool configured = false;
  if (!configured) {
    for (auto kern : {conv_igemm_kernel<1, false>, conv_igemm_kernel<1, true>, conv_igemm_kernel<2, false>, conv_igemm_kernel<2, true>})
      MDB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured = true;
  }
  const auto cdiv = [](long long a, long long b) { return (a + b - 1) / b; };
  const long long m_tiles = static_cast<long long>(ext[3]) * cdiv(ext[2], box[2]) * cdiv(ext[1], box[1]) * cdiv(ext[0], box[0]);
  const long long work = static_cast<long long>(n_classes) * cdiv(m_tiles, cg) * cdiv(N, p.BN) * splits;
  if (work >= (1ll << 30)) return 3607;
  const long long slots = static_cast<long long>(sm_count()) * ctas_per_sm / cg;
  const int grid = static_cast<int>(work < slots ? work : slots) * cg;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  auto kern = group > 1 ? (cg == 2 ? conv_igemm_kernel<2, true> : conv_igemm_kernel<1, true>)
                        : (cg == 2 ? conv_igemm_kernel<2, false> : conv_igemm_kernel<1, false>);
  MDB_CHECK_CUDA(launch_overlapped(kern, grid, NUM_THREADS, smem, stream, tx, talt, tw, p));
  if (splits > 1) {
    const long long vecs = n_classes * m_tiles * BM * (N / 8);
    MDB_CHECK_CUDA(launch_overlapped(conv_fold_kernel, static_cast<int>(cdiv(vecs, 128)), 128, 0, stream, p));
  }
  return static_cast<int>(cudaGetLastError());
}
