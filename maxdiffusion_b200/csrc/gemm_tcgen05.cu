// Persistent, warp-specialised bf16 GEMM for sm_100a:
//     D[M,N] = epilogue( A[M,K] * B[N,K]^T )
// Operands come through (non-multicast) TMA into 128-byte-swizzled shared memory, products are issued by one thread with
// tcgen05.mma, fp32 accumulators sit in TMEM and are double buffered (2 x 256 columns) so that the epilogue of tile i
// overlaps the main loop of tile i+1.
//
// What bounds it is the operand feed from L2: every shape ran at about 57 bytes per clock and SM, which a 128 x 256 tile
// of one CTA (48 KB per 512 tensor clocks) turns into 60 % of the tensor rate. So tiles of more than 128 rows are
// computed by a PAIR of CTAs (`cta_group::2`): 256 x BN, each CTA fetching its own 128 rows of A and half of B (32 KB per
// 512 clocks at BN = 256) and draining its own 128 accumulator rows. One CTA / a pair, in turn under the power cap: 32760 x
// 5120 x 5120 1400 / 1239 us, 4608 x 9216 x 3072 202 / 172 us, 4096 x 3072 x 12288 239 / 213 us.
//
// Either operand may be "MN-major" (stored transposed, i.e. A as [K,M] or B as [K,N]); this is what
// lets dgrad (dX = dY * W) and wgrad (dW = dY^T * X) run on the same kernel without transposes.
//
// Roles:  warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer (of a pair: in the even CTA), warps 2..5 and 6..9 = two
// epilogue groups that take the tile's 128-byte-wide slabs in turn.
// Covers the reference's XLA:GPU / cuBLAS matmuls behind every Dense layer
// (src/maxdiffusion/models/attention_flax.py:2471-2525, models/wan/transformers/transformer_wan.py:220-330)
// together with the elementwise fusions XLA places after them (bias, GELU-tanh, gated residual).
#include "host_common.h"

namespace mdb {

namespace gemm {
constexpr int BM = 128;  // rows of one CTA; a pair's tile has 256
constexpr int BK = 64;
constexpr int A_BYTES = BM * BK * 2;  // 16 KiB
constexpr int NUM_THREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2..5 and 6..9: two epilogue groups
constexpr int EPI_WARPS = 8;
constexpr int MAX_STAGES = 8;
constexpr int ACC_COLS = 256;     // TMEM columns of one accumulator
// Output staging of the epilogue: a slab of 32 rows x 128 bytes (64 bf16 or 32 fp32 columns) per epilogue warp, in which
// the accumulator rows that a thread owns become the 128-byte lines that 8 lanes store together. Everything a warp stages
// stays within the warp: no CTA barrier and no wait for an earlier store.
constexpr int SLAB_BYTES = 32 * 128;
constexpr int STAGING_BYTES = EPI_WARPS * SLAB_BYTES;
constexpr int BIAS_BYTES = 2 * 256 * 4;  // the tile's bias columns as fp32, for two tiles in turn
constexpr int FIXED_BYTES = STAGING_BYTES + BIAS_BYTES + 256 /*barriers*/;
constexpr int SMEM_LIMIT = 227 * 1024;
// One stage holds a k-block of A (128 rows) and of this CTA's share of B; a multiple of 1024 bytes.
__host__ __device__ constexpr int stage_bytes(int bn, int cg) { return A_BYTES + bn / cg * BK * 2; }
// As many stages as fit beside 8 KB, in which CTAs of the kernels before and after (a cut contraction's fold) can be on the SM
// too, each with a reserved kilobyte, so that launches overlap: with every byte taken 320 x 320 x 16384 took 19.3 us, 13.0 so, and
// a Flux preview step (300 launches) 3.63 and 3.50 ms; steps of long products are the same either way. One CTA's tile 256 columns
// wide takes all for its fourth stage (3 / 4: 4608 x 9216 x 3072 244 / 202 us, 8192 x 5120 x 320 43.5 / 30.7 us) unless a fold follows.
__host__ constexpr int stages_for(int bn, int cg, bool cut) {
  const int room = (SMEM_LIMIT - 8192 - FIXED_BYTES) / stage_bytes(bn, cg), all = (SMEM_LIMIT - FIXED_BYTES) / stage_bytes(bn, cg);
  const int n = cut || room > 3 ? room : all;
  return n < MAX_STAGES ? n : MAX_STAGES;
}

enum Epilogue : int {
  kEpiNone = 0,       // out = acc*alpha + bias
  kEpiGeluTanh = 1,   // out = gelu_tanh(acc*alpha + bias)
  kEpiGatedRes = 2,   // out = residual + gate[batch(row), col] * (acc*alpha + bias)
  kEpiSilu = 3,       // out = silu(acc*alpha + bias)
  kEpiAddRes = 4,     // out = residual + acc*alpha + bias
};

// Epilogues are compiled one by one: a kernel that carries all of them does not fit the instruction cache, and a short
// product then spends its time on fetching code (128 x 256 x 64: 7.5 us with one kernel for all, 6.2 us so; 8192 x 2560 x
// 64, five rounds of tiles: 23.1 and 13.3 us).
enum EpilogueKind : int {
  kPlain = 0,    // bf16 out, bias or none
  kAct = 1,      // bf16 out, bias, GELU-tanh or SiLU
  kRes = 2,      // bf16 out, bias, (gated) residual
  kPlainF32 = 3, // fp32 out or split-K partials, bias or none
  kGeglu = 5,    // bf16 out [M, N], B [2 N, K]: columns n and N + n of the product meet in a tile, out = h * gelu(gate)
  kDirect = 4,   // anything, 16-byte stores from one thread per row: the staged kernels' bit-for-bit oracle
  // fp32 out, bias and an activation / a (gated) residual. One thread per row / staged: 4608 x 3072 x 3072 66 / 62 us with
  // GELU, 78 / 66 us with a residual; 4608 x 3072 x 64 33 / 19 and 46 / 33 us.
  kActF32 = 6,
  kResF32 = 7,
};

struct Params {
  int M, N, K;
  void* out;
  long long ldo;
  const __nv_bfloat16* bias;      // [N] or nullptr
  const __nv_bfloat16* residual;  // [M, ldr] or nullptr
  long long ldr;
  const float* gate;              // [num_batches, gate_ld] fp32 or nullptr
  long long gate_ld;
  int rows_per_batch;
  int epi;
  int out_f32;
  float alpha;
  DeviceStatus* status;
  // split-K (weight gradients: a small output with a long contraction): work item w covers k-blocks
  // [split * kb_per_split, ..) of tile w % num_tiles with split = w / num_tiles and writes fp32 partials
  // [splits, M, N]; `splitk_fold_kernel` sums them in split order (deterministic, no atomics)
  int splits;
  int kb_per_split;
  float* partial;
  int mats;    // B matrices of the same shape that share A (1 .. MAX_MATS); matrix i gives columns [i N, (i + 1) N) of out
  int bn;      // columns of a tile: 64, 128, 192 or 256
  int stages;  // pipeline depth
};

constexpr int MAX_MATS = 3;
struct BMaps {
  CUtensorMap m[MAX_MATS];
};

template <int GROUP_M>
__device__ __forceinline__ void tile_coords(int tile, int num_m, int num_n, int& m_idx, int& n_idx) {
  // Grouped rasterisation: GROUP_M row-blocks share each sweep over the column-blocks so that
  // concurrently running CTAs reuse both operands out of L2.
  const int tiles_per_group = GROUP_M * num_n;
  const int group = tile / tiles_per_group;
  const int first_m = group * GROUP_M;
  const int rows = min(GROUP_M, num_m - first_m);
  const int local = tile - group * tiles_per_group;
  m_idx = first_m + local % rows;
  n_idx = local / rows;
}

template <bool A_MN, bool B_MN, int CG, int EK>
__global__ void __cluster_dims__(CG, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ BMaps maps_b, const Params p) {
  constexpr int TILE_M = CG * BM;
  constexpr int GROUP_M = 8;
  constexpr int TMEM_COLS = 2 * ACC_COLS;   // two accumulators
  const int STAGES = p.stages, BN = p.bn, BN_CTA = BN / CG;
  const int STAGE_BYTES = A_BYTES + BN_CTA * BK * 2;
  extern __shared__ __align__(1024) uint8_t smem[];  // the 128-byte swizzle repeats every 1024 bytes
  uint8_t* staging = smem + STAGES * STAGE_BYTES;  // 1024-byte aligned: every stage is a multiple of 1024 bytes
  float* bias_s = reinterpret_cast<float*>(staging + STAGING_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + STAGING_BYTES + BIAS_BYTES);
  uint64_t* full_bar = bars;                        // [MAX_STAGES]; of a pair: only the even CTA's are used
  uint64_t* empty_bar = bars + MAX_STAGES;          // [MAX_STAGES]
  uint64_t* tmem_full = bars + 2 * MAX_STAGES;      // [2]
  uint64_t* tmem_empty = bars + 2 * MAX_STAGES + 2; // [2]; of a pair: only the even CTA's are used
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const int group_id = static_cast<int>(blockIdx.x) / CG, num_groups = static_cast<int>(gridDim.x) / CG;
  const int num_m = (p.M + TILE_M - 1) / TILE_M;
  constexpr int HALVES = EK == kGeglu ? 2 : 1;  // GEGLU: half of a tile's columns are gates of the other half
  const int OUT_N = BN / HALVES;                 // output columns of a tile
  const int mat_n = (p.N + OUT_N - 1) / OUT_N;   // column tiles of one B matrix
  const int num_n = mat_n * p.mats;
  const int num_tiles = num_m * num_n;
  const int num_kb = (p.K + BK - 1) / BK;
  const int num_work = num_tiles * p.splits;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&maps_b.m[0]);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], CG * EPI_WARPS);  // every epilogue warp (of both CTAs) has read the accumulator
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    if (CG == 2) {
      tmem_alloc_pair(tmem_ptr_smem, TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_ptr_smem, TMEM_COLS);
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
        int m_idx, n_idx;
        const int split = work / num_tiles;
        tile_coords<GROUP_M>(work - split * num_tiles, num_m, num_n, m_idx, n_idx);
        const int mat = p.mats > 1 ? n_idx / mat_n : 0;
        n_idx -= mat * mat_n;
        const CUtensorMap& tmap_b = maps_b.m[mat];
        const int m0 = m_idx * TILE_M + rank * BM;
        // GEGLU (pairs only): the even CTA fetches rows n of B, the odd one rows N + n
        const int n0 = EK == kGeglu ? n_idx * OUT_N + rank * p.N : n_idx * BN + rank * BN_CTA;
        const int kb_begin = split * p.kb_per_split, kb_end = min(num_kb, kb_begin + p.kb_per_split);
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag, p.status, 10)) { ok = false; break; }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          const int k0 = kb * BK;
          if (CG == 2) {
            // both CTAs' copies complete on the even CTA's barrier, which expects the bytes of both
            if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
            const uint32_t bar = cluster_map(&full_bar[stage], 0);
            if (A_MN) {
#pragma unroll
              for (int c = 0; c < BM / 64; ++c) tma_load_2d_pair(sa + c * (BK * 128), &tmap_a, bar, m0 + c * 64, k0);
            } else {
              tma_load_2d_pair(sa, &tmap_a, bar, k0, m0);
            }
            if (B_MN) {
              for (int c = 0; c < BN_CTA / 64; ++c) tma_load_2d_pair(sb + c * (BK * 128), &tmap_b, bar, n0 + c * 64, k0);
            } else {
              tma_load_2d_pair(sb, &tmap_b, bar, k0, n0);
            }
          } else {
            mbar_expect_tx(&full_bar[stage], STAGE_BYTES);
            if (A_MN) {
#pragma unroll
              for (int c = 0; c < BM / 64; ++c) tma_load_2d(sa + c * (BK * 128), &tmap_a, &full_bar[stage], m0 + c * 64, k0);
            } else {
              tma_load_2d(sa, &tmap_a, &full_bar[stage], k0, m0);
            }
            if (B_MN) {
              for (int c = 0; c < BN_CTA / 64; ++c) tma_load_2d(sb + c * (BK * 128), &tmap_b, &full_bar[stage], n0 + c * 64, k0);
            } else {
              tma_load_2d(sb, &tmap_b, &full_bar[stage], k0, n0);
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
    // ------------------------------ MMA issuer --------------------------------
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(TILE_M, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int work = group_id; work < num_work && ok; work += num_groups, ++it) {
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1u;
        if (!mbar_wait(&tmem_empty[acc], acc_phase ^ 1u, abort_flag, p.status, 20)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
        const int kb_begin = (work / num_tiles) * p.kb_per_split, kb_end = min(num_kb, kb_begin + p.kb_per_split);
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, 21)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, BK * 128, 1024)
                                     : make_smem_desc(sa + k * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc(sb + k * 2048, BK * 128, 1024)
                                     : make_smem_desc(sb + k * 32, 16, 1024);
            const uint32_t accumulate = (kb > kb_begin || k > 0) ? 1u : 0u;
            if (CG == 2) umma_ss_pair(d_tmem, da, db, idesc, accumulate);
            else umma_ss(d_tmem, da, db, idesc, accumulate);
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
    // Two groups of four warps share a tile and take its slabs (64 bf16 or 32 fp32 columns) in turn. With short
    // contractions (10-20 K blocks) a tile's epilogue lasts as long as its main loop; two groups halve it.
    const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 are reachable from this warp
    const int row_in_tile = quarter * 32 + lane;
    const int egroup = (warp - 2) >> 2;
    const int group_thread = static_cast<int>(threadIdx.x) - 64 - egroup * 128;
    constexpr bool f32 = EK == kPlainF32 || EK == kActF32 || EK == kResF32;
    constexpr int slab_cols = f32 ? 32 : 64;
    const bool use_bias = p.bias != nullptr && p.splits == 1;
    int it = 0;
    bool ok = true;
    for (int work = group_id; work < num_work && ok; work += num_groups, ++it) {
      int m_idx, n_idx;
      const int split = work / num_tiles;
      tile_coords<GROUP_M>(work - split * num_tiles, num_m, num_n, m_idx, n_idx);
      const int mat = p.mats > 1 ? n_idx / mat_n : 0;
      n_idx -= mat * mat_n;
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1u;
      float* bias_t = bias_s + acc * 256;
      if (EK != kDirect && use_bias) {
        // the tile's bias columns once, as fp32, while the products run; a warp that still reads the previous tile's is
        // one barrier behind and reads the other buffer
        for (int c = group_thread; c < BN; c += 128) {
          const int col = n_idx * OUT_N + c % OUT_N;
          if (((c / slab_cols) & 1) == egroup)
            bias_t[c] = col < p.N ? __bfloat162float(p.bias[col + (c / OUT_N) * p.N]) : 0.0f;
        }
        named_bar_sync(1 + egroup, 128);
      }
      if (!mbar_wait(&tmem_full[acc], acc_phase, abort_flag, p.status, 30)) { ok = false; break; }
      tc_fence_after_sync();
      const long long row0 = static_cast<long long>(m_idx) * TILE_M + rank * BM;  // may lie beyond M in the odd CTA
      const long long row = row0 + row_in_tile;
      const bool row_ok = row < p.M;
      const int batch = (p.rows_per_batch > 0) ? static_cast<int>(row / p.rows_per_batch) : 0;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * ACC_COLS;
      if constexpr (EK != kDirect) {
        // ---- staged epilogue: 128 bytes of 32 rows per warp and slab, swizzled ----
        const int sw = lane & 7;
        uint8_t* slab = staging + (warp - 2) * SLAB_BYTES;
        uint8_t* my_row = slab + lane * 128;
        const long long warp_row0 = row0 + quarter * 32;
        const int rows_valid = warp_row0 < p.M ? static_cast<int>(min(32ll, p.M - warp_row0)) : 0;
        // the lines: lane l moves 16 bytes (chunk l & 7) of the rows (l >> 3) + 4 i
        const int line_row = lane >> 3, line_chunk = lane & 7;
        constexpr int esz = f32 ? 4 : 2;
        uint8_t* out_base = p.splits > 1
            ? reinterpret_cast<uint8_t*>(p.partial) + (static_cast<long long>(split) * p.M + warp_row0) * p.N * 4
            : reinterpret_cast<uint8_t*>(p.out) + (warp_row0 * p.ldo + static_cast<long long>(mat) * p.N) * esz;
        const long long out_pitch = (p.splits > 1 ? static_cast<long long>(p.N) : p.ldo) * esz;
#pragma unroll 1
        for (int c0 = egroup * slab_cols; c0 < OUT_N; c0 += 2 * slab_cols) {
          const int col0 = n_idx * OUT_N + c0;
          if (col0 >= p.N || rows_valid <= 0) break;  // uniform across the warp
          const int line_col = col0 + line_chunk * (16 / esz);
          uint32_t r[2][32];
          if constexpr (EK == kGeglu) {
            // 32 columns of h and of the gate at a time
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              tmem_ld_x32(taddr + c0 + h * 32, r[0]);
              tmem_ld_x32(taddr + OUT_N + c0 + h * 32, r[1]);
              tmem_wait_ld();
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const int c = c0 + h * 32 + v * 8 + j;
                  float hv = __uint_as_float(r[0][v * 8 + j]) * p.alpha, gv = __uint_as_float(r[1][v * 8 + j]) * p.alpha;
                  if (use_bias) {
                    hv += bias_t[c];
                    gv += bias_t[OUT_N + c];
                  }
                  x[j] = hv * (0.5f * gv * (1.0f + erff(gv * 0.7071067811865476f)));
                }
                uint4 ov;
                ov.x = pack_bf16x2(x[0], x[1]);
                ov.y = pack_bf16x2(x[2], x[3]);
                ov.z = pack_bf16x2(x[4], x[5]);
                ov.w = pack_bf16x2(x[6], x[7]);
                *reinterpret_cast<uint4*>(my_row + (((h * 4 + v) ^ sw) << 4)) = ov;
              }
            }
          } else {
          tmem_ld_x32(taddr + c0, r[0]);
          if (!f32) tmem_ld_x32(taddr + c0 + 32, r[1]);  // bf16: two 32-column loads per slab; fp32: one
          if constexpr (EK == kRes) {  // the residual passes through the slab
            uint4 rv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int rl = line_row + 4 * i;
              rv[i] = (rl < rows_valid && line_col < p.N)
                          ? *reinterpret_cast<const uint4*>(p.residual + (warp_row0 + rl) * p.ldr + line_col)
                          : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int rl = line_row + 4 * i;
              *reinterpret_cast<uint4*>(slab + rl * 128 + ((line_chunk ^ (rl & 7)) << 4)) = rv[i];
            }
            __syncwarp();
          }
          tmem_wait_ld();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (f32 && h == 1) break;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int col = col0 + h * 32 + v * 8;
              float x[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(r[h][v * 8 + j]) * p.alpha;
              if (use_bias) {  // zeros beyond N
                const float4 b0 = *reinterpret_cast<const float4*>(bias_t + c0 + h * 32 + v * 8);
                const float4 b1 = *reinterpret_cast<const float4*>(bias_t + c0 + h * 32 + v * 8 + 4);
                x[0] += b0.x; x[1] += b0.y; x[2] += b0.z; x[3] += b0.w;
                x[4] += b1.x; x[5] += b1.y; x[6] += b1.z; x[7] += b1.w;
              }
              if constexpr (EK == kAct || EK == kActF32) {
                if (p.epi == kEpiGeluTanh) {
#pragma unroll
                  for (int j = 0; j < 8; ++j) x[j] = gelu_tanh(x[j]);
                } else {
#pragma unroll
                  for (int j = 0; j < 8; ++j) x[j] = x[j] / (1.0f + __expf(-x[j]));
                }
              }
              if constexpr (EK == kRes || EK == kResF32) {
                if (row_ok && col < p.N) {
                  const uint4 rres = EK == kRes ? *reinterpret_cast<const uint4*>(my_row + (((h * 4 + v) ^ sw) << 4))
                                                : *reinterpret_cast<const uint4*>(p.residual + row * p.ldr + col);
                  const uint32_t rw[4] = {rres.x, rres.y, rres.z, rres.w};
                  float g[8];
                  if (p.epi == kEpiGatedRes) {
                    const float4 g0 = *reinterpret_cast<const float4*>(p.gate + batch * p.gate_ld + col);
                    const float4 g1 = *reinterpret_cast<const float4*>(p.gate + batch * p.gate_ld + col + 4);
                    g[0] = g0.x; g[1] = g0.y; g[2] = g0.z; g[3] = g0.w;
                    g[4] = g1.x; g[5] = g1.y; g[6] = g1.z; g[7] = g1.w;
                  } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) g[j] = 1.0f;
                  }
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    float2 f = unpack_bf16x2(rw[j]);
                    x[2 * j] = f.x + g[2 * j] * x[2 * j];
                    x[2 * j + 1] = f.y + g[2 * j + 1] * x[2 * j + 1];
                  }
                }
              }
              if (f32) {  // 8 values = two 16-byte chunks of the row's 128 bytes
                const int ch = v * 2;
                *reinterpret_cast<float4*>(my_row + (((ch) ^ sw) << 4)) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4*>(my_row + (((ch + 1) ^ sw) << 4)) = make_float4(x[4], x[5], x[6], x[7]);
              } else {
                const int ch = h * 4 + v;
                uint4 ov;
                ov.x = pack_bf16x2(x[0], x[1]);
                ov.y = pack_bf16x2(x[2], x[3]);
                ov.z = pack_bf16x2(x[4], x[5]);
                ov.w = pack_bf16x2(x[6], x[7]);
                *reinterpret_cast<uint4*>(my_row + ((ch ^ sw) << 4)) = ov;
              }
            }
          }
          }
          __syncwarp();
          if (line_col < p.N) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int rl = line_row + 4 * i;
              const uint4 ov = *reinterpret_cast<const uint4*>(slab + rl * 128 + ((line_chunk ^ (rl & 7)) << 4));
              if (rl < rows_valid)
                *reinterpret_cast<uint4*>(out_base + rl * out_pitch + static_cast<long long>(line_col) * esz) = ov;
            }
          }
          __syncwarp();  // the lines have been read before the next slab (or tile) overwrites them
        }
      } else {
#pragma unroll 1
      for (int c = egroup; c < BN / 32; c += 2) {
        const int col0 = n_idx * BN + c * 32;
        if (col0 >= p.N || row0 >= p.M) break;  // uniform across the group
        uint32_t r[32];
        tmem_ld_x32(taddr + c * 32, r);
        tmem_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {  // 4 groups of 8 columns
            const int col = col0 + v * 8;
            if (col >= p.N) break;
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(r[v * 8 + j]) * p.alpha;
            if (p.splits > 1) {
              float* o = p.partial + (static_cast<long long>(split) * p.M + row) * p.N + col;
              *reinterpret_cast<float4*>(o) = make_float4(x[0], x[1], x[2], x[3]);
              *reinterpret_cast<float4*>(o + 4) = make_float4(x[4], x[5], x[6], x[7]);
              continue;
            }
            if (p.bias) {  // single loads: a bias may start anywhere
#pragma unroll
              for (int j = 0; j < 8; ++j) x[j] += __bfloat162float(p.bias[col + j]);
            }
            if (p.epi == kEpiGeluTanh) {
#pragma unroll
              for (int j = 0; j < 8; ++j) x[j] = gelu_tanh(x[j]);
            } else if (p.epi == kEpiSilu) {
#pragma unroll
              for (int j = 0; j < 8; ++j) x[j] = x[j] / (1.0f + __expf(-x[j]));
            } else if (p.epi == kEpiGatedRes || p.epi == kEpiAddRes) {
              const uint4 rv = *reinterpret_cast<const uint4*>(p.residual + row * p.ldr + col);
              const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
              float g[8];
              if (p.epi == kEpiGatedRes) {
                const float4 g0 = *reinterpret_cast<const float4*>(p.gate + batch * p.gate_ld + col);
                const float4 g1 = *reinterpret_cast<const float4*>(p.gate + batch * p.gate_ld + col + 4);
                g[0] = g0.x; g[1] = g0.y; g[2] = g0.z; g[3] = g0.w;
                g[4] = g1.x; g[5] = g1.y; g[6] = g1.z; g[7] = g1.w;
              } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) g[j] = 1.0f;
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                float2 f = unpack_bf16x2(rw[j]);
                x[2 * j] = f.x + g[2 * j] * x[2 * j];
                x[2 * j + 1] = f.y + g[2 * j + 1] * x[2 * j + 1];
              }
            }
            if (p.out_f32) {
              float* o = reinterpret_cast<float*>(p.out) + row * p.ldo + col;
              *reinterpret_cast<float4*>(o) = make_float4(x[0], x[1], x[2], x[3]);
              *reinterpret_cast<float4*>(o + 4) = make_float4(x[4], x[5], x[6], x[7]);
            } else {
              __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + row * p.ldo + col;
              uint4 ov;
              ov.x = pack_bf16x2(x[0], x[1]);
              ov.y = pack_bf16x2(x[2], x[3]);
              ov.z = pack_bf16x2(x[4], x[5]);
              ov.w = pack_bf16x2(x[6], x[7]);
              *reinterpret_cast<uint4*>(o) = ov;
            }
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
    if (CG == 2) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// out = epilogue(sum over splits of partial[s], in split order); one thread per 8 columns.
__global__ void splitk_fold_kernel(const __grid_constant__ Params p) {
  allow_successor();
  wait_for_predecessor();
  const int n_vec = p.N / 8;
  const long long n8 = static_cast<long long>(p.M) * n_vec;
  const long long split_stride = static_cast<long long>(p.M) * p.N;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n8;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = 0; s < p.splits; ++s) {
      const float4* src = reinterpret_cast<const float4*>(p.partial + s * split_stride + i * 8);
      const float4 a = src[0], b = src[1];
      x[0] += a.x; x[1] += a.y; x[2] += a.z; x[3] += a.w;
      x[4] += b.x; x[5] += b.y; x[6] += b.z; x[7] += b.w;
    }
    const long long row = i / n_vec;
    const int col = static_cast<int>(i - row * n_vec) * 8;
    if (p.bias) {  // single loads: a bias may start anywhere
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] += __bfloat162float(p.bias[col + j]);
    }
    if (p.epi == kEpiGeluTanh) {
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = gelu_tanh(x[j]);
    } else if (p.epi == kEpiSilu) {
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = x[j] / (1.0f + __expf(-x[j]));
    } else if (p.epi == kEpiGatedRes || p.epi == kEpiAddRes) {
      const uint4 rv = *reinterpret_cast<const uint4*>(p.residual + row * p.ldr + col);
      const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
      const float* g = p.epi == kEpiGatedRes
                           ? p.gate + (p.rows_per_batch > 0 ? row / p.rows_per_batch : 0) * p.gate_ld + col
                           : nullptr;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(rw[j]);
        x[2 * j] = f.x + (g ? g[2 * j] : 1.0f) * x[2 * j];
        x[2 * j + 1] = f.y + (g ? g[2 * j + 1] : 1.0f) * x[2 * j + 1];
      }
    }
    if (p.out_f32) {
      float* o = reinterpret_cast<float*>(p.out) + row * p.ldo + col;
      *reinterpret_cast<float4*>(o) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(o + 4) = make_float4(x[4], x[5], x[6], x[7]);
    } else {
      uint4 ov;
      ov.x = pack_bf16x2(x[0], x[1]);
      ov.y = pack_bf16x2(x[2], x[3]);
      ov.z = pack_bf16x2(x[4], x[5]);
      ov.w = pack_bf16x2(x[6], x[7]);
      *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + row * p.ldo + col) = ov;
    }
  }
}

template <bool A_MN, bool B_MN, int CG, int EK>
int launch(const CUtensorMap& ta, const BMaps& tb, const Params& p, cudaStream_t stream) {
  auto kern = gemm_kernel<A_MN, B_MN, CG, EK>;
  static bool configured = false;
  if (!configured) {
    MDB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
    // all of the SM's memory as shared memory: what a CTA does not use is room for the successor's CTAs to start in
    MDB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    configured = true;
  }
  const int out_n = EK == kGeglu ? p.bn / 2 : p.bn;
  const int num_work = ((p.M + CG * BM - 1) / (CG * BM)) * ((p.N + out_n - 1) / out_n) * p.mats * p.splits;
  const int slots = sm_count() / CG;
  const int grid = (num_work < slots ? num_work : slots) * CG;
  MDB_CHECK_CUDA(launch_overlapped(kern, grid, NUM_THREADS, p.stages * stage_bytes(p.bn, CG) + FIXED_BYTES, stream, ta, tb, p));
  if (p.splits > 1) {
    const long long n8 = static_cast<long long>(p.M) * p.N / 8;
    const int blocks = static_cast<int>(n8 / 128 + 1 < sm_count() * 16 ? n8 / 128 + 1 : sm_count() * 16);
    MDB_CHECK_CUDA(launch_overlapped(splitk_fold_kernel, blocks, 128, 0, stream, p));
  }
  return static_cast<int>(cudaGetLastError());
}

template <bool A_MN, bool B_MN, int CG>
int launch_kind(int kind, const CUtensorMap& ta, const BMaps& tb, const Params& p, cudaStream_t stream) {
  switch (kind) {
    case kPlain: return launch<A_MN, B_MN, CG, kPlain>(ta, tb, p, stream);
    case kAct: return launch<A_MN, B_MN, CG, kAct>(ta, tb, p, stream);
    case kRes: return launch<A_MN, B_MN, CG, kRes>(ta, tb, p, stream);
    case kPlainF32: return launch<A_MN, B_MN, CG, kPlainF32>(ta, tb, p, stream);
    case kActF32: return launch<A_MN, B_MN, CG, kActF32>(ta, tb, p, stream);
    case kResF32: return launch<A_MN, B_MN, CG, kResF32>(ta, tb, p, stream);
    default: return launch<A_MN, B_MN, CG, kDirect>(ta, tb, p, stream);
  }
}

}  // namespace gemm
}  // namespace mdb

static int g_epilogue_mode = 0;  // 0: staged epilogue; 1: direct stores

// Tile search / benchmarks: 1 pins the direct-store epilogue (one thread per row, 16-byte stores), 0 restores the default.
extern "C" int mdb_gemm_epilogue_mode(int mode) {
  if (mode != 0 && mode != 1) return 3006;
  g_epilogue_mode = mode;
  return 0;
}

// C entry point. A is [M,K] with leading dimension lda (a_mn_major = 0) or [K,M] (a_mn_major = 1);
// B is [N,K] (b_mn_major = 0) or [K,N] (b_mn_major = 1). All leading dimensions are in elements and
// must be multiples of 8; N must be a multiple of 8; out, residual and gate start on 16-byte boundaries (they are moved 16
// bytes at a time). Returns 0 or a CUDA / encoder error code.
//
// The launch shape is the caller's (`ops/kernels.py: gemm_plan`): `ctas` per tile (1 or 2), tile width `bn` (64, 128, 192
// or 256; a transposed B needs a multiple of 64 columns per CTA), and `splits` of the contraction, which run as separate
// work items with fp32 partials (`partial`: splits * M * N values) and are summed in split order by a second kernel that
// also applies the epilogue (for products with fewer tiles than the GPU has SMs).
extern "C" int mdb_gemm_bf16(const void* A, const void* B, void* out, const void* bias, const void* residual,
                             const void* gate, int M, int N, int K, long long lda, long long ldb, long long ldo,
                             long long ldr, long long gate_ld, int rows_per_batch, int a_mn_major, int b_mn_major,
                             int epi, int out_f32, float alpha, int ctas, int bn, int splits, void* partial,
                             void* stream_ptr) {
  using namespace mdb;
  using namespace mdb::gemm;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldo & 3) || (!out_f32 && (ldo & 7))) return 3001;
  if ((epi == kEpiGatedRes || epi == kEpiAddRes) && (!residual || (ldr & 7))) return 3002;
  if (epi == kEpiGatedRes && (!gate || (gate_ld & 3))) return 3003;
  const auto misaligned = [](const void* t) { return (reinterpret_cast<uintptr_t>(t) & 15) != 0; };
  if (misaligned(out) || misaligned(partial)) return 3006;
  if ((epi == kEpiGatedRes || epi == kEpiAddRes) && (misaligned(residual) || (epi == kEpiGatedRes && misaligned(gate)))) return 3006;
  if ((ctas != 1 && ctas != 2) || (bn != 64 && bn != 128 && bn != 192 && bn != 256)) return 3004;
  if (splits < 1 || splits > 64 || (splits > 1 && partial == nullptr)) return 3005;
  const int bn_cta = bn / ctas;
  if (b_mn_major && bn_cta % 64) return 3004;
  CUtensorMap ta;
  BMaps tb = {};
  int rc;
  if (a_mn_major) {
    uint64_t dims[2] = {static_cast<uint64_t>(M), static_cast<uint64_t>(K)};
    uint64_t str[1] = {static_cast<uint64_t>(lda) * 2};
    uint32_t box[2] = {64, BK};
    rc = encode_tmap_bf16(&ta, A, 2, dims, str, box);
  } else {
    uint64_t dims[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(M)};
    uint64_t str[1] = {static_cast<uint64_t>(lda) * 2};
    uint32_t box[2] = {BK, BM};
    rc = encode_tmap_bf16(&ta, A, 2, dims, str, box);
  }
  if (rc) return rc;
  if (b_mn_major) {
    uint64_t dims[2] = {static_cast<uint64_t>(N), static_cast<uint64_t>(K)};
    uint64_t str[1] = {static_cast<uint64_t>(ldb) * 2};
    uint32_t box[2] = {64, BK};
    rc = encode_tmap_bf16(&tb.m[0], B, 2, dims, str, box);
  } else {
    uint64_t dims[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(N)};
    uint64_t str[1] = {static_cast<uint64_t>(ldb) * 2};
    uint32_t box[2] = {BK, static_cast<uint32_t>(bn_cta)};
    rc = encode_tmap_bf16(&tb.m[0], B, 2, dims, str, box);
  }
  if (rc) return rc;
  Params p;
  p.M = M; p.N = N; p.K = K;
  p.out = out; p.ldo = ldo;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.ldr = ldr;
  p.gate = static_cast<const float*>(gate);
  p.gate_ld = gate_ld;
  p.rows_per_batch = rows_per_batch;
  p.epi = epi;
  p.out_f32 = out_f32;
  p.alpha = alpha;
  p.mats = 1;
  p.bn = bn;
  p.status = status_buffer();
  {
    // every split gets at least one k-block: the count is recomputed from the rounded-up range
    const int num_kb = (K + BK - 1) / BK;
    int per = (num_kb + splits - 1) / splits;
    if (per < 1) per = 1;
    p.kb_per_split = per;
    p.splits = (num_kb + per - 1) / per;
    p.partial = static_cast<float*>(partial);
    if (p.splits <= 1) { p.splits = 1; p.kb_per_split = num_kb; }
  }
  p.stages = stages_for(bn, ctas, p.splits > 1);
  const bool f32 = out_f32 || p.splits > 1;
  const bool act = epi == kEpiGeluTanh || epi == kEpiSilu, res = epi == kEpiGatedRes || epi == kEpiAddRes;
  int kind = kDirect;
  if (g_epilogue_mode == 0) {
    if (f32) kind = p.splits > 1 ? kPlainF32 : (act ? kActF32 : (res ? kResF32 : kPlainF32));
    else kind = act ? kAct : (res ? kRes : kPlain);
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  if (ctas == 2) {
    if (a_mn_major) return b_mn_major ? launch_kind<true, true, 2>(kind, ta, tb, p, stream) : launch_kind<true, false, 2>(kind, ta, tb, p, stream);
    return b_mn_major ? launch_kind<false, true, 2>(kind, ta, tb, p, stream) : launch_kind<false, false, 2>(kind, ta, tb, p, stream);
  }
  if (a_mn_major) return b_mn_major ? launch_kind<true, true, 1>(kind, ta, tb, p, stream) : launch_kind<true, false, 1>(kind, ta, tb, p, stream);
  return b_mn_major ? launch_kind<false, true, 1>(kind, ta, tb, p, stream) : launch_kind<false, false, 1>(kind, ta, tb, p, stream);
}

// out [M, N] = h * gelu(gate) (exact GELU) of A [M, K] times B [2 N, K] transposed, plus bias [2 N]: rows n of B give h, rows
// N + n the gate (GEGLU), in one pass by pairs of CTAs: the product is not written. With bias, GEMM and GEGLU kernel / this: 2048 x (2 x 5120) x
// 1280 58 / 42 us, 8192 x (2 x 2560) x 640 85 / 60 us; at 128 rows (12.2 / 12.9 us) the caller keeps the two.
extern "C" int mdb_gemm_geglu(const void* A, const void* B, void* out, const void* bias, int M, int N, int K, long long lda,
                              long long ldb, long long ldo, void* stream_ptr) {
  using namespace mdb;
  using namespace mdb::gemm;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldo & 7)) return 3001;
  constexpr int bn = 256, ctas = 2;
  CUtensorMap ta;
  BMaps tb = {};
  uint64_t da[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(M)}, db[2] = {static_cast<uint64_t>(K), 2ull * N};
  uint64_t sa[1] = {static_cast<uint64_t>(lda) * 2}, sb[1] = {static_cast<uint64_t>(ldb) * 2};
  uint32_t box_a[2] = {BK, BM}, box_b[2] = {BK, bn / 2};
  int rc = encode_tmap_bf16(&ta, A, 2, da, sa, box_a);
  if (rc) return rc;
  rc = encode_tmap_bf16(&tb.m[0], B, 2, db, sb, box_b);
  if (rc) return rc;
  Params p = {};
  p.M = M; p.N = N; p.K = K;
  p.out = out; p.ldo = ldo;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.alpha = 1.0f;
  p.mats = 1;
  p.splits = 1;
  p.kb_per_split = (K + BK - 1) / BK;
  p.bn = bn;
  p.stages = stages_for(bn, ctas, false);
  p.status = status_buffer();
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  return launch<false, false, 2, kGeglu>(ta, tb, p, stream);
}

// out [M, mats * N] = A [M, K] times each of `mats` matrices B_i [N, K] transposed, side by side: projections of the same
// rows (q, k, v) in one launch. Apart / together: 2048 x (3 x 1280) x 1280 28.0 / 18.7 us, 154 x (2 x 1280) x 2048 16.5 / 9.1 us.
extern "C" int mdb_gemm_group(const void* A, const void* const* B, int mats, void* out, int M, int N, int K, long long lda,
                              long long ldb, long long ldo, int ctas, int bn, void* stream_ptr) {
  using namespace mdb;
  using namespace mdb::gemm;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (mats < 1 || mats > MAX_MATS) return 3008;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldo & 7)) return 3001;
  if ((ctas != 1 && ctas != 2) || (bn != 64 && bn != 128 && bn != 192 && bn != 256)) return 3004;
  CUtensorMap ta;
  BMaps tb = {};
  uint64_t da[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(M)}, db[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(N)};
  uint64_t sa[1] = {static_cast<uint64_t>(lda) * 2}, sb[1] = {static_cast<uint64_t>(ldb) * 2};
  uint32_t box_a[2] = {BK, BM}, box_b[2] = {BK, static_cast<uint32_t>(bn / ctas)};
  int rc = encode_tmap_bf16(&ta, A, 2, da, sa, box_a);
  if (rc) return rc;
  for (int i = 0; i < mats; ++i) {
    rc = encode_tmap_bf16(&tb.m[i], B[i], 2, db, sb, box_b);
    if (rc) return rc;
  }
  Params p = {};
  p.M = M; p.N = N; p.K = K;
  p.out = out; p.ldo = ldo;
  p.alpha = 1.0f;
  p.mats = mats;
  p.splits = 1;
  p.kb_per_split = (K + BK - 1) / BK;
  p.bn = bn;
  p.stages = stages_for(bn, ctas, false);
  p.status = status_buffer();
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  return ctas == 2 ? launch<false, false, 2, kPlain>(ta, tb, p, stream) : launch<false, false, 1, kPlain>(ta, tb, p, stream);
}
