// Row kernels for channels-last activations [rows, C] (a row is one pixel / voxel):
//   rms_act : y = act( x / max(||x||_2, eps) * sqrt(C) * gamma + beta ),  act = identity or SiLU
// This is the `WanRMS_norm` + SiLU that precedes every convolution of the Wan VAE's residual blocks
// (src/maxdiffusion/models/wan/autoencoder_kl_wan.py:150-183, 452-484): memory bound, one read and one write of the
// activation. A row of C channels (16 .. 1024) is handled by a group of G = 2 .. 32 lanes, each lane holding VPL
// 16-byte vectors, with G * VPL equal to the row's vector count wherever it factors that way (96 channels = 12
// vectors = 4 lanes x 3, 384 = 16 x 3, 320 = 8 x 5), so that no lane of a warp is idle; the sum of squares is
// reduced with shuffles inside the group, statistics in fp32.
#include "host_common.h"

namespace mdb {
namespace cln {

constexpr int MAX_VPL = 5;  // vectors (8 bf16) per lane

// R rows per group and iteration are loaded before any of them is reduced: a memory-bound kernel needs tens of
// kilobytes in flight per SM, and one 16-byte load per thread is not enough of them.
template <int G, int VPL, int R>
__global__ void __launch_bounds__(256)
rms_act_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, __nv_bfloat16* __restrict__ y, long long ldy,
               const float* __restrict__ gamma, const float* __restrict__ beta, long long rows, int C, float eps,
               int act, int out_w, int out_halo) {
  allow_successor();
  wait_for_predecessor();
  const int vecs = C >> 3;
  const int lane_in_group = threadIdx.x % G;
  const long long group = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / G;
  const long long n_groups = static_cast<long long>(gridDim.x) * blockDim.x / G;
  const float scale = sqrtf(static_cast<float>(C));
  // every lane of a warp runs the same number of iterations (the shuffles below name all 32 lanes)
  const long long iters = (rows + n_groups * R - 1) / (n_groups * R);
  for (long long it = 0; it < iters; ++it) {
    uint4 v[R][VPL];
    float ss[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long row = group + (it * R + r) * n_groups;
      ss[r] = 0.0f;
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int vi = lane_in_group + i * G;
        if (row < rows && vi < vecs) v[r][i] = *reinterpret_cast<const uint4*>(x + row * ldx + vi * 8);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long row = group + (it * R + r) * n_groups;
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int vi = lane_in_group + i * G;
        if (row < rows && vi < vecs) {
          const uint32_t w[4] = {v[r][i].x, v[r][i].y, v[r][i].z, v[r][i].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(w[j]);
            ss[r] += f.x * f.x + f.y * f.y;
          }
        }
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], o);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long row = group + (it * R + r) * n_groups;
      const float inv = scale / fmaxf(sqrtf(ss[r]), eps);
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int vi = lane_in_group + i * G;
        if (row < rows && vi < vecs) {
          const uint32_t w[4] = {v[r][i].x, v[r][i].y, v[r][i].z, v[r][i].w};
          float o[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(w[j]);
            o[2 * j] = f.x * inv;
            o[2 * j + 1] = f.y * inv;
          }
          const float4 g0 = *reinterpret_cast<const float4*>(gamma + vi * 8);
          const float4 g1 = *reinterpret_cast<const float4*>(gamma + vi * 8 + 4);
          o[0] *= g0.x; o[1] *= g0.y; o[2] *= g0.z; o[3] *= g0.w;
          o[4] *= g1.x; o[5] *= g1.y; o[6] *= g1.z; o[7] *= g1.w;
          if (beta != nullptr) {
            const float4 b0 = *reinterpret_cast<const float4*>(beta + vi * 8);
            const float4 b1 = *reinterpret_cast<const float4*>(beta + vi * 8 + 4);
            o[0] += b0.x; o[1] += b0.y; o[2] += b0.z; o[3] += b0.w;
            o[4] += b1.x; o[5] += b1.y; o[6] += b1.z; o[7] += b1.w;
          }
          if (act) {
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = o[j] / (1.0f + __expf(-o[j]));
          }
          uint4 ov;
          ov.x = pack_bf16x2(o[0], o[1]);
          ov.y = pack_bf16x2(o[2], o[3]);
          ov.z = pack_bf16x2(o[4], o[5]);
          ov.w = pack_bf16x2(o[6], o[7]);
          // out_w > 0: the output is the interior of a tensor whose width axis carries out_halo extra columns per side
          const long long yrow = out_w > 0 ? (row / out_w) * (out_w + 2 * out_halo) + out_halo + row % out_w : row;
          *reinterpret_cast<uint4*>(y + yrow * ldy + vi * 8) = ov;
        }
      }
    }
  }
}

}  // namespace cln
}  // namespace mdb

// x, y: bf16 [rows, C] with leading dimensions ldx / ldy (elements, multiples of 8); gamma / beta: fp32 [C]
// (beta may be null); C a multiple of 8, at most 1024. act: 0 identity, 1 SiLU. out_w > 0: x is [.., out_w, C] and y
// is the interior of a [.., out_w + 2 out_halo, C] tensor (y points at its first row, halo column included).
extern "C" int mdb_rms_act_cl(const void* x, long long ldx, void* y, long long ldy, const float* gamma,
                              const float* beta, long long rows, int C, float eps, int act, int out_w, int out_halo,
                              void* stream) {
  using namespace mdb::cln;
  if (rows <= 0) return 0;
  if ((C & 7) || C <= 0 || C > 8 * 32 * MAX_VPL || (ldx & 7) || (ldy & 7) || gamma == nullptr || out_halo < 0 ||
      (out_w > 0 && rows % out_w))
    return 3701;
  const int vecs = C >> 3;
  // widest group whose lanes are all busy; rows that do not factor fall back to a full warp with a ragged last pass
  int G = 0, vpl = 0;
  for (int g = 32; g >= 2 && G == 0; g >>= 1)
    if (vecs % g == 0 && vecs / g <= MAX_VPL && (vecs / g == 1 || vecs / g == 3 || vecs / g == 5 || g == 32)) G = g, vpl = vecs / g;
  if (G == 0) {
    G = vecs <= 8 ? 8 : (vecs <= 16 ? 16 : 32);
    vpl = (vecs + G - 1) / G;
  }
  const int R = vpl <= 2 ? 4 : (vpl <= 4 ? 2 : 1);
  const long long groups_per_block = 256 / G;
  long long blocks = (rows + groups_per_block * R - 1) / (groups_per_block * R);
  const long long cap = static_cast<long long>(mdb::sm_count()) * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  __nv_bfloat16* yp = static_cast<__nv_bfloat16*>(y);
  const int nb = static_cast<int>(blocks);
#define MDB_RMS_ACT(GG, VV, RR) \
  mdb::launch_overlapped(rms_act_kernel<GG, VV, RR>, nb, 256, 0, st, xp, ldx, yp, ldy, gamma, beta, rows, C, eps, act, out_w, out_halo)
#define MDB_RMS_ACT_G(GG)                         \
  if (G == GG) {                                  \
    if (vpl == 1) MDB_RMS_ACT(GG, 1, 4);          \
    else if (vpl == 3) MDB_RMS_ACT(GG, 3, 2);     \
    else if (vpl == 5) MDB_RMS_ACT(GG, 5, 1);     \
    else return 3701;                             \
  }
  if (G == 32) {
    if (vpl == 1) MDB_RMS_ACT(32, 1, 4);
    else if (vpl == 2) MDB_RMS_ACT(32, 2, 4);
    else if (vpl == 3) MDB_RMS_ACT(32, 3, 2);
    else if (vpl == 4) MDB_RMS_ACT(32, 4, 2);
    else MDB_RMS_ACT(32, 5, 1);
  }
  else MDB_RMS_ACT_G(16)
  else MDB_RMS_ACT_G(8)
  else MDB_RMS_ACT_G(4)
  else MDB_RMS_ACT_G(2)
  else return 3701;
#undef MDB_RMS_ACT_G
#undef MDB_RMS_ACT
  return static_cast<int>(cudaGetLastError());
}

// ---------------------------------------------------------------------------------------------------------------
// GroupNorm (+ SiLU) for channels-last activations [N, HW, C], forward and backward
// (UNet ResNet blocks and the image VAE: src/maxdiffusion/models/resnet_flax.py:97-186, vae_flax.py).
//
// A group's channels are neither contiguous over a pixel nor aligned to 16-byte vectors (320 channels in 32 groups
// are 10 channels each), so both passes work per CHANNEL and the groups appear only in a tiny fold in between:
//   sums  : partial[n, split, c] = {sum f1, sum f2} over a strip of pixels; forward (f1, f2) = (x, x^2), backward
//           (f1, f2) = (dy', dy' * x) with dy' = dy * silu'(x * scale + shift) when the activation is fused
//   fold  : (host side, on [N, C]-sized arrays) group statistics -> per-(n, c) coefficients
//   apply : forward y = act(x * a + b); backward dx = dy' * a + b + x * c, coefficients fp32 [N, C]
// One strip of pixels per CTA, a thread keeps one 8-channel vector in registers over the rows of the strip; partial
// sums are combined in a fixed order, so results are bitwise reproducible.
// ---------------------------------------------------------------------------------------------------------------
namespace mdb {
namespace cln {

__device__ __forceinline__ float silu_grad(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// grid (splits, N), block = rows_per_pass * vecs threads. act_a / act_b: forward coefficients for the fused SiLU of the
// backward pass (null: none). dy null: forward sums of x.
__global__ void __launch_bounds__(256)
gn_cl_sums_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, const float* __restrict__ act_a,
                  const float* __restrict__ act_b, float2* __restrict__ partial, int HW, int C, int rows_per_pass) {
  allow_successor();
  wait_for_predecessor();
  extern __shared__ float red[];  // [rows_per_pass][vecs][16]
  const int vecs = C >> 3;
  const int v = threadIdx.x % vecs, r = threadIdx.x / vecs;
  const int n = blockIdx.y, splits = gridDim.x;
  const int per = (HW + splits - 1) / splits;
  const int row0 = blockIdx.x * per, row1 = min(HW, row0 + per);
  float s1[8], s2[8], a[8], b[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s1[j] = s2[j] = 0.0f;
  if (dy != nullptr && act_a != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      a[j] = act_a[static_cast<long long>(n) * C + v * 8 + j];
      b[j] = act_b[static_cast<long long>(n) * C + v * 8 + j];
    }
  }
  int row = row0 + r;
  if (dy == nullptr) {
    // four rows in flight: one at a time, a strip took a memory latency per row (mean over the 56 norms of a Stable
    // Diffusion 1.5 step: 9.2 us, 4.3 us so and with strips of 16 rows)
    for (; row + 3 * rows_per_pass < row1; row += 4 * rows_per_pass) {
      uint4 u[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        u[k] = *reinterpret_cast<const uint4*>(x + (static_cast<long long>(n) * HW + row + k * rows_per_pass) * C + v * 8);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t w[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(w[j]);
          s1[2 * j] += f.x;
          s1[2 * j + 1] += f.y;
          s2[2 * j] += f.x * f.x;
          s2[2 * j + 1] += f.y * f.y;
        }
      }
    }
  }
  for (; row < row1; row += rows_per_pass) {
    const long long off = (static_cast<long long>(n) * HW + row) * C + v * 8;
    const uint4 xv = *reinterpret_cast<const uint4*>(x + off);
    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
    float xf[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(xw[j]);
      xf[2 * j] = f.x;
      xf[2 * j + 1] = f.y;
    }
    if (dy == nullptr) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s1[j] += xf[j];
        s2[j] += xf[j] * xf[j];
      }
    } else {
      const uint4 dv = *reinterpret_cast<const uint4*>(dy + off);
      const uint32_t dw[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(dw[j]);
        float d0 = f.x, d1 = f.y;
        if (act_a != nullptr) {
          d0 *= silu_grad(xf[2 * j] * a[2 * j] + b[2 * j]);
          d1 *= silu_grad(xf[2 * j + 1] * a[2 * j + 1] + b[2 * j + 1]);
        }
        s1[2 * j] += d0;
        s1[2 * j + 1] += d1;
        s2[2 * j] += d0 * xf[2 * j];
        s2[2 * j + 1] += d1 * xf[2 * j + 1];
      }
    }
  }
  float* mine = red + (static_cast<size_t>(r) * vecs + v) * 16;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    mine[j] = s1[j];
    mine[8 + j] = s2[j];
  }
  __syncthreads();
  if (r == 0) {
    for (int rr = 1; rr < rows_per_pass; ++rr) {  // fixed order
      const float* o = red + (static_cast<size_t>(rr) * vecs + v) * 16;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s1[j] += o[j];
        s2[j] += o[8 + j];
      }
    }
    float2* dst = partial + (static_cast<long long>(n) * splits + blockIdx.x) * C + v * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) dst[j] = make_float2(s1[j], s2[j]);
  }
}

// forward: y = act(x * a + b). backward (dy != null): dx = dy' * a + b + x * c, dy' = dy * silu'(x * fa + fb) if fa.
__global__ void __launch_bounds__(256)
gn_cl_apply_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ out,
                   const float* __restrict__ ca, const float* __restrict__ cb, const float* __restrict__ cc,
                   const float* __restrict__ fa, const float* __restrict__ fb, long long total_vecs, int HW, int C,
                   int act) {
  allow_successor();
  wait_for_predecessor();
  const int vecs = C >> 3;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total_vecs;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % vecs);
    const long long row = i / vecs;
    const int n = static_cast<int>(row / HW);
    const long long cbase = static_cast<long long>(n) * C + v * 8;
    const uint4 xv = *reinterpret_cast<const uint4*>(x + i * 8);
    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
    float xf[8], o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(xw[j]);
      xf[2 * j] = f.x;
      xf[2 * j + 1] = f.y;
    }
    const float4 a0 = *reinterpret_cast<const float4*>(ca + cbase), a1 = *reinterpret_cast<const float4*>(ca + cbase + 4);
    const float4 b0 = *reinterpret_cast<const float4*>(cb + cbase), b1 = *reinterpret_cast<const float4*>(cb + cbase + 4);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    if (dy == nullptr) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float z = xf[j] * av[j] + bv[j];
        o[j] = act ? z / (1.0f + __expf(-z)) : z;
      }
    } else {
      const uint4 dv = *reinterpret_cast<const uint4*>(dy + i * 8);
      const uint32_t dw[4] = {dv.x, dv.y, dv.z, dv.w};
      float df[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(dw[j]);
        df[2 * j] = f.x;
        df[2 * j + 1] = f.y;
      }
      if (fa != nullptr) {
#pragma unroll
        for (int j = 0; j < 8; ++j) df[j] *= silu_grad(xf[j] * fa[cbase + j] + fb[cbase + j]);
      }
      const float4 c0 = *reinterpret_cast<const float4*>(cc + cbase), c1 = *reinterpret_cast<const float4*>(cc + cbase + 4);
      const float cv[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = df[j] * av[j] + bv[j] + xf[j] * cv[j];
    }
    uint4 ov;
    ov.x = pack_bf16x2(o[0], o[1]);
    ov.y = pack_bf16x2(o[2], o[3]);
    ov.z = pack_bf16x2(o[4], o[5]);
    ov.w = pack_bf16x2(o[6], o[7]);
    *reinterpret_cast<uint4*>(out + i * 8) = ov;
  }
}

}  // namespace cln
}  // namespace mdb

// Per-channel partial sums over `splits` strips of pixels: partial fp32 [N, splits, C, 2]. x (and dy) bf16 [N, HW, C],
// contiguous, C a multiple of 8 and at most 2048. act_a / act_b (fp32 [N, C], may be null) select the fused-SiLU form
// of the backward sums.
extern "C" int mdb_gn_cl_sums(const void* x, const void* dy, const float* act_a, const float* act_b, float* partial, int N,
                              int HW, int C, int splits, void* stream) {
  using namespace mdb::cln;
  if (N <= 0 || HW <= 0) return 0;
  const int vecs = C >> 3;
  if ((C & 7) || vecs < 1 || vecs > 256 || splits < 1) return 3702;
  const int rows_per_pass = 256 / vecs;
  const int threads = rows_per_pass * vecs;
  const size_t smem = static_cast<size_t>(threads) * 16 * sizeof(float);
  mdb::launch_overlapped(gn_cl_sums_kernel, dim3(splits, N), threads, smem, static_cast<cudaStream_t>(stream),
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dy), act_a, act_b,
      reinterpret_cast<float2*>(partial), HW, C, rows_per_pass);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mdb_gn_cl_apply(const void* x, const void* dy, void* out, const float* ca, const float* cb, const float* cc,
                               const float* fa, const float* fb, int N, int HW, int C, int act, void* stream) {
  using namespace mdb::cln;
  if (N <= 0 || HW <= 0) return 0;
  if ((C & 7) || ca == nullptr || cb == nullptr || (dy != nullptr && cc == nullptr)) return 3703;
  const long long total = static_cast<long long>(N) * HW * (C >> 3);
  long long blocks = (total + 255) / 256;
  const long long cap = static_cast<long long>(mdb::sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  mdb::launch_overlapped(gn_cl_apply_kernel, static_cast<int>(blocks), 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dy), static_cast<__nv_bfloat16*>(out), ca, cb,
      cc, fa, fb, total, HW, C, act);
  return static_cast<int>(cudaGetLastError());
}

// The fold between the two passes, one CTA per sample: per-channel partial sums [N, splits, C, 2] -> group statistics
// -> per-(n, c) coefficients. The arithmetic is a few thousand values; as PyTorch ops it was a dozen launches per
// normalisation (twenty in the backward), which at the UNet's 176 normalisations per step cost more than the passes.
namespace mdb {
namespace cln {

__device__ __forceinline__ float param_at(const void* p, int is_bf16, int c) {
  if (p == nullptr) return 1.0f;
  return is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[c]) : static_cast<const float*>(p)[c];
}

// The folds run one CTA per (group, sample): with one per sample they were two CTAs that read up to 296 strips one after the
// other, and took longer than the passes over the images beside them (GroupNorm of 2 x 128 x 128 x 320: 57 us, 22 us so).
//
// Sums over the strips of one group's channels into ch[cg][2]; the whole CTA. `red` holds 256 float2. Strips are shared by
// 256 / cg lanes per channel; the order is fixed.
__device__ __forceinline__ void group_channel_sums(const float2* __restrict__ src, int splits, int C, int cg, float2* red,
                                                   float2* ch) {
  for (int c0 = 0; c0 < cg; c0 += 256) {
    const int width = min(256, cg - c0), lanes = 256 / width;
    const int c = threadIdx.x % width, l = threadIdx.x / width;
    float2 t = make_float2(0.0f, 0.0f);
    if (l < lanes) {
#pragma unroll 4
      for (int s = l; s < splits; s += lanes) {
        const float2 v = src[static_cast<long long>(s) * C + c0 + c];
        t.x += v.x;
        t.y += v.y;
      }
    }
    red[threadIdx.x] = t;
    __syncthreads();
    if (threadIdx.x < width) {
      for (int k = 1; k < lanes; ++k) {
        t.x += red[k * width + threadIdx.x].x;
        t.y += red[k * width + threadIdx.x].y;
      }
      ch[c0 + threadIdx.x] = t;
    }
    __syncthreads();
  }
}

// Fixed-order sum of v over the CTA (256 threads); every thread gets it.
__device__ __forceinline__ float2 cta_sum2(float2 v, float2* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float2 t = red[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) {
    t.x += red[w].x;
    t.y += red[w].y;
  }
  __syncthreads();
  return t;
}

// (mean, rstd) of a group from its channel sums; every thread gets them, the first 256 add.
__device__ __forceinline__ float2 group_stats(const float2* ch, int cg, const __nv_bfloat16* sh, float count, float eps, float2* red) {
  float2 t = make_float2(0.0f, 0.0f);
  if (threadIdx.x < 256) {
    for (int j = threadIdx.x; j < cg; j += 256) {
      if (sh != nullptr) {
        const float v = __bfloat162float(sh[j]), hw = count / cg;
        t.x += ch[j].x + hw * v;
        t.y += ch[j].y + v * (2.0f * ch[j].x + hw * v);
      } else {
        t.x += ch[j].x;
        t.y += ch[j].y;
      }
    }
  }
  t = cta_sum2(t, red);
  const float mean = t.x / count;
  return make_float2(mean, rsqrtf(fmaxf(t.y / count - mean * mean, 0.0f) + eps));
}

// (a, b) of channel c, the group's j-th
__device__ __forceinline__ float2 group_coef(float2 mr, const void* gamma, const void* beta, int params_bf16, int c, const __nv_bfloat16* sh,
                                             int j) {
  const float av = mr.y * param_at(gamma, params_bf16, c);
  const float at = sh != nullptr ? __bfloat162float(sh[j]) - mr.x : -mr.x;
  return make_float2(av, (beta != nullptr ? param_at(beta, params_bf16, c) : 0.0f) + at * av);
}

// forward: a = rstd * gamma, b = beta - mean * a; also mean / rstd [N, G] for the backward. `shift` (null: none) holds a value
// per sample and channel that is to be added to x first: the sums of x + t follow from those of x, and act((x + t) a + b) is
// act(x a + (t a + b)), so neither pass over x changes and no pass of its own adds it (an SDXL step at 1024^2: 17 passes of 16 us).
__global__ void __launch_bounds__(256)
gn_cl_fold_fwd_kernel(const float2* __restrict__ partial, int splits, int C, int groups, float count, float eps,
                      const void* gamma, const void* beta, int params_bf16, float* __restrict__ a, float* __restrict__ b,
                      float* __restrict__ mean_out, float* __restrict__ rstd_out, const __nv_bfloat16* __restrict__ shift,
                      long long shift_pitch) {
  allow_successor();
  wait_for_predecessor();
  __shared__ float2 red[256];
  extern __shared__ float2 ch[];  // [cg] channel sums
  const int g = blockIdx.x, n = blockIdx.y, cg = C / groups;
  group_channel_sums(partial + static_cast<long long>(n) * splits * C + g * cg, splits, C, cg, red, ch);
  const __nv_bfloat16* sh = shift != nullptr ? shift + n * shift_pitch + g * cg : nullptr;
  const float2 mr = group_stats(ch, cg, sh, count, eps, red);
  if (threadIdx.x == 0) {
    mean_out[n * groups + g] = mr.x;
    rstd_out[n * groups + g] = mr.y;
  }
  for (int j = threadIdx.x; j < cg; j += 256) {
    const int c = g * cg + j;
    const float2 ab = group_coef(mr, gamma, beta, params_bf16, c, sh, j);
    a[static_cast<long long>(n) * C + c] = ab.x;
    b[static_cast<long long>(n) * C + c] = ab.y;
  }
}

// backward: from d1 = sum dy', d2 = sum dy' * x per channel: dx = dy' * ca + cb + x * cc, and the per-sample terms of
// dgamma (sum dy' * xhat) and dbeta (sum dy')
__global__ void __launch_bounds__(256)
gn_cl_fold_bwd_kernel(const float2* __restrict__ partial, int splits, int C, int groups, float count, const void* gamma,
                      int params_bf16, const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                      float* __restrict__ ca, float* __restrict__ cb, float* __restrict__ cc, float* __restrict__ dgamma_n,
                      float* __restrict__ dbeta_n) {
  __shared__ float2 red[256];
  extern __shared__ float2 ch[];  // [cg] channel sums (d1, d2)
  const int g = blockIdx.x, n = blockIdx.y, cg = C / groups;
  group_channel_sums(partial + static_cast<long long>(n) * splits * C + g * cg, splits, C, cg, red, ch);
  const float mean = mean_in[n * groups + g], rstd = rstd_in[n * groups + g];
  float2 t = make_float2(0.0f, 0.0f);
  for (int j = threadIdx.x; j < cg; j += 256) {
    const int c = g * cg + j;
    const float d1 = ch[j].x, dxhat = rstd * (ch[j].y - mean * ch[j].x);
    dbeta_n[static_cast<long long>(n) * C + c] = d1;
    dgamma_n[static_cast<long long>(n) * C + c] = dxhat;
    const float gm = param_at(gamma, params_bf16, c);
    t.x += gm * d1;
    t.y += gm * dxhat;
  }
  t = cta_sum2(t, red);
  const float s1 = t.x / count, s2 = t.y / count;
  for (int j = threadIdx.x; j < cg; j += 256) {
    const int c = g * cg + j;
    const long long o = static_cast<long long>(n) * C + c;
    ca[o] = rstd * param_at(gamma, params_bf16, c);
    cb[o] = -rstd * s1 + mean * rstd * rstd * s2;
    cc[o] = -rstd * rstd * s2;
  }
}

}  // namespace cln
}  // namespace mdb

// ---------------------------------------------------------------------------------------------------------------
// GroupNorm of few pixels in one launch: a CTA per sample and group holds the group's values in shared memory, so x is read once
// and two launches and their gaps go. Every sum is taken in the order of the kernels it stands for, so the bits are theirs:
//   CF = false: up to 2048 channels, the three launches above (strips, rows of a pass, lanes of the fold);
//   CF = true:  beyond, where they do not go, the channels-first kernels (`groupnorm.cu`: leaves of 8 pixels or of one, the
//               butterfly of a warp, the one over eight warps, channels in order) without the copies to and from their layout.
// Bound by the latency of one CTA's loads and passes over shared memory (4 us and 0.12 us per KB of a group), so it wins where the
// launches of the others cost more. Microseconds, the other kernels / this one: 2 x 8^2 x 1280 7.9 / 4.4, 2 x 16^2 x 1280 9.4 / 6.1,
// 1 x 16^2 x 1920 9.7 / 6.7; channels-first with its copies 2 x 8^2 x 2560 48.5 / 6.6, 2 x 32^2 x 2560 90.2 / 23.7.
// ---------------------------------------------------------------------------------------------------------------
namespace mdb {
namespace cln {

constexpr int GN_GROUP_THREADS = 512;
constexpr int GN_GROUP_SMEM = 226 * 1024;
constexpr int GN_LEAF_CHANNELS = GN_GROUP_THREADS / 32;  // a warp per channel adds the leaves

// Shared memory: float2 [512] (sums across warps), [cg] coefficients, [cg] channel sums, [part] strip sums or leaves, then the values
// as pairs of channels, a pixel's in an odd number of words: threads of neighbouring pixels and channels meet other banks.
struct GroupLayout {
  int part, pitch;
  long long bytes;
};
__host__ __device__ inline GroupLayout group_layout(bool cf, int HW, int cg, int splits) {
  GroupLayout l;
  const int leaves = HW % 8 == 0 ? HW / 8 : HW;
  l.part = cf ? GN_LEAF_CHANNELS * ((leaves < 256 ? leaves : 256) | 1) : splits * cg;
  l.pitch = (cg / 2) | 1;
  l.bytes = (GN_GROUP_THREADS + 2ll * cg + l.part) * 8 + 4ll * HW * l.pitch;
  return l;
}

__device__ __forceinline__ float2 warp_sum2(float2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

template <bool CF>
__global__ void __launch_bounds__(GN_GROUP_THREADS)
gn_cl_group_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int HW, int C, int cg, int splits, float eps,
                   const void* gamma, const void* beta, int params_bf16, const __nv_bfloat16* __restrict__ shift, long long shift_pitch,
                   int act) {
  allow_successor();
  wait_for_predecessor();
  extern __shared__ __align__(16) float2 gn_smem[];
  constexpr int T = GN_GROUP_THREADS;
  const GroupLayout lay = group_layout(CF, HW, cg, splits);
  const int W = cg >> 1, P = lay.pitch, total = HW * W;
  float2 *red = gn_smem, *ab = red + T, *ch = ab + cg, *part = ch + cg;
  uint32_t* held = reinterpret_cast<uint32_t*>(part + lay.part);
  const int g = blockIdx.x, n = blockIdx.y, tid = threadIdx.x;
  const __nv_bfloat16* sh = shift != nullptr ? shift + n * shift_pitch + g * cg : nullptr;
  const long long base = (static_cast<long long>(n) * HW * C + g * cg) >> 1, row_words = C >> 1;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(x) + base;
  uint32_t* dst = reinterpret_cast<uint32_t*>(y) + base;
  // word i is number i % W of pixel i / W; a thread walks i in steps of the block without a division per step
  const int step_pix = T / W, step_w = T % W;
  const int pix0 = tid / W, w0 = tid % W;
  {
    int pix = pix0, w = w0;
    for (int i = tid; i < total; i += 8 * T) {
      uint32_t r[8];
      int at[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        at[u] = pix * P + w;
        if (i + u * T < total) r[u] = src[pix * row_words + w];
        pix += step_pix;
        w += step_w;
        if (w >= W) { w -= W; ++pix; }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i + u * T < total) held[at[u]] = r[u];
    }
  }
  __syncthreads();
  const float count = static_cast<float>(cg) * static_cast<float>(HW);
  if (!CF) {
    const int rows_per_pass = 256 / (C >> 3), per = (HW + splits - 1) / splits;
    for (int task = tid; task < splits * W; task += T) {
      const int s = task / W, cw = task - s * W;
      const int row0 = s * per, row1 = min(HW, row0 + per);
      float2 t0 = make_float2(0.0f, 0.0f), t1 = t0;
      for (int r = 0; r < min(rows_per_pass, per); ++r) {
        float2 s0 = make_float2(0.0f, 0.0f), s1 = s0;
        for (int row = row0 + r; row < row1; row += rows_per_pass) {
          const float2 f = unpack_bf16x2(held[row * P + cw]);
          s0.x += f.x;
          s1.x += f.y;
          s0.y += f.x * f.x;
          s1.y += f.y * f.y;
        }
        t0.x += s0.x;
        t0.y += s0.y;
        t1.x += s1.x;
        t1.y += s1.y;
      }
      part[s * cg + 2 * cw] = t0;
      part[s * cg + 2 * cw + 1] = t1;
    }
    __syncthreads();
    group_channel_sums(part, splits, cg, cg, red, ch);
    const float2 mr = group_stats(ch, cg, sh, count, eps, red);
    for (int j = tid; j < cg; j += T) ab[j] = group_coef(mr, gamma, beta, params_bf16, g * cg + j, sh, j);
  } else {
    const int vec = HW % 8 == 0 ? 8 : 1, leaves = min(256, HW / vec), LP = leaves | 1;
    const int warp = tid >> 5, lane = tid & 31;
    for (int c0 = 0; c0 < cg; c0 += GN_LEAF_CHANNELS) {
      for (int task = tid; task < leaves * (GN_LEAF_CHANNELS / 2); task += T) {
        const int k = task % (GN_LEAF_CHANNELS / 2), t = task / (GN_LEAF_CHANNELS / 2), cw = (c0 >> 1) + k;
        if (cw >= W) continue;
        float2 s0 = make_float2(0.0f, 0.0f), s1 = s0, add = s0;
        if (sh != nullptr) add = make_float2(__bfloat162float(sh[2 * cw]), __bfloat162float(sh[2 * cw + 1]));
        for (int i = t * vec; i < HW; i += 256 * vec) {
#pragma unroll 8
          for (int j = 0; j < vec; ++j) {
            float2 f = unpack_bf16x2(held[(i + j) * P + cw]);
            if (sh != nullptr) f = make_float2(f.x + add.x, f.y + add.y);
            s0.x += f.x;
            s0.y = fmaf(f.x, f.x, s0.y);
            s1.x += f.y;
            s1.y = fmaf(f.y, f.y, s1.y);
          }
        }
        part[2 * k * LP + t] = s0;
        part[(2 * k + 1) * LP + t] = s1;
      }
      __syncthreads();
      if (c0 + warp < cg) {
        float2 keep = make_float2(0.0f, 0.0f);
        for (int v = 0; v * 32 < leaves; ++v) {
          const int t = v * 32 + lane;
          const float2 sum = warp_sum2(t < leaves ? part[warp * LP + t] : make_float2(0.0f, 0.0f));
          if (lane == v) keep = sum;
        }
        keep = warp_sum2(keep);
        if (lane == 0) ch[c0 + warp] = keep;
      }
      __syncthreads();
    }
    if (tid == 0) {
      float2 t = make_float2(0.0f, 0.0f);
      for (int j = 0; j < cg; ++j) {
        t.x += ch[j].x;
        t.y += ch[j].y;
      }
      red[0] = t;
    }
    __syncthreads();
    const float2 t = red[0];
    const float mean = t.x / count;
    const float var = fmaxf(t.y / count - mean * mean, 0.0f);
    const float rstd = rsqrtf(var + eps);
    for (int j = tid; j < cg; j += T) {
      const int c = g * cg + j;
      const float ga = gamma != nullptr ? param_at(gamma, params_bf16, c) : 1.0f, be = beta != nullptr ? param_at(beta, params_bf16, c) : 0.0f;
      const float a = rstd * ga, b = be - mean * rstd * ga;
      ab[j] = make_float2(a, sh != nullptr ? fmaf(__bfloat162float(sh[j]), a, b) : b);
    }
  }
  __syncthreads();
  int pix = pix0, w = w0;
  for (int i = tid; i < total; i += T) {
    const float2 f = unpack_bf16x2(held[pix * P + w]);
    const float4 k = *reinterpret_cast<const float4*>(ab + 2 * w);
    float z0 = fmaf(f.x, k.x, k.y), z1 = fmaf(f.y, k.z, k.w);
    if (act) {
      z0 = z0 / (1.0f + __expf(-z0));
      z1 = z1 / (1.0f + __expf(-z1));
    }
    dst[pix * row_words + w] = pack_bf16x2(z0, z1);
    pix += step_pix;
    w += step_w;
    if (w >= W) { w -= W; ++pix; }
  }
}

}  // namespace cln
}  // namespace mdb

constexpr int kGnGroupElsewhere = 3705;  // `mdb_gn_cl_group`: another path is the faster one, or the only one

// x, y: bf16 [N, HW, C] contiguous; gamma / beta: [C] bf16 (params_bf16 = 1) or fp32, may be null; shift: bf16 [N, C] or null, added to x
// first; splits: the strips of `mdb_gn_cl_sums` for this size. Code 3705 (nothing was launched) where the kernel does not take the
// call; this is the only place where that is decided.
extern "C" int mdb_gn_cl_group(const void* x, void* y, int N, int HW, int C, int groups, int splits, float eps, const void* gamma,
                               const void* beta, int params_bf16, const void* shift, long long shift_pitch, int act, void* stream) {
  using namespace mdb::cln;
  if (N <= 0 || HW <= 0) return 0;
  if (groups <= 0 || C % groups || (C & 7) || splits < 1) return 3704;
  const int cg = C / groups;
  if ((cg & 1) || N > 65535 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15)) return kGnGroupElsewhere;
  const bool cf = C > 2048;
  if (cf) {
    // whatever fits is 2.2 to 18 times as fast (1 to 8 samples of 4^2 to 32^2 x 2560); from 4096 pixels on the channels-first kernels
    // may cut a channel into several sums
    if (HW >= 4096) return kGnGroupElsewhere;
  } else {
    // Three launches / one, 320 to 1920 channels in 32 groups, 4^2 to 40^2 pixels: up to 30 KB a group 1.05 to 1.8 at 32 and 64 CTAs, from 31 KB
    // on 0.91 to 1.07; up to 16 KB 0.99 to 1.5 at 128 and 256 CTAs, from 20 KB on 0.67 to 1.04; one CTA of 40 KB 0.76, 2048 of 20 KB 0.83.
    const long long ctas = static_cast<long long>(groups) * N, most = ctas >= 32 && ctas <= 74 ? 30 * 1024 : ctas <= 256 ? 16 * 1024 : 0;
    if (static_cast<long long>(HW) * cg * 2 > most) return kGnGroupElsewhere;
  }
  const GroupLayout lay = group_layout(cf, HW, cg, splits);
  if (lay.bytes > GN_GROUP_SMEM) return kGnGroupElsewhere;
  auto kern = cf ? gn_cl_group_kernel<true> : gn_cl_group_kernel<false>;
  const int smem = static_cast<int>(lay.bytes);
  if (smem > 40 * 1024) MDB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GN_GROUP_SMEM));
  return static_cast<int>(mdb::launch_overlapped(kern, dim3(groups, N), GN_GROUP_THREADS, static_cast<size_t>(smem),
      static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), HW, C, cg, splits, eps, gamma,
      beta, params_bf16, static_cast<const __nv_bfloat16*>(shift), shift_pitch, act));
}

// partial: fp32 [N, splits, C, 2] from mdb_gn_cl_sums; gamma / beta: [C] bf16 (params_bf16 = 1) or fp32, may be null;
// a, b: fp32 [N, C]; mean, rstd: fp32 [N, groups]. count = pixels * channels per group. shift: bf16 [N, C] or null, added to x.
extern "C" int mdb_gn_cl_fold_shift_fwd(const float* partial, int N, int splits, int C, int groups, float count, float eps,
                                        const void* gamma, const void* beta, int params_bf16, float* a, float* b, float* mean,
                                        float* rstd, const void* shift, long long shift_pitch, void* stream) {
  if (N <= 0) return 0;
  if (groups <= 0 || C % groups || splits < 1 || C > 8192) return 3704;
  if (N > 65535) return 3704;
  const size_t smem = static_cast<size_t>(C / groups) * sizeof(float2);  // at most 64 KB
  if (smem > 40 * 1024)
    MDB_CHECK_CUDA(cudaFuncSetAttribute(mdb::cln::gn_cl_fold_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
  mdb::launch_overlapped(mdb::cln::gn_cl_fold_fwd_kernel, dim3(groups, N), 256, smem, static_cast<cudaStream_t>(stream),
      reinterpret_cast<const float2*>(partial), splits, C, groups, count, eps, gamma, beta, params_bf16, a, b, mean, rstd,
      static_cast<const __nv_bfloat16*>(shift), shift_pitch);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mdb_gn_cl_fold_fwd(const float* partial, int N, int splits, int C, int groups, float count, float eps,
                                  const void* gamma, const void* beta, int params_bf16, float* a, float* b, float* mean,
                                  float* rstd, void* stream) {
  return mdb_gn_cl_fold_shift_fwd(partial, N, splits, C, groups, count, eps, gamma, beta, params_bf16, a, b, mean, rstd, nullptr, 0, stream);
}

// ca, cb, cc, dgamma_n, dbeta_n: fp32 [N, C] (the caller sums the last two over N).
extern "C" int mdb_gn_cl_fold_bwd(const float* partial, int N, int splits, int C, int groups, float count, const void* gamma,
                                  int params_bf16, const float* mean, const float* rstd, float* ca, float* cb, float* cc,
                                  float* dgamma_n, float* dbeta_n, void* stream) {
  if (N <= 0) return 0;
  if (groups <= 0 || C % groups || splits < 1 || C > 8192) return 3704;
  if (N > 65535) return 3704;
  const size_t smem = static_cast<size_t>(C / groups) * sizeof(float2);  // at most 64 KB
  if (smem > 40 * 1024)
    MDB_CHECK_CUDA(cudaFuncSetAttribute(mdb::cln::gn_cl_fold_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
  mdb::cln::gn_cl_fold_bwd_kernel<<<dim3(groups, N), 256, smem, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float2*>(partial), splits, C, groups, count, gamma, params_bf16, mean, rstd, ca, cb, cc, dgamma_n,
      dbeta_n);
  return static_cast<int>(cudaGetLastError());
}

// ---------------------------------------------------------------------------------------------------------------
// Row softmax, in place or out of place: y[r, :] = softmax(x[r, :]) for bf16 rows of up to 32768 columns, fp32 math.
// One CTA per row, the row lives in registers between the two reductions (one read, one write). It sits between the two
// GEMMs of attention with a head size the flash kernels are not built for (the Wan VAE's single 384-wide head,
// src/maxdiffusion/models/wan/autoencoder_kl_wan.py:487-546): scores = Q K^T on the GEMM kernel, this, then P V.
// ---------------------------------------------------------------------------------------------------------------
namespace mdb {
namespace cln {

constexpr int SM_THREADS = 256;
constexpr int SM_MAX_VPT = 16;  // vectors of 8 per thread

__device__ __forceinline__ float block_reduce(float v, bool is_max, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float w = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmaxf(v, w) : v + w;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();  // red may still be read from the previous reduction
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = red[0];
#pragma unroll
  for (int i = 1; i < SM_THREADS / 32; ++i) t = is_max ? fmaxf(t, red[i]) : t + red[i];
  return t;
}

template <int VPT>
__global__ void __launch_bounds__(SM_THREADS)
softmax_rows_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, __nv_bfloat16* __restrict__ y, long long ldy, int cols) {
  __shared__ float red[SM_THREADS / 32];
  const long long row = blockIdx.x;
  const int vecs = cols >> 3;
  float v[VPT][8];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int vi = threadIdx.x + i * SM_THREADS;
    if (vi < vecs) {
      const uint4 u = *reinterpret_cast<const uint4*>(x + row * ldx + vi * 8);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(w[j]);
        v[i][2 * j] = f.x;
        v[i][2 * j + 1] = f.y;
        mx = fmaxf(mx, fmaxf(f.x, f.y));
      }
    }
  }
  mx = block_reduce(mx, true, red);
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int vi = threadIdx.x + i * SM_THREADS;
    if (vi < vecs) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[i][j] = __expf(v[i][j] - mx);
        sum += v[i][j];
      }
    }
  }
  sum = block_reduce(sum, false, red);
  const float inv = 1.0f / sum;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int vi = threadIdx.x + i * SM_THREADS;
    if (vi < vecs) {
      uint4 o;
      o.x = pack_bf16x2(v[i][0] * inv, v[i][1] * inv);
      o.y = pack_bf16x2(v[i][2] * inv, v[i][3] * inv);
      o.z = pack_bf16x2(v[i][4] * inv, v[i][5] * inv);
      o.w = pack_bf16x2(v[i][6] * inv, v[i][7] * inv);
      *reinterpret_cast<uint4*>(y + row * ldy + vi * 8) = o;
    }
  }
}

}  // namespace cln
}  // namespace mdb

// x, y: bf16 [rows, cols] with leading dimensions ldx / ldy (multiples of 8); cols a multiple of 8, at most 32768.
extern "C" int mdb_softmax_rows(const void* x, long long ldx, void* y, long long ldy, long long rows, int cols, void* stream) {
  using namespace mdb::cln;
  if (rows <= 0) return 0;
  if ((cols & 7) || cols <= 0 || cols > 8 * SM_THREADS * SM_MAX_VPT || (ldx & 7) || (ldy & 7) || rows >= (1ll << 31)) return 3704;
  const int vpt = ((cols >> 3) + SM_THREADS - 1) / SM_THREADS;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  __nv_bfloat16* yp = static_cast<__nv_bfloat16*>(y);
  const int grid = static_cast<int>(rows);
  if (vpt <= 1) softmax_rows_kernel<1><<<grid, SM_THREADS, 0, st>>>(xp, ldx, yp, ldy, cols);
  else if (vpt <= 2) softmax_rows_kernel<2><<<grid, SM_THREADS, 0, st>>>(xp, ldx, yp, ldy, cols);
  else if (vpt <= 4) softmax_rows_kernel<4><<<grid, SM_THREADS, 0, st>>>(xp, ldx, yp, ldy, cols);
  else if (vpt <= 8) softmax_rows_kernel<8><<<grid, SM_THREADS, 0, st>>>(xp, ldx, yp, ldy, cols);
  else softmax_rows_kernel<16><<<grid, SM_THREADS, 0, st>>>(xp, ldx, yp, ldy, cols);
  return static_cast<int>(cudaGetLastError());
}
