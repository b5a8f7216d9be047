// Row softmax of fp32 scores for a second product that keeps fp32 probabilities: y = p0 + p1 + p2, three bf16 planes of `pitch`
// columns side by side, so that a bf16 product with a matrix stacked three times accumulates p to 24 bits. Columns from `cols` to
// `pitch` are zeros. The probabilities are those of a plain fp32 softmax: a rounded difference, expf, fp32 sums, a division.
//
// Built without --use_fast_math (`build.py: PRECISE`), where expf is the two-ulp function and not a flush-to-zero
// approximation. The row waits in shared memory between the passes; bound by memory (one read of 4 bytes, one write of 6).
#include "host_common.h"
#include "ptx.cuh"

namespace mdb {
namespace smsplit {

constexpr int THREADS = 256;

__device__ __forceinline__ float cta_max(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = red[0];
#pragma unroll
  for (int i = 1; i < THREADS / 32; ++i) t = fmaxf(t, red[i]);
  __syncthreads();
  return t;
}

__device__ __forceinline__ float cta_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = red[0];
#pragma unroll
  for (int i = 1; i < THREADS / 32; ++i) t += red[i];
  __syncthreads();
  return t;
}

__global__ void __launch_bounds__(THREADS)
softmax_split_kernel(const float* __restrict__ x, long long ldx, __nv_bfloat16* __restrict__ y, long long ldy, int cols, int pitch) {
  extern __shared__ float row_s[];
  __shared__ float red[THREADS / 32];
  const float* src = x + static_cast<long long>(blockIdx.x) * ldx;
  __nv_bfloat16* dst = y + static_cast<long long>(blockIdx.x) * ldy;
  float mx = -INFINITY;
  for (int c = threadIdx.x; c < cols; c += THREADS) {
    const float v = src[c];
    row_s[c] = v;
    mx = fmaxf(mx, v);
  }
  mx = cta_max(mx, red);
  float sum = 0.0f;
  for (int c = threadIdx.x; c < cols; c += THREADS) {
    const float p = expf(row_s[c] - mx);  // 0 for -inf; NaN in a row of -inf alone, for +inf and for NaN
    row_s[c] = p;
    sum += p;
  }
  sum = cta_sum(sum, red);
  for (int c = threadIdx.x; c < pitch; c += THREADS) {
    const float p = c < cols ? row_s[c] / sum : 0.0f;
    const __nv_bfloat16 p0 = __float2bfloat16(p);
    const float r1 = p - __bfloat162float(p0);
    const __nv_bfloat16 p1 = __float2bfloat16(r1);
    dst[c] = p0;
    dst[pitch + c] = p1;
    dst[2 * pitch + c] = __float2bfloat16(r1 - __bfloat162float(p1));
  }
}

}  // namespace smsplit
}  // namespace mdb

// x fp32 [rows, cols] (row pitch ldx) -> y bf16 [rows, 3 * pitch] (row pitch ldy).
extern "C" int mdb_softmax_split(const float* x, long long ldx, void* y, long long ldy, long long rows, int cols, int pitch,
                                 void* stream) {
  using namespace mdb::smsplit;
  if (rows <= 0 || cols <= 0) return 0;
  if (pitch < cols || cols > 32768 || ldy < 3ll * pitch || rows > 0x7fffffff) return 3705;
  const size_t smem = static_cast<size_t>(cols) * sizeof(float);
  if (smem > 40 * 1024)
    MDB_CHECK_CUDA(cudaFuncSetAttribute(softmax_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024));
  softmax_split_kernel<<<static_cast<unsigned int>(rows), THREADS, smem, static_cast<cudaStream_t>(stream)>>>(
      x, ldx, static_cast<__nv_bfloat16*>(y), ldy, cols, pitch);
  return static_cast<int>(cudaGetLastError());
}
