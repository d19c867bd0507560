// Sum over the rows of a bf16 matrix, accumulated in fp32 and rounded once: the gradient of a linear layer's bias.
//
// Bound by memory: one read of the matrix.  Warps read 512 contiguous bytes of a row, 8 rows in flight per thread; the rows are
// split over enough CTAs to fill the GPU, whose sums go to a workspace and meet in a second launch, always in the same order.
// With torch's reduction 12288 x 768 took 23.9 us, so 8.8 (2.9 at the rate of a copy); x 3072 29.3 and 16.6 (11.6); 49152 x 3072 66.7 and 49.4
// (46.3); 96 x 4608 6.5 and 4.4.  In one launch, clusters of 8 CTAs on 32 or 64 columns meeting through distributed shared
// memory, the first two took 12.3 and 31: 64 to 128 bytes of a row at a time are read at a third of the rate.
#include <cuda_bf16.h>

#include <algorithm>

#include "jvpattn_common.cuh"

namespace jvpattn {
namespace {

constexpr int kWarps = 8, kCols = 256, kInFlight = 8;  // of a CTA: a warp per row, 8 columns per lane

__global__ void __launch_bounds__(kWarps * 32) column_sum_kernel(const __nv_bfloat16 *x, int64_t rows, int cols, int64_t ld, int64_t rows_cta, float *part) {
  __shared__ float4 smem[kWarps][2][32];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, c0 = blockIdx.x * kCols + lane * 8;
  const int64_t r0 = blockIdx.y * rows_cta, r1 = min(rows, r0 + rows_cta);
  float s[8] = {};
  auto add = [&](uint4 v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[2 * j] += __uint_as_float(w[j] << 16);
      s[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
    }
  };
  if (c0 < cols) {
    const __nv_bfloat16 *p = x + (r0 + warp) * ld + c0;
    int64_t r = r0 + warp;
    for (; r + (kInFlight - 1) * kWarps < r1; r += kInFlight * kWarps, p += kInFlight * kWarps * ld) {
      uint4 v[kInFlight];
#pragma unroll
      for (int k = 0; k < kInFlight; ++k) v[k] = *reinterpret_cast<const uint4 *>(p + k * kWarps * ld);
#pragma unroll
      for (int k = 0; k < kInFlight; ++k) add(v[k]);
    }
    uint4 v[kInFlight - 1];
#pragma unroll
    for (int k = 0; k < kInFlight - 1; ++k) {
      v[k] = make_uint4(0, 0, 0, 0);
      if (r + k * kWarps < r1) v[k] = *reinterpret_cast<const uint4 *>(p + k * kWarps * ld);
    }
#pragma unroll
    for (int k = 0; k < kInFlight - 1; ++k) add(v[k]);
  }
  smem[warp][0][lane] = make_float4(s[0], s[1], s[2], s[3]);
  smem[warp][1][lane] = make_float4(s[4], s[5], s[6], s[7]);
  __syncthreads();
  if (threadIdx.x < 64) {
    const int l = threadIdx.x / 2, h = threadIdx.x % 2, c = blockIdx.x * kCols + l * 8 + h * 4;
    float4 t = smem[0][h][l];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) {
      const float4 u = smem[w][h][l];
      t.x += u.x, t.y += u.y, t.z += u.z, t.w += u.w;
    }
    if (c < cols) *reinterpret_cast<float4 *>(part + (int64_t)blockIdx.y * cols + c) = t;
  }
}

// 32 columns per CTA, a warp per 8th of the partial sums
__global__ void __launch_bounds__(256) column_sum_finish_kernel(const float *part, int n, int cols, __nv_bfloat16 *out) {
  __shared__ float smem[8][32];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, c = blockIdx.x * 32 + lane;
  float t = 0.f;
  if (c < cols) {
#pragma unroll 8
    for (int k = warp; k < n; k += 8) t += part[(int64_t)k * cols + c];
  }
  smem[warp][lane] = t;
  __syncthreads();
  if (warp == 0 && c < cols) {
#pragma unroll
    for (int w = 1; w < 8; ++w) t += smem[w][lane];
    out[c] = __float2bfloat16(t);
  }
}

// CTAs that share a column group's rows: four per SM in all (what an SM holds at once is five; with two 12288 x 3072 took 19.2 us, with eight
// 17.8), 32 rows each at least.
int64_t splits(int64_t rows, int cols) {
  const int64_t groups = (cols + kCols - 1) / kCols;
  return std::max<int64_t>(1, std::min<int64_t>(148 * 4 / groups, rows / 32));
}

}  // namespace

int64_t column_sum_workspace(int64_t rows, int cols) { return splits(rows, cols) * cols * 4; }

cudaError_t column_sum(const void *x, int64_t rows, int cols, int64_t ld, void *out, float *workspace, cudaStream_t stream) {
  if (cols == 0) return cudaSuccess;
  const int64_t per = (rows + splits(rows, cols) - 1) / splits(rows, cols), n = per ? (rows + per - 1) / per : 1;
  {
    LaunchScope scope(kIdDual, stream);
    const dim3 grid((unsigned)((cols + kCols - 1) / kCols), (unsigned)n);
    column_sum_kernel<<<grid, kWarps * 32, 0, stream>>>(static_cast<const __nv_bfloat16 *>(x), rows, cols, ld, per, workspace);
  }
  LaunchScope scope(kIdDual, stream);
  column_sum_finish_kernel<<<(unsigned)((cols + 31) / 32), 256, 0, stream>>>(workspace, (int)n, cols, static_cast<__nv_bfloat16 *>(out));
  return cudaGetLastError();
}

}  // namespace jvpattn
