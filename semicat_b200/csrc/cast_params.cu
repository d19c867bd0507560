// The 16-bit copies of a model's fp32 parameters that one pass under autocast needs, in one launch per 64 parameters instead
// of one each: scaled, cast and zero-padded (the vocabulary-sized matrices, whose rows the BLAS library wants on 16 bytes).
// What it saves is launches: the casts and paddings of a sampling pass of the twelve-block denoiser took 450 us in 120 of them and
// take 205 us in two (3.9 TB/s), and the pass, which is bound by the host, 3.7 -> 2.5 ms with the modulation of all blocks in
// one GEMM.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "jvpattn_common.cuh"

namespace jvpattn {
namespace {

constexpr int kEntries = 64, kThreads = 256, kChunks = 4;  // a block takes kChunks chunks of 8 outputs per thread

struct CastTable {
  jvpattn_cast e[kEntries];
  int first[kEntries + 1];  // of an entry's blocks
  int n;
};

template <typename T>
__global__ void __launch_bounds__(kThreads) cast_params_kernel(const __grid_constant__ CastTable t) {
  int lo = 0, hi = t.n - 1;  // the entry that holds this block
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (t.first[mid] <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const jvpattn_cast &e = t.e[lo];
  const int64_t n_out = (int64_t)e.rows_out * e.cols_out, base = ((int64_t)blockIdx.x - t.first[lo]) * (kThreads * kChunks);
  const bool padded = e.rows_out != e.rows || e.cols_out != e.cols;
  const bool pairs = reinterpret_cast<uintptr_t>(e.src) % 8 == 0 && (!padded || e.cols % 2 == 0);
  const bool vec = reinterpret_cast<uintptr_t>(e.src) % 16 == 0 && (!padded || e.cols % 4 == 0);
  float v[kChunks][8];
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int64_t o = (base + c * kThreads + threadIdx.x) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[c][i] = 0.f;
    if (o >= n_out) continue;
    // (a 64-bit division per chunk costs more than its arithmetic)
    const uint32_t row = !padded ? 0 : n_out <= 0xffffffffLL ? (uint32_t)o / (uint32_t)e.cols_out : (uint32_t)(o / e.cols_out);
    const uint32_t col = padded ? (uint32_t)(o - (int64_t)row * e.cols_out) : 0;
    // (cols_out is a multiple of 8 where there is padding: a chunk stays in its row)
    const int64_t left = padded ? (row < (uint32_t)e.rows ? (int64_t)e.cols - col : 0) : n_out - o;
    const float *src = e.src + (padded ? (int64_t)row * e.cols + col : o);
    if (vec && left >= 8) {
      const float4 a = reinterpret_cast<const float4 *>(src)[0], b = reinterpret_cast<const float4 *>(src)[1];
      v[c][0] = a.x, v[c][1] = a.y, v[c][2] = a.z, v[c][3] = a.w, v[c][4] = b.x, v[c][5] = b.y, v[c][6] = b.z, v[c][7] = b.w;
    } else if (pairs && left >= 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = reinterpret_cast<const float2 *>(src)[i];
        v[c][2 * i] = a.x, v[c][2 * i + 1] = a.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < left) v[c][i] = src[i];
    }
  }
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int64_t o = (base + c * kThreads + threadIdx.x) * 8;
    if (o >= n_out) continue;
    T *dst = static_cast<T *>(e.dst) + o;
    if (o + 8 <= n_out) {
      uint4 u;
      T *h = reinterpret_cast<T *>(&u);
#pragma unroll
      for (int i = 0; i < 8; ++i) h[i] = Elem<T>::from_f(v[c][i] * e.scale);
      *reinterpret_cast<uint4 *>(dst) = u;
    } else {
      for (int i = 0; i < (int)(n_out - o); ++i) dst[i] = Elem<T>::from_f(v[c][i] * e.scale);
    }
  }
}

}  // namespace

cudaError_t cast_params(const jvpattn_cast *entries, int n, int dtype, cudaStream_t stream) {
  for (int i0 = 0; i0 < n; i0 += kEntries) {
    CastTable t{};
    t.n = std::min(kEntries, n - i0);
    int64_t blocks = 0;
    for (int i = 0; i < t.n; ++i) {
      t.e[i] = entries[i0 + i];
      t.first[i] = (int)blocks;
      const int64_t chunks = ((int64_t)t.e[i].rows_out * t.e[i].cols_out + 7) / 8;
      blocks += (chunks + kThreads * kChunks - 1) / (kThreads * kChunks);
    }
    t.first[t.n] = (int)blocks;
    if (blocks == 0) continue;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    LaunchScope scope(kIdDual, stream);
    if (dtype == JVPATTN_BF16) cast_params_kernel<__nv_bfloat16><<<(unsigned)blocks, kThreads, 0, stream>>>(t);
    else cast_params_kernel<__half><<<(unsigned)blocks, kThreads, 0, stream>>>(t);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace jvpattn
