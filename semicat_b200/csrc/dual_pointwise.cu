// Dual-number pointwise kernels for the denoiser block around the attention: every op takes a primal and a tangent and
// returns both in one pass, and has a hand-written VJP for the cotangents of both outputs.  Under torch.func.jvp the same
// algebra runs as a dozen small kernels per op and per pass (primal and tangent separately), which is what bounds the
// training step once the batch is sharded over several GPUs.
//
//   ln_modulate     h = LN(x) * (1 + scale) + shift        (semicat/net/duo.py:128-135, 159: LayerNorm + adaLN modulation)
//   gated_residual  z = x + m * (g * y)                    (duo.py:157, 160: dropout(branch * gate) + skip; m = dropout keep
//                                                           mask / (1 - p): a tensor, or regenerated here from a seed)
//   gelu_dual       the tanh-form GELU of the MLP          (duo.py:118-123)
//
// LayerNorm: one warp owns one row of C channels (C = 256, 512, 768 or 1024; one element type, bf16 or fp32, for every
// tensor but the fp32 LayerNorm weight and bias): 16-byte loads, fp32 arithmetic, warp-shuffle row reductions; column
// sums that feed the gradients of per-sample or per-channel parameters are accumulated per CTA (registers, then one
// shared-memory slice per warp) and added to fp32 [B, C] buffers with one atomic per column and CTA (a CTA stays inside
// one sample); ln_finalize turns them into the parameter gradients.  Gated residual and GELU: 8 elements per thread.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "jvpattn_common.cuh"

namespace jvpattn {
namespace {

constexpr int kWarpsPerCta = 4;

template <typename T>
__device__ __forceinline__ void load8(const T *p, float (&f)[8]);
template <>
__device__ __forceinline__ void load8<float>(const float *p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
// 8 elements as loaded.  Copied as a whole before anything looks into it: bf16 pairs read through a reference to global memory
// are loads of 4 bytes each (LayerNorm forward of 32 x 128 rows of 768: 6.2 us so, 5.0 us with one load of 16 bytes).
template <typename T> struct Raw8 { uint4 q[sizeof(T) / 2]; };
template <typename T>
__device__ __forceinline__ Raw8<T> load_raw8(const T *p) {
  Raw8<T> u;
#pragma unroll
  for (int i = 0; i < (int)(sizeof(T) / 2); ++i) u.q[i] = reinterpret_cast<const uint4 *>(p)[i];
  return u;
}
__device__ __forceinline__ void unpack8(const Raw8<float> &u, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    f[4 * i] = __uint_as_float(u.q[i].x), f[4 * i + 1] = __uint_as_float(u.q[i].y);
    f[4 * i + 2] = __uint_as_float(u.q[i].z), f[4 * i + 3] = __uint_as_float(u.q[i].w);
  }
}
__device__ __forceinline__ void unpack8(const Raw8<__nv_bfloat16> &u, float (&f)[8]) {
  const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u.q[0]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(h[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16 *p, float (&f)[8]) {
  unpack8(load_raw8(p), f);
}
template <typename T> __device__ __forceinline__ float ldf(const T *p);
template <> __device__ __forceinline__ float ldf<float>(const float *p) { return *p; }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16 *p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T *p, float v);
template <> __device__ __forceinline__ void stf<float>(float *p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }
template <typename T>
__device__ __forceinline__ void store8(T *p, const float (&f)[8]);
template <>
__device__ __forceinline__ void store8<float>(float *p, const float (&f)[8]) {
  reinterpret_cast<float4 *>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4 *>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
template <>
__device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16 *p, const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4 *>(p) = u;
}

// Adds 8 adjacent sums to global memory as two 16-byte reductions.  Element by element, the lanes of each instruction are 32
// bytes apart: 32 sectors per request.  128 x 128 rows of 768: LayerNorm backward 60 -> 49 us, gated residual
// backward 61 -> 51 us.
__device__ __forceinline__ void add8(float *dst, const float (&f)[8]) {
  if (reinterpret_cast<uintptr_t>(dst) % 16 == 0) {
    atomicAdd(reinterpret_cast<float4 *>(dst), make_float4(f[0], f[1], f[2], f[3]));
    atomicAdd(reinterpret_cast<float4 *>(dst) + 1, make_float4(f[4], f[5], f[6], f[7]));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) atomicAdd(dst + i, f[i]);
  }
}

__device__ __forceinline__ float2 splat(float x) { return make_float2(x, x); }

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Channel index of element e of vector v of this lane: vectors of 8 channels, lanes interleaved (coalesced 16-byte loads).
__device__ __forceinline__ int chan(int v, int lane) { return (v * 32 + lane) * 8; }

struct LnArgs {
  const void *x, *tx;            // [rows, C]
  const float *gamma, *beta;     // [C] (beta may be null: no bias)
  const void *shift, *scale;     // [B, C] rows `mod_stride` elements apart
  const void *tshift, *tscale;   // tangents of shift / scale (null = zero)
  int64_t mod_stride, tmod_stride;
  float *mean, *rstd;            // [rows]
  void *y, *ty;                  // outputs of the forward kernels (ty: the one-pass kernel only)
  const void *g, *gt;            // cotangents (backward kernels; gt, on ty, in the one-pass kernel only)
  void *dx, *dtx;                // gradients with respect to x / tx
  float *sums;                   // [3, B, C] fp32 column sums (zeroed by the caller)
  int B, S, C;
  float eps;
  int exact;                     // backward of the tangent: bit 0 = full second-order terms (else mean / rstd held constant),
                                 // bit 1 = add to what dx holds instead of overwriting it
};

// ---- forward of y = (n gamma + beta)(1 + scale) + shift; saves mean / rstd.  A warp walks rows of one sample with the two
// per-channel factors of n in registers (gamma (1 + scale), beta (1 + scale) + shift) and the next row in flight: read per row, the
// four parameter vectors were six times the row itself on its way through L1.  Bound by memory (8 x 128 rows of 768, a launch
// among others: 3.8 -> 3.5 us).
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) ln_modulate_fwd_kernel(LnArgs a, int rows_per_cta) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int C = NV * 256;
  const int ctas_per_sample = (a.S + rows_per_cta - 1) / rows_per_cta;
  const int b = blockIdx.x / ctas_per_sample;
  const int s0 = (blockIdx.x % ctas_per_sample) * rows_per_cta + warp;
  const int s1 = min(a.S, (int)(blockIdx.x % ctas_per_sample + 1) * rows_per_cta);
  if (s0 >= s1) return;
  Raw8<T> cur[NV];
  auto load_row = [&](int s) {
    const T *x = static_cast<const T *>(a.x) + ((int64_t)b * a.S + s) * C;
#pragma unroll
    for (int v = 0; v < NV; ++v) cur[v] = load_raw8(x + chan(v, lane));
  };
  load_row(s0);
  float ga[NV][8], be[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c0 = chan(v, lane);
    float scv[8], shv[8];
    load8<float>(a.gamma + c0, ga[v]);
    if (a.beta) load8<float>(a.beta + c0, be[v]);
    load8<T>(static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride + c0, scv);
    load8<T>(static_cast<const T *>(a.shift) + (int64_t)b * a.mod_stride + c0, shv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      ga[v][i] *= 1.f + scv[i];
      be[v][i] = (a.beta ? be[v][i] * (1.f + scv[i]) : 0.f) + shv[i];
    }
  }
  for (int s = s0; s < s1; s += kWarpsPerCta) {
    const int64_t row = (int64_t)b * a.S + s;
    float xv[NV][8], t = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      unpack8(cur[v], xv[v]);
#pragma unroll
      for (int i = 0; i < 8; ++i) t += xv[v][i];
    }
    if (s + kWarpsPerCta < s1) load_row(s + kWarpsPerCta);
    const float mean = warp_sum(t) / C;
    float q = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        xv[v][i] -= mean;
        q += xv[v][i] * xv[v][i];
      }
    const float rstd = rsqrtf(warp_sum(q) / C + a.eps);
    if (lane == 0) {
      a.mean[row] = mean;
      a.rstd[row] = rstd;
    }
    T *y = static_cast<T *>(a.y) + row * C;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float out[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = xv[v][i] * rstd * ga[v][i] + be[v][i];
      store8<T>(y + chan(v, lane), out);
    }
  }
}

// The same with a row per warp and the parameter vectors read per row: half the registers, so twice the warps per SM, and no
// warp idle where a sample has fewer rows than a CTA has warps.
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) ln_modulate_fwd_row_kernel(LnArgs a) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + warp;
  if (row >= (int64_t)a.B * a.S) return;
  const int b = (int)(row / a.S);
  constexpr int C = NV * 256;
  const T *x = static_cast<const T *>(a.x) + row * C;
  float xv[NV][8];
  float s = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    load8<T>(x + chan(v, lane), xv[v]);
#pragma unroll
    for (int i = 0; i < 8; ++i) s += xv[v][i];
  }
  const float mean = warp_sum(s) / C;
  float q = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float d = xv[v][i] - mean;
      q += d * d;
    }
  const float rstd = rsqrtf(warp_sum(q) / C + a.eps);
  if (lane == 0) {
    a.mean[row] = mean;
    a.rstd[row] = rstd;
  }
  const T *sc = static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride;
  const T *sh = static_cast<const T *>(a.shift) + (int64_t)b * a.mod_stride;
  T *y = static_cast<T *>(a.y) + row * C;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c0 = chan(v, lane);
    float g[8], be[8], scv[8], shv[8], out[8];
    load8<float>(a.gamma + c0, g);
    if (a.beta) load8<float>(a.beta + c0, be);
    load8<T>(sc + c0, scv);
    load8<T>(sh + c0, shv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float ln = (xv[v][i] - mean) * rstd * g[i] + (a.beta ? be[i] : 0.f);
      out[i] = ln * (1.f + scv[i]) + shv[i];
    }
    store8<T>(y + c0, out);
  }
}

// ---- forward of the tangent alone:  ty = nd gamma (1 + scale) + (n gamma + beta) tscale + tshift,  nd = rstd P_n(tx),
//      where P_n(z) = z - mean(z) - n mean(n z)
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) ln_modulate_fwd_tangent_kernel(LnArgs a) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + warp;
  if (row >= (int64_t)a.B * a.S) return;
  const int b = (int)(row / a.S);
  constexpr int C = NV * 256;
  const T *x = static_cast<const T *>(a.x) + row * C;
  float xv[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) load8<T>(x + chan(v, lane), xv[v]);
  const float mean = a.mean[row], rstd = a.rstd[row];
  const T *sc = static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride;
  T *y = static_cast<T *>(a.y) + row * C;
  const T *tx = static_cast<const T *>(a.tx) + row * C;
  float tv[NV][8];
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    load8<T>(tx + chan(v, lane), tv[v]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      s1 += tv[v][i];
      s2 += (xv[v][i] - mean) * rstd * tv[v][i];
    }
  }
  const float m1 = warp_sum(s1) / C, m2 = warp_sum(s2) / C;
  const T *tsc = a.tscale ? static_cast<const T *>(a.tscale) + (int64_t)b * a.tmod_stride : nullptr;
  const T *tsh = a.tshift ? static_cast<const T *>(a.tshift) + (int64_t)b * a.tmod_stride : nullptr;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c0 = chan(v, lane);
    float g[8], be[8], scv[8], tscv[8], tshv[8], out[8];
    load8<float>(a.gamma + c0, g);
    if (a.beta) load8<float>(a.beta + c0, be);
    load8<T>(sc + c0, scv);
    if (tsc) load8<T>(tsc + c0, tscv);
    if (tsh) load8<T>(tsh + c0, tshv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float n = (xv[v][i] - mean) * rstd;
      const float nd = rstd * (tv[v][i] - m1 - n * m2);
      float o = nd * g[i] * (1.f + scv[i]);
      if (tsc) o += (n * g[i] + (a.beta ? be[i] : 0.f)) * tscv[i];
      if (tsh) o += tshv[i];
      out[i] = o;
    }
    store8<T>(y + c0, out);
  }
}

// y and ty of the kernel above in one pass: x is read once instead of twice (4 row-sized transfers instead of 5) and the
// statistics need not travel through memory.  Bound by memory; 128 x 128 rows of 768: 42.5 us in two kernels, 35.6 us so.
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) ln_modulate_dual_fwd_kernel(LnArgs a) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + warp;
  if (row >= (int64_t)a.B * a.S) return;
  const int b = (int)(row / a.S);
  constexpr int C = NV * 256;
  float xv[NV][8], tv[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    load8<T>(static_cast<const T *>(a.x) + row * C + chan(v, lane), xv[v]);
    if (a.tx) load8<T>(static_cast<const T *>(a.tx) + row * C + chan(v, lane), tv[v]);
    else
#pragma unroll
      for (int i = 0; i < 8; ++i) tv[v][i] = 0.f;
  }
  float s = 0.f, s1 = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      s += xv[v][i];
      s1 += tv[v][i];
    }
  const float mean = warp_sum(s) / C, m1 = warp_sum(s1) / C;
  float q = 0.f, s2 = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      xv[v][i] -= mean;
      q += xv[v][i] * xv[v][i];
      s2 += xv[v][i] * tv[v][i];
    }
  const float rstd = rsqrtf(warp_sum(q) / C + a.eps), m2 = warp_sum(s2) * rstd / C;
  if (lane == 0) {
    a.mean[row] = mean;
    a.rstd[row] = rstd;
  }
  const T *sc = static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride;
  const T *sh = static_cast<const T *>(a.shift) + (int64_t)b * a.mod_stride;
  const T *tsc = a.tscale ? static_cast<const T *>(a.tscale) + (int64_t)b * a.tmod_stride : nullptr;
  const T *tsh = a.tshift ? static_cast<const T *>(a.tshift) + (int64_t)b * a.tmod_stride : nullptr;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c0 = chan(v, lane);
    float g[8], be[8], scv[8], shv[8], tscv[8], tshv[8], o[8], to[8];
    load8<float>(a.gamma + c0, g);
    if (a.beta) load8<float>(a.beta + c0, be);
    load8<T>(sc + c0, scv);
    load8<T>(sh + c0, shv);
    if (tsc) load8<T>(tsc + c0, tscv);
    if (tsh) load8<T>(tsh + c0, tshv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float n = xv[v][i] * rstd, ln = n * g[i] + (a.beta ? be[i] : 0.f);
      o[i] = ln * (1.f + scv[i]) + shv[i];
      to[i] = rstd * (tv[v][i] - m1 - n * m2) * g[i] * (1.f + scv[i]) + (tsc ? ln * tscv[i] : 0.f) + (tsh ? tshv[i] : 0.f);
    }
    store8<T>(static_cast<T *>(a.y) + row * C + c0, o);
    store8<T>(static_cast<T *>(a.ty) + row * C + c0, to);
  }
}

// The same with a warp walking rows of one sample: four factors per channel in shared memory (gamma (1 + scale), its offset,
// gamma tscale, its offset), placed so that a warp reads 16 bytes per lane without conflicts, and the next row in flight.
// Read for every row, the six parameter vectors took as long as the row, and their latency came before the row's own: 128 x 128
// rows of 768 37.3 -> 21.1 us (4.8 TB/s), 64 x 100 of 1024 16.9 -> 12.9, 8 x 128 of 768 6.5 -> 4.5.
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) ln_modulate_dual_fwd_walk_kernel(LnArgs a, int rows_per_cta) {
  constexpr int C = NV * 256;
  __shared__ float4 fac[4][2 * NV][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ctas_per_sample = (a.S + rows_per_cta - 1) / rows_per_cta;
  const int b = blockIdx.x / ctas_per_sample;
  const int s0 = (blockIdx.x % ctas_per_sample) * rows_per_cta, s1 = min(a.S, s0 + rows_per_cta);
  Raw8<T> cx[NV], ct[NV];
  auto load_row = [&](int s) {
    const int64_t e = ((int64_t)b * a.S + s) * C;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      cx[v] = load_raw8(static_cast<const T *>(a.x) + e + chan(v, lane));
      ct[v] = a.tx ? load_raw8(static_cast<const T *>(a.tx) + e + chan(v, lane)) : Raw8<T>{};
    }
  };
  if (s0 + warp < s1) load_row(s0 + warp);
  for (int i = threadIdx.x; i < C / 8; i += kWarpsPerCta * 32) {
    const int c0 = i * 8;
    float g[8], be[8] = {}, sc[8], sh[8], tsc[8] = {}, tsh[8] = {};
    load8<float>(a.gamma + c0, g);
    if (a.beta) load8<float>(a.beta + c0, be);
    load8<T>(static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride + c0, sc);
    load8<T>(static_cast<const T *>(a.shift) + (int64_t)b * a.mod_stride + c0, sh);
    if (a.tscale) load8<T>(static_cast<const T *>(a.tscale) + (int64_t)b * a.tmod_stride + c0, tsc);
    if (a.tshift) load8<T>(static_cast<const T *>(a.tshift) + (int64_t)b * a.tmod_stride + c0, tsh);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      be[j] = a.beta ? be[j] : 0.f;
      sh[j] += be[j] * (1.f + sc[j]);
      tsh[j] += be[j] * tsc[j];
      tsc[j] *= g[j];
      g[j] *= 1.f + sc[j];
    }
    const int v = i / 32, l = i % 32;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      fac[0][2 * v + half][l] = make_float4(g[4 * half], g[4 * half + 1], g[4 * half + 2], g[4 * half + 3]);
      fac[1][2 * v + half][l] = make_float4(sh[4 * half], sh[4 * half + 1], sh[4 * half + 2], sh[4 * half + 3]);
      fac[2][2 * v + half][l] = make_float4(tsc[4 * half], tsc[4 * half + 1], tsc[4 * half + 2], tsc[4 * half + 3]);
      fac[3][2 * v + half][l] = make_float4(tsh[4 * half], tsh[4 * half + 1], tsh[4 * half + 2], tsh[4 * half + 3]);
    }
  }
  __syncthreads();
  for (int s = s0 + warp; s < s1; s += kWarpsPerCta) {
    const int64_t row = (int64_t)b * a.S + s;
    float x[NV][8], t[NV][8], sx = 0.f, st = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      unpack8(cx[v], x[v]), unpack8(ct[v], t[v]);
#pragma unroll
      for (int i = 0; i < 8; ++i) sx += x[v][i], st += t[v][i];
    }
    if (s + kWarpsPerCta < s1) load_row(s + kWarpsPerCta);
    const float mean = warp_sum(sx) / C, m1 = warp_sum(st) / C;
    float q = 0.f, s2 = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        x[v][i] -= mean;
        q += x[v][i] * x[v][i];
        s2 += x[v][i] * t[v][i];
      }
    const float rstd = rsqrtf(warp_sum(q) / C + a.eps), m2 = warp_sum(s2) * rstd / C;
    if (lane == 0) {
      a.mean[row] = mean;
      a.rstd[row] = rstd;
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float o[8], to[8];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float4 f0 = fac[0][2 * v + half][lane], f1 = fac[1][2 * v + half][lane], f2 = fac[2][2 * v + half][lane],
                     f3 = fac[3][2 * v + half][lane];
        const float gs[4] = {f0.x, f0.y, f0.z, f0.w}, bs[4] = {f1.x, f1.y, f1.z, f1.w}, gt[4] = {f2.x, f2.y, f2.z, f2.w},
                    bt[4] = {f3.x, f3.y, f3.z, f3.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = 4 * half + j;
          const float n = x[v][i] * rstd;
          o[i] = n * gs[j] + bs[j];
          to[i] = rstd * (t[v][i] - m1 - n * m2) * gs[j] + (n * gt[j] + bt[j]);
        }
      }
      store8<T>(static_cast<T *>(a.y) + row * C + chan(v, lane), o);
      store8<T>(static_cast<T *>(a.ty) + row * C + chan(v, lane), to);
    }
  }
}

// Column sums of a CTA: every warp parks its per-channel partial sums in its own slice of shared memory (plain stores),
// then the CTA adds the slices and issues one global atomic per column.  `smem` holds kWarpsPerCta * NQ * C floats.
template <int NQ, int NV>
__device__ __forceinline__ void flush_column_sums(float *smem, const float (&part)[NQ][NV][8], int lane, float *const (&dst)[NQ]) {
  constexpr int C = NV * 256;
  const int warp = threadIdx.x >> 5;
  float *mine = smem + (size_t)warp * NQ * C;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = part[q][v][i];
      store8<float>(mine + q * C + chan(v, lane), f);
    }
  __syncthreads();
  for (int q = 0; q < NQ; ++q)
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < kWarpsPerCta; ++w) t += smem[((size_t)w * NQ + q) * C + c];
      atomicAdd(dst[q] + c, t);
    }
}

// ---- backward of ty.  u = G gamma (1 + scale), w = G gamma tscale, nd = rstd P_n(tx):
//   dtx = rstd P_n(u)
//   exact:        dx = rstd P_n(w + gn) - rstd n mean(u nd),   gn = -rstd (u mean(n tx) + tx mean(u n))
//   mean / rstd held constant inside nd (what autograd does with the forward-mode formula of native_layer_norm, whose
//   saved statistics are not differentiable outputs; the w term goes through the primal output and is differentiated
//   in full):   dx = rstd P_n(w) - rstd^2 (u mean(n tx) + (tx - mean(tx)) mean(u n))
//   sums[0] += G n, sums[1] += G, sums[2] += G nd   (per sample)
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) ln_modulate_bwd_tangent_kernel(LnArgs a, int rows_per_cta) {
  extern __shared__ float smem_raw[];
  constexpr int C = NV * 256;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ctas_per_sample = (a.S + rows_per_cta - 1) / rows_per_cta;
  const int b = blockIdx.x / ctas_per_sample;
  const int s0 = (blockIdx.x % ctas_per_sample) * rows_per_cta;
  const T *sc = static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride;
  const T *tsc = a.tscale ? static_cast<const T *>(a.tscale) + (int64_t)b * a.tmod_stride : nullptr;
  float part[3][NV][8] = {};
  for (int r = warp; r < rows_per_cta && s0 + r < a.S; r += kWarpsPerCta) {
    const int64_t row = (int64_t)b * a.S + s0 + r;
    const T *x = static_cast<const T *>(a.x) + row * C;
    const T *tx = static_cast<const T *>(a.tx) + row * C;
    const T *g = static_cast<const T *>(a.g) + row * C;
    const float mean = a.mean[row], rstd = a.rstd[row];
    float n[NV][8], t[NV][8], gv[NV][8];
    float st = 0.f, snt = 0.f, su = 0.f, sun = 0.f, sw = 0.f, swn = 0.f, sut = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c0 = chan(v, lane);
      float xv[8], gam[8], scv[8], tscv[8];
      load8<T>(x + c0, xv);
      load8<T>(tx + c0, t[v]);
      load8<T>(g + c0, gv[v]);
      load8<float>(a.gamma + c0, gam);
      load8<T>(sc + c0, scv);
      if (tsc) load8<T>(tsc + c0, tscv);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        n[v][i] = (xv[i] - mean) * rstd;
        const float gg = gv[v][i] * gam[i];
        const float u = gg * (1.f + scv[i]), w = tsc ? gg * tscv[i] : 0.f;
        st += t[v][i];
        snt += n[v][i] * t[v][i];
        su += u;
        sun += u * n[v][i];
        sw += w;
        swn += w * n[v][i];
        sut += u * t[v][i];
      }
    }
    const float inv = 1.f / C;
    const float m_t = warp_sum(st) * inv, m_nt = warp_sum(snt) * inv, m_u = warp_sum(su) * inv, m_un = warp_sum(sun) * inv;
    const float m_w = warp_sum(sw) * inv, m_wn = warp_sum(swn) * inv, m_ut = warp_sum(sut) * inv;
    // nd = rstd (t - m_t - n m_nt)   =>   mean(u nd) = rstd (m_ut - m_u m_t - m_un m_nt)
    const float m_und = rstd * (m_ut - m_u * m_t - m_un * m_nt);
    // gn = -rstd (u m_nt + t m_un)   =>   mean(gn) = -rstd (m_u m_nt + m_t m_un),  mean(gn n) = -2 rstd m_un m_nt
    const float m_gn = -rstd * (m_u * m_nt + m_t * m_un), m_gnn = -2.f * rstd * m_un * m_nt;
    T *dx = static_cast<T *>(a.dx) + row * C;
    T *dtx = static_cast<T *>(a.dtx) + row * C;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c0 = chan(v, lane);
      float gam[8], scv[8], tscv[8], o1[8], o2[8];
      load8<float>(a.gamma + c0, gam);  // (cache hits: the row loop above just read them)
      load8<T>(sc + c0, scv);
      if (tsc) load8<T>(tsc + c0, tscv);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float gg = gv[v][i] * gam[i];
        const float u = gg * (1.f + scv[i]), w = tsc ? gg * tscv[i] : 0.f;
        const float nn = n[v][i], tt = t[v][i];
        const float nd = rstd * (tt - m_t - nn * m_nt);
        o2[i] = rstd * (u - m_u - nn * m_un);
        if (a.exact & 1) {
          const float gn = -rstd * (u * m_nt + tt * m_un);
          o1[i] = rstd * ((w + gn) - (m_w + m_gn) - nn * (m_wn + m_gnn)) - rstd * nn * m_und;
        } else {
          o1[i] = rstd * ((w - m_w - nn * m_wn) - rstd * (u * m_nt + (tt - m_t) * m_un));
        }
        part[0][v][i] += gv[v][i] * nn;
        part[1][v][i] += gv[v][i];
        part[2][v][i] += gv[v][i] * nd;
      }
      if (a.exact & 2) {  // dx already holds the gradient that arrived through the primal output: add to it
        float prev[8];
        load8<T>(dx + c0, prev);
#pragma unroll
        for (int i = 0; i < 8; ++i) o1[i] += prev[i];
      }
      store8<T>(dx + c0, o1);
      store8<T>(dtx + c0, o2);
    }
  }
  float *const dst[3] = {a.sums + (int64_t)b * C, a.sums + ((int64_t)a.B + b) * C, a.sums + ((int64_t)2 * a.B + b) * C};
  flush_column_sums<3, NV>(smem_raw, part, lane, dst);
}

// ---- backward of y (kTan = false).  w = G gamma (1 + scale);  dx = rstd P_n(w);  sums[0] += G n, sums[1] += G   (per sample)
// kTan = true: with the kernel above in the same pass, for the cotangents g on y and gt on ty: x is read once and dx
// written once, 6 row-sized transfers instead of 9, and dx is rounded once.  With u1 = g gamma (1 + scale) and w, u of the kernel above, dx follows
// from u1 + w in the place of w.  gamma (1 + scale) multiplies sum(g n) and sum(gt nd) alike, so those share one column
// sum: sums[0] += g n + gt nd, sums[1] += g, sums[2] += gt n, sums[3] += gt.
// Bound by memory.  A thread owns 8 channels of every row of its CTA (C / 8 threads), not a lane 8 NV of one row in four: the
// four column sums and the next row's four operands then fit the registers with room for several CTAs per SM (a warp per
// row took all 255 at C = 768 and spilled; fp32 rows would not fit here either and keep the kernels above), the per-sample factors are loaded once, and the column sums need no pass through
// shared memory.  The price is a block-wide reduction of the row's sums: one barrier per row (its buffer alternates).
// 128 x 128 rows of 768: 99 us in two kernels, 60 us so, 49 us with the column sums added 16 bytes at a time.
template <typename T, int NV, bool kTan>
__global__ void __launch_bounds__(NV * 32, (sizeof(T) == 2 ? 16 : 12) / NV) ln_modulate_bwd_kernel(LnArgs a, int rows_per_cta) {
  constexpr int C = NV * 256;
  __shared__ float scratch[2][8][NV];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = threadIdx.x * 8;
  const int ctas_per_sample = (a.S + rows_per_cta - 1) / rows_per_cta;
  const int b = blockIdx.x / ctas_per_sample;
  const int s0 = (blockIdx.x % ctas_per_sample) * rows_per_cta, s1 = min(a.S, s0 + rows_per_cta);
  const bool exact = a.exact & 1;
  float gs[8], gw[8];  // gamma (1 + scale), gamma tscale
  {
    float gam[8], scv[8];
    load8<float>(a.gamma + c0, gam);
    load8<T>(static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride + c0, scv);
    if (a.tscale) load8<T>(static_cast<const T *>(a.tscale) + (int64_t)b * a.tmod_stride + c0, gw);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      gs[i] = gam[i] * (1.f + scv[i]);
      gw[i] = a.tscale ? gam[i] * gw[i] : 0.f;
    }
  }
  struct Row {
    Raw8<T> x, g, t, gt;  // (t, gt: kTan)
    float mean, rstd;
  };
  auto load_row = [&](int s, Row &r) {
    const int64_t row = (int64_t)b * a.S + s, e = row * C + c0;
    r.x = load_raw8(static_cast<const T *>(a.x) + e);
    if (kTan) r.t = a.tx ? load_raw8(static_cast<const T *>(a.tx) + e) : Raw8<T>{};
    r.g = load_raw8(static_cast<const T *>(a.g) + e);
    if (kTan) r.gt = load_raw8(static_cast<const T *>(a.gt) + e);
    r.mean = a.mean[row];
    r.rstd = a.rstd[row];
  };
  float part[4][8] = {};
  Row cur;
  load_row(s0, cur);
  for (int s = s0; s < s1; ++s) {
    const float mean = cur.mean, rstd = cur.rstd;
    float n[8], g[8], t[8] = {}, gt[8] = {};
    unpack8(cur.x, n), unpack8(cur.g, g);
    if (kTan) unpack8(cur.t, t), unpack8(cur.gt, gt);
    if (s + 1 < s1) load_row(s + 1, cur);  // in flight across the barrier below
    float v[7] = {};  // w, w n, and with kTan t, n t, u, u n, u t
    const int nsum = !kTan ? 2 : exact ? 7 : 6;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      n[i] = (n[i] - mean) * rstd;
      const float u = gt[i] * gs[i], w = g[i] * gs[i] + (kTan ? gt[i] * gw[i] : 0.f);
      v[0] += w;
      v[1] += w * n[i];
      if (kTan) {
        v[2] += t[i];
        v[3] += n[i] * t[i];
        v[4] += u;
        v[5] += u * n[i];
        v[6] += u * t[i];
      }
    }
#pragma unroll
    for (int q = 0; q < 7; ++q) {
      if (q >= nsum) break;
      v[q] = warp_sum(v[q]);
      if (NV > 1 && lane == 0) scratch[s & 1][q][warp] = v[q];
    }
    if (NV > 1) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 7; ++q) {
        if (q >= nsum) break;
        v[q] = scratch[s & 1][q][0];
#pragma unroll
        for (int k = 1; k < NV; ++k) v[q] += scratch[s & 1][q][k];
      }
    }
    constexpr float inv = 1.f / C;
    const float m_w = v[0] * inv, m_wn = v[1] * inv, m_t = v[2] * inv, m_nt = v[3] * inv, m_u = v[4] * inv, m_un = v[5] * inv;
    const float m_und = exact ? rstd * (v[6] * inv - m_u * m_t - m_un * m_nt) : 0.f;
    const float m_gn = -rstd * (m_u * m_nt + m_t * m_un), m_gnn = -2.f * rstd * m_un * m_nt;
    float o1[8], o2[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float u = gt[i] * gs[i], w = g[i] * gs[i] + (kTan ? gt[i] * gw[i] : 0.f);
      if (!kTan) {
        o1[i] = rstd * (w - m_w - n[i] * m_wn);
        part[0][i] += g[i] * n[i];
        part[1][i] += g[i];
        continue;
      }
      const float nd = rstd * (t[i] - m_t - n[i] * m_nt);
      o2[i] = rstd * (u - m_u - n[i] * m_un);
      if (exact) {
        const float gn = -rstd * (u * m_nt + t[i] * m_un);
        o1[i] = rstd * ((w + gn) - (m_w + m_gn) - n[i] * (m_wn + m_gnn)) - rstd * n[i] * m_und;
      } else {
        o1[i] = rstd * ((w - m_w - n[i] * m_wn) - rstd * (u * m_nt + (t[i] - m_t) * m_un));
      }
      part[0][i] += g[i] * n[i] + gt[i] * nd;
      part[1][i] += g[i];
      part[2][i] += gt[i] * n[i];
      part[3][i] += gt[i];
    }
    const int64_t e = ((int64_t)b * a.S + s) * C + c0;
    store8<T>(static_cast<T *>(a.dx) + e, o1);
    if (kTan) store8<T>(static_cast<T *>(a.dtx) + e, o2);
  }
#pragma unroll
  for (int q = 0; q < (kTan ? 4 : 2); ++q) add8(a.sums + ((int64_t)q * a.B + b) * C + c0, part[q]);
}

// ---- dropout keep mask computed in the kernel instead of read from memory.  Philox-4x32-10 (Salmon et al., "Parallel
// random numbers: as easy as 1, 2, 3", 2011) keyed by a 64-bit seed that lives in device memory (drawn once per training
// step, so a replayed CUDA graph sees a new one), counter = (chunk index, call index): every kernel that touches the same
// call of the same step regenerates the same mask.  One call yields 8 x 16 bits = the masks of 8 adjacent elements.
struct DropArgs {
  const unsigned long long *seed;  // null: no generated mask
  unsigned call;
  float p;
};

__device__ __forceinline__ void dropout8(const DropArgs &d, int64_t chunk, float (&m)[8]) {
  const unsigned long long seed = *d.seed;
  unsigned k0 = (unsigned)seed, k1 = (unsigned)(seed >> 32);
  unsigned c0 = (unsigned)chunk, c1 = (unsigned)((unsigned long long)chunk >> 32), c2 = d.call, c3 = 0x5eedu;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const unsigned hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    c0 = hi1 ^ c1 ^ k0;
    c1 = lo1;
    c2 = hi0 ^ c3 ^ k1;
    c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  const float keep = 1.f - d.p, inv = 1.f / keep;
  const unsigned thr = (unsigned)(keep * 65536.f);
  const unsigned w[4] = {c0, c1, c2, c3};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[2 * i] = (w[i] & 0xffffu) < thr ? inv : 0.f;
    m[2 * i + 1] = (w[i] >> 16) < thr ? inv : 0.f;
  }
}

struct GateArgs {
  const void *x, *y;         // [rows, C]
  const void *gate;          // [B, C] rows `gate_stride` apart
  const void *mask;          // [rows, C] in the branch dtype: keep mask / (1 - p); null = all ones (or generated, see drop)
  int64_t gate_stride;
  void *z;
  int B, S, C;
  DropArgs drop;             // used when mask is null and drop.seed is not
};

// Index type of the forward kernels, which take a linear chunk index apart into (sample, row, channels): 32 bits wherever they
// hold the index and a grid stride, since two 64-bit divisions per chunk of 8 elements cost more than the chunk's arithmetic
// (128 x 128 rows of 768, pair: 30.6 -> 26.8 us).
inline bool index32(int64_t chunks) { return chunks < (int64_t(1) << 31); }

// z = x + m g y without a tangent (the passes that run outside forward-mode AD)
template <typename T, typename I>
__global__ void __launch_bounds__(256) gated_residual_fwd_kernel(GateArgs a) {
  const I total = (I)((int64_t)a.B * a.S * a.C / 8), per_row = (I)(a.C / 8);
  for (I i8 = (I)blockIdx.x * blockDim.x + threadIdx.x; i8 < total; i8 += (I)gridDim.x * blockDim.x) {
    const int64_t e = (int64_t)i8 * 8;
    const I row = i8 / per_row;
    const int c0 = (int)(i8 - row * per_row) * 8;
    const int b = (int)(row / (I)a.S);
    float xv[8], yv[8], gv[8], mv[8], out[8];
    load8<T>(static_cast<const T *>(a.x) + e, xv);
    load8<T>(static_cast<const T *>(a.y) + e, yv);
    load8<T>(static_cast<const T *>(a.gate) + (int64_t)b * a.gate_stride + c0, gv);
    const bool masked = a.mask || a.drop.seed;
    if (a.mask) load8<T>(static_cast<const T *>(a.mask) + e, mv);
    else if (a.drop.seed) dropout8(a.drop, i8, mv);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = xv[i] + (masked ? mv[i] : 1.f) * gv[i] * yv[i];
    store8<T>(static_cast<T *>(a.z) + e, out);
  }
}

// z = x + gate y and h = LN(z) (1 + scale) + shift in one pass, for passes in which nothing is recorded: the residual behind a branch
// and the LayerNorm in front of the next, with z rounded to its type before the LayerNorm as between the two kernels.  A warp
// per row; bound by launches where it is used (a sampling pass has few rows): one instead of two, and z is not read back.
struct GateLnArgs {
  const void *x, *y, *gate;
  int64_t gate_stride;
  const float *gamma, *beta;
  const void *shift, *scale;
  int64_t mod_stride;
  void *z, *h;
  int B, S;
  float eps;
};

template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) gate_ln_fwd_kernel(GateLnArgs a) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + warp;
  if (row >= (int64_t)a.B * a.S) return;
  const int64_t b = row / a.S;
  constexpr int C = NV * 256;
  Raw8<T> rx[NV], ry[NV], rg[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    rx[v] = load_raw8(static_cast<const T *>(a.x) + row * C + chan(v, lane));
    ry[v] = load_raw8(static_cast<const T *>(a.y) + row * C + chan(v, lane));
    rg[v] = load_raw8(static_cast<const T *>(a.gate) + b * a.gate_stride + chan(v, lane));
  }
  float z[NV][8], s = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    float y[8], g[8];
    unpack8(rx[v], z[v]), unpack8(ry[v], y), unpack8(rg[v], g);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      z[v][i] += g[i] * y[i];
      if constexpr (sizeof(T) == 2) z[v][i] = __bfloat162float(__float2bfloat16_rn(z[v][i]));
      s += z[v][i];
    }
    store8<T>(static_cast<T *>(a.z) + row * C + chan(v, lane), z[v]);
  }
  const float mean = warp_sum(s) / C;
  float q = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float d = z[v][i] - mean;
      q += d * d;
    }
  const float rstd = rsqrtf(warp_sum(q) / C + a.eps);
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c0 = chan(v, lane);
    float g[8], be[8], scv[8], shv[8], out[8];
    load8<float>(a.gamma + c0, g);
    if (a.beta) load8<float>(a.beta + c0, be);
    load8<T>(static_cast<const T *>(a.scale) + b * a.mod_stride + c0, scv);
    load8<T>(static_cast<const T *>(a.shift) + b * a.mod_stride + c0, shv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float ln = (z[v][i] - mean) * rstd * g[i] + (a.beta ? be[i] : 0.f);
      out[i] = ln * (1.f + scv[i]) + shv[i];
    }
    store8<T>(static_cast<T *>(a.h) + row * C + c0, out);
  }
}

// Rows of one sample that a CTA of the backward kernels walks before it adds its column sums to global memory.  Every CTA
// costs one atomic per column and sum, and at a few hundred samples those atomics (millions per launch, a dozen
// contenders per address) took longer than the rows themselves; so the count grows with the problem as long as
// eight CTAs per SM remain (four where there are no sums and the point is what a CTA loads once).  Kernels that walk their rows
// one after another (`resident` = CTAs of theirs that an SM holds) take fewer than `base` where the GPU would otherwise not be
// full: a row is then latency only (8 x 128 rows of 768, pair of LayerNorm cotangents 15.0 -> 7.4 us, gated residual 6.2 -> 4.1; 2 x 50
// rows of 256 17.1 -> 5.6).  Not fewer than four: the column sums of two-row CTAs contend (8 x 128 rows of 256, primal: 4.5 us, 3.4
// with four rows).
inline int rows_per_cta(int B, int S, int base, int ctas_per_sm = 8, int resident = 0) {
  auto ctas = [&](int rows) { return (int64_t)B * ((S + rows - 1) / rows); };
  int rows = base;
  while (rows < 64 && ctas(2 * rows) >= 148 * ctas_per_sm) rows *= 2;
  while (rows > 4 && 2 * ctas(rows) <= 148 * resident) rows /= 2;
  return rows;
}

// ---- gradients of the modulation tensors and of the LayerNorm weight / bias from the column sums of the two backward
// kernels, in one launch.  p = sums of the VJP of y ([2, B, C]: sum_s g n, sum_s g), t = sums of the VJP of ty ([3, B, C]:
// sum_s g n, sum_s g, sum_s g nd); either may be null.  One thread per channel walks the samples.
struct LnFinalArgs {
  const float *p, *t;
  const float *gamma, *beta;
  const void *scale, *tscale;
  int64_t mod_stride, tmod_stride;
  void *d_shift, *d_scale, *d_tshift, *d_tscale;  // [B, C] contiguous in the modulation dtype (null = not wanted)
  float *d_gamma, *d_beta;                        // [C], zeroed by the caller: CTAs add their samples' share
  int B, C;
};

constexpr int kFinalSamples = 4;  // samples per thread of the finalize kernel

// (All of a thread's loads go out before its first store, past which the compiler may not move them: 128 samples of 768
// channels 11.4 -> 3.1 us, 8 samples 10.1 -> 2.3.)
template <typename T>
__global__ void ln_finalize_kernel(LnFinalArgs a) {
  // (one grid axis for channels and samples: the second holds no more than 65535)
  const unsigned chunks = ((unsigned)a.C + blockDim.x - 1) / blockDim.x;
  const int c = blockIdx.x % chunks * blockDim.x + threadIdx.x;
  if (c >= a.C) return;
  const float gam = a.gamma[c], bet = a.beta ? a.beta[c] : 0.f;
  float dg = 0.f, db = 0.f;
  const int64_t BC = (int64_t)a.B * a.C;
  const int b0 = blockIdx.x / chunks * kFinalSamples;
  float sc1[kFinalSamples], tsc[kFinalSamples], p[2][kFinalSamples], t[3][kFinalSamples];
#pragma unroll
  for (int k = 0; k < kFinalSamples; ++k) {
    const int b = min(b0 + k, a.B - 1);
    const int64_t i = (int64_t)b * a.C + c;
    sc1[k] = 1.f + ldf<T>(static_cast<const T *>(a.scale) + (int64_t)b * a.mod_stride + c);
    tsc[k] = a.tscale ? ldf<T>(static_cast<const T *>(a.tscale) + (int64_t)b * a.tmod_stride + c) : 0.f;
#pragma unroll
    for (int q = 0; q < 2; ++q) p[q][k] = a.p ? a.p[q * BC + i] : 0.f;
#pragma unroll
    for (int q = 0; q < 3; ++q) t[q][k] = a.t ? a.t[q * BC + i] : 0.f;
  }
#pragma unroll
  for (int k = 0; k < kFinalSamples; ++k) {
    if (b0 + k >= a.B) break;
    const int64_t i = (int64_t)(b0 + k) * a.C + c;
    float d_scale = 0.f;
    if (a.p) {
      const float gn = p[0][k], g1 = p[1][k];
      if (a.d_shift) stf<T>(static_cast<T *>(a.d_shift) + i, g1);
      d_scale += gam * gn + bet * g1;
      dg += gn * sc1[k];
      db += g1 * sc1[k];
    }
    if (a.t) {
      const float gn = t[0][k], g1 = t[1][k], gnd = t[2][k];
      if (a.d_tshift) stf<T>(static_cast<T *>(a.d_tshift) + i, g1);
      if (a.d_tscale) stf<T>(static_cast<T *>(a.d_tscale) + i, gam * gn + bet * g1);
      d_scale += gam * gnd;
      dg += gnd * sc1[k] + gn * tsc[k];
      db += g1 * tsc[k];
    }
    if (a.d_scale) stf<T>(static_cast<T *>(a.d_scale) + i, d_scale);
  }
  // d_gamma / d_beta are zeroed by the caller (they share the zero-filled buffer of the column sums)
  atomicAdd(a.d_gamma + c, dg);
  if (a.d_beta) atomicAdd(a.d_beta + c, db);
}

// ---- gated residual on a (primal, tangent) pair in one pass each way.
//   forward   z = x + m g y,   tz = tx + m (g ty + tg y)                      (tx, ty, tg may be absent)
//   backward  from cotangents gz on z and gtz on tz (either may be absent; the skip gradients are gz and gtz themselves):
//             d_y = m (g gz + tg gtz),  d_ty = m g gtz,  d_g[b] += sum_s m (y gz + ty gtz),  d_tg[b] += sum_s m y gtz
struct GateDualArgs {
  const void *x, *tx, *y, *ty, *gate, *tgate, *mask;
  int64_t gate_stride, tgate_stride;
  void *z, *tz;
  const void *gz, *gtz;
  void *d_y, *d_ty;
  float *sums;  // [2, B, C]: gate, tgate
  int B, S, C;
  DropArgs drop;
};

template <typename T, typename I>
__global__ void __launch_bounds__(256) gated_dual_fwd_kernel(GateDualArgs a) {
  const I total = (I)((int64_t)a.B * a.S * a.C / 8), per_row = (I)(a.C / 8);
  for (I i8 = (I)blockIdx.x * blockDim.x + threadIdx.x; i8 < total; i8 += (I)gridDim.x * blockDim.x) {
    const int64_t e = (int64_t)i8 * 8;
    const I row = i8 / per_row;
    const int c0 = (int)(i8 - row * per_row) * 8;
    const int b = (int)(row / (I)a.S);
    float xv[8], txv[8], yv[8], tyv[8], gv[8], tgv[8], mv[8], o[8], to[8];
    load8<T>(static_cast<const T *>(a.x) + e, xv);
    load8<T>(static_cast<const T *>(a.y) + e, yv);
    load8<T>(static_cast<const T *>(a.gate) + (int64_t)b * a.gate_stride + c0, gv);
    if (a.tx) load8<T>(static_cast<const T *>(a.tx) + e, txv);
    if (a.ty) load8<T>(static_cast<const T *>(a.ty) + e, tyv);
    if (a.tgate) load8<T>(static_cast<const T *>(a.tgate) + (int64_t)b * a.tgate_stride + c0, tgv);
    if (a.mask) load8<T>(static_cast<const T *>(a.mask) + e, mv);
    else if (a.drop.seed) dropout8(a.drop, i8, mv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float m = (a.mask || a.drop.seed) ? mv[i] : 1.f;
      o[i] = xv[i] + m * gv[i] * yv[i];
      float br = 0.f;
      if (a.ty) br += gv[i] * tyv[i];
      if (a.tgate) br += tgv[i] * yv[i];
      to[i] = (a.tx ? txv[i] : 0.f) + m * br;
    }
    store8<T>(static_cast<T *>(a.z) + e, o);
    store8<T>(static_cast<T *>(a.tz) + e, to);
  }
}

// One thread owns 8 adjacent channels of `rows_per_cta` rows of one sample: the column sums stay in registers and leave
// with one atomic per channel and CTA; adjacent threads read adjacent 16-byte pieces of a row.  (The compiler cannot move the
// next row's loads above this row's stores by itself: 51 -> 36 us at 128 x 128 rows of 768.)
template <typename T>
__global__ void __launch_bounds__(128) gated_dual_bwd_kernel(GateDualArgs a, int rows_per_cta) {
  const int c0 = threadIdx.x * 8;
  if (c0 >= a.C) return;
  const int ctas_per_sample = (a.S + rows_per_cta - 1) / rows_per_cta;
  const int b = blockIdx.x / ctas_per_sample;
  const int s0 = (blockIdx.x % ctas_per_sample) * rows_per_cta;
  float gt[8], tgt[8], sg[8] = {}, stg[8] = {};
  load8<T>(static_cast<const T *>(a.gate) + (int64_t)b * a.gate_stride + c0, gt);
  if (a.tgate) load8<T>(static_cast<const T *>(a.tgate) + (int64_t)b * a.tgate_stride + c0, tgt);
  const int s1 = min(a.S, s0 + rows_per_cta);
  struct Row {
    Raw8<T> y, ty, g1, g2, m;
  };
  auto load_row = [&](int s, Row &r) {
    const int64_t e = ((int64_t)b * a.S + s) * a.C + c0;
    r.y = load_raw8(static_cast<const T *>(a.y) + e);
    if (a.gz) r.g1 = load_raw8(static_cast<const T *>(a.gz) + e);
    if (a.gtz) r.g2 = load_raw8(static_cast<const T *>(a.gtz) + e);
    if (a.ty && a.gtz) r.ty = load_raw8(static_cast<const T *>(a.ty) + e);
    if (a.mask) r.m = load_raw8(static_cast<const T *>(a.mask) + e);
  };
  Row cur{};
  load_row(s0, cur);
  for (int s = s0; s < s1; ++s) {
    const int64_t e = ((int64_t)b * a.S + s) * a.C + c0;
    float yv[8], tyv[8], mv[8], g1[8], g2[8], o1[8], o2[8];
    unpack8(cur.y, yv), unpack8(cur.ty, tyv), unpack8(cur.g1, g1), unpack8(cur.g2, g2), unpack8(cur.m, mv);
    if (s + 1 < s1) load_row(s + 1, cur);  // in flight across this row's arithmetic and stores
    if (!a.mask && a.drop.seed) dropout8(a.drop, e / 8, mv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float m = (a.mask || a.drop.seed) ? mv[i] : 1.f;
      const float mg1 = a.gz ? m * g1[i] : 0.f, mg2 = a.gtz ? m * g2[i] : 0.f;
      o1[i] = gt[i] * mg1 + (a.tgate ? tgt[i] * mg2 : 0.f);
      o2[i] = gt[i] * mg2;
      sg[i] += yv[i] * mg1 + (a.ty && a.gtz ? tyv[i] * mg2 : 0.f);
      stg[i] += yv[i] * mg2;
    }
    store8<T>(static_cast<T *>(a.d_y) + e, o1);
    if (a.d_ty) store8<T>(static_cast<T *>(a.d_ty) + e, o2);
  }
  float *dg = a.sums + (int64_t)b * a.C + c0, *dtg = a.sums + ((int64_t)a.B + b) * a.C + c0;
  add8(dg, sg);
  if (a.gtz) add8(dtg, stg);
}

// ------------------------------------------------------------------------------------------------ GELU (tanh form)
// g(h) = h/2 (1 + tanh u), u = k (h + a h^3).  The MLP of the block (duo.py:118-123) applies it to a (primal, tangent)
// pair; with T = tanh u, u' = k (1 + 3 a h^2), u'' = 6 a k h:
//   g'  = (1 + T) / 2 + h/2 (1 - T^2) u'
//   g'' = (1 - T^2) (u' + h/2 (u'' - 2 T u'^2))
// mode 0: y = g(h);  mode 1: out = g'(h) * v (the tangent, and the VJP of either output with respect to its own input);
// mode 2: out = g'(h) * v and out2 = g''(h) * w * v (the VJP of the tangent output: with respect to the tangent and to h);
// mode 3: out = g(h) and out2 = g'(h) * v (primal and tangent in one pass);
// mode 4: out = g'(h) * v + g''(h) * w * u and out2 = g'(h) * u (both cotangents in one pass: v on y, u on ty, w = tangent
//         of h; out = gradient of h, out2 = gradient of the tangent).
struct GeluTerms {
  float g, d1, d2;
};
__device__ __forceinline__ GeluTerms gelu_terms(float h) {
  constexpr float k = 0.7978845608028654f, a = 0.044715f;
  const float h2 = h * h, T = tanhf(k * (h + a * h2 * h));
  const float up = k * (1.f + 3.f * a * h2), upp = 6.f * a * k * h, sech2 = 1.f - T * T;
  GeluTerms r;
  r.g = 0.5f * h * (1.f + T);
  r.d1 = 0.5f * (1.f + T) + 0.5f * h * sech2 * up;
  r.d2 = sech2 * (up + 0.5f * h * (upp - 2.f * T * up * up));
  return r;
}

// The same two wide, through the logistic function s = (1 + T) / 2 = 1 / (1 + exp(-2 u)): 1 - T^2 = 4 s (1 - s), and no
// cancellation in 1 + T where h is negative.  With tanhf, element by element, the kernels on bf16 were bound by instructions.
template <bool kFirst, bool kSecond>
__device__ __forceinline__ void gelu_pair(float2 h, float2 &g, float2 &d1, float2 &d2) {
  constexpr float k = 0.7978845608028654f, a = 0.044715f, c0 = -2.f * k * 1.4426950408889634f;
  const float2 h2 = __fmul2_rn(h, h), e = __fmul2_rn(h, __ffma2_rn(h2, splat(c0 * a), splat(c0)));
  float2 x, sg;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(x.x) : "f"(e.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(x.y) : "f"(e.y));
  const float2 x1 = __fadd2_rn(x, splat(1.f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(sg.x) : "f"(x1.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(sg.y) : "f"(x1.y));
  g = __fmul2_rn(h, sg);
  if (!kFirst) return;
  // s (1 - s), the second factor as exp(-2 u) s: without cancellation on the positive side (where s is 0 the exponential overflows)
  const float2 w = __fmul2_rn(sg, __fmul2_rn(make_float2(fminf(x.x, 3e38f), fminf(x.y, 3e38f)), sg));
  const float2 up = __ffma2_rn(h2, splat(6.f * a * k), splat(2.f * k));  // 2 u'
  d1 = __ffma2_rn(__fmul2_rn(h, w), up, sg);
  if (!kSecond) return;
  const float2 mt = __fmul2_rn(__fmul2_rn(w, h), __ffma2_rn(sg, splat(-2.f), splat(1.f)));  // -h T w, 0 before u'^2 overflows
  d2 = __ffma2_rn(mt, __fmul2_rn(up, up), __fmul2_rn(w, __ffma2_rn(h2, splat(24.f * a * k), splat(4.f * k))));
}

// (bf16, 128 x 128 rows of 3072, copy rate: forward of a pair 79.3 -> 62.2 us, backward 134.7 -> 94.9; 96 x 128 rows, primal
// alone, 37.9 -> 25.8 and 56 -> 39.5.)
template <typename T, int kMode>
__global__ void __launch_bounds__(256) gelu_dual_kernel(const T *h, const T *v, const T *w, const T *u, T *out, T *out2,
                                                        int64_t n8) {
  // two chunks per iteration: all loads of both are issued before the arithmetic, so every thread keeps two 16-byte
  // loads per operand in flight (one was not enough to cover the memory latency at full occupancy)
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n8; i0 += 2 * stride) {
    const int64_t idx[2] = {i0, i0 + stride};
    Raw8<T> rh[2], rv[2], rw[2], ru[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (idx[c] >= n8) continue;
      rh[c] = load_raw8(h + idx[c] * 8);
      if (kMode >= 1) rv[c] = load_raw8(v + idx[c] * 8);
      if (kMode == 2 || kMode == 4) rw[c] = load_raw8(w + idx[c] * 8);
      if (kMode == 4) ru[c] = load_raw8(u + idx[c] * 8);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (idx[c] >= n8) continue;
      float hv[8], vv[8], wv[8], uv[8], o[8], o2[8];
      unpack8(rh[c], hv);
      if (kMode >= 1) unpack8(rv[c], vv);
      if (kMode == 2 || kMode == 4) unpack8(rw[c], wv);
      if (kMode == 4) unpack8(ru[c], uv);
      if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          float2 g, d1, d2, a, b;
          gelu_pair<(kMode >= 1), (kMode == 2 || kMode == 4)>(make_float2(hv[j], hv[j + 1]), g, d1, d2);
          const float2 v2 = make_float2(vv[j], vv[j + 1]), w2 = make_float2(wv[j], wv[j + 1]), u2 = make_float2(uv[j], uv[j + 1]);
          if (kMode == 0) a = g;
          if (kMode == 1) a = __fmul2_rn(d1, v2);
          if (kMode == 2) a = __fmul2_rn(d1, v2), b = __fmul2_rn(__fmul2_rn(d2, w2), v2);
          if (kMode == 3) a = g, b = __fmul2_rn(d1, v2);
          if (kMode == 4) a = __ffma2_rn(__fmul2_rn(d2, w2), u2, __fmul2_rn(d1, v2)), b = __fmul2_rn(d1, u2);
          o[j] = a.x, o[j + 1] = a.y;
          if (kMode >= 2) o2[j] = b.x, o2[j + 1] = b.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const GeluTerms t = gelu_terms(hv[j]);
          if (kMode == 0) o[j] = t.g;
          if (kMode == 1) o[j] = t.d1 * vv[j];
          if (kMode == 2) o[j] = t.d1 * vv[j], o2[j] = t.d2 * wv[j] * vv[j];
          if (kMode == 3) o[j] = t.g, o2[j] = t.d1 * vv[j];
          if (kMode == 4) o[j] = t.d1 * vv[j] + t.d2 * wv[j] * uv[j], o2[j] = t.d1 * uv[j];
        }
      }
      store8<T>(out + idx[c] * 8, o);
      if (kMode >= 2) store8<T>(out2 + idx[c] * 8, o2);
    }
  }
}

// Calls f(T{}, integral_constant<NV>) for the element type (dtype code 0 = bf16, 2 = fp32) and C / 256 in 1..4.
template <typename F>
cudaError_t dispatch(int dtype, int C, F &&f) {
  auto with_nv = [&](auto t) -> cudaError_t {
    switch (C / 256) {
      case 1: return f(t, std::integral_constant<int, 1>{});
      case 2: return f(t, std::integral_constant<int, 2>{});
      case 3: return f(t, std::integral_constant<int, 3>{});
      case 4: return f(t, std::integral_constant<int, 4>{});
      default: return cudaErrorInvalidValue;
    }
  };
  if (dtype == JVPATTN_BF16) return with_nv(__nv_bfloat16{});
  if (dtype == JVPATTN_FP32) return with_nv(float{});
  return cudaErrorInvalidValue;
}

}  // namespace

bool dual_shape_ok(int B, int S, int C) { return B >= 0 && S >= 1 && C >= 256 && C <= 1024 && C % 256 == 0; }

cudaError_t ln_modulate(int which, const void *x, const void *tx, const float *gamma, const float *beta, const void *shift,
                        const void *scale, const void *tshift, const void *tscale, int64_t mod_stride, int64_t tmod_stride,
                        float *mean, float *rstd, void *out, const void *g, void *dx, void *dtx, float *sums, int B, int S, int C,
                        float eps, int exact, int dtype, cudaStream_t stream) {
  LnArgs a{x, tx, gamma, beta, shift, scale, tshift, tscale, mod_stride, tmod_stride, mean, rstd, out, nullptr, g, nullptr, dx, dtx, sums,
           B, S, C, eps, exact};
  const int64_t rows = (int64_t)B * S;
  if (rows == 0) return cudaSuccess;
  LaunchScope scope(kIdDual, stream);
  return dispatch(dtype, C, [&](auto t, auto nv) -> cudaError_t {
    using T = decltype(t);
    constexpr int NV = decltype(nv)::value;
    if (which == 0 || which == 1) {
      const unsigned grid = (unsigned)((rows + kWarpsPerCta - 1) / kWarpsPerCta);
      if (which == 0) {
        const int rows_cta = rows_per_cta(B, S, kWarpsPerCta, 4);  // (four blocks fit an SM)
        if (std::min(S, rows_cta) >= (NV == 4 ? 16 : 8))
          ln_modulate_fwd_kernel<T, NV><<<(unsigned)(B * ((S + rows_cta - 1) / rows_cta)), kWarpsPerCta * 32, 0, stream>>>(a, rows_cta);
        else
          ln_modulate_fwd_row_kernel<T, NV><<<grid, kWarpsPerCta * 32, 0, stream>>>(a);
      } else {
        ln_modulate_fwd_tangent_kernel<T, NV><<<grid, kWarpsPerCta * 32, 0, stream>>>(a);
      }
    } else {
      const int rows_cta = rows_per_cta(B, S, 16, 8, which == 2 ? std::min(8, (sizeof(T) == 2 ? 16 : 12) / NV) : 0);
      const unsigned grid = (unsigned)(B * ((S + rows_cta - 1) / rows_cta));
      if (which == 2) {
        ln_modulate_bwd_kernel<T, NV, false><<<grid, NV * 32, 0, stream>>>(a, rows_cta);
      } else {
        auto k = ln_modulate_bwd_tangent_kernel<T, NV>;
        constexpr int smem = kWarpsPerCta * 3 * NV * 256 * 4;
        if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        k<<<grid, kWarpsPerCta * 32, smem, stream>>>(a, rows_cta);
      }
    }
    return cudaGetLastError();
  });
}

cudaError_t ln_modulate_dual(int which, const void *x, const void *tx, const float *gamma, const float *beta, const void *shift,
                             const void *scale, const void *tshift, const void *tscale, int64_t mod_stride, int64_t tmod_stride,
                             float *mean, float *rstd, void *y, void *ty, const void *g, const void *gt, void *dx, void *dtx,
                             float *sums, int B, int S, int C, float eps, int exact, int dtype, cudaStream_t stream) {
  LnArgs a{x, tx, gamma, beta, shift, scale, tshift, tscale, mod_stride, tmod_stride, mean, rstd, y, ty, g, gt, dx, dtx, sums,
           B, S, C, eps, exact};
  const int64_t rows = (int64_t)B * S;
  if (rows == 0) return cudaSuccess;
  LaunchScope scope(kIdDual, stream);
  return dispatch(dtype, C, [&](auto t, auto nv) -> cudaError_t {
    using T = decltype(t);
    constexpr int NV = decltype(nv)::value;
    if constexpr (!std::is_same<T, __nv_bfloat16>::value) {
      return cudaErrorInvalidValue;
    } else if (which == 0) {
      // Below four rows a sample most warps of a CTA of its own would idle (rows of 768: 16384 x 1 52 us a row per warp, 70 so;
      // 4096 x 4 46 and 29; 8 x 128 6.5 and 4.5).
      const int rows_cta = rows_per_cta(B, S, kWarpsPerCta, 4);
      if (S >= kWarpsPerCta)
        ln_modulate_dual_fwd_walk_kernel<T, NV><<<(unsigned)(B * ((S + rows_cta - 1) / rows_cta)), kWarpsPerCta * 32, 0, stream>>>(a, rows_cta);
      else
        ln_modulate_dual_fwd_kernel<T, NV><<<(unsigned)((rows + kWarpsPerCta - 1) / kWarpsPerCta), kWarpsPerCta * 32, 0, stream>>>(a);
    } else {
      const int rows_cta = rows_per_cta(B, S, 16, 8, 16 / NV);
      ln_modulate_bwd_kernel<T, NV, true><<<(unsigned)(B * ((S + rows_cta - 1) / rows_cta)), NV * 32, 0, stream>>>(a, rows_cta);
    }
    return cudaGetLastError();
  });
}

cudaError_t gated_residual(const void *x, const void *y, const void *gate, const void *mask, int64_t gate_stride, void *z, int B,
                           int S, int C, int dtype, const unsigned long long *drop_seed, unsigned drop_call, float drop_p,
                           cudaStream_t stream) {
  const int64_t total = (int64_t)B * S * C / 8;
  if (total == 0) return cudaSuccess;
  if (C % 8) return cudaErrorInvalidValue;
  GateArgs a{x, y, gate, mask, gate_stride, z, B, S, C, {drop_seed, drop_call, drop_p}};
  LaunchScope scope(kIdDual, stream);
  const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 8);
  auto launch = [&](auto tag) -> cudaError_t {
    using T = decltype(tag);
    // (fp32 operands that L2 does not hold together run faster through the 64-bit kernel, which keeps fewer of them in flight:
    // 128 x 128 rows of 768 with a mask 33.7 -> 31.1 us, of 1024 45.9 -> 40.5; 64 x 128 rows without one 10.3 against 10.9 us)
    const bool in_l2 = sizeof(T) == 2 || total * 8 * (int64_t)sizeof(T) * (mask ? 4 : 3) < (int64_t(96) << 20);
    if (index32(total) && in_l2) gated_residual_fwd_kernel<T, uint32_t><<<grid, 256, 0, stream>>>(a);
    else gated_residual_fwd_kernel<T, int64_t><<<grid, 256, 0, stream>>>(a);
    return cudaGetLastError();
  };
  if (dtype == JVPATTN_BF16) return launch(__nv_bfloat16{});
  if (dtype == JVPATTN_FP32) return launch(float{});
  return cudaErrorInvalidValue;
}

cudaError_t gate_ln(const void *x, const void *y, const void *gate, int64_t gate_stride, const float *gamma, const float *beta, const void *shift,
                    const void *scale, int64_t mod_stride, void *z, void *h, int B, int S, int C, float eps, int dtype, cudaStream_t stream) {
  const int64_t rows = (int64_t)B * S;
  if (rows == 0) return cudaSuccess;
  const GateLnArgs a{x, y, gate, gate_stride, gamma, beta, shift, scale, mod_stride, z, h, B, S, eps};
  LaunchScope scope(kIdDual, stream);
  return dispatch(dtype, C, [&](auto t, auto nv) -> cudaError_t {
    gate_ln_fwd_kernel<decltype(t), decltype(nv)::value><<<(unsigned)((rows + kWarpsPerCta - 1) / kWarpsPerCta), kWarpsPerCta * 32, 0, stream>>>(a);
    return cudaGetLastError();
  });
}

cudaError_t ln_finalize(const float *p, const float *t, const float *gamma, const float *beta, const void *scale,
                        const void *tscale, int64_t mod_stride, int64_t tmod_stride, void *d_shift, void *d_scale, void *d_tshift,
                        void *d_tscale, float *d_gamma, float *d_beta, int B, int C, int dtype, cudaStream_t stream) {
  if (C == 0) return cudaSuccess;
  LnFinalArgs a{p, t, gamma, beta, scale, tscale, mod_stride, tmod_stride, d_shift, d_scale, d_tshift, d_tscale, d_gamma, d_beta, B, C};
  LaunchScope scope(kIdDual, stream);
  if (B == 0) return cudaSuccess;
  const int64_t grid = (int64_t)((C + 127) / 128) * (((int64_t)B + kFinalSamples - 1) / kFinalSamples);
  if (grid > INT32_MAX) return cudaErrorInvalidValue;
  if (dtype == JVPATTN_BF16) ln_finalize_kernel<__nv_bfloat16><<<(unsigned)grid, 128, 0, stream>>>(a);
  else if (dtype == JVPATTN_FP32) ln_finalize_kernel<float><<<(unsigned)grid, 128, 0, stream>>>(a);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t gated_residual_dual(int which, const void *x, const void *tx, const void *y, const void *ty, const void *gate,
                                const void *tgate, const void *mask, int64_t gate_stride, int64_t tgate_stride, void *z, void *tz,
                                const void *gz, const void *gtz, void *d_y, void *d_ty, float *sums, int B, int S, int C, int dtype,
                                const unsigned long long *drop_seed, unsigned drop_call, float drop_p, cudaStream_t stream) {
  if ((int64_t)B * S * C == 0) return cudaSuccess;
  if (C % 8 || C > 1024) return cudaErrorInvalidValue;
  GateDualArgs a{x, tx, y, ty, gate, tgate, mask, gate_stride, tgate_stride, z, tz, gz, gtz, d_y, d_ty, sums, B, S, C,
                 {drop_seed, drop_call, drop_p}};
  LaunchScope scope(kIdDual, stream);
  auto launch = [&](auto tag) -> cudaError_t {
    using T = decltype(tag);
    if (which == 0) {
      const int64_t n8 = (int64_t)B * S * C / 8;
      const unsigned grid = (unsigned)std::min<int64_t>((n8 + 255) / 256, 148 * 16);
      if (index32(n8)) gated_dual_fwd_kernel<T, uint32_t><<<grid, 256, 0, stream>>>(a);
      else gated_dual_fwd_kernel<T, int64_t><<<grid, 256, 0, stream>>>(a);
    } else {
      const int threads = (C / 8 + 31) / 32 * 32;
      const int rows_cta = rows_per_cta(B, S, 16, 8, 512 / threads);
      gated_dual_bwd_kernel<T><<<(unsigned)(B * ((S + rows_cta - 1) / rows_cta)), threads, 0, stream>>>(a, rows_cta);
    }
    return cudaGetLastError();
  };
  if (dtype == JVPATTN_BF16) return launch(__nv_bfloat16{});
  if (dtype == JVPATTN_FP32) return launch(float{});
  return cudaErrorInvalidValue;
}

cudaError_t gelu_dual(int mode, const void *h, const void *v, const void *w, const void *u, void *out, void *out2, int64_t n,
                      int dtype, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (n % 8) return cudaErrorInvalidValue;
  const int64_t n8 = n / 8;
  const unsigned grid = (unsigned)std::min<int64_t>((n8 + 511) / 512, 148 * 8);
  LaunchScope scope(kIdDual, stream);
  auto launch = [&](auto tag) -> cudaError_t {
    using T = decltype(tag);
    auto H = static_cast<const T *>(h), V = static_cast<const T *>(v), W = static_cast<const T *>(w), U = static_cast<const T *>(u);
    auto O = static_cast<T *>(out), O2 = static_cast<T *>(out2);
    switch (mode) {
      case 0: gelu_dual_kernel<T, 0><<<grid, 256, 0, stream>>>(H, V, W, U, O, O2, n8); break;
      case 1: gelu_dual_kernel<T, 1><<<grid, 256, 0, stream>>>(H, V, W, U, O, O2, n8); break;
      case 2: gelu_dual_kernel<T, 2><<<grid, 256, 0, stream>>>(H, V, W, U, O, O2, n8); break;
      case 3: gelu_dual_kernel<T, 3><<<grid, 256, 0, stream>>>(H, V, W, U, O, O2, n8); break;
      case 4: gelu_dual_kernel<T, 4><<<grid, 256, 0, stream>>>(H, V, W, U, O, O2, n8); break;
      default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
  };
  if (dtype == JVPATTN_BF16) return launch(__nv_bfloat16{});
  if (dtype == JVPATTN_FP32) return launch(float{});
  return cudaErrorInvalidValue;
}

}  // namespace jvpattn
