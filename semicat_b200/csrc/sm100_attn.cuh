// Small device/host helpers shared by the tcgen05 attention kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "jvpattn_common.cuh"

namespace jvpattn {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}

// What the pair (a, b) is above its 16-bit rounding `hi` = pack2(a, b), rounded to 16 bits itself: hi + rest carries 16
// significant bits where bf16 carries 8.  Nothing above an infinite value, where inf - inf would make it NaN (one packed compare
// and an AND: 32 x 8 heads of 32 channels at length 256, backward 72 -> 76 us, 79 with a compare per element; kFinite
// leaves them out for P, which no finite scores make infinite).
template <typename T, bool kFinite = false>
__device__ __forceinline__ uint32_t pack2_rest(float a, float b, uint32_t hi) {
  static_assert(std::is_same<T, __nv_bfloat16>::value, "fp16 parts do not have the exponent range");
  const uint32_t lo = pack2<T>(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
  if (kFinite) return lo;
  const uint32_t largest = 0x7f7f7f7fu;  // both halves the largest finite value
  return lo & __hle2_mask(__habs2(*reinterpret_cast<const __nv_bfloat162 *>(&hi)), *reinterpret_cast<const __nv_bfloat162 *>(&largest));
}

template <typename T> struct IsBf16 { static constexpr bool value = false; };
template <> struct IsBf16<__nv_bfloat16> { static constexpr bool value = true; };

// Head dimensions of the tcgen05 kernels.  Their tiles are 64 or 128 channels wide.  A bf16 head of another width (a
// multiple of 8, so that rows stay 16-byte aligned) runs on the next wider tile: the tensor maps carry the true width, a
// load fills the channels past it with zeros (no memory is read for them), which add nothing to any product, and a
// store drops them.  The portable kernels that these widths had before keep P, U and the backward's weights in
// fp32, so here each such operand goes into its product as two bf16 parts (16 significant bits, below the rounding of
// the bf16 result by 2^-8) instead of one.  fp16 heads of other widths stay on the portable kernels: fp16 parts do not have
// the exponent range of the fp32 values.  Forward and backward of 32 x 8 heads of 32 channels at length 256: 5.0 ms on the
// portable kernels, 0.16 ms of device time here.
inline bool sm100_native_head_dim(int D) { return D == 64 || D == 128; }
inline bool sm100_head_dim_ok(int D, int dtype) {
  return sm100_native_head_dim(D) || (D >= 16 && D < 128 && D % 8 == 0 && dtype == JVPATTN_BF16);
}

// A view the TMA / vector-store paths can take: 16-byte aligned base, strides that keep every row 16-byte
// aligned, rows that do not overlap, and a positive stride below 2^40 bytes on every axis that has more than one
// entry (a tensor map cannot describe a broadcast axis; an expanded tensor takes the SIMT kernels instead).
inline bool tma_view_ok(const View &v, int B, int H, int L, int D) {
  if (!v.ptr) return false;
  if (reinterpret_cast<uintptr_t>(v.ptr) % 16 != 0) return false;
  auto axis_ok = [](int64_t stride, int n) { return n <= 1 || (stride > 0 && stride % 8 == 0 && stride < (int64_t(1) << 39)); };
  return axis_ok(v.sl, L) && axis_ok(v.sh, H) && axis_ok(v.sb, B) && (L <= 1 || v.sl >= D);
}

}  // namespace jvpattn
