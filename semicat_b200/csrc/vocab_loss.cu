// Vocabulary-side ends of the flow-map training step, each as one pass family over (rows, V) with nothing of that
// size materialised in fp32 (semicat/models/semicat.py:70-85 interpolation, :89-110 cross-entropy step, :112-167
// self-distillation step with sd_type "lag", :210-229 flow map):
//
//   interp       xt   = (1 - t) x0 + t onehot(id)                            -> 16-bit, row pitch padded for the embedding GEMM
//   xst          xst  = xs + dt (softmax(l) - xs),  xs = (1 - s) x0 + s onehot(id),  dt = (t - s) / (1 - s + 1e-8)
//                                                                             -> 16-bit padded (input of the target pass); lse
//   ce_fwd/bwd   cross-entropy of padded 16-bit logits against ids (label smoothing eps), per-row loss and d loss / d logits
//   sd_fwd/bwd   sum_v ((1 - t) dv - softmax(l_target) + xst)^2 per row, with
//                dv = ddt (p - xs) + dt p o (tl - sum(p tl)),  ddt = 1 / (1 - s + 1e-8)   (the t-derivative of the flow map
//                by forward mode: l are the logits, tl their tangent), and its gradient with respect to l and tl.
//
// x0 is the fp32 noise (row pitch ldx), everything else is recomputed per element, so the only (rows, V) traffic is the
// operands themselves.  One CTA per (b, l) row; rows are walked in chunks of 8 columns with 16-byte accesses; columns at
// or beyond V (the padding of the GEMM operands) read as -inf logits / zero inputs and are written as zeros.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <utility>

#include "jvpattn_common.cuh"

namespace jvpattn {
namespace {

constexpr int kThreads = 256;
constexpr float kNegInf = -INFINITY;

template <typename T> struct Pack8;
template <> struct Pack8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16 *p, float (&v)[8]) {
    const uint4 u = *reinterpret_cast<const uint4 *>(p);
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16 *p, const float (&v)[8]) {
    uint4 u;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4 *>(p) = u;
  }
};
template <> struct Pack8<float> {
  static __device__ __forceinline__ void load(const float *p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  }
  static __device__ __forceinline__ void store(float *p, const float (&v)[8]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4 *>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
};

// fp32 noise row: 16-byte loads where the pitch allows (kVec), element loads with a bound otherwise
template <bool kVec>
__device__ __forceinline__ void load_x0(const float *row, int v0, int V, float (&x)[8]) {
  if (kVec) {
    Pack8<float>::load(row + v0, x);  // the padded pitch covers the whole chunk
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = v0 + i < V ? row[v0 + i] : 0.f;
  }
}

template <int NQ, int NT = kThreads>
__device__ __forceinline__ void block_sum(float (&v)[NQ], float *scratch) {
  constexpr int kWarps = NT / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  __syncthreads();  // scratch may still be read from an earlier reduction
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) scratch[q * kWarps + warp] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    float r = scratch[q * kWarps];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) r += scratch[q * kWarps + w];
    v[q] = r;
  }
}

// (exp(a + c), exp(b + c)), the sums and the scaling two wide: issue slots, not the exponential unit, bound the passes over the
// logits.
__device__ __forceinline__ float2 exp2x(float a, float b, float c) {
  const float2 e = __fmul2_rn(__fadd2_rn(make_float2(a, b), make_float2(c, c)), make_float2(1.4426950408889634f, 1.4426950408889634f));
  float2 r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(e.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(e.y));
  return r;
}

// Calls f(first column, whole) for this thread's chunks of 8 columns.  Only the row's last chunk can reach past V: `whole` is a
// compile-time constant that takes the per-element checks of the arithmetic out of all others (what remains is one test per
// chunk in load_logits, and load_x0's own for noise off the 16-byte pitch).  With them and scalar exponents the passes over 16-bit
// logits were bound by instructions: 6144 rows of 30522, cross-entropy forward 112 -> 72 us (57 us at the memory rate),
// backward 148 -> 124 us (115 us), 2048 rows of the flow map 112 -> 102 us (77 us).  The last chunk goes to another warp than the
// one before it, beside which it runs (256 rows of 27: self-distillation forward 6.2 -> 5.8 us).
template <typename F>
__device__ __forceinline__ void for_chunks(int V, F &&f) {
  const int nfull = V / 8;
  for (int c = threadIdx.x; c < nfull; c += kThreads) f(c * 8, std::true_type{});
  if (V % 8 && threadIdx.x == (nfull + 32) % kThreads) f(nfull * 8, std::false_type{});
}

// Running (max, sum of exp) of one thread's elements, then across the block: returns the row's log-sum-exp.
struct OnlineLse {
  float mx = kNegInf, sm = 0.f;
  __device__ __forceinline__ void add8(const float (&l)[8]) {
    float cm = l[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) cm = fmaxf(cm, l[i]);
    if (cm == kNegInf) return;
    if (cm > mx) {
      sm *= __expf(mx - cm);  // exp(-inf) = 0 on the first chunk
      mx = cm;
    }
    float2 t = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) t = __fadd2_rn(t, exp2x(l[2 * i], l[2 * i + 1], -mx));
    sm += t.x + t.y;
  }
  template <int NT = kThreads>
  __device__ __forceinline__ float finish(float *scratch) {
    float m = mx;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = m;
    __syncthreads();
    float M = scratch[0];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) M = fmaxf(M, scratch[w]);
    float s[1] = {mx == kNegInf ? 0.f : sm * __expf(mx - M)};
    block_sum<1, NT>(s, scratch);
    return M + __logf(s[0]);
  }
};

template <typename T>
__device__ __forceinline__ void load_logits(const T *row, int v0, int V, float (&l)[8]) {
  Pack8<T>::load(row + v0, l);
  if (v0 + 8 > V) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (v0 + i >= V) l[i] = kNegInf;
  }
}

// Log-sum-exp of a row, two chunks in flight per thread.
template <typename T>
__device__ __forceinline__ void add_row(OnlineLse &acc, const T *l, int V) {
  const int nfull = V / 8;
  int c = threadIdx.x;
  for (; c + kThreads < nfull; c += 2 * kThreads) {
    float a[8], b[8];
    Pack8<T>::load(l + c * 8, a);
    Pack8<T>::load(l + (c + kThreads) * 8, b);
    acc.add8(a);
    acc.add8(b);
  }
  for (; c * 8 < V; c += kThreads) {
    float a[8];
    load_logits<T>(l, c * 8, V, a);
    acc.add8(a);
  }
}

// Zeros in the chunks of an output row behind the one that holds column V - 1.
template <typename T>
__device__ __forceinline__ void zero_tail(T *out, int V, int64_t ldo) {
  const float o[8] = {};
  for (int64_t c = (V + 7) / 8 + threadIdx.x; c < ldo / 8; c += kThreads) Pack8<T>::store(out + c * 8, o);
}

struct VocabArgs {
  const void *l, *tl, *lt;     // logits, their tangent, target logits: 16-bit or fp32, row pitch ld (elements, multiple of 8)
  int64_t ld;
  const float *x0;             // noise, row pitch ldx
  int64_t ldx;
  const int64_t *ids;          // [rows]
  const float *s, *t;          // [batch]
  float *lse;                  // [rows]
  float *stats;                // [rows, 4]: lse of the target logits, m = sum(p tl), sum(p r), sum(p r tl)
  float *loss;                 // [rows]
  const float *g;              // scalar cotangent of the MEAN of the row losses (device memory)
  void *out, *out2;            // 16-bit / fp32 outputs, row pitch ldo
  int64_t ldo;
  float eps;                   // label smoothing
  int rows_per_sample, V;
  int64_t rows;
};

// ------------------------------------------------------------------------------------------------ interpolation
template <typename T, bool kVec>
__global__ void __launch_bounds__(kThreads) interp_kernel(VocabArgs a) {
  const int64_t row = blockIdx.x;
  const float t = a.t[row / a.rows_per_sample];
  const int id = (int)a.ids[row];
  const float *x0 = a.x0 + row * a.ldx;
  T *out = static_cast<T *>(a.out) + row * a.ldo;
  const int nchunk = (int)(a.ldo / 8);
  for (int c = threadIdx.x; c < nchunk; c += kThreads) {
    const int v0 = c * 8;
    float x[8];
    if (v0 < a.V) {
      load_x0<kVec>(x0, v0, a.V, x);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = v0 + i < a.V ? (1.f - t) * x[i] + (v0 + i == id ? t : 0.f) : 0.f;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = 0.f;
    }
    Pack8<T>::store(out + v0, x);
  }
}

// ------------------------------------------------------------------------------------------------ rows held in shared memory between two passes
// A persistent CTA walks rows; each thread copies the chunks that it will itself read (16 bytes of each of NTENS bf16 rows, chunk
// c of a row at column 8 (c NT + thread)) into shared memory of its own and waits for its own copies alone, so they need no
// barrier.  The next row's chunk is requested as soon as the second pass has read this one's.  A row takes kChunks places whatever
// its length; those past its end hold nothing.  One place more, to keep memory busy while the block reduces the first pass, was no
// faster, nor was any other split of the row over threads (512 of 8 chunks, 1024 of 4).
template <int NT, int NTENS>
struct RowStage {
  static constexpr int kChunks = 6;
  static constexpr size_t kBytes = (size_t)kChunks * NTENS * NT * 16;
  uint4 *buf;
  const __nv_bfloat16 *src[NTENS];  // this thread's next chunk
  int64_t row, rows, step;          // step: from a row's last place to the first of this CTA's next row
  int nchunk, c = 0;
  __device__ __forceinline__ void start(uint4 *buf_, const VocabArgs &a, const void *const (&tensors)[NTENS]) {
    buf = buf_;
    row = blockIdx.x, rows = a.rows, nchunk = (a.V + 7) / 8;
    step = (int64_t)gridDim.x * a.ld - (int64_t)(kChunks - 1) * NT * 8;
#pragma unroll
    for (int k = 0; k < NTENS; ++k) src[k] = static_cast<const __nv_bfloat16 *>(tensors[k]) + row * a.ld + threadIdx.x * 8;
#pragma unroll
    for (int i = 0; i < kChunks; ++i) request();
  }
  __device__ __forceinline__ void request() {
    if (row < rows && c * NT + (int)threadIdx.x < nchunk) {
#pragma unroll
      for (int k = 0; k < NTENS; ++k) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(buf + (c * NTENS + k) * NT + threadIdx.x);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src[k]) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const bool wrap = ++c == kChunks;
#pragma unroll
    for (int k = 0; k < NTENS; ++k) src[k] += wrap ? step : (int64_t)NT * 8;
    if (wrap) c = 0, row += gridDim.x;
  }
  template <int C>
  __device__ __forceinline__ void wait() const {  // for chunk C of the first pass: the row's later ones may be under way
    asm volatile("cp.async.wait_group %0;" ::"n"(kChunks - 1 - C) : "memory");
  }
  __device__ __forceinline__ void read(int chunk, int k, float (&v)[8]) const {
    Pack8<__nv_bfloat16>::load(reinterpret_cast<const __nv_bfloat16 *>(buf + (chunk * NTENS + k) * NT + threadIdx.x), v);
  }
};
// f(0), f(1), ... with compile-time arguments
template <int... I, typename F>
__device__ __forceinline__ void unrolled(std::integer_sequence<int, I...>, F &&f) {
  (f(std::integral_constant<int, I>{}), ...);
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ------------------------------------------------------------------------------------------------ flow map, primal
template <typename T, bool kVec>
__global__ void __launch_bounds__(kThreads) xst_kernel(VocabArgs a) {
  __shared__ float scratch[8];
  const int64_t row = blockIdx.x;
  const int b = (int)(row / a.rows_per_sample);
  const float s = a.s[b], t = a.t[b], dt = (t - s) / (1.f - s + 1e-8f);
  const int id = (int)a.ids[row], V = a.V;
  const T *l = static_cast<const T *>(a.l) + row * a.ld;
  const float *x0 = a.x0 + row * a.ldx;
  T *out = static_cast<T *>(a.out) + row * a.ldo;
  OnlineLse acc;
  add_row<T>(acc, l, V);
  const float lse = acc.finish(scratch);
  if (threadIdx.x == 0) a.lse[row] = lse;
  for_chunks(V, [&](int v0, auto tag) {
    constexpr bool whole = decltype(tag)::value;
    float lv[8], x[8], o[8];
    load_logits<T>(l, v0, V, lv);
    load_x0<kVec>(x0, v0, V, x);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const float2 p = exp2x(lv[i], lv[i + 1], -lse);
      const float xs0 = (1.f - s) * x[i] + (v0 + i == id ? s : 0.f), xs1 = (1.f - s) * x[i + 1] + (v0 + i + 1 == id ? s : 0.f);
      o[i] = xs0 + dt * (p.x - xs0);
      o[i + 1] = xs1 + dt * (p.y - xs1);
    }
    if (!whole) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (v0 + i >= V) o[i] = 0.f;
    }
    Pack8<T>::store(out + v0, o);
  });
  zero_tail<T>(out, V, a.ldo);
}

// xst_kernel for bf16 rows that fit: l is read once, and the next row's while this one's results leave; the one-hot term is
// added to the one chunk that holds it.  30522 columns: 2048 rows 101 -> 85 us, 6144 273 -> 238 us (229 us at the copy rate);
// 8192 rows of 512 columns 21 -> 17 us.
template <int NT, bool kVec>
__global__ void __launch_bounds__(NT, 1536 / NT) xst_staged_kernel(VocabArgs a) {
  using Stage = RowStage<NT, 1>;
  constexpr int kWarps = NT / 32, NC = Stage::kChunks;
  extern __shared__ uint4 stage_raw[];
  __shared__ float s_max[kWarps], s_sum[kWarps];
  const int V = a.V, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Stage stage;
  stage.start(stage_raw, a, {a.l});
  for (int64_t row = blockIdx.x; row < a.rows; row += gridDim.x) {
    const unsigned b = (unsigned)row / (unsigned)a.rows_per_sample;
    const float s = a.s[b], t = a.t[b];
    const int id = (int)a.ids[row];
    OnlineLse acc;
    unrolled(std::make_integer_sequence<int, NC>{}, [&](auto ci) {
      constexpr int c = decltype(ci)::value;
      stage.template wait<c>();
      const int v0 = (c * NT + threadIdx.x) * 8;
      if (v0 >= V) return;
      float lv[8];
      stage.read(c, 0, lv);
      if (v0 + 8 > V) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (v0 + i >= V) lv[i] = kNegInf;
      }
      acc.add8(lv);
    });
    const float wmax = warp_max(acc.mx);
    if (lane == 0) s_max[warp] = wmax;
    __syncthreads();
    float M = s_max[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, s_max[w]);
    float sum = acc.mx == kNegInf ? 0.f : acc.sm * __expf(acc.mx - M);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    sum = s_sum[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) sum += s_sum[w];
    const float lse = M + __logf(sum), dt = (t - s) / (1.f - s + 1e-8f);
    if (threadIdx.x == 0) a.lse[row] = lse;
    const float *x0 = a.x0 + row * a.ldx;
    __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(a.out) + row * a.ldo;
    unrolled(std::make_integer_sequence<int, NC>{}, [&](auto ci) {
      constexpr int c = decltype(ci)::value;
      const int v0 = (c * NT + threadIdx.x) * 8;
      if (v0 < V) {
        float lv[8], x[8], o[8];
        load_x0<kVec>(x0, v0, V, x);
        stage.read(c, 0, lv);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] *= 1.f - s;
        if ((unsigned)(id - v0) < 8u) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (v0 + i == id) x[i] += s;
        }
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          const float2 p = exp2x(lv[i], lv[i + 1], -lse), xs = make_float2(x[i], x[i + 1]);
          const float2 r = __ffma2_rn(make_float2(dt, dt), __fadd2_rn(p, make_float2(-xs.x, -xs.y)), xs);
          o[i] = r.x, o[i + 1] = r.y;
        }
        if (v0 + 8 > V) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (v0 + i >= V) o[i] = 0.f;
        }
        Pack8<__nv_bfloat16>::store(out + v0, o);
      }
      stage.request();  // over the chunk just read
    });
    for (int64_t c = (V + 7) / 8 + threadIdx.x; c < a.ldo / 8; c += NT) {
      const float zero[8] = {};
      Pack8<__nv_bfloat16>::store(out + c * 8, zero);
    }
  }
}

// ------------------------------------------------------------------------------------------------ cross-entropy
// (eight CTAs per SM: fp32 logits otherwise take 37 registers and six; 2048 rows of 30522 with smoothing 49 -> 43.5 us)
template <typename T>
__global__ void __launch_bounds__(kThreads, 8) ce_fwd_kernel(VocabArgs a) {
  __shared__ float scratch[16];
  const int64_t row = blockIdx.x;
  const int id = (int)a.ids[row], V = a.V;
  const T *l = static_cast<const T *>(a.l) + row * a.ld;
  OnlineLse acc;
  float sums[1] = {0.f};  // sum of the logits (label smoothing)
  if (a.eps == 0.f) {
    add_row<T>(acc, l, V);
  } else {
    for_chunks(V, [&](int v0, auto tag) {
    constexpr bool whole = decltype(tag)::value;
      float lv[8];
      load_logits<T>(l, v0, V, lv);
      acc.add8(lv);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (whole || v0 + i < V) sums[0] += lv[i];
    });
  }
  const float lse = acc.finish(scratch);
  if (a.eps != 0.f) block_sum<1>(sums, scratch);
  if (threadIdx.x == 0) {
    const float target = id >= 0 && id < V ? (float)l[id] : 0.f;
    a.lse[row] = lse;
    a.loss[row] = a.eps == 0.f ? lse - target : (1.f - a.eps) * (lse - target) + a.eps * (lse - sums[0] / (float)V);
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) ce_bwd_kernel(VocabArgs a) {
  const int64_t row = blockIdx.x;
  const int id = (int)a.ids[row], V = a.V;
  const T *l = static_cast<const T *>(a.l) + row * a.ld;
  T *dl = static_cast<T *>(a.out) + row * a.ldo;
  const float lse = a.lse[row], gs = a.g[0] / (float)a.rows, off = a.eps / (float)V, hit = 1.f - a.eps;
  for_chunks(V, [&](int v0, auto tag) {
    constexpr bool whole = decltype(tag)::value;
    float lv[8], o[8];
    load_logits<T>(l, v0, V, lv);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const float2 p = exp2x(lv[i], lv[i + 1], -lse);
      o[i] = p.x;
      o[i + 1] = p.y;
    }
    if (id >= v0 && id < v0 + 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (v0 + i == id) o[i] -= hit;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = whole || v0 + i < V ? gs * (o[i] - off) : 0.f;
    Pack8<T>::store(dl + v0, o);
  });
  zero_tail<T>(dl, V, a.ldo);
}

// ------------------------------------------------------------------------------------------------ self-distillation ("lag")
// The residual of one element, (1 - t) dv - q + xst with q = softmax(l_target), in the form shared by the forward and the
// backward.  In the interpolated input its coefficient is 1 - dt - (1 - t) ddt = 1e-8 ddt and in p it is dt + (1 - t) ddt =
// (1 - s) ddt, so that
//   r = p ((1 - s) ddt - beta m + beta tl) - q + 1e-8 ddt xs,     beta = (1 - t) dt.
// Written out term by term, sums of the size of the noise cancel and leave their rounding (1e-7 |x0|) in r.  Here the last term
// is all that is left of the noise; where its coefficient is below 2^-24 (s < 0.83) it is below that rounding, and the row does
// without the noise.
struct SdRow {
  float s, beta, ddt, dt, k, lse, lse_t, m, ap;
  int id;
  bool noise;
  __device__ __forceinline__ void load(float s_, float t, float lse_, int id_) {
    s = s_, lse = lse_, id = id_;
    ddt = 1.f / (1.f - s + 1e-8f);
    dt = (t - s) * ddt;
    beta = (1.f - t) * dt;
    k = 1e-8f * ddt;
    noise = !(fabsf(k) <= 5.9604645e-8f);
  }
  __device__ __forceinline__ void target(float lse_t_, float m_) {
    lse_t = lse_t_, m = m_;
    ap = (1.f - s) * ddt - beta * m;
  }
  // residuals of columns v and v + 1 of probability p (x0: their noise, used where `kNoise`)
  template <bool kNoise>
  __device__ __forceinline__ float2 residual(float2 p, float2 tl, float2 lt, float2 x0, int v) const {
    const float2 q = exp2x(lt.x, lt.y, -lse_t);
    float2 r = __ffma2_rn(p, __ffma2_rn(make_float2(beta, beta), tl, make_float2(ap, ap)), make_float2(-q.x, -q.y));
    if (kNoise) {
      r.x += k * ((1.f - s) * x0.x + (v == id ? s : 0.f));
      r.y += k * ((1.f - s) * x0.y + (v + 1 == id ? s : 0.f));
    }
    return r;
  }
};

// (2048 rows of 30522 in bf16 169 -> 120 us, 8192 of 512 33 -> 31 us with the residual's form above, in fp32 252 -> 211 us.
// Five CTAs per SM: 48 registers.  Fewer rows at a time, so that the second pass finds them in L2, is slower: 186 against 172 us
// at four CTAs by registers, 208 / 211 / 245 at four / three / two by shared memory, before that form.  Noise off the 16-byte
// pitch needs 64 registers.)
template <typename T, bool kVec>
__global__ void __launch_bounds__(kThreads, kVec ? 5 : 4) sd_fwd_kernel(VocabArgs a) {
  __shared__ float scratch[24];
  const int64_t row = blockIdx.x;
  const int b = (int)(row / a.rows_per_sample), V = a.V;
  SdRow r;
  r.load(a.s[b], a.t[b], a.lse[row], (int)a.ids[row]);
  const T *l = static_cast<const T *>(a.l) + row * a.ld;
  const T *tl = static_cast<const T *>(a.tl) + row * a.ld;
  const T *lt = static_cast<const T *>(a.lt) + row * a.ld;
  const float *x0 = a.x0 + row * a.ldx;
  OnlineLse acc;
  float m[1] = {0.f};
  for_chunks(V, [&](int v0, auto tag) {
    constexpr bool whole = decltype(tag)::value;
    float lv[8], tv[8], qv[8];
    load_logits<T>(l, v0, V, lv);
    Pack8<T>::load(tl + v0, tv);
    load_logits<T>(lt, v0, V, qv);
    acc.add8(qv);
    float2 t = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; i += 2)
      t = __ffma2_rn(exp2x(lv[i], lv[i + 1], -r.lse),
                     make_float2(whole || v0 + i < V ? tv[i] : 0.f, whole || v0 + i + 1 < V ? tv[i + 1] : 0.f), t);
    m[0] += t.x + t.y;
  });
  const float lse_t = acc.finish(scratch);
  block_sum<1>(m, scratch);
  r.target(lse_t, m[0]);
  float sums[3] = {0.f, 0.f, 0.f};  // sum r^2, sum p r, sum p r tl
  auto second = [&](auto noise) {
    constexpr bool kNoise = decltype(noise)::value;
    for_chunks(V, [&](int v0, auto tag) {
      constexpr bool whole = decltype(tag)::value;
      float lv[8], tv[8], qv[8], x[8] = {};
      load_logits<T>(l, v0, V, lv);
      Pack8<T>::load(tl + v0, tv);
      load_logits<T>(lt, v0, V, qv);
      if (kNoise) load_x0<kVec>(x0, v0, V, x);
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const float2 p = exp2x(lv[i], lv[i + 1], -r.lse);
        const float2 res = r.residual<kNoise>(p, make_float2(tv[i], tv[i + 1]), make_float2(qv[i], qv[i + 1]),
                                              make_float2(x[i], x[i + 1]), v0 + i);
        if (whole || v0 + i < V) sums[0] += res.x * res.x, sums[1] += p.x * res.x, sums[2] += p.x * res.x * tv[i];
        if (whole || v0 + i + 1 < V) sums[0] += res.y * res.y, sums[1] += p.y * res.y, sums[2] += p.y * res.y * tv[i + 1];
      }
    });
  };
  r.noise ? second(std::true_type{}) : second(std::false_type{});
  block_sum<3>(sums, scratch);
  if (threadIdx.x == 0) {
    a.loss[row] = sums[0];
    float4 st = make_float4(r.lse_t, r.m, sums[1], sums[2]);
    *reinterpret_cast<float4 *>(a.stats + row * 4) = st;
  }
}

// sd_fwd_kernel for bf16 rows of which one fills an SM's shared memory (one CTA of 768 threads): its second pass reads 183 KB
// per row of 30522 from L2.  2048 such rows 120 -> 107 us, 6144 336 -> 304 us (172 us at the copy rate; issue slots, the
// reductions between the passes and 24 warps per SM are what is left).  Two or four CTAs on shorter rows are no faster than
// the plain kernel (2048 rows of 16000: 59 against 58 us), nor is keeping p in registers for the second pass.
constexpr int kSdStagedThreads = 768;
template <bool kVec>
__global__ void __launch_bounds__(kSdStagedThreads, 1) sd_fwd_staged_kernel(VocabArgs a) {
  constexpr int NT = kSdStagedThreads;
  using Stage = RowStage<NT, 3>;
  constexpr int kWarps = NT / 32, NC = Stage::kChunks;
  extern __shared__ uint4 stage_raw[];
  __shared__ float s_max[kWarps], s_one[2][kWarps], s_two[3][kWarps];  // one area per reduction: one barrier each
  const int V = a.V, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Stage stage;
  stage.start(stage_raw, a, {a.l, a.tl, a.lt});
  auto fetch = [&](int64_t row, float &s, float &t, float &lse, int &id) {
    if (row >= a.rows) return;
    const unsigned b = (unsigned)row / (unsigned)a.rows_per_sample;
    s = a.s[b], t = a.t[b], lse = a.lse[row], id = (int)a.ids[row];
  };
  float ns = 0.f, nt = 0.f, nlse = 0.f;
  int nid = 0;
  fetch(blockIdx.x, ns, nt, nlse, nid);
  for (int64_t row = blockIdx.x; row < a.rows; row += gridDim.x) {
    SdRow r;
    r.load(ns, nt, nlse, nid);
    OnlineLse acc;
    float2 m2 = make_float2(0.f, 0.f);
    unrolled(std::make_integer_sequence<int, NC>{}, [&](auto ci) {
      constexpr int c = decltype(ci)::value;
      stage.template wait<c>();
      const int v0 = (c * NT + threadIdx.x) * 8;
      if (v0 >= V) return;
      float lv[8], tv[8], qv[8];
      stage.read(c, 0, lv);
      stage.read(c, 1, tv);
      stage.read(c, 2, qv);
      if (v0 + 8 > V) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (v0 + i >= V) lv[i] = qv[i] = kNegInf, tv[i] = 0.f;
      }
      acc.add8(qv);
#pragma unroll
      for (int i = 0; i < 8; i += 2) m2 = __ffma2_rn(exp2x(lv[i], lv[i + 1], -r.lse), make_float2(tv[i], tv[i + 1]), m2);
    });
    const float wmax = warp_max(acc.mx);
    if (lane == 0) s_max[warp] = wmax;
    fetch(row + gridDim.x, ns, nt, nlse, nid);
    __syncthreads();
    float M = s_max[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, s_max[w]);
    float one[2] = {acc.mx == kNegInf ? 0.f : acc.sm * __expf(acc.mx - M), m2.x + m2.y};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) one[q] += __shfl_xor_sync(0xffffffffu, one[q], o);
      if (lane == 0) s_one[q][warp] = one[q];
    }
    __syncthreads();
    one[0] = one[1] = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) one[0] += s_one[0][w], one[1] += s_one[1][w];
    r.target(M + __logf(one[0]), one[1]);

    float2 rr = make_float2(0.f, 0.f), pr = rr, prt = rr;  // sum r^2, sum p r, sum p r tl
    auto second = [&](auto noise) {
      constexpr bool kNoise = decltype(noise)::value;
      const float *x0 = a.x0 + row * a.ldx;
      unrolled(std::make_integer_sequence<int, NC>{}, [&](auto ci) {
        constexpr int c = decltype(ci)::value;
        const int v0 = (c * NT + threadIdx.x) * 8;
          if (v0 < V) {
          float lv[8], tv[8], qv[8], x[8] = {};
          stage.read(c, 0, lv);
          stage.read(c, 1, tv);
          stage.read(c, 2, qv);
          if (kNoise) load_x0<kVec>(x0, v0, V, x);
          if (v0 + 8 > V) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (v0 + i >= V) lv[i] = qv[i] = kNegInf, tv[i] = x[i] = 0.f;  // p = q = 0
          }
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const float2 p = exp2x(lv[i], lv[i + 1], -r.lse), tl2 = make_float2(tv[i], tv[i + 1]);
            const float2 res = r.residual<kNoise>(p, tl2, make_float2(qv[i], qv[i + 1]), make_float2(x[i], x[i + 1]), v0 + i);
            const float2 w = __fmul2_rn(p, res);
            rr = __ffma2_rn(res, res, rr);
            pr = __fadd2_rn(pr, w);
            prt = __ffma2_rn(w, tl2, prt);
          }
        }
        stage.request();  // over the chunk just read
      });
    };
    r.noise ? second(std::true_type{}) : second(std::false_type{});
    float two[3] = {rr.x + rr.y, pr.x + pr.y, prt.x + prt.y};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) two[q] += __shfl_xor_sync(0xffffffffu, two[q], o);
      if (lane == 0) s_two[q][warp] = two[q];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        two[q] = lane < kWarps ? s_two[q][lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) two[q] += __shfl_xor_sync(0xffffffffu, two[q], o);
      }
      if (lane == 0) {
        a.loss[row] = two[0];
        *reinterpret_cast<float4 *>(a.stats + row * 4) = make_float4(r.lse_t, r.m, two[1], two[2]);
      }
    }
  }
}

// (2048 rows of 30522 in bf16: 138 -> 109 us, of 625 MB)
template <typename T, bool kVec>
__global__ void __launch_bounds__(kThreads) sd_bwd_kernel(VocabArgs a) {
  const int64_t row = blockIdx.x;
  const int b = (int)(row / a.rows_per_sample), V = a.V;
  SdRow r;
  r.load(a.s[b], a.t[b], a.lse[row], (int)a.ids[row]);
  const float4 st = *reinterpret_cast<const float4 *>(a.stats + row * 4);
  r.target(st.x, st.y);
  // cotangent on dv: H = gamma * residual, gamma = 2 (1 - t) g / rows; its row sums follow from the forward's
  const float gamma = 2.f * (1.f - a.t[b]) * a.g[0] / (float)a.rows;
  const float sH = gamma * st.z, sHt = gamma * st.w;
  const float spc = r.ddt * sH + r.dt * sHt - 2.f * r.dt * r.m * sH;
  const T *l = static_cast<const T *>(a.l) + row * a.ld;
  const T *tl = static_cast<const T *>(a.tl) + row * a.ld;
  const T *lt = static_cast<const T *>(a.lt) + row * a.ld;
  const float *x0 = a.x0 + row * a.ldx;
  T *dl = static_cast<T *>(a.out) + row * a.ldo;
  T *dtl = static_cast<T *>(a.out2) + row * a.ldo;
  auto pass = [&](auto noise) {
    constexpr bool kNoise = decltype(noise)::value;
    for_chunks(V, [&](int v0, auto tag) {
      constexpr bool whole = decltype(tag)::value;
      float lv[8], tv[8], qv[8], x[8] = {}, o1[8], o2[8];
      load_logits<T>(l, v0, V, lv);
      Pack8<T>::load(tl + v0, tv);
      load_logits<T>(lt, v0, V, qv);
      if (kNoise) load_x0<kVec>(x0, v0, V, x);
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const float2 p = exp2x(lv[i], lv[i + 1], -r.lse), tl2 = make_float2(tv[i], tv[i + 1]);
        const float2 res = r.residual<kNoise>(p, tl2, make_float2(qv[i], qv[i + 1]), make_float2(x[i], x[i + 1]), v0 + i);
        const float2 H = __fmul2_rn(make_float2(gamma, gamma), res);
        // ddt H + dt H (tl - m) - dt sH tl - spc
        const float2 c1 = __ffma2_rn(make_float2(r.dt, r.dt), __fadd2_rn(tl2, make_float2(-r.m, -r.m)), make_float2(r.ddt, r.ddt));
        const float2 c2 = __ffma2_rn(make_float2(-r.dt * sH, -r.dt * sH), tl2, make_float2(-spc, -spc));
        const float2 d1 = __fmul2_rn(p, __ffma2_rn(H, c1, c2));
        const float2 d2 = __fmul2_rn(__fmul2_rn(make_float2(r.dt, r.dt), p), __fadd2_rn(H, make_float2(-sH, -sH)));
        o1[i] = d1.x, o1[i + 1] = d1.y;
        o2[i] = d2.x, o2[i + 1] = d2.y;
      }
      if (!whole) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (v0 + i >= V) o1[i] = o2[i] = 0.f;
      }
      Pack8<T>::store(dl + v0, o1);
      Pack8<T>::store(dtl + v0, o2);
    });
  };
  r.noise ? pass(std::true_type{}) : pass(std::false_type{});
  zero_tail<T>(dl, V, a.ldo);
  zero_tail<T>(dtl, V, a.ldo);
}

template <typename K>
cudaError_t launch_staged(K kernel, int threads, size_t smem, int ctas_per_sm, const VocabArgs &a, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kernel<<<(unsigned)std::min<int64_t>(a.rows, (int64_t)sm_count() * ctas_per_sm), threads, smem, stream>>>(a);
  return cudaGetLastError();
}
template <int NT, bool kVec>
cudaError_t launch_xst_staged(const VocabArgs &a, cudaStream_t stream) {
  return launch_staged(xst_staged_kernel<NT, kVec>, NT, RowStage<NT, 1>::kBytes, 1536 / NT, a, stream);
}
// Whether the bf16 instance of `op` has a staged form for rows of V columns, see the kernels.
bool staged(int op, int V) {
  constexpr int kMost = 8 * RowStage<kSdStagedThreads, 3>::kChunks * kSdStagedThreads;  // 36864 columns
  return V <= kMost && (op == 1 || (op == 4 && V > kMost / 2));
}
template <bool kVec>
cudaError_t run_staged(int op, const VocabArgs &a, cudaStream_t stream) {
  if (op == 4) return launch_staged(sd_fwd_staged_kernel<kVec>, kSdStagedThreads, RowStage<kSdStagedThreads, 3>::kBytes, 1, a, stream);
  const int threads = (a.V + 47) / 48;  // that six chunks each would take
  return threads <= 128   ? launch_xst_staged<128, kVec>(a, stream)
         : threads <= 256 ? launch_xst_staged<256, kVec>(a, stream)
         : threads <= 512 ? launch_xst_staged<512, kVec>(a, stream) : launch_xst_staged<768, kVec>(a, stream);
}

bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

// op: 0 interp, 1 xst, 2 ce forward, 3 ce backward, 4 sd forward, 5 sd backward
cudaError_t vocab_loss(int op, const void *l, const void *tl, const void *lt, int64_t ld, const float *x0, int64_t ldx,
                       const int64_t *ids, const float *s, const float *t, float *lse, float *stats, float *loss, const float *g,
                       void *out, void *out2, int64_t ldo, float eps, int batch, int rows_per_sample, int V, int dtype,
                       cudaStream_t stream) {
  const int64_t rows = (int64_t)batch * rows_per_sample;
  if (rows == 0) return cudaSuccess;
  if (rows > 0x7fffffffLL) return cudaErrorInvalidValue;
  const int64_t Vp = (V + 7) & ~7;
  // 16-byte accesses: every 16-bit / fp32 operand row must start on a 16-byte boundary and cover the padded width
  for (const void *p : {l, tl, lt})
    if (p && (!aligned16(p) || ld % 8 || ld < Vp)) return cudaErrorInvalidValue;
  for (const void *p : {(const void *)out, (const void *)out2})
    if (p && (!aligned16(p) || ldo % 8 || ldo < Vp)) return cudaErrorInvalidValue;
  if (stats && !aligned16(stats)) return cudaErrorInvalidValue;
  const bool vec = x0 && aligned16(x0) && ldx % 4 == 0 && ldx >= Vp;
  VocabArgs a{l, tl, lt, ld, x0, ldx, ids, s, t, lse, stats, loss, g, out, out2, ldo, eps, rows_per_sample, V, rows};
  LaunchScope scope(kIdDual, stream);
  auto launch = [&](auto tag) -> cudaError_t {
    using T = decltype(tag);
    const dim3 grid((unsigned)rows), block(kThreads);
    if (std::is_same<T, __nv_bfloat16>::value && staged(op, V)) return vec ? run_staged<true>(op, a, stream) : run_staged<false>(op, a, stream);
    switch (op) {
      case 0: vec ? interp_kernel<T, true><<<grid, block, 0, stream>>>(a) : interp_kernel<T, false><<<grid, block, 0, stream>>>(a); break;
      case 1: vec ? xst_kernel<T, true><<<grid, block, 0, stream>>>(a) : xst_kernel<T, false><<<grid, block, 0, stream>>>(a); break;
      case 2: ce_fwd_kernel<T><<<grid, block, 0, stream>>>(a); break;
      case 3: ce_bwd_kernel<T><<<grid, block, 0, stream>>>(a); break;
      case 4: vec ? sd_fwd_kernel<T, true><<<grid, block, 0, stream>>>(a) : sd_fwd_kernel<T, false><<<grid, block, 0, stream>>>(a); break;
      case 5: vec ? sd_bwd_kernel<T, true><<<grid, block, 0, stream>>>(a) : sd_bwd_kernel<T, false><<<grid, block, 0, stream>>>(a); break;
      default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
  };
  if (dtype == JVPATTN_BF16) return launch(__nv_bfloat16{});
  if (dtype == JVPATTN_FP32) return launch(float{});
  return cudaErrorInvalidValue;
}

}  // namespace jvpattn
