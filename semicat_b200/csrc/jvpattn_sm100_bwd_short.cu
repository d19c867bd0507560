// Attention-JVP backward for sequences that fit one tile (Lq and Lk up to 128, head_dim 64): all gradients of a (batch, head)
// pair from one CTA, which forms each score tile once.  The kernels of jvpattn_sm100_bwd.cu pass over such a pair three times
// (row dots, query owner, key owner), read its tensors two and three times and form the scores twice.
//
// Maths as there.  The whole key axis is at hand, so the row sums need no pass of their own and no O / Od:
//   delta = rowsum(P o A)          dsum = rowsum(P o (A o N + C))
// and the 16-bit operands P, PoN, W1, W2 go to shared memory, where one copy serves both contractions: K-major (rows = queries)
// for dQ, MN-major (rows = keys) for dK and dV.
//
//   warp 0      TMA loads and stores        warp 1   MMA issuer        warps 2..   score algebra, kParts threads per query row
//
// Tensor memory: S | Sd | A | C of 128 columns each (without tangents S | C); the accumulators take the place of what has been
// read: [dVd | dV] over S once P is written, [dQd | dQ] over A and [dKd | dK] over C once W1, W2 are.  So the next item's S and
// Sd are formed behind this one's last products, under the epilogue.
// Shared memory: five places for pairs of tiles and the operands: 224 KB with tangents (one CTA per SM), 112 KB without (two).
// W1 | W2 overwrite P | PoN when dV has been formed; dV, dVd are staged over V, Vd, dK, dKd over Q, Qd and dQ, dQd over W1.
// (Q, Qd) and (V, Vd) take three places in turn, (K, Kd) and (G, gO) two, such that the next item's Q, K can be requested when dV
// has been formed (its G is dead, and so is the V of the item before), its G when the last products have read K and its V when
// dK has left Q's place.
//
// Bound by memory, and where a CTA has few items by its chain of phases.  Row dots, query owner and key owner together against this
// kernel, us: 64 x 12 pairs of length 128 62.6 -> 43.9 (27 at the copy rate), of 96 55 -> 37, of 64 44 -> 29; 12 x 12 of 128
// 16.6 -> 9.1; without tangents 192 x 12 of 128 87.7 -> 49.1 (40 at the copy rate), of 64 63 -> 36, of 40 59 -> 32.
#include <algorithm>

#include "jvpattn_common.cuh"
#include "sm100_attn.cuh"
#include "sm100_ptx.cuh"

namespace jvpattn {
namespace {

using namespace ptx;

constexpr int kRows = 128;
constexpr uint32_t kTile = kRows * 128;  // bytes of a 128 x 64 tile of 16-bit elements

// Threads per query row, and score columns that a thread has in registers at a time.  Shared memory takes all of L1, so what spills
// goes to L2: with N held beside P the score algebra took twice as long as with N formed again from Sd (51.4 -> 43.9 us for
// 64 x 12 pairs of length 128).
__host__ __device__ constexpr int short_parts(bool has_t) { return has_t ? 4 : 2; }
__host__ __device__ constexpr int short_chunk(bool has_t) { return has_t ? 8 : 16; }
__host__ __device__ constexpr int short_threads(bool has_t) { return 64 + 128 * short_parts(has_t); }

template <bool kHasT>
struct ShortSmem {
  static constexpr int kT = kHasT ? 2 : 1;
  static constexpr int kParts = short_parts(kHasT);
  alignas(1024) uint16_t qv[3][kT][kRows * 64];  // item n: (Q, Qd) in place n % 3, (V, Vd), then (dV, dVd), in place (n + 2) % 3
  uint16_t kg[2][kT][kRows * 64];                // (K, Kd) in place n % 2; with tangents (G, gO), without gO, in the other
  uint16_t w[kT][2][kRows * 64];                 // P | PoN, then W1 | W2 (without: P, then W2), boxes of 64 keys; then dQ, dQd
  alignas(16) float stat[kT][kRows];             // lse, mu
  uint64_t qk_full, vg_full, s1_full, s2_full, p_done, sums_read, v_done, v_staged, w_done, k_done, k_staged, done, acc_free, o_staged, w_free;
  uint32_t tmem_base;
};

struct ShortMaps {
  CUtensorMap q[2], k[2], v[2], g[2];
  CUtensorMap dq[2], dk[2], dv[2];  // [1]: of the tangent
};

struct ShortArgs {
  const float *lse, *mu;  // [B, H, stat_len]
  unsigned int *status;
  long long wait_cycles;
  int items, H, Lq, Lk, stat_len, has_o;
  float scale;
};

// kWhole: more than 112 queries and keys, so that every 16-row step and every warp has its share: without the tests that leave the
// others out (192 x 12 pairs of length 128 without tangents 54.4 -> 49.1 us; with tangents there is no difference and no such instance).
template <typename T, bool kHasT, bool kWhole>
__global__ void __launch_bounds__(short_threads(kHasT), kHasT ? 1 : 2) sm100_bwd_short_kernel(const __grid_constant__ ShortMaps maps, ShortArgs a) {
  using Smem = ShortSmem<kHasT>;
  constexpr int kT = Smem::kT, kParts = Smem::kParts, kCompute = 128 * kParts;
  constexpr bool kBf16 = IsBf16<T>::value;
  constexpr uint32_t kColS = 0, kColSd = 128, kColA = 256, kColC = kHasT ? 384 : 128;
  constexpr uint32_t kColV = 0, kColQ = kHasT ? 256 : 128, kColK = kHasT ? 384 : 192;  // with tangents [dXd | dX]
  constexpr uint32_t kTmemCols = kHasT ? 512 : 256;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Smem &s = *reinterpret_cast<Smem *>(smem_raw);
  if (reinterpret_cast<uintptr_t>(smem_raw) % 1024 != 0) {  // two CTAs leave no room to round up
    if (threadIdx.x == 0) atomicCAS(a.status, 0u, 300u);
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool has_o = !kHasT || a.has_o != 0;

  if (threadIdx.x == 0) {
    mbar_init(&s.qk_full, 1);
    mbar_init(&s.vg_full, 2);  // V, Vd and G, gO are requested separately
    mbar_init(&s.s1_full, 1);
    mbar_init(&s.s2_full, 1);
    mbar_init(&s.p_done, kCompute);
    mbar_init(&s.sums_read, kCompute);
    mbar_init(&s.v_done, 1);
    mbar_init(&s.v_staged, kCompute);
    mbar_init(&s.w_done, kCompute);
    mbar_init(&s.k_done, 1);
    mbar_init(&s.k_staged, kCompute);
    mbar_init(&s.done, 1);
    mbar_init(&s.acc_free, kCompute);
    mbar_init(&s.o_staged, kCompute);
    mbar_init(&s.w_free, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&s.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem_base;
  // every wait of item n (the n-th of this CTA) is for phase n of its barrier
  auto wait = [&](uint64_t *bar, int n, unsigned code) -> bool {
    if (mbar_wait_for(a.wait_cycles, bar, n & 1)) return true;
    atomicCAS(a.status, 0u, code);
    return false;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    if (lane == 0) {
      const int ng = kHasT && has_o ? 2 : 1;
      auto load_qk = [&](int it, int n) {
        const int h = it % a.H, b = it / a.H;
        mbar_expect_tx(&s.qk_full, 2 * kT * kTile + kT * kRows * 4);
        for (int t = 0; t < kT; ++t) {
          tma_load_4d(s.qv[n % 3][t], &maps.q[t], &s.qk_full, 0, 0, h, b);
          tma_load_4d(s.kg[n % 2][t], &maps.k[t], &s.qk_full, 0, 0, h, b);
        }
        const size_t si = (size_t)it * a.stat_len;  // stat_len is a multiple of 128: always in bounds
        bulk_load_1d(s.stat[0], a.lse + si, kRows * 4, &s.qk_full);
        if (kHasT) bulk_load_1d(s.stat[kT - 1], a.mu + si, kRows * 4, &s.qk_full);
      };
      auto load_v = [&](int it, int n) {
        mbar_expect_tx(&s.vg_full, kT * kTile);
        for (int t = 0; t < kT; ++t) tma_load_4d(s.qv[(n + 2) % 3][t], &maps.v[t], &s.vg_full, 0, 0, it % a.H, it / a.H);
      };
      auto load_g = [&](int it, int n) {
        mbar_expect_tx(&s.vg_full, ng * kTile);
        for (int t = 0; t < ng; ++t) tma_load_4d(s.kg[(n + 1) % 2][t], &maps.g[t], &s.vg_full, 0, 0, it % a.H, it / a.H);
      };
      int it = blockIdx.x;
      load_qk(it, 0);
      load_v(it, 0);
      load_g(it, 0);
      for (int n = 0;; ++n) {
        const int h = it % a.H, b = it / a.H, next = it + gridDim.x;
        const bool more = next < a.items;
        if (!wait(&s.v_done, n, 301)) break;  // dV formed: G is dead, and S has been formed from this item's Q and K
        if (more) {
          load_qk(next, n + 1);
          const int h2 = next % a.H, b2 = next / a.H;
          for (int t = 0; t < kT; ++t) tma_prefetch_4d(&maps.v[t], 0, 0, h2, b2);
          for (int t = 0; t < ng; ++t) tma_prefetch_4d(&maps.g[t], 0, 0, h2, b2);
        }
        if (!wait(&s.v_staged, n, 302)) break;
        for (int t = 0; t < kT; ++t) tma_store_4d(&maps.dv[t], s.qv[(n + 2) % 3][t], 0, 0, h, b);
        tma_store_commit();
        if (!wait(&s.k_staged, n, 303)) break;
        for (int t = 0; t < kT; ++t) tma_store_4d(&maps.dk[t], s.qv[n % 3][t], 0, 0, h, b);
        tma_store_commit();
        if (!wait(&s.done, n, 304)) break;
        if (more) load_g(next, n + 1);
        if (!wait(&s.o_staged, n, 305)) break;
        for (int t = 0; t < kT; ++t) tma_store_4d(&maps.dq[t], s.w[0][t], 0, 0, h, b);
        tma_store_commit();
        if (!more) break;
        tma_store_wait_read_but<1>();  // dK has left
        load_v(next, n + 1);
        tma_store_wait_read();
        mbar_arrive(&s.w_free);
        it = next;
      }
      tma_store_wait_all();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t kN1 = 128 * kT;
      constexpr uint32_t idesc_s2 = make_idesc(kRows, kN1, kBf16, false, false);     // two score tiles at once
      constexpr uint32_t idesc_s = make_idesc(kRows, kRows, kBf16, false, false);
      constexpr uint32_t idesc_q2 = make_idesc(kRows, 64 * kT, kBf16, false, true);  // A rows = queries
      constexpr uint32_t idesc_q = make_idesc(kRows, 64, kBf16, false, true);
      constexpr uint32_t idesc_k2 = make_idesc(kRows, 64 * kT, kBf16, true, true);   // A rows = keys
      constexpr uint32_t idesc_k = make_idesc(kRows, 64, kBf16, true, true);
      const uint32_t base = smem_u32(&s) >> 4;
      // Operands from byte offset `member` of shared memory.  K-major: 16 channels per step (a box of 64 is a tile); MN-major: 16 rows
      // per step, 64-element column blocks a tile apart.
      auto km = [&](uint32_t member, int kk) { return base + ((member + (kk >> 2) * kTile + (kk & 3) * 32) >> 4) + kDescLoKMajor; };
      auto mn = [&](uint32_t member, int kk) { return base + ((member + kk * 2048) >> 4) + desc_lo_mn_major(kTile); };
      // steps of the contractions over queries and keys (what lies beyond is not written either)
      const int nq = kWhole ? 8 : (a.Lq + 15) / 16, nk = kWhole ? 8 : (a.Lk + 15) / 16;
      constexpr int kUnroll = kWhole ? 8 : 1;
      constexpr uint32_t kPlace = kT * kTile, ow = offsetof(Smem, w), ow2 = ow + (kT - 1) * 2 * kTile;
      for (int it = blockIdx.x, n = 0; it < a.items; it += gridDim.x, ++n) {
        const uint32_t oq = offsetof(Smem, qv) + n % 3 * kPlace, ov = offsetof(Smem, qv) + (n + 2) % 3 * kPlace;
        const uint32_t ok_ = offsetof(Smem, kg) + n % 2 * kPlace, og = offsetof(Smem, kg) + (n + 1) % 2 * kPlace;
        const uint32_t oqd = oq + kTile, ogo = og + (kT - 1) * kTile;
        if (!wait(&s.qk_full, n, 311) || (n > 0 && !wait(&s.v_staged, n - 1, 312))) break;  // dV has left its columns
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma_ss_lo(tmem + kColS, km(oq, kk), km(ok_, kk), idesc_s2, kk > 0);  // [S | Sd] = Q [K ; Kd]^T
        if (kHasT) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) mma_ss_lo(tmem + kColSd, km(oqd, kk), km(ok_, kk), idesc_s, true);  // Sd += Qd K^T
        }
        tc_commit(&s.s1_full);
        if (!wait(&s.vg_full, n, 313) || (n > 0 && !wait(&s.acc_free, n - 1, 316))) break;  // and so have dQ and dK
        tc_fence_after();
        if (kHasT) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) mma_ss_lo(tmem + kColA, km(og, kk), km(ov, kk), idesc_s2, kk > 0);  // [A | C] = G [V ; Vd]^T
        }
        if (has_o) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) mma_ss_lo(tmem + kColC, km(ogo, kk), km(ov, kk), idesc_s, kHasT || kk > 0);  // C += gO V^T
        }
        tc_commit(&s.s2_full);
        if (!wait(&s.p_done, n, 314)) break;
        tc_fence_after();
        if (!kHasT) {
#pragma unroll kUnroll
          for (int kk = 0; kk < nq; ++kk) mma_ss_lo(tmem + kColV, mn(ow, kk), mn(og, kk), idesc_k, kk > 0);  // dV = P^T gO
        } else if (has_o) {
#pragma unroll kUnroll
          for (int kk = 0; kk < nq; ++kk) {
            mma_ss_lo(tmem + kColV, mn(ow, kk), mn(og, kk), idesc_k2, kk > 0);     // [dVd | dV] = P^T [G | gO]
            mma_ss_lo(tmem + kColV + 64, mn(ow2, kk), mn(og, kk), idesc_k, true);  // dV += PoN^T G
          }
        } else {
#pragma unroll kUnroll
          for (int kk = 0; kk < nq; ++kk) {
            mma_ss_lo(tmem + kColV, mn(ow, kk), mn(og, kk), idesc_k, kk > 0);
            mma_ss_lo(tmem + kColV + 64, mn(ow2, kk), mn(og, kk), idesc_k, kk > 0);
          }
        }
        tc_commit(&s.v_done);
        if (!wait(&s.w_done, n, 315)) break;
        tc_fence_after();
#pragma unroll kUnroll
        for (int kk = 0; kk < nq; ++kk) {
          mma_ss_lo(tmem + kColK, mn(ow, kk), mn(oq, kk), idesc_k2, kk > 0);                // [dKd | dK] = W1^T [Q | Qd]
          if (kHasT) mma_ss_lo(tmem + kColK + 64, mn(ow2, kk), mn(oq, kk), idesc_k, true);  // dK += W2^T Q
        }
        tc_commit(&s.k_done);
#pragma unroll kUnroll
        for (int kk = 0; kk < nk; ++kk) {
          mma_ss_lo(tmem + kColQ, km(ow, kk), mn(ok_, kk), idesc_q2, kk > 0);                // [dQd | dQ] = W1 [K | Kd]
          if (kHasT) mma_ss_lo(tmem + kColQ + 64, km(ow2, kk), mn(ok_, kk), idesc_q, true);  // dQ += W2 K
        }
        tc_commit(&s.done);
      }
    }
  } else {
    // ------------------------------------------------------------------ score algebra
    constexpr int CH = kRows / kParts;  // key columns per thread
    const int quad = warp & 3, part = (warp - 2) >> 2, row = quad * 32 + lane, col0 = part * CH;
    const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16);
    const float sl2 = a.scale * kLog2e, inv_scale = 1.f / a.scale;
    const float2 sl2x2 = make_float2(sl2, sl2), scx2 = make_float2(a.scale, a.scale);
    unsigned char *const w0 = reinterpret_cast<unsigned char *>(s.w[0][0]), *const w1 = reinterpret_cast<unsigned char *>(s.w[kT - 1][0]);
    constexpr int kChunk = short_chunk(kHasT);
    auto load = [&](uint32_t col, uint32_t (&r)[kChunk]) {
      if constexpr (kChunk == 16) tmem_ld16(tlane + col, r);
      else tmem_ld8(tlane + col, r);
    };
    // operand columns from `col` of this row, 16 bytes at a time, in a box of 64
    auto put = [&](unsigned char *tile, int col, const uint32_t (&r)[kChunk / 2]) {
      unsigned char *box = tile + (col >> 6) * kTile;
#pragma unroll
      for (int i = 0; i < kChunk / 8; ++i)
        *reinterpret_cast<uint4 *>(box + swizzle128_offset(row, (col & 63) / 8 + i)) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
    };
    auto pair = [](const uint32_t *r, int i) { return make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])); };
    // accumulator columns [c, c + 32) of this row -> 32 channels from `ch` of a staging tile
    auto stage32 = [&](uint32_t c, unsigned char *tile, int ch) {
      uint32_t r[32];
      tmem_ld32(tlane + c, r);
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 u;
        u.x = pack2<T>(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1]));
        u.y = pack2<T>(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
        u.z = pack2<T>(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]));
        u.w = pack2<T>(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
        *reinterpret_cast<uint4 *>(tile + swizzle128_offset(row, ch / 8 + i)) = u;
      }
    };
    constexpr int kOut = 64 * kT / kParts;  // accumulator columns per thread and output pair
    static_assert(kOut % 32 == 0, "32 columns at a time");
    // columns from the last 16 that hold a key on, and warps without a query, have nothing to do (nor to write: see `steps`)
    const int ncol = kWhole ? CH : min(CH, (a.Lk + 15) / 16 * 16 - col0);
    const bool live = kWhole || quad * 32 < a.Lq, live_k = kWhole || quad * 32 < a.Lk;
    bool ok = true;
    auto wait_all = [&](uint64_t *bar, int n, unsigned code) {
      if (ok && !__all_sync(0xffffffffu, mbar_wait_for(a.wait_cycles, bar, n & 1))) {
        atomicCAS(a.status, 0u, code);
        ok = false;
      }
      tc_fence_after();
    };
    for (int it = blockIdx.x, n = 0; it < a.items; it += gridDim.x, ++n) {
      uint16_t(*const vplace)[kRows * 64] = s.qv[(n + 2) % 3];
      float2 *const sums = reinterpret_cast<float2 *>(vplace[0]);  // (V is dead when they are written, and they are when dV is)
      wait_all(&s.qk_full, n, 321);
      float lse2 = INFINITY, mu = 0.f;  // a row past the end: P = 0
      if (ok && row < a.Lq) {
        lse2 = s.stat[0][row] * kLog2e;
        if (kHasT) mu = s.stat[kT - 1][row];
      }
      if (n > 0) wait_all(&s.w_free, n - 1, 322);  // the last item's outputs have left the operands' place
      wait_all(&s.s1_full, n, 323);
      // ---- P = exp(scale S - lse), N = scale Sd - mu (formed again where it is used: Sd stays in place until dV has left)
      float2 sp[CH / 2];  // scale * P
      if (ok) {
#pragma unroll
        for (int c = 0; c < CH; c += kChunk) {
          if (!live || c >= ncol) continue;
          uint32_t rs[kChunk], rd[kChunk], kp[kChunk / 2], kpn[kChunk / 2];
          load(kColS + col0 + c, rs);
          if (kHasT) load(kColSd + col0 + c, rd);
          tc_wait_ld();
          if (a.Lk < kRows) {
#pragma unroll
            for (int i = 0; i < kChunk; ++i)
              if (col0 + c + i >= a.Lk) rs[i] = __float_as_uint(-INFINITY);  // key past the end: P = 0
          }
#pragma unroll
          for (int i = 0; i < kChunk / 2; ++i) {
            const float2 t = __ffma2_rn(pair(rs, i), sl2x2, make_float2(-lse2, -lse2));
            const float2 p = make_float2(fast_exp2(t.x), fast_exp2(t.y));
            sp[c / 2 + i] = __fmul2_rn(p, scx2);
            kp[i] = pack2<T>(p.x, p.y);
            if (kHasT) {
              const float2 pn = __fmul2_rn(p, __ffma2_rn(pair(rd, i), scx2, make_float2(-mu, -mu)));
              kpn[i] = pack2<T>(pn.x, pn.y);
            }
          }
          put(w0, col0 + c, kp);
          if (kHasT) put(w1, col0 + c, kpn);
        }
        fence_proxy_async();
        tc_fence_before();
        mbar_arrive(&s.p_done);
      }
      // ---- row sums over this thread's columns, then over the row's threads
      wait_all(&s.s2_full, n, 324);
      float2 acc1 = make_float2(0.f, 0.f), acc2 = acc1;
      if (ok) {
#pragma unroll
        for (int c = 0; c < CH; c += kChunk) {
          if (!live || c >= ncol) continue;
          uint32_t ra[kChunk], rc[kChunk], rd[kChunk];
          if (kHasT) load(kColA + col0 + c, ra), load(kColSd + col0 + c, rd);
          load(kColC + col0 + c, rc);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < kChunk / 2; ++i) {
            float2 inner = pair(rc, i);
            if (kHasT) {
              acc1 = __ffma2_rn(sp[c / 2 + i], pair(ra, i), acc1);
              inner = __ffma2_rn(pair(ra, i), __ffma2_rn(pair(rd, i), scx2, make_float2(-mu, -mu)), inner);
            }
            acc2 = __ffma2_rn(sp[c / 2 + i], inner, acc2);
          }
        }
      }
      if (ok) sums[part * kRows + row] = make_float2(acc1.x + acc1.y, acc2.x + acc2.y);
      asm volatile("bar.sync %0, %1;" ::"r"(1 + quad), "n"(32 * kParts) : "memory");
      float delta = 0.f, dsum = 0.f;
#pragma unroll
      for (int p = 0; p < kParts; ++p) {
        const float2 t = sums[p * kRows + row];
        delta += t.x;
        dsum += t.y;
      }
      delta *= inv_scale, dsum *= inv_scale;
      if (ok) mbar_arrive(&s.sums_read);
      // ---- W1 = scale P (A - delta), W2 = scale P ((A - delta) N + C - dsum), over P and PoN
      wait_all(&s.v_done, n, 325);
      if (ok) {
#pragma unroll
        for (int c = 0; c < CH; c += kChunk) {
          if (!live || c >= ncol) continue;
          uint32_t ra[kChunk], rc[kChunk], rd[kChunk], kw1[kChunk / 2], kw2[kChunk / 2];
          if (kHasT) load(kColA + col0 + c, ra), load(kColSd + col0 + c, rd);
          load(kColC + col0 + c, rc);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < kChunk / 2; ++i) {
            float2 inner = __fadd2_rn(pair(rc, i), make_float2(-dsum, -dsum));
            if (kHasT) {
              const float2 da = __fadd2_rn(pair(ra, i), make_float2(-delta, -delta));
              const float2 v1 = __fmul2_rn(sp[c / 2 + i], da);
              kw1[i] = pack2<T>(v1.x, v1.y);
              inner = __ffma2_rn(da, __ffma2_rn(pair(rd, i), scx2, make_float2(-mu, -mu)), inner);
            }
            const float2 v2 = __fmul2_rn(sp[c / 2 + i], inner);
            kw2[i] = pack2<T>(v2.x, v2.y);
          }
          if (kHasT) put(w0, col0 + c, kw1);
          put(w1, col0 + c, kw2);
        }
        fence_proxy_async();
        tc_fence_before();
        mbar_arrive(&s.w_done);
      }
      // ---- dVd, dV (columns kColV ..) -> over Vd, V, and over every thread's sums
      wait_all(&s.sums_read, n, 327);
      if (ok) {
#pragma unroll
        for (int c = 0; c < kOut; c += 32) {
          const int col = part * kOut + c, t = kHasT ? 1 - (col >> 6) : 0;  // [dVd | dV]: the tangent's first
          if (live_k) stage32(kColV + col, reinterpret_cast<unsigned char *>(vplace[t]), col & 63);
        }
        fence_proxy_async();
        tc_fence_before();
        mbar_arrive(&s.v_staged);
      }
      // ---- dKd, dK -> over Qd, Q; dQd, dQ -> over W1
      wait_all(&s.k_done, n, 328);
      if (ok) {
#pragma unroll
        for (int c = 0; c < kOut; c += 32) {
          const int col = part * kOut + c, t = kHasT ? 1 - (col >> 6) : 0;
          if (live_k) stage32(kColK + col, reinterpret_cast<unsigned char *>(s.qv[n % 3][t]), col & 63);
        }
        fence_proxy_async();
        mbar_arrive(&s.k_staged);
      }
      wait_all(&s.done, n, 326);
      if (ok) {
#pragma unroll
        for (int c = 0; c < kOut; c += 32) {
          const int col = part * kOut + c, t = kHasT ? 1 - (col >> 6) : 0;
          if (live) stage32(kColQ + col, w0 + t * kTile, col & 63);
        }
        tc_fence_before();
        mbar_arrive(&s.acc_free);
        fence_proxy_async();
        mbar_arrive(&s.o_staged);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

template <typename T, bool kHasT, bool kWhole>
cudaError_t launch_short(const BwdArgs &a, cudaStream_t stream) {
  ShortMaps maps;
  bool ok = true;
  auto map = [&](CUtensorMap *m, const View &v, int L) {
    ok = ok && make_tensor_map(m, v.ptr, a.dtype, a.B, a.H, L, a.D, v.sb, v.sh, v.sl, kRows);
  };
  const bool has_o = a.g_o.ptr != nullptr;
  map(&maps.q[0], a.q, a.Lq), map(&maps.k[0], a.k, a.Lk), map(&maps.v[0], a.v, a.Lk);
  map(&maps.dq[0], a.dq, a.Lq), map(&maps.dk[0], a.dk, a.Lk), map(&maps.dv[0], a.dv, a.Lk);
  map(&maps.g[0], kHasT ? a.g_to : a.g_o, a.Lq);
  if (kHasT) {
    map(&maps.q[1], a.tq, a.Lq), map(&maps.k[1], a.tk, a.Lk), map(&maps.v[1], a.tv, a.Lk);
    map(&maps.dq[1], a.dtq, a.Lq), map(&maps.dk[1], a.dtk, a.Lk), map(&maps.dv[1], a.dtv, a.Lk);
    if (has_o) map(&maps.g[1], a.g_o, a.Lq);
  }
  if (!ok) return cudaErrorInvalidValue;
  ShortArgs ka{a.lse, a.mu, a.status, a.wait_cycles, a.B * a.H, a.H, a.Lq, a.Lk, a.stat_len, has_o, a.scale};
  auto kernel = sm100_bwd_short_kernel<T, kHasT, kWhole>;
  constexpr size_t smem = sizeof(ShortSmem<kHasT>);
  static_assert(smem <= (228 * 1024 - (kHasT ? 1 : 2) * 1024) / (kHasT ? 1 : 2), "shared memory of one SM");
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  {
    LaunchScope scope(kIdBwdShortTc, stream);
    kernel<<<(unsigned)std::min(ka.items, sm_count() * (kHasT ? 1 : 2)), short_threads(kHasT), smem, stream>>>(maps, ka);
  }
  return cudaGetLastError();
}

}  // namespace

// The line at 16 pairs is not where the kernels cross.  In a graph this one is faster from the first pair on: 1, 8 and 15 pairs of
// length 128 8.2, 8.4, 8.4 us against 10.2, 10.4, 10.4 in three kernels, of length 32 6.3 against 8.3, without tangents 6.2 against
// 8.4.  Fewer pairs keep the kernels that split a pair because the PyTorch call around either takes 250 us.  From 16 on it is the
// faster one at every length (24 to 3072 pairs, queries x keys 1 x 1: 5.6-61 us against 8.1-120; 1 x 128 7.8-104 against 9.1-159;
// 128 x 1 7.1-87 against 9.6-181; 100 x 100 8.2-122 against 10.8-222).
bool sm100_bwd_short_ok(const BwdArgs &a) {
  return a.D == 64 && a.Lq <= kRows && a.Lk <= kRows && (int64_t)a.B * a.H >= 16 && (int64_t)a.B * a.H < (int64_t(1) << 30);
}

cudaError_t sm100_bwd_short(const BwdArgs &a, cudaStream_t stream) {
  auto launch = [&](auto elem, auto has_t) {
    using T = decltype(elem);
    constexpr bool kHasT = decltype(has_t)::value;
    if constexpr (!kHasT)
      if (a.Lq > 112 && a.Lk > 112) return launch_short<T, false, true>(a, stream);
    return launch_short<T, kHasT, false>(a, stream);
  };
  auto typed = [&](auto elem) { return a.g_to.ptr ? launch(elem, std::true_type{}) : launch(elem, std::false_type{}); };
  return a.dtype == JVPATTN_BF16 ? typed(__nv_bfloat16{}) : typed(__half{});
}

}  // namespace jvpattn
