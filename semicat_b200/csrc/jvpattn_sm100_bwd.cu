// Attention-JVP backward for sm_100a: the VJPs of cotangents gO (on O) and G (on Od) with respect to
// q, k, v and their tangents, from the saved row statistics (lse, mu).  tcgen05 MMAs with TMEM
// accumulators, TMA-staged tiles, warp-specialised load / MMA / softmax-algebra roles.
//
// Maths (closed form of what semicat/jvp_utils/flash_jvp_backward.py:87-2290 and
// semicat/jvp_utils/flash_attn_triton.py:406-685 compute), per (batch, head):
//   P  = exp(scale QK^T - lse)            N = scale (Qd K^T + Q Kd^T) - mu
//   A  = G V^T                            C = G Vd^T + gO V^T
//   delta = rowsum(G o O)                 dsum = rowsum(G o Od) + rowsum(gO o O)
//   W1 = scale P o (A - delta)            W2 = scale P o ((A - delta) o N + C - dsum)
//   dQd = W1 K      dQ = W1 Kd + W2 K     dKd = W1^T Q     dK = W1^T Qd + W2^T Q
//   dVd = P^T G     dV = (P o N)^T G + P^T gO
// The reference gets delta / dsum from an extra L^2 pass (flash_jvp_backward.py:2012-2290); here they are
// d-length row dot products computed by a small bandwidth-bound kernel into the caller's workspace.
//
// One kernel template serves both sides.  A CTA owns 128 rows of the "resident" side X and streams tiles of
// the other side Y:
//   query owner   X = (Q, Qd, G, gO)   Y = (K, Kd, V, Vd)     -> dQ, dQd
//   key owner     X = (K, Kd, V, Vd)   Y = (Q, Qd, G, gO)     -> dK, dKd, dV, dVd
// For either owner the score tiles are S = X0 Y0^T, Sd = X1 Y0^T + X0 Y1^T, A = X2 Y2^T, C = X2 Y3^T + X3 Y2^T
// (for the key owner these are the transposes, rows = keys), and the outputs are
//   dX1 = W1 Y0,  dX0 = W1 Y1 + W2 Y0,  and for the key owner dVd = P Y2, dV = (P o N) Y2 + P Y3.
// The 16-bit operands P, PoN, W1, W2 are written over the fp32 score columns in TMEM and fed back to the
// tensor core as the A operand; the Y tiles are read MN-major as the B operand.
//
//   warp 0      TMA producer (X once per item, Y through rings of one to three stages, see BwdSmem)
//   warp 1      MMA issuer (query owner: the score products)
//   last warp   query owner only: second MMA issuer (the output products)
//   warps 2..   kParts threads per owned row (each on 1/kParts of the tile's columns): score algebra, operand
//               write-back over consumed score columns, epilogue
//
// kPair = true serves head dimensions between the two tile widths (see sm100_head_dim_ok): the four operands go into
// the output products as a 16-bit value plus the 16-bit rounding of what is left of it, two products per operand.
#include <algorithm>

#include "jvpattn_common.cuh"
#include "sm100_attn.cuh"
#include "sm100_ptx.cuh"

namespace jvpattn {
namespace {

using namespace ptx;

constexpr int kRows = 128;
// threads of a CTA: TMA warp, MMA warp, 4 * parts score-algebra warps, and the second MMA warp of the head_dim 64 query owner
__host__ __device__ constexpr int bwd_threads(int parts, bool two_issuers) { return 64 + 128 * parts + (two_issuers ? 32 : 0); }
// score-algebra threads per owned row: each handles at least 16 columns of a streamed tile
#ifndef JVPATTN_BWD_PARTS_WIDE
#define JVPATTN_BWD_PARTS_WIDE 2
#endif
__host__ __device__ constexpr int bwd_parts(int tile) { return tile >= 64 ? JVPATTN_BWD_PARTS_WIDE : 2; }

// head_dim 128 streams 64-row tiles as two pairs with barriers of their own, (Y0, Y1) and (Y2, Y3).  Shared memory holds the
// owned rows (128 KB with dK, 64 KB without) and three or four pairs of 32 KB, not two stages of all four tensors; but
// (Y2, Y3) of a tile are last read by its A / C products, long before (Y0, Y1) by dK / dQ, so one stage of the former
// and two of the latter keep the tensor core fed.  64-row tiles rather than two whole stages of 32-row ones, because a product
// whose A operand comes from shared memory re-reads all of A for every N: at 128 B / clk a 16-channel step of N = 64 takes
// 48 cycles for 32 cycles of arithmetic and N = 32 takes 40 for 16, while N = 128 ([S | Sd], [A | C] of a 64-row tile)
// reads as long as it multiplies.  Forward and backward of 128 heads at length 2048: 5.42 ms with 32-row tiles, 4.30 ms so.
// The query owner of head_dim 64 (with tangents) streams pairs for another reason: two whole stages fit, but (Y0, Y1) of a tile are
// released by its last products and were wanted again right after them, so every second tile waited 1400 cycles for its load.
// It has three stages of (Y0, Y1) and two of (Y2, Y3): 564 -> 507 us for 128 heads at length 2048.
__host__ __device__ constexpr bool bwd_pair_ring(int D, bool kv, bool has_t) { return D == 128 || (!kv && has_t); }
// Without tangents two of the four tensors on either side, one of the two score products per region and the tangent
// accumulators are absent.  At head_dim 64 two CTAs then share an SM, one's products beside the other's score algebra
// (192 x 12 heads of length 128: key owner 55 -> 41 us, query owner 42 -> 35 us).
__host__ __device__ constexpr bool bwd_compact(int D, bool has_t) { return D == 64 && !has_t; }
__host__ __device__ constexpr bool bwd_two_issuers(int D, bool kv, bool has_t) { return D == 64 && !kv && !bwd_compact(D, has_t); }

template <int D, int TILE, bool kKV, bool kDoK, bool kHasT>
struct BwdSmem {
  static constexpr int kBoxes = D / 64;
  static constexpr int kXBuf = D == 64 ? 2 : 1;  // owned-row tiles are double buffered where shared memory allows
  static constexpr bool kRing = bwd_pair_ring(D, kKV, kHasT);
  static constexpr int kStages = kRing && D == 64 ? 3 : 2;           // stages (kRing: of (Y0, Y1))
  static constexpr int kStages2 = kRing && D == 128 && kDoK ? 1 : 2;  // stages of (Y2, Y3)
  static constexpr bool kCompact = bwd_compact(D, kHasT);  // tensor 0 and the one of 2 and 3 that is there, in slots 0 and 1
  static constexpr int kXTensors = kDoK && !kCompact ? 4 : 2;  // the dV / dVd pass reads X0 and X1 only
  static constexpr int kPer = kRing || kCompact ? 2 : 4;       // streamed tensors of a stage
  static __host__ __device__ constexpr int slot(int t) { return kCompact ? t >> 1 : t; }
  alignas(1024) uint16_t x[kXBuf][kXTensors][kBoxes][kRows * 64];
  // Streamed tiles.  Within a stage the 64-channel box is outermost and the four tensors of a box (kRing: the two of a pair)
  // are adjacent, so that [Y0 ; Y1] and [Y2 ; Y3] are each one K-major B operand of 2 TILE rows (merged score products) at
  // any head dimension.  kRing: the stages of (Y0, Y1), then those of (Y2, Y3).
  alignas(1024) uint16_t y[(kStages + (kRing ? kStages2 : 0)) * kPer * kBoxes][TILE * 64];
  float4 stats[kKV ? 2 : 1][kKV ? TILE : 1];  // key owner only: per query column {lse*log2e, mu, delta, dsum} (double buffered)
  // Query owner: the owned rows' statistics {lse, mu, delta, dsum} as four float arrays, brought in by bulk copies
  // that complete on the same barrier as the rows.  Its compute warps then issue no global loads at all: a load in
  // flight holds a scoreboard slot that the tensor-memory reads of the score algebra also wait on, which exposed
  // the memory latency once per item even with nothing depending on the load.
  alignas(16) float xstat[kKV ? 1 : kXBuf][4][kKV ? 4 : kRows];
  uint64_t x_full[kXBuf], x_empty[kXBuf], acc_free, y_full[kStages], y_empty[kStages], y2_full[kStages], y2_empty[kStages], s1_full[2],
      s2_full, c1_done[2], c2_done[2], r2_free, done, vdone;
  uint32_t tmem_base;
};


struct BwdMaps {
  CUtensorMap x[4], y[4];
  CUtensorMap out[4];  // dX0, dX1, dV, dVd as 128-row x 64-channel store boxes (D = 64 only)
};

struct BwdKernelArgs {
  View out[4];            // dX0, dX1, dV, dVd (unused entries have ptr == nullptr)
  const float *lse, *mu;  // [B, H, stat_len]
  const float *delta, *dsum;
  unsigned int *status;
  long long wait_cycles;           // budget of every bounded wait
  int D;                           // channels of a head (the tiles may be wider)
  int B, H, Lx, Ly, Lq, stat_len;  // Lx rows on the owner side, Ly on the streamed side
  int xmask, ymask;             // which of the four X / Y tensors are loaded
  int has_o;
  float scale;
};

// rows of (G o O), (G o Od) + (gO o O): D/8 threads per row, 16-byte loads.  Bound by memory; a grid over (rows, heads,
// batch), because taking a linear row index apart with 64-bit divisions cost more instructions than everything else here
// (64 x 12 heads of 128 rows: 14.4 -> 10.5 us; 192 x 12 without tangents: 28.3 -> 19.0 us).
template <int D, typename T>
__global__ void __launch_bounds__(256) row_dots_kernel(BwdArgs a, float *delta, float *dsum) {
  constexpr int kTpr = D / 8;
  ptx::griddep_launch_dependents();  // the query-owner launch may set up while this kernel drains
  const int part = threadIdx.x % kTpr;
  const int b = blockIdx.z, h = blockIdx.y;
  const int64_t row = (int64_t)blockIdx.x * (256 / kTpr) + threadIdx.x / kTpr;
  const int i = (int)row;
  float d1 = 0.f, d2 = 0.f;
  const bool live = row < a.Lq && part * 8 < a.D;  // heads narrower than the tile: the threads past the end add zero
  if (live) {
    auto load8 = [&](const View &v, float (&f)[8]) {
      const uint4 u = *reinterpret_cast<const uint4 *>(static_cast<const T *>(v.ptr) + v.offset(b, h, i) + part * 8);
      const T *e = reinterpret_cast<const T *>(&u);
#pragma unroll
      for (int t = 0; t < 8; ++t) f[t] = Elem<T>::to_f(e[t]);
    };
    float o[8], x[8], g[8];
    load8(a.o, o);
    if (a.g_to.ptr) {
      load8(a.g_to, g);
      load8(a.to, x);
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        d1 = fmaf(g[t], o[t], d1);
        d2 = fmaf(g[t], x[t], d2);
      }
    }
    if (a.g_o.ptr) {
      load8(a.g_o, g);
#pragma unroll
      for (int t = 0; t < 8; ++t) d2 = fmaf(g[t], o[t], d2);
    }
  }
#pragma unroll
  for (int off = kTpr / 2; off > 0; off >>= 1) {
    d1 += __shfl_xor_sync(0xffffffffu, d1, off);
    d2 += __shfl_xor_sync(0xffffffffu, d2, off);
  }
  if (live && part == 0) {
    const size_t si = ((size_t)b * a.H + h) * a.stat_len + i;
    delta[si] = d1;
    dsum[si] = d2;
  }
}

template <int D, int TILE, bool kKV, bool kDoK, bool kDoV, typename T, bool kPair, bool kHasT>
__global__ void __launch_bounds__(bwd_threads(bwd_parts(TILE), bwd_two_issuers(D, kKV, kHasT)), bwd_compact(D, kHasT) ? 2 : 1) sm100_bwd_kernel(const __grid_constant__ BwdMaps maps, BwdKernelArgs a) {
  constexpr int kParts = bwd_parts(TILE);
  constexpr int kComputeThreads = 128 * kParts;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  using Smem = BwdSmem<D, TILE, kKV, kDoK, kHasT>;
  Smem &s = *reinterpret_cast<Smem *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if constexpr (D == 128 && kDoK) {  // no room was left to round up: the base must have been aligned
    if (reinterpret_cast<uintptr_t>(smem_raw) % 1024 != 0) {
      if (threadIdx.x == 0) atomicCAS(a.status, 0u, 220u);
      return;
    }
  }
  constexpr int kBoxes = D / 64;
  constexpr int kStages = Smem::kStages;
  constexpr bool kRing = Smem::kRing;
  constexpr int kStages2 = Smem::kStages2;
  constexpr int kPairs = kHasT ? 2 : 1;  // a gradient and its tangent's
  constexpr int kAcc = (kDoK ? kPairs : 0) + (kDoV ? kPairs : 0);
  // accumulators; the tangent-gradient tile sits below its partner so that one N = 2D instruction can update both
  constexpr uint32_t kColKd = 0, kColK = kHasT ? D : 0;                                   // dX1, dX0
  constexpr uint32_t kColVd = kDoK ? kPairs * D : 0, kColV = kColVd + (kHasT ? D : 0);  // dVd, dV
  // two score regions that are in different phases of the pipeline: (S | Sd) and (A | C)
  constexpr uint32_t kColS = kAcc * D, kColA = kColS + kPairs * TILE, kColC = kColS + (2 * kPairs - 1) * TILE;
  // Query owner: its two accumulators leave room for a separate, double-buffered home of the W1 / W2 operands
  // (TILE / 2 packed columns each), so that the (A | C) region is free again as soon as the score algebra has read it
  // instead of when the output products have consumed the operands written over it.
  // (Not at head_dim 128: accumulators and score regions of 64 columns fill tensor memory.)
  constexpr bool kSplit = bwd_two_issuers(D, kKV, kHasT);
  // The dV / dVd pass at head_dim 128 has no (A | C): (S | Sd) takes both regions in turn, so that the tensor core forms the next
  // tile's scores while the compute warps work on this one's.
  // Scores and score algebra then run up to two tiles ahead of each other's waits, which a parity wait on one barrier would
  // mistake for none: their barriers alternate with the region.  (Tile g + 2 cannot complete either before tile g has been
  // waited for: its products are issued behind the wait for the algebra of tile g.)
  constexpr bool kAlternate = kRing && !kDoK;
  auto alt = [](int g) { return kAlternate ? g & 1 : 0; };
  auto alt_parity = [](int g) { return (kAlternate ? g >> 1 : g) & 1; };
  constexpr uint32_t kColW = kAcc * D + 2 * kPairs * TILE;
  constexpr uint32_t kWBuf = kPair ? 2 * TILE : TILE;  // columns of one buffer: W1, W2, each with its low parts where kPair
  constexpr uint32_t kUsed = kColW + (kSplit ? 2 * kWBuf : 0);
  static_assert(kUsed <= 512, "TMEM budget");
  constexpr uint32_t kTmemCols = kUsed <= 256 ? 256 : 512;
  constexpr bool kBf16 = IsBf16<T>::value;
  constexpr uint32_t kTileBytes = TILE * D * 2;
  constexpr int CH = TILE / kParts;  // score columns per compute thread and tile
  static_assert(CH % 16 == 0, "a compute thread reads its score columns 16 at a time");
  // d = 64 key owner: dV / dVd are final one group before dK / dKd (their last products are issued ahead of the last
  // tile's second half), so they are staged for the output stores while the tensor core finishes dK / dKd
  constexpr bool kEarlyV = kKV && kDoK && kDoV && kBoxes == 1;

  constexpr int kXBuf = Smem::kXBuf;
  constexpr int kWarpB = 2 + 4 * kParts;  // the second MMA issuer sits behind the score-algebra warps
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntiles = (a.Ly + TILE - 1) / TILE;
  // (compile-time: as a kernel argument it left a branch at every use in the score algebra, and those showed in its stalls:
  // 128 heads of 64 channels at length 2048: key owner 772 -> 693 us, query owner 622 -> 568 us)
  constexpr bool has_t = kHasT;
  const bool has_o = a.has_o != 0;
  // Persistent CTA: work item = 128 owned rows of one (batch, head); items blockIdx.x, + gridDim.x, ...
  // Counters shared by all roles: n = items done by this CTA, g = streamed tiles done (across items).
  const int nx = (a.Lx + kRows - 1) / kRows;
  const int items = a.B * a.H * nx;
  auto decode = [&](int it, int &bb, int &hh, int &xx0) {
    // Short sequences (a step's tensors are a few L2 sizes): the query owner walks the items from the back, the key
    // owner from the front, so that each launch starts with the (batch, head) pairs that the launch before it (the
    // forward front to back, then the query owner back to front) touched last, while their tensors are still in L2.
    // At long sequences a launch outlives the cache many times over and the order is the plain one.
    if (!kKV && ntiles <= 8) it = items - 1 - it;
    xx0 = (it % nx) * kRows;
    const int bh = it / nx;
    hh = bh % a.H;
    bb = bh / a.H;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kXBuf; ++i) {
      mbar_init(&s.x_full[i], 1);
      // MMA issuer, plus the thread whose output stores read the buffer; single row buffer of the query owner: plus
      // each compute warp once it has its rows' statistics (see there)
      mbar_init(&s.x_empty[i], kBoxes == 1 ? 2 : kKV ? 1 : 1 + kComputeThreads / 32);
    }
    mbar_init(&s.acc_free, kComputeThreads);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&s.y_full[i], 1);
      mbar_init(&s.y_empty[i], 1);
      mbar_init(&s.y2_full[i], 1);
      mbar_init(&s.y2_empty[i], 1);
    }
    mbar_init(&s.s1_full[0], 1);
    mbar_init(&s.s1_full[1], 1);
    mbar_init(&s.s2_full, 1);
    mbar_init(&s.c1_done[0], kComputeThreads);
    mbar_init(&s.c1_done[1], kComputeThreads);
    mbar_init(&s.c2_done[0], kComputeThreads);
    mbar_init(&s.c2_done[1], kComputeThreads);
    mbar_init(&s.r2_free, kComputeThreads);
    mbar_init(&s.done, 1);
    mbar_init(&s.vdone, 1);
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
  // Launch overlap (programmatic dependent launch).  The row-dot kernel is launched normally, so everything earlier
  // in the stream has completed when it runs, and it releases its dependents at once.  The query owner, launched
  // with the programmatic-serialization attribute, sets up and requests its first row tiles while the row-dot
  // kernel drains; only its producer thread reads what that kernel wrote (delta, dsum), so that thread alone
  // waits for it, and it releases the key-owner launches right after.  Those read nothing the query owner writes:
  // their CTAs move onto SMs as query-owner CTAs leave, which hides their start-up and fills the tail in which
  // only some SMs still hold a query-owner item.  A key-owner CTA can only exist after every query-owner producer
  // has passed its wait, hence after the row dots are complete.
  if (kKV) griddep_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      prefetch_tensormap(&maps.x[0]);
      prefetch_tensormap(&maps.y[0]);
      int n = 0, g = 0;
      bool ok = true;
      // owned-row tiles of work item `it_` (the n_-th of this CTA) into X buffer n_ % kXBuf
      auto load_x = [&](int it_, int n_) -> bool {
        int b, h, x0;
        decode(it_, b, h, x0);
        const int xb = n_ % kXBuf;
        if (!mbar_wait_for(a.wait_cycles, &s.x_empty[xb], ((n_ / kXBuf) & 1) ^ 1)) {
          atomicCAS(a.status, 0u, 209u);
          return false;
        }
        mbar_expect_tx(&s.x_full[xb], __popc(a.xmask) * kRows * D * 2 + (kKV ? 0 : (has_t ? 4 : 3) * kRows * 4));
        for (int t = 0; t < (kDoK ? 4 : 2); ++t)
          if (a.xmask >> t & 1)
            for (int x = 0; x < kBoxes; ++x) tma_load_4d(s.x[xb][Smem::slot(t)][x], &maps.x[t], &s.x_full[xb], 64 * x, x0, h, b);
        if (!kKV) {
          if (n_ == 0) griddep_wait();  // delta / dsum are the row-dot kernel's output
          const size_t si = ((size_t)b * a.H + h) * a.stat_len + x0;  // stat_len is a multiple of 128: always in bounds
          bulk_load_1d(s.xstat[xb][0], a.lse + si, kRows * 4, &s.x_full[xb]);
          if (has_t) bulk_load_1d(s.xstat[xb][1], a.mu + si, kRows * 4, &s.x_full[xb]);
          bulk_load_1d(s.xstat[xb][2], a.delta + si, kRows * 4, &s.x_full[xb]);
          bulk_load_1d(s.xstat[xb][3], a.dsum + si, kRows * 4, &s.x_full[xb]);
          if (n_ == 0) griddep_launch_dependents();
        }
        if (kXBuf == 1 && it_ + (int)gridDim.x < items) {  // single X buffer: at least bring the next item's rows into L2
          decode(it_ + gridDim.x, b, h, x0);
          for (int t = 0; t < 4; ++t)
            if (a.xmask >> t & 1)
              for (int x = 0; x < kBoxes; ++x) tma_prefetch_4d(&maps.x[t], 64 * x, x0, h, b);
        }
        return true;
      };
      // A streamed tile can only be requested once its stage is free, one tile ahead at best, which is less
      // than the DRAM latency when an item has few tiles: the tile `kAhead` positions further down this CTA's
      // stream is therefore pulled into L2 when a tile is requested.
      constexpr int kAhead = 2;
      auto prefetch_y = [&](int n_, int j_) {
        const int pos = j_ + kAhead;
        const int it_ = blockIdx.x + (n_ + pos / ntiles) * (int)gridDim.x;
        if (it_ >= items) return;
        int b, h, x0;
        decode(it_, b, h, x0);
        for (int t = 0; t < 4; ++t)
          if (a.ymask >> t & 1)
            for (int x = 0; x < kBoxes; ++x) tma_prefetch_4d(&maps.y[t], 64 * x, (pos % ntiles) * TILE, h, b);
      };
      // With two X buffers the next item's rows are requested as soon as this item's first two streamed tiles
      // are on their way, so they are resident long before the item starts.
      const int jx = kXBuf == 2 ? (ntiles < 2 ? ntiles - 1 : 1) : -1;
      if (blockIdx.x < items) ok = load_x(blockIdx.x, 0);
      for (int it = blockIdx.x; ok && it < items; it += gridDim.x, ++n) {
        int b, h, x0;
        decode(it, b, h, x0);
        if (kXBuf == 1 && n > 0 && !(ok = load_x(it, n))) break;
        for (int j = 0; j < ntiles; ++j, ++g) {
          const int st = g % kStages;
          if (!mbar_wait_for(a.wait_cycles, &s.y_empty[st], ((g / kStages) & 1) ^ 1)) {
            atomicCAS(a.status, 0u, 201u);
            ok = false;
            break;
          }
          constexpr int kOne = kRing ? 2 : 4;  // tensors that complete on one barrier
          mbar_expect_tx(&s.y_full[st], __popc(a.ymask & ((1 << kOne) - 1)) * kTileBytes);
          for (int t = 0; t < kOne; ++t)
            if (a.ymask >> t & 1)
              for (int x = 0; x < kBoxes; ++x)
                tma_load_4d(s.y[(st * kBoxes + x) * Smem::kPer + Smem::slot(t)], &maps.y[t], &s.y_full[st], 64 * x, j * TILE, h, b);
          if constexpr (kRing) {
            const int st2 = g % kStages2;
            if (!mbar_wait_for(a.wait_cycles, &s.y2_empty[st2], ((g / kStages2) & 1) ^ 1)) {
              atomicCAS(a.status, 0u, 217u);
              ok = false;
              break;
            }
            mbar_expect_tx(&s.y2_full[st2], __popc(a.ymask >> 2) * kTileBytes);
            for (int t = 2; t < 4; ++t)
              if (a.ymask >> t & 1)
                for (int x = 0; x < kBoxes; ++x)
                  tma_load_4d(s.y[((kStages + st2) * kBoxes + x) * 2 + t - 2], &maps.y[t], &s.y2_full[st2], 64 * x, j * TILE, h, b);
          }
          prefetch_y(n, j);
          if (j == jx && it + (int)gridDim.x < items && !(ok = load_x(it + gridDim.x, n + 1))) break;
        }
      }
    }
  } else if (warp == 1 || warp == kWarpB) {
    // ------------------------------------------------------------------ MMA issuer
    // Per streamed tile j the tensor core runs four groups, interleaved with the two halves of the score
    // algebra so that it always has the next group queued while the compute warps work:
    //   scores1(j): S, Sd            -> compute1(j): P, PoN (operands), keeps scale*P and N in registers
    //   scores2(j): A, C             -> compute2(j): W1, W2 (operands)
    //   outV(j):    dVd, dV += ...   needs compute1(j)         outK(j): dX1, dX0 += ...   needs compute2(j)
    // issue order: scores1(0) scores2(0) | outV(j) scores1(j+1) outK(j) scores2(j+1) | ...
    // (elect.sync, not `lane == 0`: the branch is then known to be uniform and descriptors stay in uniform registers.  128
    // heads of 64 channels at length 2048: key owner 855 -> 772 us, query owner 633 -> 622 us, forward 444 -> 387 us)
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc(kRows, TILE, kBf16, false, false);
      constexpr uint32_t idesc_o = make_idesc(kRows, D, kBf16, false, true);
      // Pairs of products that share their A operand and whose B tiles / accumulators are adjacent are issued as
      // one instruction of twice the width: fewer instructions for the single issuing thread, and N = 128
      // instructions run at the full tensor rate where N = 64 ones reach about two thirds of it.
      constexpr bool kMergeS = 2 * TILE <= 256;                   // score products: [S | Sd], [A | C]
      constexpr bool kMerge = (kBoxes == 1) && (2 * D <= 256);    // output products: [dX1 | dX0], [dVd | dV]
      constexpr uint32_t idesc_s2 = make_idesc(kRows, 2 * TILE, kBf16, false, false);
      constexpr uint32_t idesc_o2 = make_idesc(kRows, 2 * D, kBf16, false, true);
      // the X2 Y3^T term of C carries G Vd^T for the query owner but V gO^T for the key owner, and vice versa
      const bool term23 = kKV ? has_o : has_t;
      const bool term32 = kKV ? has_t : has_o;
      // Low descriptor words: one runtime base (shared memory offset >> 4) plus compile-time tile offsets, so
      // that issuing an MMA costs a handful of instructions (the issue rate of this one thread bounds the kernel).
      const uint32_t base16 = smem_u32(&s) >> 4;
      constexpr uint32_t kXTile = kRows * 128, kYTile = TILE * 128;  // bytes of one 64-channel box
      constexpr int kPer = Smem::kPer;  // adjacent tensors of a box
      auto xbase = [&](int xb) { return base16 + (uint32_t)((offsetof(Smem, x) + (size_t)xb * Smem::kXTensors * kBoxes * kXTile) >> 4); };
      auto ybase = [&](int st) { return base16 + (uint32_t)((offsetof(Smem, y) + (size_t)st * kPer * kBoxes * kYTile) >> 4); };
      // base for tensors 2 and 3 of tile g (their place follows from their index as in a stage of four)
      auto ybase2 = [&](int g) { return kRing ? ybase(kStages + g % kStages2) - (2 * kYTile >> 4) : ybase(g % kStages); };
      auto xd = [&](uint32_t xlo, int t, int kk) {
        return xlo + (uint32_t)(((Smem::slot(t) * kBoxes + (kk >> 2)) * kXTile + (kk & 3) * 32) >> 4) + kDescLoKMajor;
      };
      auto yd = [&](uint32_t ylo, int t, int kk) {
        return ylo + (uint32_t)((((kk >> 2) * kPer + Smem::slot(t)) * kYTile + (kk & 3) * 32) >> 4) + kDescLoKMajor;
      };
      // one accumulator at a time, 16 channels per instruction.  g = tile counter (stage / parity), xb = X buffer,
      // last = this is the item's last tile (its X tiles are released once no later score MMA needs them)
      auto scores1 = [&](int g, int xb, bool last) -> bool {
        const int st = g % kStages;
        if (!mbar_wait_for(a.wait_cycles, &s.y_full[st], (g / kStages) & 1)) return false;
        tc_fence_after();
        const uint32_t xlo = xbase(xb), ylo = ybase(st);
        const uint32_t sc = kColS + (kAlternate ? (uint32_t)(g & 1) * kPairs * TILE : 0);
        if (kMergeS && has_t) {
          // [S | Sd] = X0 [Y0 ; Y1]^T in one N = 2 TILE instruction per step, then Sd += X1 Y0^T
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_ss_lo(tmem + sc, xd(xlo, 0, kk), yd(ylo, 0, kk), idesc_s2, kk > 0);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_ss_lo(tmem + sc + TILE, xd(xlo, 1, kk), yd(ylo, 0, kk), idesc_s, true);
        } else {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_ss_lo(tmem + sc, xd(xlo, 0, kk), yd(ylo, 0, kk), idesc_s, kk > 0);
          if (has_t) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              mma_ss_lo(tmem + sc + TILE, xd(xlo, 1, kk), yd(ylo, 0, kk), idesc_s, kk > 0);
              mma_ss_lo(tmem + sc + TILE, xd(xlo, 0, kk), yd(ylo, 1, kk), idesc_s, true);
            }
          }
        }
        tc_commit(&s.s1_full[alt(g)]);
        if (kRing && !kDoK) tc_commit(&s.y_empty[st]);  // the dV / dVd products read (Y2, Y3) only
        if (!kDoK && last) tc_commit(&s.x_empty[xb]);
        return true;
      };
      auto scores2 = [&](int g, int xb, bool last) -> bool {
        if (!kDoK) return true;
        if constexpr (kRing) {
          if (!mbar_wait_for(a.wait_cycles, &s.y2_full[g % kStages2], (g / kStages2) & 1)) return false;
          tc_fence_after();
        }
        // (not kRing: already resident, scores1 waited for the whole stage)
        const uint32_t xlo = xbase(xb), ylo = ybase2(g);
        bool c_started = false;
        if (kMergeS && has_t && term23) {
          // [A | C] = X2 [Y2 ; Y3]^T in one N = 2 TILE instruction per step
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_ss_lo(tmem + kColA, xd(xlo, 2, kk), yd(ylo, 2, kk), idesc_s2, kk > 0);
          c_started = true;
        } else if (has_t) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_ss_lo(tmem + kColA, xd(xlo, 2, kk), yd(ylo, 2, kk), idesc_s, kk > 0);
        }
        if (term23 && !c_started) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            mma_ss_lo(tmem + kColC, xd(xlo, 2, kk), yd(ylo, 3, kk), idesc_s, c_started || kk > 0);
          c_started = true;
        }
        if (term32) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            mma_ss_lo(tmem + kColC, xd(xlo, 3, kk), yd(ylo, 2, kk), idesc_s, c_started || kk > 0);
        }
        tc_commit(&s.s2_full);
        if (kRing) tc_commit(&s.y2_empty[g % kStages2]);
        if (last) tc_commit(&s.x_empty[xb]);
        return true;
      };
      // Y tiles as MN-major B operands of the output products: consecutive 64-channel blocks are the two boxes of
      // one tensor (d = 128: kPer tiles apart) or, for the merged d = 64 products, two adjacent tensors
      constexpr uint32_t lbo = (kBoxes == 1 ? 1 : kPer) * TILE * 128;
      auto yb = [&](uint32_t ylo, int t, int kk) {
        return ylo + (uint32_t)((Smem::slot(t) * kYTile + kk * 2048) >> 4) + desc_lo_mn_major(lbo);
      };
      // the thread that owned score columns [16 kk, 16 kk + 16) left its 8 packed operand columns at the start
      // of its own column range (see the score-algebra warps)
      // (kPair: every 16 score columns became 8 packed columns of high parts and 8 of low parts, in place)
      auto oa = [&](int kk) -> uint32_t { return kPair ? 16 * kk : ((16 * kk) / CH) * CH + ((16 * kk) % CH) / 2; };
      if constexpr (kSplit) {
        // ---- query owner: two issuers and a chain-free schedule.
        // Measured per 64-key tile with one issuer: the score algebra needed ~1570 cycles, the tensor pipe ~1280, but a
        // tile took ~3280, because (A | C) of the next tile could only be issued behind the output products of this
        // one (which read W1 / W2 from that region), and those wait for the second half of the score algebra: a serial
        // chain of algebra -> 8 MMAs -> 8 MMAs -> algebra, with every tcgen05.commit on the way holding back its
        // thread's later MMAs until the earlier ones have drained.  Here W1 / W2 have a home of their own, so
        //   issuer A (warp 1):    scores1(j+1) once compute1(j) has read (S | Sd); scores2(j+1) once compute2(j) has
        //                         read (A | C) - neither waits for an output product;
        //   issuer B (last warp): outK(j) once compute2(j) has written W1 / W2; its commits (stage free, item done)
        //                         drain only its own queue.
        // Hazards: W[g & 1] is rewritten by compute2(g + 2), which therefore waits for outK(g) (y_empty of its stage; that barrier
        // cannot complete again before outK(g + 3), so the parity is unambiguous).
        int it = blockIdx.x, j = 0, n = 0, g = 0;
        bool ok = it < items;
        if (warp == 1) {
          if (ok && !mbar_wait_for(a.wait_cycles, &s.x_full[0], 0)) {
            atomicCAS(a.status, 0u, 202u);
            ok = false;
          }
          if (ok) {
            if (!scores1(0, 0, false)) {
              atomicCAS(a.status, 0u, 203u);
              ok = false;
            } else {
              scores2(0, 0, ntiles == 1);
            }
          }
          while (ok) {
            int it2 = it, j2 = j + 1, n2 = n;
            if (j2 == ntiles) {
              it2 = it + gridDim.x;
              j2 = 0;
              n2 = n + 1;
            }
            if (it2 >= items) break;
            if (!mbar_wait_for(a.wait_cycles, &s.c1_done[alt(g)], alt_parity(g))) {  // (S | Sd) of tile g has been read
              atomicCAS(a.status, 0u, 204u);
              break;
            }
            if (j2 == 0 && !mbar_wait_for(a.wait_cycles, &s.x_full[n2 % kXBuf], (n2 / kXBuf) & 1)) {
              atomicCAS(a.status, 0u, 202u);
              break;
            }
            if (!scores1(g + 1, n2 % kXBuf, false)) {
              atomicCAS(a.status, 0u, 203u);
              break;
            }
            if (!mbar_wait_for(a.wait_cycles, &s.r2_free, g & 1)) {  // (A | C) of tile g has been read
              atomicCAS(a.status, 0u, 215u);
              break;
            }
            tc_fence_after();
            scores2(g + 1, n2 % kXBuf, j2 == ntiles - 1);
            it = it2; j = j2; n = n2; ++g;
          }
        } else {
          static_assert(kMerge && kHasT, "[dX1 | dX0] are one accumulator");
          for (; ok; ) {
            const int st = g % kStages;
            // Two barriers, by tile parity.  Nothing that this thread issues gates the second half of the score algebra,
            // so the compute warps can complete two tiles (g and g + 1) while this thread is still held up behind the
            // other issuer's MMAs, and a parity wait on a single barrier would then take the incomplete phase g + 2
            // for phase g and never return.  Tile g + 2 cannot complete before outK(g) (the score algebra waits for it
            // before it overwrites W), so with one barrier per parity the wait is unambiguous.
            if (!mbar_wait_for(a.wait_cycles, &s.c2_done[g & 1], (g >> 1) & 1)) {  // W1 / W2 of tile g are in place
              atomicCAS(a.status, 0u, 216u);
              break;
            }
            if (j == 0 && !mbar_wait_for(a.wait_cycles, &s.acc_free, (n & 1) ^ 1)) {  // previous item's accumulators have been read out
              atomicCAS(a.status, 0u, 210u);
              break;
            }
            tc_fence_after();
            const uint32_t ylo_out = ybase(st);
            const uint32_t w1 = tmem + kColW + (uint32_t)(g & 1) * kWBuf, w2 = w1 + kWBuf / 2;
            if constexpr (kPair) {
              constexpr uint32_t kLow = TILE / 2;  // low parts behind the high parts
              const bool acc = j > 0;
#pragma unroll
              for (int kk = 0; kk < TILE / 16; ++kk) {
#pragma unroll
                for (uint32_t part = 0; part <= kLow; part += kLow) {
                  mma_ts_lo(tmem + kColKd, w1 + part + 8 * kk, yb(ylo_out, 0, kk), idesc_o2, acc || kk > 0 || part > 0);
                  mma_ts_lo(tmem + kColK, w2 + part + 8 * kk, yb(ylo_out, 0, kk), idesc_o, true);
                }
              }
            } else {
              const bool acc = j > 0;
#pragma unroll
              for (int kk = 0; kk < TILE / 16; ++kk) {
                mma_ts_lo(tmem + kColKd, w1 + 8 * kk, yb(ylo_out, 0, kk), idesc_o2, acc || kk > 0);  // [dX1 | dX0] += W1 [Y0 | Y1]
                mma_ts_lo(tmem + kColK, w2 + 8 * kk, yb(ylo_out, 0, kk), idesc_o, true);          // dX0 += W2 Y0
              }
            }
            tc_commit(&s.y_empty[st]);
            if (j == ntiles - 1) tc_commit(&s.done);
            if (++j == ntiles) {
              it += gridDim.x;
              j = 0;
              ++n;
            }
            ++g;
            if (it >= items) break;
          }
        }
      } else {
      // the stream of (item, tile) pairs this CTA walks; `n` counts items, `g` tiles
      int it = blockIdx.x, j = 0, n = 0, g = 0;
      bool ok = it < items;
      if (ok && !mbar_wait_for(a.wait_cycles, &s.x_full[0], 0)) {
        atomicCAS(a.status, 0u, 202u);
        ok = false;
      }
      if (ok) {
        if (!scores1(0, 0, ntiles == 1) || !scores2(0, 0, ntiles == 1)) {
          atomicCAS(a.status, 0u, 203u);
          ok = false;
        }
      }
      bool init0 = false, init1 = false, initv = false, initvd = false;  // accumulators written in this item
      while (ok) {
        const int st = g % kStages;
        // successor in the stream
        int it2 = it, j2 = j + 1, n2 = n;
        if (j2 == ntiles) {
          it2 = it + gridDim.x;
          j2 = 0;
          n2 = n + 1;
        }
        const bool has_next = it2 < items;
        if (j == 0) init0 = init1 = initv = initvd = false;
        auto next_scores1 = [&]() -> bool {
          if (j2 == 0 && !mbar_wait_for(a.wait_cycles, &s.x_full[n2 % kXBuf], (n2 / kXBuf) & 1)) {
            atomicCAS(a.status, 0u, 202u);
            return false;
          }
          if (!scores1(g + 1, n2 % kXBuf, j2 == ntiles - 1)) {
            atomicCAS(a.status, 0u, 203u);
            return false;
          }
          return true;
        };
        // kAlternate: the other region's operands were read by the products of tile g - 1, which are ahead in the queue
        if (kAlternate && has_next && !next_scores1()) break;
        if (!mbar_wait_for(a.wait_cycles, &s.c1_done[alt(g)], alt_parity(g))) {
          atomicCAS(a.status, 0u, 204u);
          break;
        }
        if (j == 0 && !mbar_wait_for(a.wait_cycles, &s.acc_free, (n & 1) ^ 1)) {  // previous item's accumulators have been read out
          atomicCAS(a.status, 0u, 210u);
          break;
        }
        if (kAlternate && !mbar_wait_for(a.wait_cycles, &s.y2_full[g % kStages2], (g / kStages2) & 1)) {
          atomicCAS(a.status, 0u, 218u);
          break;
        }
        tc_fence_after();
        const uint32_t ylo_out = ybase(st), ylo_v = ybase2(g);
        const uint32_t sp_ = tmem + kColS + (kAlternate ? (uint32_t)(g & 1) * kPairs * TILE : 0), spn_ = sp_ + TILE;
        // (the common case, both cotangents present, is issued as straight-line code: a run-time condition between
        //  two instructions of a group costs this thread tens of cycles per instruction)
        if constexpr (kPair) {
          if (kDoV) {
#pragma unroll
            for (int kk = 0; kk < TILE / 16; ++kk) {
#pragma unroll
              for (uint32_t part = 0; part <= 8; part += 8) {
                const uint32_t p = sp_ + oa(kk) + part, pn = spn_ + oa(kk) + part;
                if (kMerge && has_t && has_o) {
                  mma_ts_lo(tmem + kColVd, p, yb(ylo_v, 2, kk), idesc_o2, initvd);
                  mma_ts_lo(tmem + kColV, pn, yb(ylo_v, 2, kk), idesc_o, true);
                  initv = initvd = true;
                } else {
                  if (has_t) {
                    mma_ts_lo(tmem + kColVd, p, yb(ylo_v, 2, kk), idesc_o, initvd);
                    mma_ts_lo(tmem + kColV, pn, yb(ylo_v, 2, kk), idesc_o, initv);
                    initv = initvd = true;
                  }
                  if (has_o) {
                    mma_ts_lo(tmem + kColV, p, yb(ylo_v, 3, kk), idesc_o, initv);
                    initv = true;
                  }
                }
              }
            }
          }
        } else if (kDoV && kMerge && has_t && has_o) {
          const bool acc = j > 0;
#pragma unroll
          for (int kk = 0; kk < TILE / 16; ++kk) {
            mma_ts_lo(tmem + kColVd, sp_ + oa(kk), yb(ylo_v, 2, kk), idesc_o2, acc || kk > 0);  // [dVd | dV] += P [G | gO]
            mma_ts_lo(tmem + kColV, spn_ + oa(kk), yb(ylo_v, 2, kk), idesc_o, true);          // dV += (P o N) G
          }
          initv = initvd = true;
        } else if (kDoV) {
#pragma unroll
          for (int kk = 0; kk < TILE / 16; ++kk) {
            if (has_t) {
              mma_ts_lo(tmem + kColVd, sp_ + oa(kk), yb(ylo_v, 2, kk), idesc_o, initvd);  // dVd += P G
              mma_ts_lo(tmem + kColV, spn_ + oa(kk), yb(ylo_v, 2, kk), idesc_o, initv);   // dV  += (P o N) G
              initv = initvd = true;
            }
            if (has_o) {
              mma_ts_lo(tmem + kColV, sp_ + oa(kk), yb(ylo_v, 3, kk), idesc_o, initv);    // dV  += P gO
              initv = true;
            }
          }
        }
        if (kEarlyV && j == ntiles - 1) tc_commit(&s.vdone);  // dV / dVd of this item are final
        if (!kAlternate && has_next && !next_scores1()) break;
        if (kDoK) {
          if (!mbar_wait_for(a.wait_cycles, &s.c2_done[0], g & 1)) {
            atomicCAS(a.status, 0u, 207u);
            break;
          }
          tc_fence_after();
          if constexpr (kPair) {
#pragma unroll
            for (int kk = 0; kk < TILE / 16; ++kk) {
#pragma unroll
              for (uint32_t part = 0; part <= 8; part += 8) {
                const uint32_t w1 = tmem + kColA + oa(kk) + part, w2 = tmem + kColC + oa(kk) + part;
                if (kMerge && has_t) {
                  mma_ts_lo(tmem + kColKd, w1, yb(ylo_out, 0, kk), idesc_o2, init1);
                  init0 = init1 = true;
                } else if (has_t) {
                  mma_ts_lo(tmem + kColKd, w1, yb(ylo_out, 0, kk), idesc_o, init1);
                  mma_ts_lo(tmem + kColK, w1, yb(ylo_out, 1, kk), idesc_o, init0);
                  init0 = init1 = true;
                }
                mma_ts_lo(tmem + kColK, w2, yb(ylo_out, 0, kk), idesc_o, init0);
                init0 = true;
              }
            }
          } else if (kMerge && has_t) {
            const bool acc = j > 0;
#pragma unroll
            for (int kk = 0; kk < TILE / 16; ++kk) {
              mma_ts_lo(tmem + kColKd, tmem + kColA + oa(kk), yb(ylo_out, 0, kk), idesc_o2, acc || kk > 0);  // [dX1 | dX0] += W1 [Y0 | Y1]
              mma_ts_lo(tmem + kColK, tmem + kColC + oa(kk), yb(ylo_out, 0, kk), idesc_o, true);          // dX0 += W2 Y0
            }
            init0 = init1 = true;
          } else {
#pragma unroll
            for (int kk = 0; kk < TILE / 16; ++kk) {
              if (has_t) {
                mma_ts_lo(tmem + kColKd, tmem + kColA + oa(kk), yb(ylo_out, 0, kk), idesc_o, init1);  // dX1 += W1 Y0
                mma_ts_lo(tmem + kColK, tmem + kColA + oa(kk), yb(ylo_out, 1, kk), idesc_o, init0);   // dX0 += W1 Y1
                init0 = init1 = true;
              }
              mma_ts_lo(tmem + kColK, tmem + kColC + oa(kk), yb(ylo_out, 0, kk), idesc_o, init0);     // dX0 += W2 Y0
              init0 = true;
            }
          }
        }
        tc_commit(kAlternate ? &s.y2_empty[g % kStages2] : &s.y_empty[st]);
        if (j == ntiles - 1) tc_commit(&s.done);
        if (!has_next) break;
        if (!scores2(g + 1, n2 % kXBuf, j2 == ntiles - 1)) {
          atomicCAS(a.status, 0u, 219u);
          break;
        }
        it = it2; j = j2; n = n2; ++g;
      }
      }  // single issuer
    }
  } else {
    // ------------------------------------------------------------------ score algebra: two threads per owned row
    const int quad = warp & 3;
    const int part = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    const int col0 = part * CH;
    const int ctid = threadIdx.x - 64;  // 0..255 among the compute threads
    const uint32_t tlane = tmem + ((uint32_t)(quad * 32) << 16);
    const float sl2 = a.scale * kLog2e;
    // without dV only scale * P is needed: the scale goes into the exponent
    const float lscale = kDoV ? 0.f : __log2f(a.scale);
    const float2 sl2x2 = make_float2(sl2, sl2), scx2 = make_float2(a.scale, a.scale);
    // Score columns [c, c + 16) of this warp's 32 rows in 16 registers, and 16-bit operands back as 8 packed columns.
    // Query owner: a thread has its own row.  Key owner: two fragments of 16 rows, so that a thread meets 4 of the 16
    // columns in 4 rows.  The statistics go with the columns there, and a thread that had a row of its own read those of every
    // column from shared memory: 64 broadcast reads of 8 bytes per thread and tile, each as wide as 32 lanes on the way to
    // the registers - 35 % of the shared-memory pipe (128 heads at
    // length 2048: 907 -> 855 us without them).  Pair i of a thread is columns
    // 8 ((i >> 1) & 1) + 2 (lane % 4) and the next, in either form's order of registers.
    auto load_cols = [&](uint32_t col, uint32_t (&r)[16]) {
      if constexpr (kKV) {
        tmem_ld16_frag(col, &r[0]);
        tmem_ld16_frag(col + (16u << 16), &r[8]);
      } else {
        tmem_ld16(col, r);
      }
    };
    auto store_cols = [&](uint32_t col, const uint32_t (&r)[8]) {
      if constexpr (kKV) {
        tmem_st8_frag(col, &r[0]);
        tmem_st8_frag(col + (16u << 16), &r[4]);
      } else {
        tmem_st8(col, r);
      }
    };
    const int fcol = 2 * (lane & 3);
    // per-column statistics of the key owner: the first TILE compute threads fetch one query column each,
    // one tile ahead (also across items), and publish it through shared memory
    // (bh: the item's (batch, head) row of the statistics.  Taking the item apart at every tile kept all warps in front of the barrier
    // below: 4 x 16 heads of length 2048 at head_dim 64 573.9k -> 567.5k cycles.)
    auto fetch_stat = [&](int bh, int j_) -> float4 {
      const int col = j_ * TILE + ctid;
      if (ctid >= TILE || col >= a.Lq) return make_float4(INFINITY, 0.f, 0.f, 0.f);  // padded query: P = 0
      const size_t si = (size_t)bh * a.stat_len + col;
      // raw values: nothing may depend on these loads until they are published a tile later (a dependent
      // instruction here would stall the warp, and with it the barrier below, for the full memory latency)
      return make_float4(a.lse[si], has_t ? a.mu[si] : 0.f, a.delta[si], a.dsum[si]);
    };
    float4 pre = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kKV && blockIdx.x < items) pre = fetch_stat(blockIdx.x / nx, 0);
    bool ok = true;
    int n = 0, g = 0;
    int pending_xb = -1;  // compute thread 0: X buffer whose output stores have been issued but not yet released
   for (int it = blockIdx.x; it < items; it += gridDim.x, ++n) {
    int b, h, x0;
    decode(it, b, h, x0);
    // query owner: this thread's row statistics {lse * log2e, mu, delta, dsum}, delivered with the item's rows
    float4 rstat = make_float4(INFINITY, 0.f, 0.f, 0.f);  // row past the end: P = 0
    if (!kKV) {
      const int xb_ = n % kXBuf;
      if (ok && !__all_sync(0xffffffffu, mbar_wait_for(a.wait_cycles, &s.x_full[xb_], (n / kXBuf) & 1))) {
        atomicCAS(a.status, 0u, 211u);
        ok = false;
      }
      if (ok && x0 + row < a.Lx)
        rstat = make_float4(s.xstat[xb_][0][row] * kLog2e - lscale, has_t ? s.xstat[xb_][1][row] : 0.f, s.xstat[xb_][2][row],
                            s.xstat[xb_][3][row]);
      if (kXBuf == 1) {
        // The issuer's release does not cover these reads: with one streamed tile per item its last score products are
        // queued while these warps are still in the epilogue of the item before, and the rows of the item after next
        // could land here first.  (Two buffers: the release behind the output stores comes after every warp's reads.)
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.x_empty[xb_]);
      }
    }
    for (int j = 0; j < ntiles; ++j, ++g) {
      if (kKV) {
        if (ctid < TILE) s.stats[g & 1][ctid] = make_float4(pre.x * kLog2e - lscale, pre.y, pre.z, pre.w);
        if (j + 1 < ntiles) pre = fetch_stat(b * a.H + h, j + 1);
        else if (it + (int)gridDim.x < items) pre = fetch_stat((it + (int)gridDim.x) / nx, 0);
        asm volatile("bar.sync 1, %0;" ::"n"(kComputeThreads) : "memory");
      }
      // a warp whose wait ran out keeps walking the loops without touching TMEM so that the barrier above still matches
      if (ok && !__all_sync(0xffffffffu, mbar_wait_for(a.wait_cycles, &s.s1_full[alt(g)], alt_parity(g)))) {
        atomicCAS(a.status, 0u, 205u);
        ok = false;
      }
      if (!ok) continue;
      tc_fence_after();
      const float4 *st = s.stats[g & 1];
      const int nvalid = a.Ly - j * TILE;  // streamed rows in this tile (masking for the query owner)
      const uint32_t tS = tlane + kColS + (kAlternate ? (uint32_t)(g & 1) * kPairs * TILE : 0), tSd = tS + TILE;
      // ---- first half: P = exp2(s*scale*log2e - lse*log2e), N = scale*sd - mu
      float2 sp[CH / 2], nn[CH / 2];  // scale * P and N, carried into the second half
#pragma unroll
      for (int c = 0; c < CH; c += 16) {
        const int cs = col0 + c;  // first score column of this chunk
        uint32_t rs[16], rd[16];
        load_cols(tS + cs, rs);
        if (has_t) load_cols(tSd + cs, rd);
        tc_wait_ld();
        if (!kDoV && c + 16 >= CH) {
          // nothing is written back over the scores: the region is free once this thread's last read has landed
          tc_fence_before();
          mbar_arrive(&s.c1_done[alt(g)]);
        }
        if (!kKV && nvalid < TILE) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (cs + i >= nvalid) rs[i] = __float_as_uint(-INFINITY);  // key past the end: P = 0
        }
        uint32_t kp[8], kpn[8];
        uint32_t kpl[kPair ? 8 : 1], kpnl[kPair ? 8 : 1];  // low parts
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int sc = cs + 8 * ((i >> 1) & 1) + fcol;  // key owner: this pair's first column
          const float4 s0 = kKV ? st[sc] : rstat, s1 = kKV ? st[sc + 1] : rstat;
          const float2 t = __ffma2_rn(make_float2(__uint_as_float(rs[2 * i]), __uint_as_float(rs[2 * i + 1])), sl2x2,
                                      make_float2(-s0.x, -s1.x));
          const float2 p = make_float2(fast_exp2(t.x), fast_exp2(t.y));
          float2 n = make_float2(0.f, 0.f);
          if (has_t)
            n = __ffma2_rn(make_float2(__uint_as_float(rd[2 * i]), __uint_as_float(rd[2 * i + 1])), scx2,
                           make_float2(-s0.y, -s1.y));
          sp[c / 2 + i] = kDoV ? __fmul2_rn(p, scx2) : p;
          nn[c / 2 + i] = n;
          if (kDoV) {
            kp[i] = pack2<T>(p.x, p.y);
            if constexpr (kPair) kpl[i] = pack2_rest<T, true>(p.x, p.y, kp[i]);
            if (has_t) {
              const float2 pn = __fmul2_rn(p, n);
              kpn[i] = pack2<T>(pn.x, pn.y);
              if constexpr (kPair) kpnl[i] = pack2_rest<T>(pn.x, pn.y, kpn[i]);
            }
          }
        }
        if (kDoV) {
          // 16 score columns become 8 packed operand columns, written at the start of this thread's own
          // column range, over columns it has already consumed
          if constexpr (kPair) {
            store_cols(tS + cs, kp);
            store_cols(tS + cs + 8, kpl);
            if (has_t) {
              store_cols(tSd + cs, kpn);
              store_cols(tSd + cs + 8, kpnl);
            }
          } else {
            store_cols(tS + col0 + c / 2, kp);
            if (has_t) store_cols(tSd + col0 + c / 2, kpn);
          }
        }
      }
      if (kDoV) {
        tc_wait_st();
        tc_fence_before();
        mbar_arrive(&s.c1_done[alt(g)]);  // S / Sd consumed (the region may be refilled) and P / PoN in place
      }
      if (pending_xb >= 0) {
        // the previous item's output stores have long finished reading its X buffer: hand it back to the producer
        tma_store_wait_read();
        mbar_arrive(&s.x_empty[pending_xb]);
        pending_xb = -1;
      }
      if (!kDoK) continue;
      // ---- second half: W1 = scale P (A - delta), W2 = scale P ((A - delta) N + C - dsum)
      if (!__all_sync(0xffffffffu, mbar_wait_for(a.wait_cycles, &s.s2_full, g & 1))) {
        atomicCAS(a.status, 0u, 208u);
        ok = false;
        continue;
      }
      // W1 / W2 of tile g go where those of tile g - 2 were: its output products must have read them
      if (kSplit && g >= 2 &&
          !__all_sync(0xffffffffu, mbar_wait_for(a.wait_cycles, &s.y_empty[(g - 2) % kStages], ((g - 2) / kStages) & 1))) {
        atomicCAS(a.status, 0u, 221u);
        ok = false;
        continue;
      }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < CH; c += 16) {
        const int cs = col0 + c;
        uint32_t ra[16], rc[16];
        if (has_t) load_cols(tlane + kColA + cs, ra);
        load_cols(tlane + kColC + cs, rc);
        tc_wait_ld();
        if (kSplit && c + 16 >= CH) {
          tc_fence_before();
          mbar_arrive(&s.r2_free);  // (A | C) read: the next tile's products may overwrite the region
        }
        uint32_t kw1[8], kw2[8];
        uint32_t kw1l[kPair ? 8 : 1], kw2l[kPair ? 8 : 1];  // low parts
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int sc = cs + 8 * ((i >> 1) & 1) + fcol;  // key owner: this pair's first column
          const float4 s0 = kKV ? st[sc] : rstat, s1 = kKV ? st[sc + 1] : rstat;
          float2 inner = __fadd2_rn(make_float2(__uint_as_float(rc[2 * i]), __uint_as_float(rc[2 * i + 1])),
                                    make_float2(-s0.w, -s1.w));
          if (has_t) {
            const float2 da = __fadd2_rn(make_float2(__uint_as_float(ra[2 * i]), __uint_as_float(ra[2 * i + 1])),
                                         make_float2(-s0.z, -s1.z));
            const float2 w1 = __fmul2_rn(sp[c / 2 + i], da);
            kw1[i] = pack2<T>(w1.x, w1.y);
            if constexpr (kPair) kw1l[i] = pack2_rest<T>(w1.x, w1.y, kw1[i]);
            inner = __ffma2_rn(da, nn[c / 2 + i], inner);
          }
          const float2 w2 = __fmul2_rn(sp[c / 2 + i], inner);
          kw2[i] = pack2<T>(w2.x, w2.y);
          if constexpr (kPair) kw2l[i] = pack2_rest<T>(w2.x, w2.y, kw2[i]);
        }
        if (kSplit) {
          // contiguous packing in the operands' own buffer: key column k of the tile sits in packed column k / 2
          const uint32_t wbase = tlane + kColW + (uint32_t)(g & 1) * kWBuf + (col0 + c) / 2;
          if (has_t) tmem_st8(wbase, kw1);
          tmem_st8(wbase + kWBuf / 2, kw2);
          if constexpr (kPair) {
            if (has_t) tmem_st8(wbase + TILE / 2, kw1l);
            tmem_st8(wbase + kWBuf / 2 + TILE / 2, kw2l);
          }
        } else if constexpr (kPair) {
          if (has_t) {
            store_cols(tlane + kColA + cs, kw1);
            store_cols(tlane + kColA + cs + 8, kw1l);
          }
          store_cols(tlane + kColC + cs, kw2);
          store_cols(tlane + kColC + cs + 8, kw2l);
        } else {
          if (has_t) store_cols(tlane + kColA + col0 + c / 2, kw1);
          store_cols(tlane + kColC + col0 + c / 2, kw2);
        }
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&s.c2_done[kSplit ? (g & 1) : 0]);
    }
    // ---- epilogue of the item: accumulators -> 16-bit outputs, each thread 1/kParts of the channels of its row
    {
      const int xr = x0 + row;
      const bool live = xr < a.Lx;
      constexpr int kChan = D / kParts;  // channels per thread
      const int cbase = part * kChan;
      auto store_acc = [&](uint32_t col, const View &v) {
        static_assert(kBoxes == 1 || kChan % 32 == 0, "per-lane stores move 32 channels at a time");
        T *dst = static_cast<T *>(v.ptr) + v.offset(b, h, live ? xr : 0) + cbase;
#pragma unroll
        for (int c = 0; c < kChan; c += 32) {
          uint32_t r[32], pk[16];
          tmem_ld32(tlane + col + cbase + c, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = pack2<T>(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          if (live) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (!kPair || cbase + c + 8 * i < a.D)  // heads narrower than the tile
                reinterpret_cast<uint4 *>(dst + c)[i] = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
          }
        }
      };
      // D = 64: accumulators -> registers -> swizzled shared tiles -> one TMA store per tensor (coalesced, and rows
      // past the end are clipped by the hardware); per-lane 16-byte global stores are far slower.  The item's own
      // X tiles are dead by now (every MMA of the item has retired), so they serve as the staging tiles; the buffer
      // goes back to the producer only after the stores have read it (see `pending_xb`).  The barrier is executed
      // by every compute thread, whether or not its waits succeeded.
      const int xb = n % kXBuf;
      auto stage_acc = [&](uint32_t col, int which) {
        static_assert(kBoxes != 1 || kChan == 16 || kChan == 32, "staging moves 16 or 32 channels per thread");
        uint32_t r[kChan];
        if constexpr (kChan == 32) {
          tmem_ld32(tlane + col + cbase, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
        } else {
          tmem_ld16(tlane + col + cbase, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
        }
        tc_wait_ld();
        unsigned char *tile = reinterpret_cast<unsigned char *>(s.x[xb][Smem::slot(which)][0]);
#pragma unroll
        for (int i = 0; i < kChan / 8; ++i) {
          uint4 v;
          v.x = pack2<T>(__uint_as_float(r[8 * i + 0]), __uint_as_float(r[8 * i + 1]));
          v.y = pack2<T>(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
          v.z = pack2<T>(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]));
          v.w = pack2<T>(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
          *reinterpret_cast<uint4 *>(tile + swizzle128_offset(row, part * (kChan / 8) + i)) = v;
        }
      };
      if (kEarlyV) {
        if (ok && !__all_sync(0xffffffffu, mbar_wait_for(a.wait_cycles, &s.vdone, n & 1))) {
          atomicCAS(a.status, 0u, 214u);
          ok = false;
        }
        tc_fence_after();
        if (ok) {
          stage_acc(kColV, 2);
          if (has_t) stage_acc(kColVd, 3);
        }
      }
      if (ok && !__all_sync(0xffffffffu, mbar_wait_for(a.wait_cycles, &s.done, n & 1))) {
        atomicCAS(a.status, 0u, 206u);
        ok = false;
      }
      tc_fence_after();
      if (kBoxes == 1) {
        const bool w0 = kDoK, w1 = kDoK && has_t, w2 = kDoV, w3 = kDoV && has_t;
        if (ok) {
          if (w0) stage_acc(kColK, 0);
          if (w1) stage_acc(kColKd, 1);
          if (w2 && !kEarlyV) stage_acc(kColV, 2);
          if (w3 && !kEarlyV) stage_acc(kColVd, 3);
          fence_proxy_async();
        }
        asm volatile("bar.sync 2, %0;" ::"n"(kComputeThreads) : "memory");
        if (ctid == 0) {
          if (ok) {
            if (w0) tma_store_4d(&maps.out[0], s.x[xb][0][0], 0, x0, h, b);
            if (w1) tma_store_4d(&maps.out[1], s.x[xb][Smem::slot(1)][0], 0, x0, h, b);
            if (w2) tma_store_4d(&maps.out[2], s.x[xb][Smem::slot(2)][0], 0, x0, h, b);
            if (w3) tma_store_4d(&maps.out[3], s.x[xb][Smem::slot(3)][0], 0, x0, h, b);
            tma_store_commit();
          }
          pending_xb = xb;
        }
      } else if (ok) {
        if (kDoK) {
          store_acc(kColK, a.out[0]);
          if (has_t) store_acc(kColKd, a.out[1]);
        }
        if (kDoV) {
          store_acc(kColV, a.out[2]);
          if (has_t) store_acc(kColVd, a.out[3]);
        }
      }
      tc_fence_before();
      mbar_arrive(&s.acc_free);  // the next item may overwrite the accumulators
    }
   }  // items
  }

  if (threadIdx.x == 64) tma_store_wait_all();  // the thread that issued the output stores (nobody waits on x_empty any more)
  // A key-owner grid may finish before the query-owner grid it was allowed to start beside.  Work that follows the
  // call in the stream is ordered after this (the last) grid only, so one thread of every key-owner CTA waits for the
  // grid before it here: the call's completion then implies the query owner's (and, at head_dim 128, the first key
  // pass's).  Every CTA of the earlier grid is resident or done by the time a CTA of this one exists, so the wait
  // cannot deadlock; it costs nothing unless this grid really is the faster one.
  if (kKV && threadIdx.x == 32) griddep_wait();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

template <int D, int TILE, bool kKV, bool kDoK, bool kDoV, typename T, bool kPair, bool kHasT>
cudaError_t launch_side(const BwdArgs &a, const float *delta, const float *dsum, cudaStream_t stream) {
  constexpr bool has_t = kHasT;
  const bool has_o = a.g_o.ptr != nullptr;
  const View qside[4] = {a.q, a.tq, a.g_to, a.g_o};
  const View kside[4] = {a.k, a.tk, a.v, a.tv};
  const View *xs = kKV ? kside : qside, *ys = kKV ? qside : kside;
  const int Lx = kKV ? a.Lk : a.Lq, Ly = kKV ? a.Lq : a.Lk;
  // which tensors each mode reads: the tangent-side ones only with a cotangent on Od, gO only when given
  const int qmask = 1 | (has_t ? 2 | 4 : 0) | (has_o ? 8 : 0);
  int kmask = 1 | (has_t ? 2 | 8 : 0) | 4;
  if (kKV && !kDoK) kmask &= 1 | 2;  // the dV / dVd pass of a split launch needs no value tiles
  BwdMaps maps;
  BwdKernelArgs ka{};
  ka.xmask = kKV ? kmask : qmask;
  ka.ymask = kKV ? qmask : kmask;
  for (int t = 0; t < 4; ++t) {
    if ((ka.xmask >> t & 1) &&
        !make_tensor_map(&maps.x[t], xs[t].ptr, a.dtype, a.B, a.H, Lx, a.D, xs[t].sb, xs[t].sh, xs[t].sl, kRows))
      return cudaErrorInvalidValue;
    if ((ka.ymask >> t & 1) &&
        !make_tensor_map(&maps.y[t], ys[t].ptr, a.dtype, a.B, a.H, Ly, a.D, ys[t].sb, ys[t].sh, ys[t].sl, TILE))
      return cudaErrorInvalidValue;
  }
  if (kKV) {
    ka.out[0] = a.dk; ka.out[1] = a.dtk; ka.out[2] = a.dv; ka.out[3] = a.dtv;
  } else {
    ka.out[0] = a.dq; ka.out[1] = a.dtq;
  }
  if (D == 64) {
    for (int t = 0; t < 4; ++t)
      if (ka.out[t].ptr &&
          !make_tensor_map(&maps.out[t], ka.out[t].ptr, a.dtype, a.B, a.H, Lx, a.D, ka.out[t].sb, ka.out[t].sh, ka.out[t].sl, kRows))
        return cudaErrorInvalidValue;
  }
  ka.lse = a.lse; ka.mu = a.mu; ka.delta = delta; ka.dsum = dsum; ka.status = a.status; ka.wait_cycles = a.wait_cycles;
  ka.D = a.D;
  ka.B = a.B; ka.H = a.H; ka.Lx = Lx; ka.Ly = Ly; ka.Lq = a.Lq; ka.stat_len = a.stat_len;
  ka.has_o = has_o; ka.scale = a.scale;
  auto kernel = sm100_bwd_kernel<D, TILE, kKV, kDoK, kDoV, T, kPair, kHasT>;
  using Smem = BwdSmem<D, TILE, kKV, kDoK, kHasT>;
  // room to round the base up to 1 KB, as far as the SM has it (the kernel checks that it fits)
  const size_t smem = std::min<size_t>(sizeof(Smem) + 1024, 227 * 1024);
  static_assert(sizeof(Smem) <= 227 * 1024, "shared memory of one SM");
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int64_t items = (int64_t)a.B * a.H * ((Lx + kRows - 1) / kRows);
  // persistent: one CTA (two where they fit) per SM walks the items
  dim3 grid((unsigned)std::min<int64_t>(items, sm_count() * (Smem::kCompact ? 2 : 1)));
  {
    LaunchScope scope(kKV ? kIdBwdKeyTc : kIdBwdQueryTc, stream);
    e = launch_overlapped(kernel, grid, dim3(bwd_threads(bwd_parts(TILE), bwd_two_issuers(D, kKV, kHasT))), smem, stream, maps, ka);
  }
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <int D, typename T, bool kPair, bool kHasT>
cudaError_t launch_bwd(const BwdArgs &a, cudaStream_t stream) {
  float *delta = static_cast<float *>(a.workspace);
  float *dsum = delta + (size_t)a.B * a.H * a.stat_len;
  {
    constexpr int kTpr = D / 8;
    const dim3 grid((unsigned)((a.Lq + 256 / kTpr - 1) / (256 / kTpr)), a.H, a.B);
    {
      LaunchScope scope(kIdRowDots, stream);
      row_dots_kernel<D, T><<<grid, 256, 0, stream>>>(a, delta, dsum);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  cudaError_t e = cudaSuccess;
  if constexpr (D == 64) {
    // (query owner with operand pairs: two accumulators, a 64-column score tile and both W buffers would take 640 columns)
    e = launch_side<D, kPair && kHasT ? 32 : 64, false, true, false, T, kPair, kHasT>(a, delta, dsum, stream);
    if (e != cudaSuccess) return e;
    return launch_side<D, 64, true, true, true, T, kPair, kHasT>(a, delta, dsum, stream);
  } else {
  // head_dim 128: four fp32 accumulators of 128 columns do not fit TMEM next to the score tiles, so the
  // key side runs as two passes (dK, dKd | dV, dVd)
  e = launch_side<D, 64, false, true, false, T, kPair, kHasT>(a, delta, dsum, stream);
  if (e != cudaSuccess) return e;
  e = launch_side<D, 64, true, true, false, T, kPair, kHasT>(a, delta, dsum, stream);
  if (e != cudaSuccess) return e;
  return launch_side<D, 64, true, false, true, T, kPair, kHasT>(a, delta, dsum, stream);
  }
}

}  // namespace

// Number of SMs of the current device (cached per device id).
int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

size_t sm100_bwd_workspace_bytes(int B, int H, int Lq, int Lk, int D, int stat_len) {
  (void)Lq; (void)Lk; (void)D;
  size_t bytes = (size_t)2 * B * H * stat_len * sizeof(float);
  return (bytes + 255) / 256 * 256;
}

bool sm100_bwd_supported(const BwdArgs &a) {
  if (!sm100_head_dim_ok(a.D, a.dtype)) return false;
  if (a.Lq < 1 || a.Lk < 1 || a.H > 65535 || a.B > 65535) return false;
  const bool has_t = a.g_to.ptr != nullptr, has_o = a.g_o.ptr != nullptr;
  auto ok_q = [&](const View &v) { return tma_view_ok(v, a.B, a.H, a.Lq, a.D); };
  auto ok_k = [&](const View &v) { return tma_view_ok(v, a.B, a.H, a.Lk, a.D); };
  if (!ok_q(a.q) || !ok_q(a.o) || !ok_q(a.dq) || !ok_k(a.k) || !ok_k(a.v) || !ok_k(a.dk) || !ok_k(a.dv)) return false;
  if (has_t && (!ok_q(a.tq) || !ok_q(a.to) || !ok_q(a.g_to) || !ok_q(a.dtq) || !ok_k(a.tk) || !ok_k(a.tv) || !ok_k(a.dtk) ||
                !ok_k(a.dtv)))
    return false;
  if (has_o && !ok_q(a.g_o)) return false;
  // the query owner's row statistics travel by 16-byte-granular bulk copies
  if (reinterpret_cast<uintptr_t>(a.lse) % 16 || reinterpret_cast<uintptr_t>(a.workspace) % 16 || a.stat_len % 4) return false;
  if (has_t && reinterpret_cast<uintptr_t>(a.mu) % 16) return false;
  return true;
}

template <bool kHasT>
cudaError_t dispatch_bwd(const BwdArgs &a, cudaStream_t stream) {
  if (!sm100_native_head_dim(a.D))
    return a.D < 64 ? launch_bwd<64, __nv_bfloat16, true, kHasT>(a, stream) : launch_bwd<128, __nv_bfloat16, true, kHasT>(a, stream);
  if (a.dtype == JVPATTN_BF16)
    return a.D == 64 ? launch_bwd<64, __nv_bfloat16, false, kHasT>(a, stream) : launch_bwd<128, __nv_bfloat16, false, kHasT>(a, stream);
  return a.D == 64 ? launch_bwd<64, __half, false, kHasT>(a, stream) : launch_bwd<128, __half, false, kHasT>(a, stream);
}

cudaError_t sm100_bwd(const BwdArgs &a, cudaStream_t stream) {
  if (sm100_bwd_short_ok(a)) return sm100_bwd_short(a, stream);
  return a.g_to.ptr ? dispatch_bwd<true>(a, stream) : dispatch_bwd<false>(a, stream);
}

}  // namespace jvpattn
