// Backward of the attention kernel of swa.cuh (causal sliding window, or - causal = 0 - every key of the batch entry
// visible to every query) for sm_100a.  With P = softmax(q k^T * scale) restricted to the visible keys, recomputed from
// the forward's log-sum-exp L, and Delta_i = sum_d dO_i O_i:
//   dV_j = sum_i P_ij dO_i,   dS_ij = P_ij (dO_i . v_j - Delta_i) * scale,   dK_j = sum_i dS_ij q_i,   dQ_i = sum_j dS_ij k_j.
// One kernel, two modes (a CTA owns a 128-row OUTER tile and walks the 128-row INNER tiles of its band):
//   MODE 0  outer = key tile j, inner = query tiles i:  dV_j += P^T dO_i,  dK_j += dS^T Q_i   (two accumulators)
//   MODE 1  outer = query tile i, inner = key tiles j:  dQ_i += dS K_j                        (one accumulator)
// The OUTER rows are the tensor-memory lanes in both modes: per inner tile the first products are
// [128 outer x 128 inner] (mode 0: S^T = K Q^T and dP^T = V dO^T; mode 1: S = Q K^T and dP = dO V^T), four softmax
// threads per lane (32 columns each) turn them into bf16 P and dS, which go back to tensor memory, into the columns the
// thread has just read, and are the A operands of the second products from there (the shared memory that tiles of them
// would take holds a third inner stage, and the second products read half as many operand bytes).  The inner tiles
// serve as K-major B operands of the first products and as MN-major B operands (rows = k) of the second.
// Order of the products, all issued by one thread and executed in that order:
//   mode 0  ... dV(t), S(t + 1), dK(t), dP(t + 1) ...   P(t + 1) is worked out while dK(t), dP(t + 1) run, dS(t) during dV(t),
//                                                       S(t + 1); S and dP have one set of columns each
//   mode 1  ... dP(t + 1), dQ(t), S(t + 2) ...          S has two sets of columns, dP one
// The first inner operand (Q or K) is held from its first product to the second products a tile later and goes through a
// three-stage ring, the other through two stages.  Every mbarrier wait is bounded.
// Measured (2 x 32768 tokens, 12 heads of 128, window 2048; 128 x 128 pairs): keys' side 1469 us, queries' side 1059, where
// 64-row inner tiles with P and dS in shared memory took 1698 and 1288.  About 2800 and 2300 clocks a tile for 2050 and 1540 of
// products; 1030 of them are exponentials (16 a clock), which no other phase of the same tile can hide.  One tile of 64 tokens is
// where the old tiles stay ahead on the queries' side (64 x 8 heads: 21.3 / 18.5, keys' side 24.8 / 24.9).
#pragma once
#include "swa.cuh"

namespace lact {

struct SwaBwdArgs {
  CUtensorMap q, k, v, dout;           // 4-D maps (feature, token, head, batch), box {64, 128, 1, 1}
  CUtensorMap q16, k16, v16, dout16;   // the same, box {64, 16, 1, 1}
  const float* lse;            // [b][h][l]: log2-domain log-sum-exp of the forward (m + log2(l))
  const float* delta;          // [b][h][l]: sum_d dO O
  const int32_t* seq_start;    // optional [l], as in the forward
  bf16* out0;                  // MODE 0: dK, MODE 1: dQ   ([b][l][h][d], strides below)
  bf16* out1;                  // MODE 0: dV
  int64_t o_bs, o_ts, o_hs;
  int32_t L, window, heads, tiles;   // L: queries per batch entry; tiles: outer tiles per (batch, head) of this launch
  int32_t Lk, causal;                // keys per batch entry (= L when causal); causal = 0: every query sees every key
  float scale_log2, scale;
  int32_t* status;
};

// softmax warps: four per tensor-memory lane quarter, 32 columns of a tile each
constexpr int kSwaBwdWarps = 16, kSwaBwdThreads = 64 + 32 * kSwaBwdWarps + 32;  // + loads, products, per-query values

template <int HD>
struct SwaBwdSmem {
  static constexpr uint32_t kTile = 128 * HD * 2;
  static constexpr int kStagesA = 3, kStagesB = 2;
  // outer pair | first inner operand x 3 | second inner operand x 2 | 2 stages x (lse, delta) of 128 queries (mode 0) | barriers
  static constexpr uint32_t kOuter = 0, kA = 2 * kTile, kB = kA + kStagesA * kTile, kStats = kB + kStagesB * kTile,
                            kBars = kStats + 2 * 2 * 128 * 4;
  static constexpr uint32_t kBytes = kBars + 256;
};

// Packed sequences: the end of the sequence that holds `row`, at most `limit` (> row); the same answer in all lanes of a full warp.
// (seq_start never falls; 32 places are looked at together: 3 rounds for 2048 of them.)
__device__ __forceinline__ int sequence_end(const int32_t* seq_start, int row, int limit) {
  int lo = row, hi = limit;   // the end is in (lo, hi]
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) >> 5, at = lo + (static_cast<int>(threadIdx.x & 31) + 1) * step;
    const int f = __ffs(__ballot_sync(0xFFFFFFFFu, at >= hi || seq_start[at] > row)) - 1;
    hi = min(hi, lo + (f + 1) * step);
    lo += f * step;
  }
  return hi;
}

template <int HD, int MODE>
__global__ void __launch_bounds__(kSwaBwdThreads, 1) swa_bwd_kernel(const __grid_constant__ SwaBwdArgs a) {
  static_assert(HD == 64 || HD == 128, "head dimensions 64 and 128");
  using SM = SwaBwdSmem<HD>;
  constexpr int KBD = HD / 64, NA = SM::kStagesA, NB = SM::kStagesB;
  constexpr uint32_t kBox = 128 * 128;    // [128 rows][64 features] box of a tile
  constexpr uint32_t kTmemCols = 512;
  // tensor memory: S at 0 (mode 1: two sets, 0 and 128), dP at 128 (mode 1: 256), accumulators behind them
  constexpr uint32_t kDP = MODE == 0 ? 128 : 256, kAcc = kDP + 128;
  extern __shared__ __align__(1024) uint8_t swa_bwd_smem[];   // (no room for alignment slack: the array itself is aligned)
  const uint32_t base = smem_u32(swa_bwd_smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(swa_bwd_smem + SM::kBars);
  uint64_t* outer_full = bars;        // the CTA's own two tiles have landed
  uint64_t* a_full = bars + 1;        // [3] first inner operand (mode 0: Q, mode 1: K)
  uint64_t* a_empty = bars + 4;       // [3]
  uint64_t* b_full = bars + 7;        // [2] second inner operand (mode 0: dO, mode 1: V)
  uint64_t* b_empty = bars + 9;       // [2]
  uint64_t* s_full = bars + 11;       // [2] S is in tensor memory (mode 0: the first alone)
  uint64_t* dp_full = bars + 13;      // dP is in tensor memory
  uint64_t* p_full = bars + 14;       // an arrival per softmax warp, mode 0: S has been read, P written
  uint64_t* ds_full = bars + 15;      // likewise: dP (and S, mode 1) has been read, dS written
  uint64_t* acc_full = bars + 16;     // all products of this CTA done
  uint64_t* st_full = bars + 17;      // [2] mode 0: a tile's per-query values are in shared memory
  uint64_t* st_empty = bars + 19;     // [2] an arrival per softmax warp: it has read them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(outer_full, 1);
    for (int s = 0; s < NA; ++s) { mbar_init(&a_full[s], 1); mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < NB; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&st_full[s], 1); mbar_init(&st_empty[s], kSwaBwdWarps); }
    mbar_init(dp_full, 1);
    mbar_init(p_full, kSwaBwdWarps);
    mbar_init(ds_full, kSwaBwdWarps);
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);

  const int ot = blockIdx.x % a.tiles;
  const int head = (blockIdx.x / a.tiles) % a.heads;
  const int batch = blockIdx.x / (a.tiles * a.heads);
  const int o0 = ot * 128;   // first row of the outer tile (keys in mode 0, queries in mode 1)
  const int window = a.window > 0 ? a.window : a.L;
  // inner rows [i_lo, i_hi] that any row of this tile meets, in 128-row tiles from t_lo
  int i_lo = 0, i_hi = (MODE == 0 ? a.L : a.Lk) - 1;   // block attention: all
  if (a.causal && MODE == 0) {   // queries that see any key of this tile: key <= q <= key + window - 1, of the key's sequence
    const int64_t past = static_cast<int64_t>(o0) + 127 + window;
    i_lo = o0;
    if (past <= i_hi) i_hi = static_cast<int>(past) - 1;
    if (a.seq_start != nullptr) i_hi = sequence_end(a.seq_start, min(o0 + 127, a.L - 1), i_hi + 1) - 1;
  } else if (a.causal) {         // keys this query tile sees: not before the window of its first query, nor before that query's sequence
    i_lo = max(o0 - (window - 1), a.seq_start != nullptr ? a.seq_start[o0] : 0);
    if (o0 + 127 < i_hi) i_hi = o0 + 127;
  }
  const int t_lo = i_lo / 128, T = i_hi / 128 - t_lo + 1;
  // (swizzled tiles need the alignment asked for above)
  bool failed = uniform(static_cast<uint32_t>(*reinterpret_cast<volatile int32_t*>(a.status))) != kStatusOk || (base & 1023u) != 0;
  const CUtensorMap* outer_a = MODE == 0 ? &a.k : &a.q;          // outer pair: (K, V) or (Q, dO)
  const CUtensorMap* outer_b = MODE == 0 ? &a.v : &a.dout;
  const CUtensorMap* inner_a = MODE == 0 ? &a.q : &a.k;          // inner pair: (Q, dO) or (K, V)
  const CUtensorMap* inner_b = MODE == 0 ? &a.dout : &a.v;
  float* const stats = reinterpret_cast<float*>(swa_bwd_smem + SM::kStats);   // [stage][lse | delta * scale][128]
  const int64_t stat_base = (static_cast<int64_t>(batch) * a.heads + head) * a.L;

  if (warp == 0) {
    const uint32_t leader = elect_leader();
    if (!failed) {
      auto load = [&](uint32_t dst, const CUtensorMap* map, uint64_t* bar, int row) {
        for (int j = 0; j < KBD; ++j) tma_load_4d_if(leader, dst + j * kBox, map, bar, 64 * j, row, head, batch);
      };
      // Groups of 16 inner rows that no row of the outer tile meets arrive as zeros (from behind the tensor's end): their
      // probabilities are zero, but a NaN or an infinity in such a row would reach all rows of the tile, up to 127 past the band.
      const int rows = MODE == 0 ? a.L : a.Lk;
      auto load_inner = [&](uint32_t dst, const CUtensorMap* map, const CUtensorMap* map16, uint64_t* bar, int t) {
        const int row = (t_lo + t) * 128;
        if (row + 15 >= i_lo && (row + 112 <= i_hi || i_hi == rows - 1)) {
          load(dst, map, bar, row);
        } else {
#pragma unroll 1
          for (int g = 0; g < 128; g += 16) {
            const int from = row + g + 15 < i_lo || row + g > i_hi ? rows : row + g;
            for (int j = 0; j < KBD; ++j) tma_load_4d_if(leader, dst + j * kBox + g * 128, map16, bar, 64 * j, from, head, batch);
          }
        }
      };
      mbar_expect_tx_if(leader, outer_full, 2 * SM::kTile);
      load(base + SM::kOuter, outer_a, outer_full, o0);
      load(base + SM::kOuter + SM::kTile, outer_b, outer_full, o0);
      for (int t = 0; t < T && !failed; ++t) {
        const int sa = t % NA, sb = t % NB;
        if (t >= NA && !mbar_wait_warp(&a_empty[sa], (t / NA - 1) & 1, abort_flag)) { failed = true; break; }
        mbar_expect_tx_if(leader, &a_full[sa], SM::kTile);
        load_inner(base + SM::kA + sa * SM::kTile, inner_a, MODE == 0 ? &a.q16 : &a.k16, &a_full[sa], t);
        if (t >= NB && !mbar_wait_warp(&b_empty[sb], (t / NB - 1) & 1, abort_flag)) { failed = true; break; }
        mbar_expect_tx_if(leader, &b_full[sb], SM::kTile);
        load_inner(base + SM::kB + sb * SM::kTile, inner_b, MODE == 0 ? &a.dout16 : &a.v16, &b_full[sb], t);
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_leader();
    if (!failed) {
      const uint32_t idesc_first = make_idesc_bf16(128, 128, 0, 0);  // [outer x inner], both operands K-major (features)
      const uint32_t idesc_acc = make_idesc_bf16(128, HD, 0, 1);     // [outer x HD]: A = P / dS, B = inner tile MN-major
      const SmemDescBase desc(kBox);   // MN-major: 64-feature atoms a box apart (K-major descriptors ignore it)
      // 128 x 128 product of two K-major tiles into columns `col`
      auto first = [&](uint32_t col, uint32_t x, uint32_t y) {
#pragma unroll
        for (int kk = 0; kk < KBD; ++kk)
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4)
            umma_bf16_if(leader, col, desc.at((x + kk * kBox + k4 * 32) >> 4), desc.at((y + kk * kBox + k4 * 32) >> 4), idesc_first,
                         (kk | k4) != 0);
      };
      // accumulator at `col` += A (tensor memory: 32 inner rows in 16 columns from `ta` and every 32 columns on) x inner tile
      auto second = [&](uint32_t col, uint32_t ta, uint32_t y, bool fresh) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ta_if(leader, col, ta + (k >> 1) * 32 + (k & 1) * 8, desc.at((y + k * 2048) >> 4), idesc_acc, !fresh || k != 0);
      };
      const uint32_t o_a = base + SM::kOuter, o_b = o_a + SM::kTile;
      auto tile_a = [&](int t) { return base + SM::kA + (t % NA) * SM::kTile; };
      auto tile_b = [&](int t) { return base + SM::kB + (t % NB) * SM::kTile; };
      auto issue_s = [&](int t) -> bool {
        if (!mbar_wait_warp(&a_full[t % NA], (t / NA) & 1, abort_flag)) return false;
        tc_fence_after();
        const int set = MODE == 0 ? 0 : t & 1;
        first(tmem + set * 128, o_a, tile_a(t));
        umma_commit_if(leader, &s_full[set]);
        return true;
      };
      auto issue_dp = [&](int t) -> bool {
        if (!mbar_wait_warp(&b_full[t % NB], (t / NB) & 1, abort_flag)) return false;
        tc_fence_after();
        first(tmem + kDP, o_b, tile_b(t));
        umma_commit_if(leader, dp_full);
        if (MODE == 1) umma_commit_if(leader, &b_empty[t % NB]);
        return true;
      };
      failed = !mbar_wait_warp(outer_full, 0, abort_flag) || !issue_s(0) || !issue_dp(0) || (MODE == 1 && T > 1 && !issue_s(1));
      for (int t = 0; t < T && !failed; ++t) {
        if (MODE == 0) {
          if (!mbar_wait_warp(p_full, t & 1, abort_flag)) { failed = true; break; }
          tc_fence_after();
          second(tmem + kAcc, tmem, tile_b(t), t == 0);                // dV += P^T dO
          umma_commit_if(leader, &b_empty[t % NB]);
          if (t + 1 < T && !issue_s(t + 1)) { failed = true; break; }
          if (!mbar_wait_warp(ds_full, t & 1, abort_flag)) { failed = true; break; }
          tc_fence_after();
          second(tmem + kAcc + HD, tmem + kDP, tile_a(t), t == 0);     // dK += dS^T Q
          umma_commit_if(leader, &a_empty[t % NA]);
          if (t + 1 < T && !issue_dp(t + 1)) { failed = true; break; }
        } else {
          if (!mbar_wait_warp(ds_full, t & 1, abort_flag)) { failed = true; break; }
          tc_fence_after();
          if (t + 1 < T && !issue_dp(t + 1)) { failed = true; break; }
          second(tmem + kAcc, tmem + (t & 1) * 128, tile_a(t), t == 0);  // dQ += dS K
          umma_commit_if(leader, &a_empty[t % NA]);
          if (t + 2 < T && !issue_s(t + 2)) { failed = true; break; }
        }
      }
      if (!failed) umma_commit_if(leader, acc_full);
    }
  } else if (warp == 2 + kSwaBwdWarps) {
    // ---------------- mode 0: the per-query values of an inner tile, fetched a tile ahead.  A stage has a barrier of its own for
    // its way back: the softmax warps may be two tiles past this warp (their tile t - 1 needs nothing more from it), and a wait by
    // parity on a barrier that completes once per tile, such as ds_full, would then stand for a tile that waits for this warp.
    if (MODE == 0) {
      // (queries that no key of the tile meets have values like those behind the end: theirs need not be finite)
      float x[8];   // lse and delta of queries lane, lane + 32, ...
      auto fetch = [&](int t) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int qi = (t_lo + t) * 128 + lane + 32 * i;
          x[i] = qi <= i_hi ? a.lse[stat_base + qi] : INFINITY;
          x[4 + i] = qi <= i_hi ? a.delta[stat_base + qi] : 0.f;
        }
      };
      if (!failed) fetch(0);
      for (int t = 0; t < T && !failed; ++t) {
        if (t >= 2 && !mbar_wait_warp(&st_empty[t & 1], ((t >> 1) - 1) & 1, abort_flag)) { failed = true; break; }  // tile t - 2
        float* st = stats + (t & 1) * 256 + lane;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          st[32 * i] = x[i];
          st[128 + 32 * i] = x[4 + i] * a.scale;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&st_full[t & 1]);
        if (t + 1 < T) fetch(t + 1);
      }
    }
  } else {
    // ---------------- softmax / epilogue: four threads per tensor-memory lane (outer row), 32 inner columns each
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const int row = o0 + r;             // this thread's key (mode 0) or query (mode 1)
    const int c0 = part * 32;
    float lse_r = INFINITY, delta_r = 0.f;
    int row_start = 0;
    if (MODE == 1 && row < a.L) {
      lse_r = a.lse[stat_base + row];
      delta_r = a.delta[stat_base + row] * a.scale;
      if (a.seq_start != nullptr) row_start = a.seq_start[row];
    }
    // first / last inner row that this outer row meets: mode 0, queries row .. row + window - 1 of its sequence; mode 1, the keys of
    // its window and sequence.  (The bounds once per thread: tests of every pair took 8500 clocks in each of the two tiles of a
    // band that are cut by it, a quarter of the kernel at a window of 2048.)
    int in_lo = 0, in_hi = -1;
    if (MODE == 0 && row < a.Lk) {
      const int64_t last = a.causal ? static_cast<int64_t>(row) + window - 1 : a.L - 1;
      in_lo = a.causal ? row : 0;
      in_hi = static_cast<int>(last < a.L - 1 ? last : a.L - 1);
    } else if (MODE == 1 && row < a.L) {
      in_lo = a.causal ? max(row - (window - 1), row_start) : 0;
      in_hi = a.causal ? row : a.Lk - 1;
    }
    if (MODE == 0 && a.seq_start != nullptr) {   // sequence after sequence of this warp's 32 keys
      const int first = o0 + quarter * 32;
      const int limit = static_cast<int>(min(static_cast<int64_t>(a.L), static_cast<int64_t>(first) + 31 + window));
      for (int end = min(first, a.L); __any_sync(0xFFFFFFFFu, end <= row && row < a.L);) {
        end = sequence_end(a.seq_start, end, limit);
        if (row < end && in_hi >= end) in_hi = end - 1;
      }
    }
    for (int t = 0; t < T && !failed; ++t) {
      const int i0 = (t_lo + t) * 128, set = MODE == 0 ? 0 : t & 1;
      const float* st = stats + (t & 1) * 256 + c0;
      if ((MODE == 0 && !mbar_wait_warp(&st_full[t & 1], (t >> 1) & 1, abort_flag)) ||
          !mbar_wait_warp(&s_full[set], (MODE == 0 ? t : t >> 1) & 1, abort_flag)) {
        failed = true;
        break;
      }
      tc_fence_after();
      const int lo = in_lo - i0 - c0, hi = in_hi - i0 - c0;          // this row's share of the warp's 32 columns
      const bool interior = __all_sync(0xFFFFFFFFu, lo <= 0 && hi >= 31);   // every pair visible: no masks
      if (!__any_sync(0xFFFFFFFFu, lo <= 31 && hi >= 0)) {
        // None is: zeros without the exponentials.  (Tiles of 128 rows are mostly that where sequences or windows are short: 16384
        // tokens, window 64, 85.1 -> 76.9 and 66.6 -> 60.5 us, 64 sequences of 64 tokens 27.8 -> 24.8 and 23.9 -> 21.2.  As a case
        // of the code below instead of a path of its own it took 640 and 438 us instead of 624 and 419 for 32768 tokens of 64.)
        uint32_t zero[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) zero[j] = 0;
        if (MODE == 0) {
          tmem_st16(tmem + lane_off + c0, zero);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full);
        }
        if (!mbar_wait_warp(dp_full, t & 1, abort_flag)) {
          failed = true;
          break;
        }
        tc_fence_after();
        tmem_st16(tmem + lane_off + (MODE == 0 ? kDP : set * 128u) + c0, zero);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(ds_full);
          if (MODE == 0) mbar_arrive(&st_empty[t & 1]);
        }
        continue;
      }
      uint32_t bits[32];
      tmem_ld32(tmem + lane_off + set * 128 + c0, bits);
      tmem_ld_wait();
      // p = 2^(s c - lse)
      float p[32];
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        float lv[4] = {lse_r, lse_r, lse_r, lse_r};
        if (MODE == 0) {
          const float4 l4 = *reinterpret_cast<const float4*>(st + g * 4);
          lv[0] = l4.x; lv[1] = l4.y; lv[2] = l4.z; lv[3] = l4.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) p[g * 4 + e] = exp2_ftz(fmaf(__uint_as_float(bits[g * 4 + e]), a.scale_log2, -lv[e]));
      }
      if (!interior) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < lo || j > hi) p[j] = 0.f;
      }
      uint32_t w[16];
      if (MODE == 0) {
#pragma unroll
        for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2(p[2 * j], p[2 * j + 1]);
        tmem_st16(tmem + lane_off + c0, w);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (!mbar_wait_warp(dp_full, t & 1, abort_flag)) {
        failed = true;
        break;
      }
      tc_fence_after();
      // dS = p (dP scale - Delta scale)
      tmem_ld32(tmem + lane_off + kDP + c0, bits);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        float dv[4] = {delta_r, delta_r, delta_r, delta_r};
        if (MODE == 0) {
          const float4 d4 = *reinterpret_cast<const float4*>(st + 128 + g * 4);
          dv[0] = d4.x; dv[1] = d4.y; dv[2] = d4.z; dv[3] = d4.w;
        }
        float ds[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) ds[e] = p[g * 4 + e] * fmaf(__uint_as_float(bits[g * 4 + e]), a.scale, -dv[e]);
        w[g * 2] = pack_bf16x2(ds[0], ds[1]);
        w[g * 2 + 1] = pack_bf16x2(ds[2], ds[3]);
      }
      tmem_st16(tmem + lane_off + (MODE == 0 ? kDP : set * 128u) + c0, w);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(ds_full);
        if (MODE == 0) mbar_arrive(&st_empty[t & 1]);
      }
    }
    if (failed) *abort_flag = 1;
    // accumulators: row = outer-tile row (key in mode 0, query in mode 1); this thread stores HD / 4 features of it
    if (!failed && !mbar_wait_warp(acc_full, 0, abort_flag)) failed = true;
    if (!failed) {
      tc_fence_after();
      constexpr int OC = HD / 4;
#pragma unroll
      for (int acc = 0; acc < (MODE == 0 ? 2 : 1); ++acc) {
        // mode 0: accumulator 0 = dV, accumulator 1 = dK; mode 1: dQ
        bf16* dst_base = MODE == 0 ? (acc == 0 ? a.out1 : a.out0) : a.out0;
        bf16* dst = dst_base + batch * a.o_bs + static_cast<int64_t>(row) * a.o_ts + head * a.o_hs + part * OC;
#pragma unroll
        for (int c = 0; c < OC; c += 16) {
          uint32_t bits[16];
          tmem_ld16(tmem + lane_off + kAcc + acc * HD + part * OC + c, bits);
          tmem_ld_wait();
          if (row < (MODE == 0 ? a.Lk : a.L)) {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              uint4 u;
              u.x = pack_bf16x2(__uint_as_float(bits[g * 8 + 0]), __uint_as_float(bits[g * 8 + 1]));
              u.y = pack_bf16x2(__uint_as_float(bits[g * 8 + 2]), __uint_as_float(bits[g * 8 + 3]));
              u.z = pack_bf16x2(__uint_as_float(bits[g * 8 + 4]), __uint_as_float(bits[g * 8 + 5]));
              u.w = pack_bf16x2(__uint_as_float(bits[g * 8 + 6]), __uint_as_float(bits[g * 8 + 7]));
              *reinterpret_cast<uint4*>(dst + c + g * 8) = u;
            }
          }
        }
      }
    }
  }
  if (failed && *reinterpret_cast<volatile int32_t*>(a.status) == kStatusOk) {
    *abort_flag = 1;
    report_timeout(a.status);
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 256; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// Delta[b][h][i] = sum_d dO[b][i][h][d] * O[b][i][h][d]: one warp per (batch, token, head) row.
struct SwaDeltaArgs {
  const bf16 *o, *dout;      // [b][l][h][d], token / batch strides below, head stride d
  int64_t o_ts, o_bs, d_ts, d_bs;
  float* delta;              // [b][h][l]
  int32_t b, L, heads, d;
};

}  // namespace lact
