// The attention forward of swa.cuh on pairs of query tiles, for calls with enough of them (swa_takes_pairs).  A work item is a pair of
// 128-query tiles of one (batch, head), "groups" 0 and 1, which share the key and value tiles; persistent CTAs walk items (SwaPairArgs
// says which).
//   warp 0      TMA producer: the queries of an item, then key and value tiles of 128 rows through two-stage rings that run
//               on across items;
//   warps 1, 2  MMA issuers, one per group: S = Q K^T (128 x 128 fp32) and O += P V (128 x d) per key tile, all in tensor memory;
//               P, two bf16 to a column, takes the place of the S it was made from and is the A operand of O += P V there;
//   warps 8-15  softmax:      four warps per group, one thread per query row (a row is a tensor-memory lane): maximum, then
//               exponentials, sum and P;
//   warps 4-7   correction:   where the maximum of a row has grown, O of the rows of its warp is multiplied by exp2(m_old - m_new)
//               before the next P V; at an item's end they divide by the sums and write the rows.
// While one group's softmax runs, the tensor pipe works on the other group's P V and next S; products of one group follow each
// other in the pipe, so S complete means the P V before it is complete and O may be changed.
// What bounds it (clocks inside the kernel, per key tile of one group): S 570, reading 128 scores and their maximum 370, exponentials 1700
// to 2000 (1190 with nothing else on the SM: 128 per thread at four lanes a clock), P V and hand-overs 700; two groups 3500 when
// they alternate and 4300 when they run in step.  An item's first and last tile (masks, loads from memory, rows written) cost about four
// tiles more.  With one tile per CTA, P through shared memory and O in registers a tile took 2900 clocks, 1800 of them what it moved
// through shared memory (224 KB; here 128).  24 x 32768 queries, window 2048, d = 128: 1201 -> 816 us
// (663 -> 976 TFLOP/s of the band's products).
// Code size counts: roles in 107 KB of code took 919 us, in 78 KB 836, in 67 KB 820 (a quarter of the stalls waits for
// instructions), which is why rarely run loops are not unrolled and masks are applied in tensor memory.
// Key and value tiles share one shared-memory layout ([128 rows][64 features] boxes, 128-byte swizzle): the first
// product reads it K-major (features = k), the second MN-major (keys = k).  The roles wait for each
// other at mbarriers alone, every wait with a limit.
#pragma once
#include <type_traits>
#include "swa.cuh"

namespace lact {

struct SwaPairArgs {
  CUtensorMap q, k, v;   // 4-D maps (feature, token, head, batch), box {64, 128, 1, 1}
  CUtensorMap k2, v2;    // keys and values behind the first `Lk1` (block attention over a cache and new tokens), if Lk1 > 0
  bf16* o;               // [b][l][h][d], strides below (elements); feature stride 1
  int64_t o_bs, o_ts, o_hs;
  int32_t L, window;     // queries per batch entry; window <= 0: unbounded (plain causal attention)
  int32_t Lk, causal;    // keys per batch entry (= L when causal); causal = 0: every query sees every key of its entry
  int32_t Lk1;           // two runs of keys: the second begins at the next whole tile behind Lk1, and Lk counts from there on
  int32_t heads, entries;  // heads x batch entries
  int32_t pairs;             // items per (batch, head)
  float scale_log2;      // log2(e) / sqrt(d)
  const int32_t* seq_start;  // optional [l]: first token of the packed sequence every token belongs to (nondecreasing;
                             // keys before it are invisible), or nullptr: one sequence per batch entry
  float* lse;            // optional [b][h][l]: log2-domain log-sum-exp of every row (the backward's input), or nullptr
  int32_t* status;
  // Items are numbered with the (batch, head) fastest and the last queries first (the longest items of causal attention without a
  // window).  The first `whole` are dealt to the CTAs in snake order.  The `rest`, fewer than SMs, would leave SMs idle: their key
  // tiles, `span` per item, are laid end to end and cut into `cutters` shares, one per CTA of the first `cutters`: the first
  // `longer` have share + 1 tiles, the others `share`.  A share meets two items at most.  A CTA leaves the unnormalised output rows,
  // maxima and sums of its piece of an item in `part` / `ml`, and swa_combine_kernel puts the pieces together.
  // (Pieces in their order step to the next cutter, the next item or both: the sum of the two numbers is a piece's own.)
  int32_t whole, rounds, rest, cutters, span, share, longer;   // rounds: of whole items over the grid
  float* part;   // [cutter + item - whole][group][128 rows][HD], a multiple of 32 bytes
  float2* ml;    // [cutter + item - whole][group][128 rows]: maximum, sum
};

constexpr int kSwaPairThreads = 512;
// Registers per thread: the block is launched with 128 for all; 128 * (56 + 104 + 2 * 176) are the 65536 it then has.
constexpr int kSwaPairIssueRegs = 56, kSwaPairCorrectionRegs = 104, kSwaPairSoftmaxRegs = 176;
static_assert(128 * (kSwaPairIssueRegs + kSwaPairCorrectionRegs + 2 * kSwaPairSoftmaxRegs) <= 512 * 128, "register split");

template <int HD>
struct SwaPairSmem {
  static constexpr uint32_t kTile = 128 * HD * 2;          // one Q / K / V tile
  static constexpr uint32_t kQ = 0, kK = 2 * kTile, kV = 4 * kTile, kBars = 6 * kTile;
  static constexpr uint32_t kBytes = kBars + 256 + 4096 + 1024;   // + barriers + what softmax tells correction + alignment slack
};

// As mbar_wait_warp, in as little code as it takes: the roles' loops share the instruction cache.
__device__ __forceinline__ bool swa_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag) {
  WaitClock clock;
  uint32_t i = 0;
  while (!__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity))) {
    if ((++i & 63u) == 0 && __any_sync(0xFFFFFFFFu, *abort_flag != 0 || !clock.within_limit())) return false;
  }
  return true;
}

// One item (or piece of one) of a CTA.
struct SwaItem {
  int batch, head, q0;
  int lo[2], hi[2];   // key tiles of either group (lo == hi: none)
  int first, last;    // key tiles of the item
  int piece;          // number of the piece of a cut item, or -1: whole
  __device__ __forceinline__ bool has(int g, int t) const { return t >= lo[g] && t < hi[g]; }
};
// first key tile (of all cut items, end to end) of a cutter's share, and the cutter whose share holds a tile
__device__ __forceinline__ uint32_t swa_share(const SwaPairArgs& a, uint32_t cutter) { return cutter * a.share + min(cutter, static_cast<uint32_t>(a.longer)); }
__device__ __forceinline__ uint32_t swa_cutter(const SwaPairArgs& a, uint32_t tile) {
  const uint32_t longer = static_cast<uint32_t>(a.longer) * (a.share + 1);
  return tile < longer ? tile / (a.share + 1) : a.longer + (tile - longer) / a.share;
}
// the (batch, head), first query and key tiles of an item
__device__ __forceinline__ void swa_place(const SwaPairArgs& a, int item, SwaItem& w) {
  const uint32_t bh = a.heads * a.entries, row = static_cast<uint32_t>(item) / bh, at = item - row * bh;
  w.batch = static_cast<int>(at / static_cast<uint32_t>(a.heads));
  w.head = static_cast<int>(at) - w.batch * a.heads;
  w.q0 = (a.pairs - 1 - static_cast<int>(row)) * 256;
  const int window = a.window > 0 ? a.window : a.L;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int q0 = w.q0 + 128 * g;
    w.lo[g] = w.hi[g] = 0;
    if (q0 >= a.L) continue;
    if (a.causal) {
      int lo = max(q0 - (window - 1), 0);
      // packed sequences: no row of this tile sees a key before the first row's sequence start
      if (a.seq_start != nullptr) lo = max(lo, a.seq_start[q0]);
      w.lo[g] = lo / 128;
      w.hi[g] = (min(q0 + 128, a.L) + 127) / 128;
    } else {
      w.hi[g] = (a.Lk + 127) / 128;
    }
  }
  w.first = w.lo[0];
  w.last = max(w.hi[0], w.hi[1]);
}
// 1: item `it` of this CTA is in `w`; 0: it has none, but may have a later one; -1: there are no more.
__device__ __forceinline__ int swa_item(const SwaPairArgs& a, int it, SwaItem& w) {
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  const int rounds = a.rounds;
  w.piece = -1;
  if (it < rounds) {
    const int item = snake_tile(it, grid, cta);
    if (item >= a.whole) return 0;
    swa_place(a, item, w);
    return 1;
  }
  if (cta >= a.cutters) return -1;
  const uint32_t u0 = swa_share(a, cta), u1 = swa_share(a, cta + 1);
  const uint32_t rest = u0 / static_cast<uint32_t>(a.span) + (it - rounds), begin = rest * a.span;
  if (begin >= u1) return -1;
  swa_place(a, a.whole + static_cast<int>(rest), w);
  w.piece = cta + static_cast<int>(rest);
  // (an item at the start of a sequence has fewer tiles than `span`: its later pieces are empty)
  const int T = w.last - w.first;
  w.last = w.first + min(static_cast<int>(min(u1 - begin, static_cast<uint32_t>(a.span))), T);
  w.first += min(static_cast<int>(max(u0, begin) - begin), T);
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    w.lo[g] = max(w.lo[g], w.first);
    w.hi[g] = max(w.lo[g], min(w.hi[g], w.last));
  }
  return 1;
}

// Puts the pieces of the cut items together: a warp per query row, four features (two at HD = 64) per lane.
template <int HD>
__global__ void __launch_bounds__(256) swa_combine_kernel(const __grid_constant__ SwaPairArgs a) {
  using Vec = typename std::conditional<HD == 128, float4, float2>::type;
  griddep_launch_dependents();
  griddep_wait();
  if (*reinterpret_cast<volatile int32_t*>(a.status) != kStatusOk) return;
  const int lane = threadIdx.x & 31, row = (blockIdx.x & 31) * 8 + (threadIdx.x >> 5);   // of the item's 256
  const uint32_t rest = blockIdx.x >> 5, begin = rest * a.span;
  SwaItem w;
  swa_place(a, a.whole + static_cast<int>(rest), w);
  const int qi = w.q0 + row;
  if (qi >= a.L) return;
  const int piece0 = static_cast<int>(swa_cutter(a, begin) + rest), pieces = static_cast<int>(swa_cutter(a, begin + a.span - 1) + rest) - piece0 + 1;
  const float2* const ml = a.ml + static_cast<int64_t>(piece0) * 256 + row;
  float m = -INFINITY, l = 0.f;
  for (int s = 0; s < pieces; ++s) m = fmaxf(m, ml[s * 256].x);
  const Vec* src = reinterpret_cast<const Vec*>(a.part + (static_cast<int64_t>(piece0) * 256 + row) * HD) + lane;
  float o[HD / 32] = {};
#pragma unroll 4
  for (int s = 0; s < pieces; ++s, src += 256 * 32) {
    const Vec x = *src;
    const float2 ms = ml[s * 256];
    // (a maximum of -inf is a share without a visible key, all zeros, or one whose scores are all NaN: those pass through)
    const float f = ms.x == -INFINITY ? 1.f : exp2_ftz(ms.x - m);
    l = fmaf(ms.y, f, l);
    const float* const v = reinterpret_cast<const float*>(&x);
#pragma unroll
    for (int j = 0; j < HD / 32; ++j) o[j] = fmaf(v[j], f, o[j]);
  }
  const float inv = l > 0.f ? 1.0f / l : 0.f;
  if (a.lse != nullptr && lane == 0) a.lse[(static_cast<int64_t>(w.batch) * a.heads + w.head) * a.L + qi] = m + log2f(l);
  uint32_t* const dst = reinterpret_cast<uint32_t*>(a.o + w.batch * a.o_bs + static_cast<int64_t>(qi) * a.o_ts + w.head * a.o_hs) + lane * (HD / 64);
#pragma unroll
  for (int j = 0; j < HD / 64; ++j) dst[j] = pack_bf16x2(o[2 * j] * inv, o[2 * j + 1] * inv);
}

template <int HD>
__global__ void __launch_bounds__(kSwaPairThreads, 1) swa_pairs_kernel(const __grid_constant__ SwaPairArgs a) {
  static_assert(HD == 64 || HD == 128, "head dimensions 64 and 128");
  using SM = SwaPairSmem<HD>;
  constexpr int KBD = HD / 64;                // 64-feature blocks of a tile
  constexpr uint32_t kBox = 128 * 128;        // bytes of one [128][64] box
  constexpr uint32_t kTmemCols = 512;         // S / P of group g: columns 128 g; O: 256 + 128 g
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + SM::kBars);
  uint64_t* q_full = bars;            // [2] groups
  uint64_t* k_full = bars + 2;        // [2] stages
  uint64_t* k_empty = bars + 4;       // [2], an arrival per group
  uint64_t* v_full = bars + 6;        // [2]
  uint64_t* v_empty = bars + 8;       // [2], an arrival per group
  uint64_t* s_full = bars + 10;       // [2] groups: S of the tile is complete (and all products of the group before it)
  uint64_t* p_half = bars + 12;       // [2] groups, 8 arrivals: P of the first 64 keys is written (4), O brought to the new maximum
                                      // (4; an item's first tile has no O yet: the softmax warps arrive for both)
  uint64_t* o_full = bars + 14;       // [2] groups: the item's last product is complete
  uint64_t* o_empty = bars + 16;      // [2] groups, 4 arrivals: O and the row's maximum and sum have been read
  uint64_t* a_full = bars + 18;       // [2] groups, 4 arrivals: the factors of O are in `factor`
  uint64_t* ml_full = bars + 20;      // [2] groups, 4 arrivals: the item's maxima and sums are in `row_ml`
  uint64_t* p_full = bars + 22;       // [2] groups, 4 arrivals: all of P is written
  uint64_t* q_empty = bars + 24;      // [2] groups
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* factor = reinterpret_cast<float*>(aligned + SM::kBars + 256);           // [2 groups][128 rows]
  float2* row_ml = reinterpret_cast<float2*>(aligned + SM::kBars + 256 + 1024);  // [2 groups][128 rows]

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 2);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 2);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_half[s], 8);
      mbar_init(&p_full[s], 4);
      mbar_init(&o_full[s], 1);
      mbar_init(&o_empty[s], 4);
      mbar_init(&a_full[s], 4);
      mbar_init(&ml_full[s], 4);
    }
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
  griddep_launch_dependents();
  griddep_wait();

  bool failed = uniform(static_cast<uint32_t>(*reinterpret_cast<volatile int32_t*>(a.status))) != kStatusOk;
  const int second = a.Lk1 > 0 ? (a.Lk1 + 127) / 128 * 128 : 0x7FFFFFFF;  // where the second run of keys begins
  SwaItem w;

  if (warp >= 8) {
    registers_grow<kSwaPairSoftmaxRegs>();
    // ---------------- softmax: a thread per query row
    const int g = (warp - 8) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
    const uint32_t s_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + g * 128;
    uint32_t tiles = 0, parts = 0;
    for (int it = 0; !failed; ++it) {
      const int have = swa_item(a, it, w);
      if (have < 0) break;
      const int q0 = w.q0 + 128 * g;
      const int lo = g == 0 ? w.lo[0] : w.lo[1], hi = g == 0 ? w.hi[0] : w.hi[1];
      if (have == 0 || lo >= hi) continue;
      const int qi = q0 + r;
      const int window = a.window > 0 ? a.window : a.L;
      const int row_start = (a.seq_start != nullptr && qi < a.L) ? a.seq_start[qi] : 0;
      const int tile_start = a.seq_start != nullptr ? a.seq_start[min(q0 + 127, a.L - 1)] : 0;  // last row's
      float m = -INFINITY, l = 0.f;
      for (int t = lo; t < hi; ++t) {
        const int kv0 = t * 128;
        // every (row, key) pair of the tile inside the band and the sequence: no masks
        const int keys = kv0 < second && a.Lk1 > 0 ? a.Lk1 : a.Lk;  // (not causal) end of the run this tile belongs to
        const bool interior = a.causal ? (kv0 + 127 <= q0 && kv0 >= q0 + 127 - (window - 1) && kv0 + 127 < a.L && kv0 >= tile_start)
                                       : kv0 + 127 < keys;
        // first / last column of the tile this row may see
        const int j_lo = (a.causal ? max(qi - (window - 1), row_start) : 0) - kv0;
        const int j_hi = (a.causal ? min(qi, a.L - 1) : keys - 1) - kv0;
        if (!swa_wait(&s_full[g], tiles & 1, abort_flag)) { failed = true; break; }
        ++tiles;
        tc_fence_after();
        if (__builtin_expect(!interior, 0)) {   // the scores that the row does not see become -inf, in place (a loop: code that few tiles run stays short)
#pragma unroll 1
          for (int c = 0; c < 128; c += 32) {
            uint32_t y[32];
            tmem_ld32(s_addr + c, y);
            tmem_ld_wait();
            const int from = min(max(j_lo - c, 0), 32), to = min(max(j_hi + 1 - c, 0), 32);
            const uint32_t seen = static_cast<uint32_t>((1ull << to) - 1) & ~static_cast<uint32_t>((1ull << from) - 1);
#pragma unroll
            for (int j = 0; j < 32; ++j) y[j] = (seen >> j) & 1u ? y[j] : 0xFF800000u;
            tmem_st32(s_addr + c, y);
          }
          tmem_st_wait();
        }
        uint32_t x[4][32];   // the row's scores
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + 32 * c, x[c]);
        tmem_ld_wait();
        float top[4];   // four chains
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          top[c] = fmaxf(__uint_as_float(x[c][0]), __uint_as_float(x[c][1]));
#pragma unroll
          for (int j = 2; j < 32; j += 2) top[c] = fmax3(top[c], __uint_as_float(x[c][j]), __uint_as_float(x[c][j + 1]));
        }
        const float mx = fmaxf(fmax3(top[0], top[1], top[2]), top[3]);
        const float m_new = fmaxf(m, mx * a.scale_log2);
        const float alpha = m_new == -INFINITY ? 1.f : exp2_ftz(m - m_new);
        if (t > lo) {
          factor[g * 128 + r] = alpha;
          __syncwarp();
          if (lane == 0) mbar_arrive(&a_full[g]);
        }
        const float shift = m_new == -INFINITY ? 0.f : -m_new;
        const F32x2 scale2 = f32x2(a.scale_log2, a.scale_log2), shift2 = f32x2(shift, shift);
        F32x2 sum2 = f32x2(0.f, 0.f);
        // 32 scores to probabilities
        uint32_t p[32];
        auto exp_chunk = [&](int c) {
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            float u, v;
            f32x2_split(f32x2_fma(f32x2(__uint_as_float(x[c][j]), __uint_as_float(x[c][j + 1])), scale2, shift2), u, v);
            u = exp2_ftz(u);
            v = exp2_ftz(v);
            sum2 = f32x2_add(sum2, f32x2(u, v));
            p[(c & 1) * 16 + (j >> 1)] = pack_bf16x2(u, v);
          }
        };
        exp_chunk(0);
        exp_chunk(1);
        tmem_st32(s_addr, p);   // P goes over scores that this thread has read
        exp_chunk(2);
        tmem_st_wait();   // the products of the first 64 keys need not wait for the others
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (t > lo) mbar_arrive(&p_half[g]);
          else mbar_arrive_twice(&p_half[g]);
        }
        exp_chunk(3);
        tmem_st32(s_addr + 32, p);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[g]);
        float even, odd;
        f32x2_split(sum2, even, odd);
        l = l * alpha + (even + odd);
        m = m_new;
      }
      // (the item before has been read out)
      if (failed || (parts > 0 && !swa_wait(&o_empty[g], (parts - 1) & 1, abort_flag))) { failed = true; break; }
      ++parts;
      row_ml[g * 128 + r] = make_float2(m, l);
      __syncwarp();
      if (lane == 0) mbar_arrive(&ml_full[g]);
    }
  } else if (warp >= 4) {
    registers_shrink<kSwaPairCorrectionRegs>();
    // ---------------- correction
    const int quarter = warp & 3, r = quarter * 32 + lane;
    const uint32_t o_lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + 256;
    const bool wide = ((reinterpret_cast<uintptr_t>(a.o) | (a.o_ts * 2) | (a.o_bs * 2)) & 31) == 0;
    uint32_t tiles0 = 0, tiles1 = 0, parts0 = 0, parts1 = 0;
    for (int it = 0;; ++it) {
      const int have = swa_item(a, it, w);
      if (have < 0) break;
      if (have == 0) continue;
      // a group's rows are read out a tile behind its last, and at the end
      const int done0 = w.lo[0] < w.hi[0] ? w.hi[0] : w.last, done1 = w.q0 + 128 >= a.L ? -1 : w.lo[1] < w.hi[1] ? w.hi[1] : w.last;
      for (int t = w.first; t <= w.last; ++t) {
        // the output rows of the groups that have ended, 32 features at a time (a piece without key tiles has none)
#pragma unroll 1
        for (int g = 0; g < 2; ++g) {
          if (t != (g == 0 ? done0 : done1)) continue;
          const int qi = w.q0 + 128 * g + r;
          const bool any = g == 0 ? w.lo[0] < w.hi[0] : w.lo[1] < w.hi[1];
          float m = -INFINITY, l = 0.f;
          if (any && !failed) {
            const uint32_t ph = (g == 0 ? parts0++ : parts1++) & 1;
            if (!swa_wait(&ml_full[g], ph, abort_flag) || !swa_wait(&o_full[g], ph, abort_flag)) {
              failed = true;
            } else {
              const float2 x = row_ml[g * 128 + r];
              m = x.x;
              l = x.y;
              tc_fence_after();
            }
          }
          auto own = [&](int c, float (&v)[32]) {
            uint32_t x[32];
            if (any) {
              tmem_ld32(o_lanes + g * 128 + c, x);
              tmem_ld_wait();
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = any ? __uint_as_float(x[j]) : 0.f;
          };
          auto free_o = [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && any && !failed) mbar_arrive(&o_empty[g]);
          };
          bf16* const dst = a.o + w.batch * a.o_bs + static_cast<int64_t>(qi) * a.o_ts + w.head * a.o_hs;
          auto store_rows = [&](int c, const float (&v)[32], float inv) {
            if (failed || qi >= a.L) return;
            uint32_t x[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = pack_bf16x2(v[2 * j] * inv, v[2 * j + 1] * inv);
            if (wide) {
              st_global_32(dst + c, x);
              st_global_32(dst + c + 16, x + 8);
            } else {
#pragma unroll
              for (int j = 0; j < 16; j += 4) st_global_16(dst + c + 2 * j, x[j], x[j + 1], x[j + 2], x[j + 3]);
            }
          };
          auto finish_row = [&]() -> float {   // 1 / the row's sum; its log-sum-exp
            if (a.lse != nullptr && !failed && qi < a.L)
              a.lse[(static_cast<int64_t>(w.batch) * a.heads + w.head) * a.L + qi] = m + log2f(l);
            return l > 0.f ? 1.0f / l : 0.f;
          };
          if (w.piece < 0) {
            const float inv = finish_row();
            __syncwarp();   // (rows past the end have stored nothing)
#pragma unroll 1
            for (int c = 0; c < HD; c += 32) {
              float v[32];
              own(c, v);
              store_rows(c, v, inv);
              __syncwarp();
            }
            free_o();
            continue;
          }
          // a piece of a cut item
          const int64_t mine = static_cast<int64_t>(w.piece) * 256 + g * 128 + r;
#pragma unroll 1
          for (int c = 0; c < HD; c += 32) {
            float v[32];
            own(c, v);
            float* const to = a.part + mine * HD + c;
#pragma unroll
            for (int j = 0; j < 32; j += 8) st_global_32(to + j, reinterpret_cast<const uint32_t*>(v + j));
            __syncwarp();
          }
          free_o();
          a.ml[mine] = make_float2(m, l);
        }
#pragma unroll 1
        for (int g = 0; g < 2; ++g) {
          if (failed || t <= (g == 0 ? w.lo[0] : w.lo[1]) || t >= (g == 0 ? w.hi[0] : w.hi[1])) continue;
          if (!swa_wait(&a_full[g], (g == 0 ? tiles0 : tiles1) & 1, abort_flag)) { failed = true; continue; }
          if (g == 0) ++tiles0;
          else ++tiles1;
          const float alpha = factor[g * 128 + r];
          if (__any_sync(0xFFFFFFFFu, alpha != 1.f)) {
            tc_fence_after();
            const F32x2 alpha2 = f32x2(alpha, alpha);
#pragma unroll 1
            for (int c = 0; c < HD; c += 32) {
              uint32_t x[32];
              tmem_ld32(o_lanes + g * 128 + c, x);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; j += 2) {
                float y, z;
                f32x2_split(f32x2_mul(f32x2(__uint_as_float(x[j]), __uint_as_float(x[j + 1])), alpha2), y, z);
                x[j] = __float_as_uint(y);
                x[j + 1] = __float_as_uint(z);
              }
              tmem_st32(o_lanes + g * 128 + c, x);
            }
            tmem_st_wait();
            tc_fence_before();
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_half[g]);
        }
      }
    }
  } else {
    registers_shrink<kSwaPairIssueRegs>();
    if (warp == 0) {
      const uint32_t leader = elect_leader();
      uint32_t n = 0, parts0 = 0, parts1 = 0;   // key tiles so far; per group, items with any tile
      for (int it = 0; !failed; ++it) {
        const int have = swa_item(a, it, w);
        if (have < 0) break;
        if (have == 0) continue;
        for (int t = w.first; t < w.last && !failed; ++t) {
#pragma unroll 1
          for (int g = 0; g < 2; ++g) {   // a group's queries before the first key tile it meets
            if (t != (g == 0 ? w.lo[0] : w.lo[1]) || t >= (g == 0 ? w.hi[0] : w.hi[1]) || failed) continue;
            const uint32_t part = g == 0 ? parts0++ : parts1++;
            if (part > 0 && !swa_wait(&q_empty[g], (part - 1) & 1, abort_flag)) { failed = true; continue; }
            mbar_expect_tx_if(leader, &q_full[g], SM::kTile);
            for (int j = 0; j < KBD; ++j)
              tma_load_4d_if(leader, base + SM::kQ + g * SM::kTile + j * kBox, &a.q, &q_full[g], 64 * j, w.q0 + 128 * g, w.head, w.batch);
          }
          const uint32_t sb = n & 1, ph = ((n >> 1) & 1) ^ 1;
          const bool behind = t * 128 >= second;
          const int row = t * 128 - (behind ? second : 0);
          const CUtensorMap* const km = behind ? &a.k2 : &a.k;
          const CUtensorMap* const vm = behind ? &a.v2 : &a.v;
          if (failed || !swa_wait(&k_empty[sb], ph, abort_flag)) { failed = true; break; }
          mbar_expect_tx_if(leader, &k_full[sb], SM::kTile);
          for (int j = 0; j < KBD; ++j)
            tma_load_4d_if(leader, base + SM::kK + sb * SM::kTile + j * kBox, km, &k_full[sb], 64 * j, row, w.head, w.batch);
          if (!swa_wait(&v_empty[sb], ph, abort_flag)) { failed = true; break; }
          mbar_expect_tx_if(leader, &v_full[sb], SM::kTile);
          for (int j = 0; j < KBD; ++j)
            tma_load_4d_if(leader, base + SM::kV + sb * SM::kTile + j * kBox, vm, &v_full[sb], 64 * j, row, w.head, w.batch);
          ++n;
        }
      }
    } else if (warp < 3) {
      // ---------------- products of one group
      const int g = warp - 1;
      const uint32_t leader = elect_leader();
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0), idesc_o = make_idesc_bf16(128, HD, 0, 1);
      const SmemDescBase k_desc(0), v_desc(kBox);
      const uint32_t s_col = tmem + g * 128, o_col = s_col + 256;
      const uint32_t q_at = (base + SM::kQ + g * SM::kTile) >> 4, k_at = (base + SM::kK) >> 4, v_at = (base + SM::kV) >> 4;
      uint32_t n = 0, tiles = 0, parts = 0;   // key tiles; those of this group whose P V has been issued; its items begun
      bool pending = false, fresh = false, ends = false;   // a tile of this group waits for its P V; as its item's first, last tile
      uint32_t stage = 0, parity = 0;                      // ... and its place in the ring
      int it = 0, t = 0, last = 0, lo = 0, hi = 0;
      bool over = false;   // no items are left
      while (!failed) {
        while (t >= last && !over) {
          const int have = swa_item(a, it++, w);
          over = have < 0;
          if (have <= 0) continue;
          t = uniform(w.first);
          last = uniform(w.last);
          lo = uniform(g == 0 ? w.lo[0] : w.lo[1]);
          hi = uniform(g == 0 ? w.hi[0] : w.hi[1]);
        }
        const uint32_t sb = n & 1, ph = (n >> 1) & 1;
        if (!over && !swa_wait(&k_full[sb], ph, abort_flag)) { failed = true; break; }
        if (pending) {
          if (!swa_wait(&v_full[stage], parity, abort_flag) || (fresh && parts > 1 && !swa_wait(&o_empty[g], parts & 1, abort_flag)) ||
              !swa_wait(&p_half[g], tiles & 1, abort_flag)) {
            failed = true;
            break;
          }
          tc_fence_after();
          // A = probabilities in tensor memory, 8 columns per 16 keys; B = values, MN-major: atoms of 64 features, each
          // [128 key rows][64] (one box), 16 key rows = 2048 bytes per MMA step
          const uint32_t vb = v_at + stage * (SM::kTile >> 4), keep = fresh ? 0u : 1u;
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ta_if(leader, o_col, s_col + k * 8, v_desc.at(vb + k * 128), idesc_o, k != 0 ? 1u : keep);
          if (!swa_wait(&p_full[g], tiles & 1, abort_flag)) { failed = true; break; }
          tc_fence_after();
#pragma unroll
          for (int k = 4; k < 8; ++k) umma_bf16_ta_if(leader, o_col, s_col + k * 8, v_desc.at(vb + k * 128), idesc_o, 1u);
          umma_commit_if(leader, &v_empty[stage]);
          if (ends) umma_commit_if(leader, &o_full[g]);
          ++tiles;
          pending = false;
        }
        if (over) break;
        if (t < lo || t >= hi) {   // the other group's alone
          if (!swa_wait(&v_full[sb], ph, abort_flag)) { failed = true; break; }
          if (lane == 0) {
            mbar_arrive(&k_empty[sb]);
            mbar_arrive(&v_empty[sb]);
          }
        } else {
          if (t == lo) {
            if (!swa_wait(&q_full[g], parts++ & 1, abort_flag)) { failed = true; break; }
            // Groups that begin together come to their exponentials at the same time, then both to their products, and stay so: 4300 clocks
            // per pair of tiles.  Half a tile apart, they alternate: 3500 (d = 128; tiles of d = 64, a fifth shorter, wait as long).
            if (g == 1 && lo == uniform(w.lo[0]) && hi - lo >= 4)
              for (const uint32_t begin = clock(); clock() - begin < 1700u;) __nanosleep(64);
          }
          tc_fence_after();
          const uint32_t kb = k_at + sb * (SM::kTile >> 4);
#pragma unroll
          for (int kk = 0; kk < KBD; ++kk)
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4)
              umma_bf16_if(leader, s_col, k_desc.at(q_at + kk * (kBox >> 4) + k4 * 2), k_desc.at(kb + kk * (kBox >> 4) + k4 * 2), idesc_s, (kk | k4) != 0);
          umma_commit_if(leader, &s_full[g]);
          umma_commit_if(leader, &k_empty[sb]);
          pending = true;
          fresh = t == lo;
          ends = t + 1 == hi;
          stage = sb;
          parity = ph;
          if (ends) umma_commit_if(leader, &q_empty[g]);
        }
        ++t;
        ++n;
      }
    }
  }
  // a wait that ran out: raise the flag so the other roles stop, record the status
  if (failed && *reinterpret_cast<volatile int32_t*>(a.status) == kStatusOk) {
    *abort_flag = 1;
    report_timeout(a.status);
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 256; ++i) __nanosleep(1000);  // bulk copies still in flight land before shared memory goes
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace lact
