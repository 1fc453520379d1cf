// Token x weight products on pairs of SMs, with the weights kept in shared memory.
//
//   gate       [y0 | y2] = x [W0; W2]^T, SwiGLU in the epilogue
//   pointwise  [y0 | y2] = k [W0; W2]^T and dh = v W1, lr-weighted backward of SwiGLU in the epilogue
//   store      c = a b^T, bf16
//
// All of them multiply many tokens by the same few weights with a short contraction (K <= 512).  The one-SM kernel
// (umma_gemm.cuh) streams both operands; what limits it there is how many bytes 227 KB of ring can have in flight: a ring
// stage is taken for about 3000 clocks (load from L2 or memory, its products, the way back to the producer), so 168 KB of
// stages bring 50 bytes a clock, where a tile of the pointwise stage wants 336 KB and its products take 2300 clocks.
// Here two SMs work on one tile of 256 tokens (tcgen05 cta_group::2): each holds half of the weight rows for as long as its
// run of tiles needs them, and loads nothing but its own 128 tokens: 192 KB for the same pointwise tile.
// Measured (us per launch, pairs against single SMs): 32 entries of 384, 2048 tokens: gate 43 / 48, down 28.8 / 31.5, pointwise
// 96 / 99 (6130 / 6730 clocks per 128 tokens and 64 hidden features, 3400 of them waiting for tokens from memory); 16 of 192,
// 49152 tokens: pointwise 314 / 347 (3660 / 4390 clocks, the epilogue's 3700).
// A pair keeps its column tile and walks a contiguous run of token tiles.  Both CTAs run
// the same program: warp 0 loads the CTA's own operands, warps 2-9 are its epilogue; warp 1 of the leader (rank 0) issues the
// products of both.  Full barriers live in the leader's shared memory (both CTAs' loads complete there), every other barrier
// in both, signalled by multicast commits.  All mbarrier waits are bounded; the cluster barriers at either end are reached by
// every thread whatever its waits returned, and no commit is still on its way then.
#pragma once
#include "ops.cuh"

namespace lact {

constexpr int kPairMaxKb = 8;    // k-blocks of a resident operand (K <= 512)
constexpr int kPairMaxRing = 8;
constexpr int kPairRows = 2 * kBM;          // tokens of a tile
constexpr uint32_t kPairPanel = kBM * 128;  // a staged output panel: 128 rows x 64 columns
constexpr uint32_t kPairBars = 512;         // barriers and flags

// Wiring of a pair kernel on top of an op of the one-SM engine (accumulators, epilogue, outputs, operand maps):
//   b_map(t, rank), b_col(t, rank)  which B map CTA `rank` loads for term t, and where its share of the columns starts
//   b_rows(t)                       rows of B per CTA (half of the term's N)
//   kHalfAtom                       the last term's share is 32 columns wide and MN-major: 64-byte swizzle
struct PairGateWiring {
  template <class Op> __host__ __device__ static constexpr int b_rows(int) { return Op::BT; }
  template <class Op> __device__ static int b_map(int, int rank) { return rank; }
  template <class Op> __device__ static int b_col(int, int) { return 0; }
  static constexpr bool kHalfAtom = false;
};
struct PairPointwiseWiring {
  template <class Op> __host__ __device__ static constexpr int b_rows(int t) { return t == 0 ? Op::BT : Op::BT / 2; }
  template <class Op> __device__ static int b_map(int t, int rank) { return t == 0 ? rank : 2; }
  template <class Op> __device__ static int b_col(int t, int rank) { return t == 0 ? 0 : rank * (Op::BT / 2); }
  static constexpr bool kHalfAtom = true;
};
struct PairStoreWiring {
  template <class Op> __host__ __device__ static constexpr int b_rows(int) { return Op::BT / 2; }
  template <class Op> __device__ static int b_map(int, int) { return 0; }
  template <class Op> __device__ static int b_col(int, int rank) { return rank * (Op::BT / 2); }
  static constexpr bool kHalfAtom = false;
};
template <class Op> struct PairWiring { using type = PairStoreWiring; };
template <int BT> struct PairWiring<OpSwigluGate<BT>> { using type = PairGateWiring; };
template <> struct PairWiring<OpFwGradPointwise> { using type = PairPointwiseWiring; };

// a CTA's share of the weights
template <class Op>
__host__ __device__ constexpr uint32_t pair_b_bytes(int num_kb) {
  uint32_t rows = 0;
  for (int t = 0; t < Op::NTERMS; ++t) rows += PairWiring<Op>::type::template b_rows<Op>(t);
  return rows * 128u * static_cast<uint32_t>(num_kb);
}
// staged panels in rotation: panel i is written while the stores of the panels before it are still being read out
template <class Op>
__host__ __device__ constexpr int pair_panels() { return Op::NOUT > 1 ? 3 : 2; }
// a ring stage: this CTA's tokens, one k-block of every A operand
template <class Op>
__host__ __device__ constexpr uint32_t pair_stage_bytes() { return Op::NA * kATileBytes; }
// depth of the activation ring that fits beside them
template <class Op>
__host__ __device__ constexpr int pair_ring(int num_kb) {
  const int64_t left = 232448ll - 1024 - kPairBars - pair_panels<Op>() * static_cast<int64_t>(kPairPanel) - pair_b_bytes<Op>(num_kb);
  const int64_t n = left / static_cast<int64_t>(pair_stage_bytes<Op>());
  return n < 0 ? 0 : static_cast<int>(n > kPairMaxRing ? kPairMaxRing : n);
}

template <class Op>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreadsV2, 1)
pair_gemm_kernel(const __grid_constant__ GemmArgs<Op, 1> args, const int ring) {
  using Wire = typename PairWiring<Op>::type;
  static_assert(Op::NOUT > 0 && Op::NTERMS <= 2, "staged ops");
  constexpr int BT = Op::BT, NACC = Op::NACC, NOUT = Op::NOUT, PANELS = pair_panels<Op>();
  constexpr uint32_t kAccCols = NACC * BT;
  constexpr uint32_t kTmemCols = tmem_cols_pow2(2 * kAccCols);
  static_assert(2 * kAccCols <= 512, "double-buffered accumulators exceed tensor memory");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const GemmProblem<Op>& P = args.prob[0];
  const int num_kb = (P.K + kBK - 1) / kBK;
  const uint32_t b_base = base, a_base = base + pair_b_bytes<Op>(num_kb), stg = a_base + ring * pair_stage_bytes<Op>();
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem_raw + (stg - raw) + PANELS * kPairPanel);
  uint64_t* const full = bars;                         // [ring]           leader's: both CTAs' loads
  uint64_t* const empty = full + kPairMaxRing;         // [ring]           in both
  uint64_t* const b_full = empty + kPairMaxRing;       // [k-blocks]       leader's
  uint64_t* const b_empty = b_full + kPairMaxKb;       // [k-blocks]       in both
  uint64_t* const acc_full = b_empty + kPairMaxKb;     // [2]              in both
  uint64_t* const acc_empty = acc_full + 2;            // [2]              leader's: both CTAs' epilogue warps
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* const abort_flag = tmem_slot + 1;  // [0] raised by anyone, [1 + tile parity] by epilogue warps only
  static_assert((2 * kPairMaxRing + 2 * kPairMaxKb + 4) * 8 + 16 <= kPairBars, "barrier space");

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairMaxRing; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < kPairMaxKb; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 2 * kEpiWarps); }
    for (int s = 0; s < 3; ++s) abort_flag[s] = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, kTmemCols);
    tmem_relinquish_pair();
  }
  if (threadIdx.x == 64) {
#pragma unroll
    for (int i = 0; i < Op::NA; ++i) tma_prefetch_desc(&P.a[i]);
#pragma unroll
    for (int i = 0; i < Op::NB; ++i) tma_prefetch_desc(&P.b[i]);
#pragma unroll
    for (int i = 0; i < NOUT; ++i) tma_prefetch_desc(&P.out[i]);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the peer's barriers are initialised, both halves of tensor memory are there
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);
  griddep_launch_dependents();
  griddep_wait();

  // The column tiles of one stretch of tokens belong to neighbouring pairs (a team of `tn`), which walk the same tokens at the
  // same time: they are read from memory once, and whole rows are written together.  The stretches, batch entry after batch
  // entry, are dealt to the teams in contiguous shares.
  const int tn = (P.N + BT - 1) / BT, tm = (P.M + kPairRows - 1) / kPairRows, total = tm * P.batch;
  const int pair = blockIdx.x >> 1, teams = (gridDim.x >> 1) / tn, team = pair / tn;
  const int t_begin = static_cast<int>(static_cast<int64_t>(total) * team / teams);
  const int t_end = static_cast<int>(static_cast<int64_t>(total) * (team + 1) / teams);
  const int n0 = (pair - team * tn) * BT;
  struct Run { int batch, m; };
  auto locate = [&](int tile) {
    Run r;
    if constexpr (Op::kReverseBatch) tile = total - 1 - tile;
    r.batch = tile / tm;
    r.m = tile - r.batch * tm;
    return r;
  };
  // first / last tile of a stretch over the same weights
  auto begins = [&](const Run& r) { return r.m == (Op::kReverseBatch ? tm - 1 : 0); };
  auto ends = [&](const Run& r) { return r.m == (Op::kReverseBatch ? 0 : tm - 1); };
  // (the CTAs of a pair may differ: every wait for the other has a limit)
  bool failed = earlier_launch_failed(args.status);
  const bool work = !failed;
  constexpr bool SEG = op_segments<Op>::value;
  auto load = [](uint32_t leader, uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int entry, int segment) {
    if constexpr (SEG) tma_load_4d_pair_if(leader, dst, map, bar, c0, c1, entry, segment);
    else tma_load_3d_pair_if(leader, dst, map, bar, c0, c1, entry);
  };
  auto term_bytes = [](int t) { return static_cast<uint32_t>(Wire::template b_rows<Op>(t)) * 128u; };  // a k-block of B, per CTA
  constexpr uint32_t b_bytes = pair_b_bytes<Op>(1);
  auto term_base = [&](int t) { return b_base + (t == 0 ? 0u : term_bytes(0) * num_kb); };

  if (warp == 0) {
    // ---------------- TMA producer: this CTA's tokens through the ring; its weight rows when a run begins, k-block by k-block
    // as the products of the run before let go of them
    const uint32_t leader = elect_leader(), signaller = rank == 0 ? leader : 0u;
    int s = 0;
    uint32_t ph = 0, bph = 0;
    for (int tile = t_begin; tile < t_end && !failed; ++tile) {
      const Run r = locate(tile);
      const bool first = tile == t_begin || begins(r);
      // coordinates of this tile's boxes, per term; one k-block on per stage
      int a_row[Op::NTERMS], a_batch[Op::NTERMS], a_k[Op::NTERMS], b_mn[Op::NTERMS], b_batch[Op::NTERMS], b_k[Op::NTERMS];
      bool b_major[Op::NTERMS];
      int entry, segment;
      entry_of(P, r.batch, entry, segment);
#pragma unroll
      for (int t = 0; t < Op::NTERMS; ++t) {
        const OperandInfo& ai = P.ai[Op::term_a(t)];
        a_row[t] = ai.mn_off + r.m * kPairRows + static_cast<int>(rank) * kBM;
        a_batch[t] = ai.batch_off + entry;
        a_k[t] = ai.k_off;
        const OperandInfo& bi = P.bi[Wire::template b_map<Op>(t, rank)];
        b_mn[t] = bi.mn_off + n0 + Wire::template b_col<Op>(t, rank);
        b_batch[t] = bi.batch_off + entry;
        b_k[t] = bi.k_off;
        b_major[t] = bi.mn_major != 0;
      }
      for (int kb = 0; kb < num_kb; ++kb) {
        if (first) {
          if (!mbar_wait_warp(&b_empty[kb], bph ^ 1, abort_flag)) { failed = true; break; }
          mbar_expect_tx_if(signaller, &b_full[kb], 2 * b_bytes);
          const uint32_t bar = leader_address(&b_full[kb]);
#pragma unroll
          for (int t = 0; t < Op::NTERMS; ++t) {
            const CUtensorMap* const map = &P.b[Wire::template b_map<Op>(t, rank)];
            const uint32_t dst = term_base(t) + kb * term_bytes(t);
            if (!b_major[t]) load(leader, dst, map, bar, b_k[t], b_mn[t], b_batch[t], segment);
            else if (Wire::kHalfAtom && t == Op::NTERMS - 1) load(leader, dst, map, bar, b_mn[t], b_k[t], b_batch[t], segment);
            else {
#pragma unroll
              for (int j = 0; j < Wire::template b_rows<Op>(t) / 64; ++j)
                load(leader, dst + j * kAtomBytes, map, bar, b_mn[t] + 64 * j, b_k[t], b_batch[t], segment);
            }
            b_k[t] += kBK;
          }
        }
        if (!mbar_wait_warp(&empty[s], ph ^ 1, abort_flag)) { failed = true; break; }
        mbar_expect_tx_if(signaller, &full[s], 2 * pair_stage_bytes<Op>());
        const uint32_t bar = leader_address(&full[s]), st = a_base + s * pair_stage_bytes<Op>();
#pragma unroll
        for (int t = 0; t < Op::NTERMS; ++t) {
          load(leader, st + Op::term_a(t) * kATileBytes, &P.a[Op::term_a(t)], bar, a_k[t], a_row[t], a_batch[t], segment);
          a_k[t] += kBK;
        }
        if (++s == ring) { s = 0; ph ^= 1; }
      }
      if (first) bph ^= 1;
    }
    // The last products' commits arrive in this CTA's shared memory too: they are waited for, stage by stage, before it goes.
    for (int i = 0; i < ring && !failed; ++i) {
      failed = !mbar_wait_warp(&empty[s], ph ^ 1, abort_flag);
      if (++s == ring) { s = 0; ph ^= 1; }
    }
    for (int kb = 0; kb < num_kb && !failed; ++kb) failed = !mbar_wait_warp(&b_empty[kb], bph ^ 1, abort_flag);
  } else if (warp == 1) {
    // ---------------- MMA issuer of the pair
    if (rank == 0) {
      const uint32_t leader = elect_leader();
      int s = 0;
      uint32_t ph = 0, bph = 0, n = 0;
      const SmemDescBase desc(kAtomBytes);
      for (int tile = t_begin; tile < t_end && !failed; ++tile, ++n) {
        const Run r = locate(tile);
        const bool first = tile == t_begin || begins(r), last = tile == t_end - 1 || ends(r);
        const uint32_t as = n & 1;
        const uint32_t acc = tmem + as * kAccCols;
        if (!mbar_wait_warp(&acc_empty[as], ((n >> 1) & 1) ^ 1, abort_flag)) { failed = true; break; }
        tc_fence_after();
        uint32_t idesc[Op::NTERMS], step_b[Op::NTERMS];
#pragma unroll
        for (int t = 0; t < Op::NTERMS; ++t) {
          const bool half_atom = Wire::kHalfAtom && t == Op::NTERMS - 1;
          const int b_mn = half_atom ? 1 : P.bi[Wire::template b_map<Op>(t, 0)].mn_major;
          idesc[t] = make_idesc_bf16(kPairRows, Op::term_n(t), 0, b_mn);
          step_b[t] = half_atom ? 64 : (b_mn ? 128 : 2);  // 16 k-rows of 64 or 128 bytes, or 32 bytes inside a row
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          if (first && !mbar_wait_warp(&b_full[kb], bph, abort_flag)) { failed = true; break; }
          if (!mbar_wait_warp(&full[s], ph, abort_flag)) { failed = true; break; }
          tc_fence_after();
#pragma unroll
          for (int t = 0; t < Op::NTERMS; ++t) {
            const SmemDescBase descb = Wire::kHalfAtom && t == Op::NTERMS - 1 ? SmemDescBase::half_atom() : desc;
            const uint32_t a_tile = (a_base + s * pair_stage_bytes<Op>() + Op::term_a(t) * kATileBytes) >> 4;
            const uint32_t b_tile = (term_base(t) + kb * term_bytes(t)) >> 4;
#pragma unroll
            for (int k4 = 0; k4 < kBK / kUmmaK; ++k4)
              umma_bf16_pair_if(leader, acc + Op::term_col(t), desc.at(a_tile + k4 * 2), descb.at(b_tile + k4 * step_b[t]), idesc[t],
                                (kb > 0 || k4 > 0 || !Op::term_first(t)) ? 1u : 0u);
          }
          umma_commit_pair_if(leader, &empty[s]);
          if (last) umma_commit_pair_if(leader, &b_empty[kb]);
          if (++s == ring) { s = 0; ph ^= 1; }
        }
        if (!failed) umma_commit_pair_if(leader, &acc_full[as]);
        if (first) bph ^= 1;
      }
    }
  } else if (work) {
    // ---------------- epilogue of this CTA's 128 tokens: the two warps of a lane quarter take the two 32-column halves of every
    // 64-column panel; each panel of each output goes through a staging buffer and out by TMA
    const int quarter = warp & 3, half = (warp - 2) >> 2, row_local = quarter * 32 + lane;
    const bool elected = threadIdx.x == 64;
    uint32_t n = 0, buf = 0;
    bool stop = false;
    typename Op::Prefetch pf_next;  // the epilogue's own operands, fetched a tile ahead
    auto fetch = [&](int tile) {
      if (tile >= t_end) return;
      const Run r = locate(tile);
      Op::prefetch(P.ep, r.batch, r.m * kPairRows + static_cast<int>(rank) * kBM + row_local, n0, half, P.M, P.N, pf_next);
    };
    fetch(t_begin);
    for (int tile = t_begin; tile < t_end && !stop; ++tile, ++n) {
      const Run r = locate(tile);
      const int m0 = r.m * kPairRows + static_cast<int>(rank) * kBM, row = m0 + row_local;
      const uint32_t as = n & 1;
      typename Op::Prefetch pf = pf_next;
      fetch(tile + 1);
      // A warp whose wait ran out tells the others at the tile's first named barrier, in the word of the tile's parity: by the
      // time it could raise that word for another tile, all of them have looked.
      if (!mbar_wait(&acc_full[as], (n >> 1) & 1, abort_flag)) abort_flag[1 + as] = 1;
      tc_fence_after();
      const uint32_t acc = tmem + as * kAccCols + (static_cast<uint32_t>(quarter * 32) << 16) + half * 32;
      const int panels = min(BT / 64, (P.N - n0 + 63) / 64);
      int entry, segment;
      entry_of(P, r.batch, entry, segment);
      for (int pnl = 0; pnl < panels && !stop; ++pnl) {
        uint32_t packed[NOUT][16];
        {
          float v[NACC][32], ov[NOUT][32];
          {
            uint32_t bits[NACC][32];
#pragma unroll
            for (int a = 0; a < NACC; ++a) tmem_ld32(acc + a * BT + pnl * 64, bits[a]);
            tmem_ld_wait();
#pragma unroll
            for (int a = 0; a < NACC; ++a)
#pragma unroll
              for (int j = 0; j < 32; ++j) v[a][j] = __uint_as_float(bits[a][j]);
          }
          if (pnl == panels - 1) {  // everything has been read: the accumulators are free
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(&acc_empty[as]);
          }
          Op::epilogue_staged(P.ep, r.batch, row, n0 + pnl * 64 + half * 32, P.M, P.N, v, ov, pf);
#pragma unroll
          for (int o = 0; o < NOUT; ++o)
#pragma unroll
            for (int j = 0; j < 16; ++j) packed[o][j] = pack_bf16x2(ov[o][2 * j], ov[o][2 * j + 1]);
        }
#pragma unroll
        for (int o = 0; o < NOUT; ++o) {
          const uint32_t line = stg + buf * kPairPanel + row_local * 128;
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const uint32_t addr = line + (((half * 4 + g) ^ (row_local & 7)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(packed[o][g * 4]), "r"(packed[o][g * 4 + 1]),
                         "r"(packed[o][g * 4 + 2]), "r"(packed[o][g * 4 + 3])
                         : "memory");
          }
          fence_async_proxy();
          // after this barrier the buffer of the next panel is free: the stores issued up to PANELS - 1 panels ago have read theirs
          if (elected) bulk_wait_read<PANELS - 2>();
          named_barrier_sync(2, kEpiWarps * 32);
          if (pnl == 0 && o == 0 && abort_flag[1 + as] != 0) { stop = true; break; }
          if (elected && m0 < P.M) {
            const int col = P.oi[o].col_off + n0 + pnl * 64, at = P.oi[o].row_off + m0, b = P.oi[o].batch_off + entry;
            if constexpr (SEG) tma_store_4d(&P.out[o], stg + buf * kPairPanel, col, at, b, segment);
            else tma_store_3d(&P.out[o], stg + buf * kPairPanel, col, at, b);
          }
          if (elected) bulk_commit_group();
          if (++buf == PANELS) buf = 0;
        }
      }
    }
    if (elected) bulk_wait_all();
    failed = stop;
  }
  if (failed && work) {
    *abort_flag = 1;
    report_timeout(args.status);
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 256; ++i) __nanosleep(1000);  // bulk copies still in flight land before shared memory goes
  }
  __syncthreads();
  cluster_sync();  // the peer's products, commits and arrivals on this CTA's shared and tensor memory are through
  if (warp == 1) tmem_dealloc_pair(tmem, kTmemCols);
}

}  // namespace lact
