// Batched bf16 GEMM engine for sm_100a: TMA-fed shared-memory tiles, tcgen05.mma into tensor
// memory, warp-specialised (1 TMA warp, 1 MMA warp, 4 epilogue warps), pluggable fp32 epilogue.
//
// One CTA computes one 128 x BN output tile of one batch entry of one problem:
//     acc[c] (+)= A[term_a] * B[term_b]^T          for every term of the op
// where A operands are (M x K) and B operands are (N x K), each either K-major (k contiguous
// in global memory) or MN-major (m / n contiguous).  Several terms may share operands (SwiGLU
// gate + up projection share the activations) or accumulators (split-precision products).
// Out-of-range parts of a tile are zero-filled by TMA, so ragged M, N and K need no masks in
// the main loop; the epilogue clips its stores.
#pragma once
#include "ptx.cuh"

namespace lact {

using bf16 = __nv_bfloat16;

constexpr int kBM = 128;   // UMMA M (rows of the accumulator = TMEM lanes)
constexpr int kBK = 64;    // k-block: 64 bf16 = 128 bytes = one swizzle row
constexpr int kUmmaK = 16; // K of one tcgen05.mma for 16-bit operands
constexpr uint32_t kATileBytes = kBM * kBK * 2;
constexpr uint32_t kAtomBytes = 64 * kBK * 2;  // one 64(mn) x 64(k) MN-major atom column

struct OperandInfo {
  int32_t mn_major;   // 0: global [mn][k] (k contiguous); 1: global [k][mn] (mn contiguous)
  int32_t mn_off;     // added to the mn coordinate
  int32_t k_off;      // added to the k coordinate
  int32_t batch_off;  // added to the batch coordinate
};

// Where a staged (TMA-stored) output tile lands: tile (m0, n0) of batch entry b is stored at
// coordinates (col_off + n0, row_off + m0, batch_off + b) of the output map, whose extents clip it.
// Dataflow kernels store from registers instead: element (r, c) of entry b at ptr[b * bs + r * ld + c].
struct OutInfo {
  int32_t row_off, col_off, batch_off, enabled;
  void* ptr;
  int64_t bs;
  int32_t ld, wide;  // wide: rows start on 32 bytes
};

template <class Op>
struct GemmProblem {
  CUtensorMap a[Op::NA];
  CUtensorMap b[Op::NB];
  CUtensorMap out[Op::NOUT > 0 ? Op::NOUT : 1];  // bf16 outputs written by TMA store (NOUT == 0: none)
  OperandInfo ai[Op::NA];
  OperandInfo bi[Op::NB];
  OutInfo oi[Op::NOUT > 0 ? Op::NOUT : 1];
  int32_t M, N, K, batch;
  int32_t entries;  // ops with `kSegments`: batch index x is entry x % entries of segment x / entries (0: one segment)
  typename Op::Epi ep;
  // Split contraction (ops with `kSplitK`; `splits` > 1): the k-blocks of every output tile are dealt to `splits` units of
  // `kb_per_split` k-blocks each.  A unit leaves its fp32 sums in `part`; the unit that finds the tile's word of `count` at
  // splits - 1 is the last to arrive, adds all of them in their order (the same result whoever is last), runs the epilogue
  // and sets the word back to zero.  Nothing waits for another unit.
  int32_t splits, kb_per_split;
  float* part;      // [tile of the launch][split][128 * BT]
  uint32_t* count;  // [tile of the launch], zero before and after the launch
};

template <class Op, int NPROB>
struct GemmArgs {
  using OpType = Op;
  GemmProblem<Op> prob[NPROB];
  int32_t* status;  // device status word (0 = ok)
};

__host__ __device__ constexpr uint32_t tmem_cols_pow2(uint32_t n) {
  return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512;
}

// An op describes the wiring of one GEMM kernel:
//   NA, NB        operand tiles loaded per pipeline stage (A tiles: 128 rows; B tiles: BT rows)
//   BT            width of the output tile in logical columns (= rows of every B operand tile)
//   NACC          accumulators handed to the epilogue, accumulator a at TMEM columns [a*BT, (a+1)*BT)
//   terms         each term issues MMAs  acc[cols term_col .. term_col + term_n) (+)= A[term_a] * B[term_b..]^T;
//                 term_n may span several consecutive B tiles (they are adjacent in shared memory)
//   STAGES        depth of the shared-memory ring
// Accumulators are double-buffered in tensor memory (2 * NACC * BT <= 512 columns), so the epilogue
// of tile i overlaps the main loop of tile i + 1.
template <class Op>
__host__ __device__ constexpr uint32_t gemm_stage_bytes() {
  return Op::NA * kATileBytes + Op::NB * Op::BT * kBK * 2;
}
// bf16 staging tiles for TMA-stored outputs: NOUT x [128 rows][BT columns], 128-byte swizzled in
// 64-column panels (the layout the output tensor maps expect)
template <class Op>
__host__ __device__ constexpr uint32_t gemm_staging_bytes();
template <class Op>
__host__ __device__ constexpr uint32_t gemm_smem_bytes() {
  return Op::STAGES * gemm_stage_bytes<Op>() + gemm_staging_bytes<Op>() + 1024 /*alignment slack*/ + 256 /*barriers*/;
}

constexpr int kEpiWarps = 8;
constexpr int kGemmThreadsV2 = 64 + 32 * kEpiWarps;  // producer warp + MMA warp + epilogue warps
// dataflow kernels add a scout warp that walks the tile sequence ahead of the producer and checks
// every tile's dependency, so that the global-memory latency of that check never stalls the loads
constexpr int kGemmThreadsFlow = kGemmThreadsV2 + 32;
constexpr uint32_t kFlowScratch = kEpiWarps * 32 * 80;  // a 32 x 32 bf16 block (rows padded to 80 bytes) per epilogue warp
// ring stages of `stride` bytes beside that scratch
__host__ __device__ constexpr int flow_ring(uint32_t stride) {
  return static_cast<int>((232448u - 1024u - 256u - kFlowScratch) / stride) > 8
             ? 8
             : static_cast<int>((232448u - 1024u - 256u - kFlowScratch) / stride);
}

// One operand tile of a ring stage: ROWS (mn) x one k-block.  Shared-memory layout:
//   K-major:  [ROWS rows][64 k];
//   MN-major: per 64-wide mn atom [64 k rows][64 mn] (atoms 8 KB apart).
// (A ring of four or five small stages refills sooner than one of two stages of two k-blocks: 72 tiles of the token contraction, 25
// k-blocks each, 19.4 -> 17.3 us.)
// The cursor holds the coordinates of an operand's next boxes: they are worked out once per output tile, so that between two
// stages the issuing warp only adds.  (What that warp spends per box is what the loads can reach: see gemm_phase.)
// SEG: the maps are 4-D (inner, row, entry, segment), see op_segments.
template <int ROWS, bool SEG>
struct OperandCursor {
  const CUtensorMap* map;
  int32_t inner, row, batch, segment;  // first box of the stage
  int32_t d_inner, d_row;     // advance per stage
  int32_t mn_major;           // 0: K-major, one box; 1: MN-major, a box per atom
  __device__ __forceinline__ void start(const CUtensorMap* m, const OperandInfo& oi, int mn0, int kc, int b, int seg) {
    map = m;
    batch = oi.batch_off + b;
    segment = seg;
    mn_major = oi.mn_major;
    if (mn_major) {
      inner = oi.mn_off + mn0; row = oi.k_off + kc;
      d_inner = 0; d_row = kBK;
    } else {
      inner = oi.k_off + kc; row = oi.mn_off + mn0;
      d_inner = kBK; d_row = 0;
    }
  }
  __device__ __forceinline__ void box(uint32_t leader, uint32_t dst, uint32_t bar, int at) const {
    if constexpr (SEG) tma_load_4d_if(leader, dst, map, bar, at, row, batch, segment);
    else tma_load_3d_if(leader, dst, map, bar, at, row, batch);
  }
  __device__ __forceinline__ void load(uint32_t leader, uint32_t dst, uint32_t bar) {
    if (!mn_major) {
      box(leader, dst, bar, inner);
    } else {
#pragma unroll
      for (int j = 0; j < ROWS / 64; ++j) box(leader, dst + j * kAtomBytes, bar, inner + 64 * j);
    }
    inner += d_inner;
    row += d_row;
  }
};

struct TileCoord {
  int prob, batch, m0, n0;
  int slot, split;  // split contractions: running number of the output tile, and which share of its k-blocks
};

// Ops whose output is a symmetric M x M matrix (both operands the same rows) may declare `kSymmetric`: only the
// 128 x 128 tiles on and above the diagonal are computed, and every off-diagonal tile is stored twice, as it is and
// transposed.  Needs BT = 128, one staged output, dataflow mode.
// On the diagonal the B tiles are the very rows of the A tiles, read the same way: they are not loaded a second time, the
// products read A tile `diag_a(b)` in place of B tile b.  At three row blocks half of the computed tiles lie on the diagonal: a
// quarter of the operand bytes of these phases, worth 0.4 % of a forward and 0.8 % of a training step at 32 units of 384 (the
// kernels wait for stages in flight and for each other's tiles more than for bytes).
template <class Op, class = void>
struct op_symmetric { static constexpr bool value = false; };
template <class Op>
struct op_symmetric<Op, decltype(void(Op::kSymmetric))> { static constexpr bool value = Op::kSymmetric; };

template <class Op>
__host__ __device__ constexpr uint32_t gemm_staging_bytes() {
  return Op::NOUT * kBM * Op::BT * 2 + Op::kEpiScratch;
}

// Ops whose launches may cover several runs of tokens ("segments") of the same entries, each with weights of its own, declare
// `kSegments`: all their maps are 4-D, (columns, rows, entry, segment).
template <class Op, class = void>
struct op_segments { static constexpr bool value = false; };
template <class Op>
struct op_segments<Op, decltype(void(Op::kSegments))> { static constexpr bool value = Op::kSegments; };
// batch index -> entry and segment
template <class Op>
__device__ __forceinline__ void entry_of(const GemmProblem<Op>& P, int batch, int& entry, int& segment) {
  entry = batch;
  segment = 0;
  if constexpr (op_segments<Op>::value) {
    if (P.entries > 0) {
      segment = batch / P.entries;
      entry = batch - segment * P.entries;
    }
  }
}

// Ops whose contraction may be split over several units (see GemmProblem): direct epilogues, single-phase kernels.
template <class Op, class = void>
struct op_split { static constexpr bool value = false; };
template <class Op>
struct op_split<Op, decltype(void(Op::kSplitK))> { static constexpr bool value = Op::kSplitK; };

// Ops whose epilogue reads per-row values from global memory may declare `kFetchAhead`: `prefetch` then only issues the loads
// and is called a tile ahead.  Where the epilogue sets the pace (the pointwise stage at 192 features, 4570 clocks a tile) 2000
// of them went on waiting for the learning rates of the tile in hand.
template <class Op, class = void>
struct op_fetch_ahead { static constexpr bool value = false; };
template <class Op>
struct op_fetch_ahead<Op, decltype(void(Op::kFetchAhead))> { static constexpr bool value = Op::kFetchAhead; };

// Per-thread view of the CTA's pipeline resources and of this thread's progress counters.  The
// producer thread advances the ring stage, the MMA thread stage and `tcount`, epilogue threads `tcount`;
// all three walk the same tile sequence, so their private copies stay consistent.  The counters
// run on across phases of a multi-phase kernel.
struct GemmCtx {
  uint32_t smem_base;     // 1024-byte aligned start of the stage ring
  uint32_t stage_stride;  // bytes between ring stages (>= the op's stage bytes)
  uint32_t staging;       // 1024-byte aligned start of the output staging tiles
  uint64_t *full_bar, *empty_bar, *acc_full_bar, *acc_empty_bar;
  volatile uint32_t* abort_flag;  // [0] raised by anyone, [1], [2] by epilogue warps only
  uint32_t tmem_base;
  uint32_t slot = 0, phase = 0, tcount = 0;  // ring stage in turn and its phase; output tiles so far
  // dataflow mode (multi-phase kernels whose phases are ordered by completion counters, see FlowDeps)
  uint32_t rot = 0;              // tiles handed out by earlier phases, modulo the grid size
  uint32_t ptile = 0;            // tiles whose dependency has been verified (scout) / consumed (producer)
  uint32_t* dep_ok = nullptr;    // shared-memory word: tiles verified by the scout warp, read by the producer thread
  volatile uint32_t* last_unit = nullptr;  // shared-memory word: this unit completes its tile (split contractions)
  template <int RING>
  __device__ __forceinline__ void next_stage() {
    if (++slot == RING) { slot = 0; phase ^= 1; }
  }
};

struct NoPatch {
  template <class Epi>
  __device__ __forceinline__ void operator()(Epi&, int) const {}
};

// Phase ordering of a multi-phase kernel without grid-wide barriers.  Every (problem, batch entry)
// owns a completion counter in global memory; a tile's stores are followed by one releasing increment
// of its batch entry's counter, and a tile of a later phase may load only after the
// counter of its batch entry has reached `need` = the number of tiles all earlier phases produce for
// that entry.  The phases of a batch entry must form a chain (each phase reads only what earlier
// phases of the same entry wrote, and overwrites only what earlier phases of the same entry read).
// All CTAs walk the phases in the same order and must be co-resident; every wait is bounded.
struct NoDeps {
  static constexpr bool kOn = false;
};
struct FlowDeps {
  static constexpr bool kOn = true;
  uint32_t* counter[2];  // per problem: [batch] counters
  uint32_t need[2];      // per problem: value required before a tile of this phase loads
};

__device__ __forceinline__ uint32_t ld_acquire_gpu_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_u32(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_cta_shared_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cta_shared_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
// Bounded spin until *ctr >= need (global memory, written by other CTAs).
__device__ __forceinline__ bool dep_wait(const uint32_t* ctr, uint32_t need, volatile uint32_t* abort_flag) {
  if (need == 0 || ld_acquire_gpu_u32(ctr) >= need) return true;
  WaitClock clock;
  for (uint32_t i = 1;; ++i) {
    if (ld_acquire_gpu_u32(ctr) >= need) return true;
    if ((i & 31u) == 0 && (*abort_flag != 0 || !clock.within_limit())) return false;
  }
}
// Producer thread: bounded wait until the scout warp has verified the dependency of the tile with
// running number `seq` (0-based).
__device__ __forceinline__ bool flow_wait_verified(const GemmCtx& cx, uint32_t seq) {
  if (ld_acquire_cta_shared_u32(cx.dep_ok) > seq) return true;
  WaitClock clock;
  for (uint32_t i = 1;; ++i) {
    if (ld_acquire_cta_shared_u32(cx.dep_ok) > seq) return true;
    if ((i & 255u) == 0 && (*cx.abort_flag != 0 || !clock.within_limit())) return false;
  }
}

// Round r of the persistent loop hands CTA c tile r*G + c in even rounds and r*G + (G-1-c) in odd
// rounds ("snake"): with the problems listed heaviest first, a CTA that drew an expensive tile in
// one round draws a cheap one (or none) in the next.
__device__ __forceinline__ int snake_tile(int round, int grid, int cta) {
  return round * grid + ((round & 1) ? (grid - 1 - cta) : cta);
}

// One GEMM phase: CTA c processes its snake sequence of tiles of the concatenated tile lists of
// `nprob` problems.  Tiles of one batch entry are consecutive (n fastest), so CTAs that run at
// the same time share operand tiles in L2.  Warp 0 = TMA producer, warp 1 = MMA issuer, warps
// 2.. = epilogue.  Returns true if a bounded wait ran out.  No CTA-wide sync inside.
// With Deps = FlowDeps tiles are dealt round-robin continuing from the previous phase (no snake) and
// ordered by the completion counters described above.
template <class Op, int RING, class EpiPatch, class Deps = NoDeps>
__device__ __forceinline__ bool gemm_phase(GemmCtx& cx, const GemmProblem<Op>* probs, const int nprob,
                                           EpiPatch patch, Deps deps = Deps{}) {
  constexpr int BT = Op::BT, NA = Op::NA, NB = Op::NB, NACC = Op::NACC;
  constexpr uint32_t kBTileBytes = BT * kBK * 2;  // one k-block of a B tile
  constexpr uint32_t kStageBytes = gemm_stage_bytes<Op>();
  constexpr uint32_t kAccCols = NACC * BT;
  constexpr int kMaxProb = 2;
  static_assert(2 * kAccCols <= 512, "double-buffered accumulators exceed tensor memory");
  // Multi-phase (dataflow) kernels run ops of different tile widths back to back without draining the pipeline: the two
  // accumulator buffers sit at fixed halves of the 512 allocated columns there, so that buffer 0 of one op can never
  // overlap buffer 1 of the previous op while its epilogue is still reading it.
  constexpr uint32_t kAccStride = Deps::kOn ? 256u : kAccCols;
  static_assert(BT % 64 == 0 && BT <= 256, "BT must be 64, 128, 192 or 256");

  constexpr bool SYM = op_symmetric<Op>::value;
  static_assert(!SYM || (BT == kBM && Op::NOUT == 1 && Deps::kOn), "symmetric ops: 128-wide tiles, one staged output, dataflow");
  constexpr bool SEG = op_segments<Op>::value;
  static_assert(!SEG || !Deps::kOn, "segments: one phase");
  constexpr bool SPLIT = op_split<Op>::value;
  static_assert(!SPLIT || (Op::NOUT == 0 && Op::kWarpTranspose && !Deps::kOn), "split contractions: direct epilogue, one phase");
  int tiles_of[kMaxProb], tn_of[kMaxProb], tm_of[kMaxProb], per_batch_of[kMaxProb], splits_of[kMaxProb];
  int total_tiles = 0;
#pragma unroll
  for (int p = 0; p < kMaxProb; ++p) {
    if (p < nprob) {
      tn_of[p] = (probs[p].N + BT - 1) / BT;
      tm_of[p] = (probs[p].M + kBM - 1) / kBM;
      per_batch_of[p] = SYM ? tm_of[p] * (tm_of[p] + 1) / 2 : tn_of[p] * tm_of[p];
      splits_of[p] = SPLIT && probs[p].splits > 1 ? probs[p].splits : 1;
      tiles_of[p] = per_batch_of[p] * probs[p].batch * splits_of[p];
    } else {
      tn_of[p] = tm_of[p] = per_batch_of[p] = splits_of[p] = 1;
      tiles_of[p] = 0;
    }
    total_tiles += tiles_of[p];
  }
  auto coord = [&](int tile) {
    TileCoord c;
    c.prob = 0;
    c.slot = c.split = 0;
    if (tile >= tiles_of[0]) {
      tile -= tiles_of[0];
      c.prob = 1;
      if constexpr (SPLIT) c.slot = tiles_of[0] / splits_of[0];
    }
    const int per_batch = per_batch_of[c.prob];
    c.batch = tile / per_batch;
    int r = tile - c.batch * per_batch;
    if constexpr (SPLIT) {  // the units of one batch entry and split are consecutive: they share operand tiles
      const int unit = c.batch;
      c.batch = unit / splits_of[c.prob];
      c.split = unit - c.batch * splits_of[c.prob];
      c.slot += c.batch * per_batch + r;
    }
    // a consumer of large intermediates walks the batch entries backwards: the entries its producer wrote last
    // are the ones still in L2
    if constexpr (Op::kReverseBatch) c.batch = probs[c.prob].batch - 1 - c.batch;
    if constexpr (SYM) {
      // tiles on and above the diagonal, row by row: row i holds the tiles (i, i) .. (i, T - 1)
      int i = 0, len = tm_of[c.prob];
      while (r >= len) { r -= len; ++i; --len; }
      c.m0 = i * kBM;
      c.n0 = (i + r) * BT;
    } else {
      c.m0 = (r / tn_of[c.prob]) * kBM;
      c.n0 = (r % tn_of[c.prob]) * BT;
    }
    return c;
  };

  // the k-blocks [first, last) of a unit
  auto k_range = [&](const GemmProblem<Op>& P, const TileCoord& tc, int& first, int& last) {
    first = 0;
    last = (P.K + kBK - 1) / kBK;
    if constexpr (SPLIT) {
      if (splits_of[tc.prob] > 1) {
        first = tc.split * P.kb_per_split;
        last = min(last, first + P.kb_per_split);
      }
    }
  };

  const int rounds = (total_tiles + gridDim.x - 1) / gridDim.x;
  const uint32_t rot0 = cx.rot;
  auto tile_at = [&](int r) {
    if constexpr (Deps::kOn) return r * static_cast<int>(gridDim.x) + static_cast<int>((blockIdx.x + gridDim.x - rot0) % gridDim.x);
    else return snake_tile(r, gridDim.x, blockIdx.x);
  };
  if constexpr (Deps::kOn) cx.rot = (cx.rot + static_cast<uint32_t>(total_tiles)) % gridDim.x;

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  bool failed = false;
  if (warp == 0) {
    // ---------------- TMA producer (warp-uniform, issued by its leader lane); the ring keeps running across tiles.
    // With the coordinates of every box worked out from the operand's description at the box itself this warp spent 200 to
    // 250 clocks per box (clocks inside the kernel), more than the products of a k-block take: a 64-wide pointwise tile of
    // 384 features, 30 boxes, took 7570 clocks, and takes 6740 with the cursors.
    const uint32_t leader = elect_leader();
    {
      for (int tile_i = 0; tile_i < rounds && !failed; ++tile_i) {
        const int tile = tile_at(tile_i);
        if (tile >= total_tiles) continue;
        const TileCoord tc = coord(tile);
        const GemmProblem<Op>& P = probs[tc.prob];
        int kb0, kb1;
        k_range(P, tc, kb0, kb1);
        const bool diagonal = SYM && tc.m0 == tc.n0;
        OperandCursor<kBM, SEG> ca[NA];
        OperandCursor<BT, SEG> cb[NB];
        int entry, segment;
        entry_of(P, tc.batch, entry, segment);
#pragma unroll
        for (int i = 0; i < NA; ++i) ca[i].start(&P.a[i], P.ai[i], tc.m0, kb0 * kBK, entry, segment);
#pragma unroll
        for (int i = 0; i < NB; ++i) cb[i].start(&P.b[i], P.bi[i], tc.n0, kb0 * kBK, entry, segment);
        const uint32_t bytes = diagonal ? NA * kATileBytes : kStageBytes;
        if constexpr (Deps::kOn) {
          if (!__all_sync(0xFFFFFFFFu, flow_wait_verified(cx, cx.ptile++))) { failed = true; break; }  // the scout warp checked this tile
          asm volatile("fence.proxy.async.global;" ::: "memory");
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&cx.empty_bar[cx.slot], cx.phase ^ 1, cx.abort_flag)) { failed = true; break; }
          const uint32_t bar = smem_u32(&cx.full_bar[cx.slot]);
          mbar_expect_tx_if(leader, bar, bytes);
          const uint32_t st = cx.smem_base + cx.slot * cx.stage_stride;
#pragma unroll
          for (int i = 0; i < NA; ++i) ca[i].load(leader, st + i * kATileBytes, bar);
          if (!diagonal) {
#pragma unroll
            for (int i = 0; i < NB; ++i) cb[i].load(leader, st + NA * kATileBytes + i * kBTileBytes, bar);
          }
          cx.next_stage<RING>();
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (warp-uniform, issued by its leader lane)
    const uint32_t leader = elect_leader();
    {
      for (int tile_i = 0; tile_i < rounds && !failed; ++tile_i) {
        const int tile = tile_at(tile_i);
        if (tile >= total_tiles) continue;
        const TileCoord tc = coord(tile);
        const GemmProblem<Op>& P = probs[tc.prob];
        int kb0, kb1;
        k_range(P, tc, kb0, kb1);
        const int num_kb = kb1 - kb0;
        const uint32_t as = cx.tcount & 1, aph = (cx.tcount >> 1) & 1;
        if (!mbar_wait_warp(&cx.acc_empty_bar[as], aph ^ 1, cx.abort_flag)) { failed = true; break; }
        tc_fence_after();
        const uint32_t acc_base = cx.tmem_base + as * kAccStride;
        const bool diagonal = SYM && tc.m0 == tc.n0;
        // K-major tiles: 16 elements = 32 bytes on inside the swizzled 128-byte row; MN-major tiles: 16 k-rows of 128 bytes on, 64-wide
        // atoms 8 KB apart (the leading offset)
        uint32_t idesc[Op::NTERMS], step_a[Op::NTERMS], step_b[Op::NTERMS];
#pragma unroll
        for (int t = 0; t < Op::NTERMS; ++t) {
          const int a_mn = P.ai[Op::term_a(t)].mn_major, b_mn = P.bi[Op::term_b(t)].mn_major;
          idesc[t] = make_idesc_bf16(kBM, Op::term_n(t), a_mn, b_mn);
          step_a[t] = a_mn ? 128 : 2;
          step_b[t] = b_mn ? 128 : 2;
        }
        const SmemDescBase desc(kAtomBytes);  // (K-major descriptors ignore the leading offset)
        for (int kb = 0; kb < num_kb; ++kb) {
          const uint32_t s = cx.slot;
          if (!mbar_wait_warp(&cx.full_bar[s], cx.phase, cx.abort_flag)) { failed = true; break; }
          tc_fence_after();
          const uint32_t st = (cx.smem_base + s * cx.stage_stride) >> 4;
#pragma unroll
          for (int t = 0; t < Op::NTERMS; ++t) {
            const uint32_t a_tile = st + Op::term_a(t) * (kATileBytes >> 4);
            uint32_t b_off = NA * kATileBytes + Op::term_b(t) * kBTileBytes;
            if constexpr (SYM) {
              if (diagonal) b_off = Op::diag_a(Op::term_b(t)) * kATileBytes;
            }
            const uint32_t b_tile = st + (b_off >> 4);
#pragma unroll
            for (int k4 = 0; k4 < kBK / kUmmaK; ++k4) {
              const uint32_t acc = (kb > 0 || k4 > 0 || !Op::term_first(t)) ? 1u : 0u;
              umma_bf16_if(leader, acc_base + Op::term_col(t), desc.at(a_tile + k4 * step_a[t]), desc.at(b_tile + k4 * step_b[t]),
                           idesc[t], acc);
            }
          }
          umma_commit_if(leader, &cx.empty_bar[s]);  // frees the stage once these MMAs have read it
          cx.next_stage<RING>();
        }
        if (!failed) umma_commit_if(leader, &cx.acc_full_bar[as]);
        ++cx.tcount;
      }
    }
  } else if constexpr (Deps::kOn) {
    if (warp == 2 + kEpiWarps) {
      // ---------------- dependency scout (dataflow kernels only): one thread verifies, in tile order,
      // that every tile's inputs are complete and publishes the count of verified tiles
      if (lane == 0) {
        for (int tile_i = 0; tile_i < rounds && !failed; ++tile_i) {
          const int tile = tile_at(tile_i);
          if (tile >= total_tiles) continue;
          const TileCoord tc = coord(tile);
          if (!dep_wait(deps.counter[tc.prob] + tc.batch, deps.need[tc.prob], cx.abort_flag)) { failed = true; break; }
          st_release_cta_shared_u32(cx.dep_ok, ++cx.ptile);
        }
      }
      return failed;
    }
    // ---------------- epilogue of a dataflow tile: rounded rows go from registers straight to global memory, 64 bytes per thread
    // and 32 columns.  What counts here is how soon the next phase of the matrix may load.  Clocks inside the kernel at 8 matrices of
    // side 384 (a tile per SM and phase): bulk stores from a staging tile took 3170 clocks from the hand-over to the counter, and
    // 5300 with the chip full; stores from registers and the release take 1470.  The loading warp's fence between counter and
    // loads, for global memory alone, costs 900 clocks less than one for all proxies' state spaces.  Without staging tiles the
    // ring takes all of shared memory.  8 matrices 97.6 -> 72.9 us a launch, 64 of them (power-limited in a long call) 197 -> 160.
    static_assert(Op::NOUT == 1, "one output");
    const int quarter = warp & 3, half = (warp - 2) >> 2, row_local = quarter * 32 + lane;
    const uint32_t scratch = cx.staging + (warp - 2) * (32 * 80);
    for (int tile_i = 0; tile_i < rounds; ++tile_i) {
      const int tile = tile_at(tile_i);
      if (tile >= total_tiles) continue;
      const TileCoord tc = coord(tile);
      const GemmProblem<Op>& P = probs[tc.prob];
      typename Op::Epi ep = P.ep;
      patch(ep, tc.prob);
      const uint32_t as = cx.tcount & 1, aph = (cx.tcount >> 1) & 1;
      const int row = tc.m0 + row_local;
      typename Op::Prefetch pf;
      Op::prefetch(ep, tc.batch, row, tc.n0, half, P.M, P.N, pf);
      // A warp whose wait ran out tells the others at the tile's barrier, in the word of the tile's parity: by the time it could
      // raise that word for another tile, all of them have looked.
      const bool got = mbar_wait(&cx.acc_full_bar[as], aph, cx.abort_flag);
      if (!got) cx.abort_flag[1 + as] = 1;
      tc_fence_after();
      const uint32_t acc_base = cx.tmem_base + as * kAccStride + (static_cast<uint32_t>(quarter * 32) << 16);
      const int64_t ld = P.oi[0].ld;
      bf16* const out = static_cast<bf16*>(P.oi[0].ptr) + tc.batch * P.oi[0].bs;
      const bool wide = P.oi[0].wide != 0;
      auto release = [&]() {  // all TMEM reads of this warp are complete: hand the buffer back
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&cx.acc_empty_bar[as]);
      };
      if (tc.n0 + half * 32 >= P.N) release();
      for (int c = half * 32; c < BT; c += 64) {
        const int left = P.N - (tc.n0 + c);  // columns; a multiple of 8
        if (left <= 0) break;                // warp-uniform
        float v[1][32], ov[1][32];
        {
          uint32_t bits[32];
          tmem_ld32(acc_base + c, bits);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[0][j] = __uint_as_float(bits[j]);
        }
        if (c + 64 >= BT || left <= 64) release();
        Op::epilogue_staged(ep, tc.batch, row, tc.n0 + c, P.M, P.N, v, ov, pf);
        uint32_t w[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2(ov[0][2 * j], ov[0][2 * j + 1]);
        if (got && row < P.M) {
          bf16* const p = out + row * ld + tc.n0 + c;
          if (wide && left >= 32) {
            st_global_32(p, w);
            st_global_32(p + 16, w + 8);
          } else {
#pragma unroll
            for (int g = 0; g < 4; ++g)
              if (g * 8 < left) st_global_16(p + g * 8, w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
          }
        }
        if constexpr (SYM) {
          if (tc.m0 != tc.n0) {  // the block transposed: through the warp's scratch, four lanes per row of 64 bytes
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const uint16_t h = static_cast<uint16_t>((j & 1) ? w[j >> 1] >> 16 : w[j >> 1]);
              asm volatile("st.shared.b16 [%0], %1;" ::"r"(scratch + j * 80 + lane * 2), "h"(h) : "memory");
            }
            __syncwarp();
            const int u = lane & 3, col = tc.m0 + quarter * 32 + u * 8;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int rr = i * 8 + (lane >> 2), at = tc.n0 + c + rr;
              uint32_t x[4];
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3])
                           : "r"(scratch + rr * 80 + u * 16)
                           : "memory");
              if (got && at < P.N && col < P.M) st_global_16(out + at * ld + col, x[0], x[1], x[2], x[3]);
            }
          }
        }
        __syncwarp();  // (scratch; and the next tensor-memory load wants the warp together, whose last rows may lie past M)
      }
      // (the loading warps of other SMs have the proxy fence between the counter and their bulk loads of these rows)
      named_barrier_sync(2, kEpiWarps * 32);
      if (cx.abort_flag[1 + as] != 0) { failed = true; break; }
      if (threadIdx.x == 64) red_release_gpu_u32(deps.counter[tc.prob] + tc.batch, 1u);
      ++cx.tcount;
    }
  } else {
    // ---------------- epilogue: warp w may only touch TMEM lanes [32*(w%4), 32*(w%4)+32); the two
    // warps of a lane quarter take alternate 32-column chunks.  Ops with NOUT > 0 round their
    // results to bf16 into swizzled shared-memory tiles that one thread hands to TMA stores
    // (full-line writes, clipped by the output map); other ops store from registers.
    constexpr int NOUT = Op::NOUT;
    constexpr int NSTG = NOUT;  // staging tiles
    constexpr int kEpiThreads = kEpiWarps * 32;
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const bool elected = threadIdx.x == 64;
    const int row_local = quarter * 32 + lane;
    auto tile_of_round = [&](int r) {
      if (r >= rounds) return -1;
      const int t = tile_at(r);
      return t < total_tiles ? t : -1;
    };
    [[maybe_unused]] typename Op::Prefetch pf_next;
    [[maybe_unused]] auto fetch = [&](int tile) {
      if (tile < 0) return;
      const TileCoord tc = coord(tile);
      const GemmProblem<Op>& P = probs[tc.prob];
      Op::prefetch(P.ep, tc.batch, tc.m0 + row_local, tc.n0, half, P.M, P.N, pf_next);
    };
    if constexpr (op_fetch_ahead<Op>::value) fetch(tile_of_round(0));
    for (int tile_i = 0; tile_i < rounds; ++tile_i) {
      const int tile = tile_of_round(tile_i);
      if (tile < 0) continue;
      const TileCoord tc = coord(tile);
      const GemmProblem<Op>& P = probs[tc.prob];
      typename Op::Epi ep = P.ep;
      patch(ep, tc.prob);
      const uint32_t stg = cx.staging;
      const uint32_t as = cx.tcount & 1, aph = (cx.tcount >> 1) & 1;
      const int row = tc.m0 + row_local;
      // global operands of the epilogue are fetched while the tile's MMAs are still running, or a tile ahead
      typename Op::Prefetch pf;
      if constexpr (op_fetch_ahead<Op>::value) {
        pf = pf_next;
        fetch(tile_of_round(tile_i + 1));
      } else {
        Op::prefetch(ep, tc.batch, row, tc.n0, half, P.M, P.N, pf);
      }
      bool got = mbar_wait(&cx.acc_full_bar[as], aph, cx.abort_flag);
      tc_fence_after();
      const uint32_t acc_base = cx.tmem_base + as * kAccStride + (static_cast<uint32_t>(quarter * 32) << 16);
      if constexpr (NOUT > 0) {
        // A warp whose wait ran out must not leave the others stuck at a named barrier: it raises
        // a flag that only epilogue warps write, and every warp decides after the barrier.
        if (!got) cx.abort_flag[1] = 1;
        // the previous tile's stores must have finished reading the staging tile
        if (elected) bulk_wait_read_all();
        named_barrier_sync(1, kEpiThreads);
        if (cx.abort_flag[1] != 0) { failed = true; break; }
      } else {
        if constexpr (SPLIT) {
          // (as above: the warps of a split tile meet at named barriers, so they give up together)
          if (splits_of[tc.prob] > 1) {
            if (!got) cx.abort_flag[1] = 1;
            named_barrier_sync(1, kEpiThreads);
            got = cx.abort_flag[1] == 0;
          }
        }
        if (!got) { failed = true; break; }
      }
      if constexpr (SPLIT) {
        if (splits_of[tc.prob] > 1) {
          // this unit's sums: 32 x 32 blocks, sixteen bytes per lane and store
          const int splits = splits_of[tc.prob];
          constexpr int kTileF4 = kBM * BT / 4;
          float4* const tile_part = reinterpret_cast<float4*>(P.part) + static_cast<int64_t>(tc.slot) * splits * kTileF4;
          float4* const mine = tile_part + static_cast<int64_t>(tc.split) * kTileF4;
          for (int c = half * 32; c < BT; c += 64) {
            if (tc.n0 + c >= P.N) break;
            uint32_t bits[32];
            tmem_ld32(acc_base + c, bits);
            tmem_ld_wait();
            float4* const blk = mine + (quarter * (BT / 32) + (c >> 5)) * 256 + lane;
#pragma unroll
            for (int g = 0; g < 8; ++g)
              __stcg(blk + g * 32, make_float4(__uint_as_float(bits[g * 4]), __uint_as_float(bits[g * 4 + 1]),
                                               __uint_as_float(bits[g * 4 + 2]), __uint_as_float(bits[g * 4 + 3])));
          }
          tc_fence_before();
          __threadfence();
          __syncwarp();
          if (lane == 0) mbar_arrive(&cx.acc_empty_bar[as]);
          named_barrier_sync(2, kEpiThreads);
          if (elected) {
            const bool last = atomicAdd(P.count + tc.slot, 1u) == static_cast<uint32_t>(splits - 1);
            __threadfence();
            if (last) P.count[tc.slot] = 0;
            *cx.last_unit = last;
          }
          named_barrier_sync(1, kEpiThreads);
          if (*cx.last_unit != 0) {
            for (int c = half * 32; c < BT; c += 64) {
              if (tc.n0 + c >= P.N) break;
              float v[NACC][32];
#pragma unroll
              for (int j = 0; j < 32; ++j) v[0][j] = 0.f;
              const float4* blk = tile_part + (quarter * (BT / 32) + (c >> 5)) * 256 + lane;
              for (int s = 0; s < splits; ++s, blk += kTileF4) {
                float4 x[8];
#pragma unroll
                for (int g = 0; g < 8; ++g) x[g] = __ldcg(blk + g * 32);
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                  v[0][g * 4] += x[g].x; v[0][g * 4 + 1] += x[g].y; v[0][g * 4 + 2] += x[g].z; v[0][g * 4 + 3] += x[g].w;
                }
              }
              Op::epilogue_warp(ep, tc.batch, tc.m0 + quarter * 32, tc.n0 + c, P.M, P.N, v, pf,
                                cx.staging + (warp - 2) * (32 * 144), lane);
            }
            if constexpr (Op::kTileReduce) {
              float tv = Op::tile_value(pf);
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) tv += __shfl_xor_sync(0xFFFFFFFFu, tv, o);
              if (lane == 0) Op::tile_store(ep, tc.batch, tc.m0 / kBM, tc.n0 / BT, warp - 2, tv);
            }
          }
          ++cx.tcount;
          continue;
        }
      }
      for (int c = half * 32; c < BT; c += 64) {
        if (tc.n0 + c >= P.N) break;  // warp-uniform
        float v[NACC][32];
        {
          uint32_t bits[NACC][32];
#pragma unroll
          for (int a = 0; a < NACC; ++a) tmem_ld32(acc_base + a * BT + c, bits[a]);
          tmem_ld_wait();  // one wait for the loads of all accumulators
#pragma unroll
          for (int a = 0; a < NACC; ++a)
#pragma unroll
            for (int j = 0; j < 32; ++j) v[a][j] = __uint_as_float(bits[a][j]);
        }
        if constexpr (NOUT > 0) {
          float ov[NSTG > 0 ? NSTG : 1][32];
          const uint32_t rowaddr = (c >> 6) * (kBM * 128) + row_local * 128;
          const uint32_t unit0 = (c & 63) >> 3;
          Op::epilogue_staged(ep, tc.batch, row, tc.n0 + c, P.M, P.N, v, ov, pf);
#pragma unroll
          for (int o = 0; o < NSTG; ++o) {
            const uint32_t base = stg + o * (kBM * BT * 2) + rowaddr;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint32_t addr = base + (((unit0 + g) ^ (row_local & 7)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
                           "r"(pack_bf16x2(ov[o][g * 8 + 0], ov[o][g * 8 + 1])),
                           "r"(pack_bf16x2(ov[o][g * 8 + 2], ov[o][g * 8 + 3])),
                           "r"(pack_bf16x2(ov[o][g * 8 + 4], ov[o][g * 8 + 5])),
                           "r"(pack_bf16x2(ov[o][g * 8 + 6], ov[o][g * 8 + 7]))
                           : "memory");
            }
          }
        } else {
          if constexpr (Op::kWarpTranspose)
            Op::epilogue_warp(ep, tc.batch, tc.m0 + quarter * 32, tc.n0 + c, P.M, P.N, v, pf,
                              cx.staging + (warp - 2) * (32 * 144), lane);
          else
            Op::epilogue(ep, tc.batch, row, tc.n0 + c, P.M, P.N, v, pf, c >> 6);
        }
      }
      // all TMEM reads of this warp are complete (wait::ld above): hand the buffer back
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&cx.acc_empty_bar[as]);
      if constexpr (Op::kTileReduce) {
        // per-tile, per-warp reduction of a per-thread value (no cross-warp synchronisation: the
        // consumer adds the eight warp partials of every tile in a fixed order)
        float tv = Op::tile_value(pf);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tv += __shfl_xor_sync(0xFFFFFFFFu, tv, o);
        if (lane == 0) Op::tile_store(ep, tc.batch, tc.m0 / kBM, tc.n0 / BT, warp - 2, tv);
      }
      if constexpr (NOUT > 0) {
        fence_async_proxy();
        named_barrier_sync(2, kEpiThreads);
        if (elected) {
          int entry, segment;
          entry_of(P, tc.batch, entry, segment);
#pragma unroll
          for (int o = 0; o < NOUT; ++o) {
            if (!P.oi[o].enabled || Op::skip_store(ep, o)) continue;
            for (int pnl = 0; pnl < BT / 64; ++pnl) {
              if (tc.n0 + pnl * 64 >= P.N) break;
              const uint32_t src = stg + o * (kBM * BT * 2) + pnl * (kBM * 128);
              const int col = P.oi[o].col_off + tc.n0 + pnl * 64, at = P.oi[o].row_off + tc.m0, b = P.oi[o].batch_off + entry;
              if constexpr (SEG) tma_store_4d(&P.out[o], src, col, at, b, segment);
              else tma_store_3d(&P.out[o], src, col, at, b);
            }
          }
          bulk_commit_group();
        }
      }
      ++cx.tcount;
    }
    if constexpr (NOUT > 0) {
      if (elected) bulk_wait_all();  // this CTA's output tiles are in global memory
    }
  }
  return failed;
}

// Carves barriers out of shared memory behind a ring of `ring` stages of `stage_stride` bytes,
// initialises them and allocates `tmem_cols` columns of tensor memory.  Ends with a CTA-wide sync.
__device__ __forceinline__ void gemm_setup(GemmCtx& cx, uint8_t* smem_raw, int ring, uint32_t stage_stride,
                                           uint32_t staging_bytes, uint32_t tmem_cols) {
  const uint32_t raw_addr = smem_u32(smem_raw);
  cx.smem_base = (raw_addr + 1023u) & ~1023u;
  cx.stage_stride = stage_stride;
  cx.staging = cx.smem_base + ring * stage_stride;
  uint8_t* aligned = smem_raw + (cx.smem_base - raw_addr);
  cx.full_bar = reinterpret_cast<uint64_t*>(aligned + ring * stage_stride + staging_bytes);
  cx.empty_bar = cx.full_bar + ring;
  cx.acc_full_bar = cx.empty_bar + ring;    // [2]
  cx.acc_empty_bar = cx.acc_full_bar + 2;   // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(cx.acc_empty_bar + 2);
  cx.abort_flag = tmem_slot + 1;  // [3]
  cx.dep_ok = tmem_slot + 4;
  cx.last_unit = tmem_slot + 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ring; ++s) {
      mbar_init(&cx.full_bar[s], 1);
      mbar_init(&cx.empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&cx.acc_full_bar[s], 1);
      mbar_init(&cx.acc_empty_bar[s], kEpiWarps);
    }
    cx.abort_flag[0] = 0;
    cx.abort_flag[1] = 0;
    cx.abort_flag[2] = 0;
    *cx.dep_ok = 0;
    fence_mbar_init();
  }
  if ((threadIdx.x >> 5) == 1) {
    tmem_alloc(tmem_slot, tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cx.tmem_base = uniform(*tmem_slot);
}

__device__ __forceinline__ void gemm_teardown(GemmCtx& cx, bool failed, int32_t* status, uint32_t tmem_cols) {
  if (failed) {
    *cx.abort_flag = 1;
    report_timeout(status);
  }
  tc_fence_before();
  __syncthreads();
  if (*cx.abort_flag && threadIdx.x == 0) {
    // let bulk copies still in flight land before shared memory is released
    for (int i = 0; i < 256; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if ((threadIdx.x >> 5) == 1) tmem_dealloc(cx.tmem_base, tmem_cols);
}

// Whether an earlier launch has given up.  Calls on other streams may share the word, so it can change while a CTA reads it:
// the epilogue warps decide together (they would wait for one another at named barriers, which have no time limit; the barrier
// here costs nothing, they have to wait for the first tile anyway).  The other warps wait at mbarriers alone, with a limit.
// The answer has to be uniform for the compiler too: with a decision per thread, or one barrier for all warps, the launches of
// small calls took 0.2 to 0.7 us longer (4 entries of 384, 2048 tokens: apply 15.5 us, 16.1 and 16.1 that way).
__device__ __forceinline__ bool earlier_launch_failed(const int32_t* status) {
  bool set = *reinterpret_cast<const volatile int32_t*>(status) != kStatusOk;
  if (uniform_warp_index() >= 2) set = named_barrier_any(1, kEpiWarps * 32, set);
  return uniform(set) != 0;
}

// Persistent single-phase kernel.  The prologue (barriers, tensor memory, descriptor prefetch)
// touches no global memory and may overlap the tail of the previous kernel in the stream.
template <class Op, int NPROB>
__global__ void __launch_bounds__(kGemmThreadsV2, 1)
umma_gemm_kernel(const __grid_constant__ GemmArgs<Op, NPROB> args, const int nprob) {
  static_assert(NPROB <= 2, "at most two problems per launch");
  extern __shared__ uint8_t smem_raw[];
  constexpr uint32_t kTmemCols = tmem_cols_pow2(2 * Op::NACC * Op::BT);
  GemmCtx cx;
  gemm_setup(cx, smem_raw, Op::STAGES, gemm_stage_bytes<Op>(), gemm_staging_bytes<Op>(), kTmemCols);
  if (threadIdx.x == 32) {
    for (int p = 0; p < nprob; ++p) {
#pragma unroll
      for (int i = 0; i < Op::NA; ++i) tma_prefetch_desc(&args.prob[p].a[i]);
#pragma unroll
      for (int i = 0; i < Op::NB; ++i) tma_prefetch_desc(&args.prob[p].b[i]);
#pragma unroll
      for (int i = 0; i < Op::NOUT; ++i) tma_prefetch_desc(&args.prob[p].out[i]);
    }
  }
  griddep_launch_dependents();
  griddep_wait();
  bool failed = false;
  // an earlier launch gave up: do nothing but release the resources
  if (!earlier_launch_failed(args.status))
    failed = gemm_phase<Op, Op::STAGES>(cx, args.prob, nprob, NoPatch{});
  gemm_teardown(cx, failed, args.status, kTmemCols);
}

}  // namespace lact
