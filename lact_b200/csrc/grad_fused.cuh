// Fast-weight gradient of heads of 128 features in one launch: the pointwise stage and the token contraction of one (entry, slice of 32
// hidden features) per CTA, the planes between them in shared memory.  Per tile of 128 tokens:
//   y0 | y2 = k [w0; w2]^T (128 x 64), dh = v w1 (128 x 32)                     tensor memory, two buffers of 96 columns
//   dy0 | dy2, hidden * lr1 (as in OpFwGradPointwise), bf16, [128 tokens][64] and [128][32], shared memory
//   [dw0; dw2]^T += k^T [dy0 | dy2] (128 x 64), dw1 += v^T hidden (128 x 32)     tensor memory
// Warp 0 loads the slice's weights once and the tiles of k and v through rings of three and two; warp 1 issues the products of the first stage, warp 10
// those of the second (one warp for both spent 800 of 2200 clocks per tile on looking at barriers); warps 2-9 are the epilogue (two
// threads per token).  k and v serve both
// stages from the same shared memory: K-major for the first, MN-major (tokens = k) for the second.  A CTA takes all tokens of the update in
// their order, as a tile of the contraction alone does, so the gradient has the bits of the two launches.  So have the sums of squares
// that Newton-Schulz divides by (one flipped rounding of that norm is carried far by the updates that follow): they are added up in the
// order of the contraction's tiles, 128 columns wide, whose warps take blocks of 32 columns two apart.  For dw1 these are slices two
// apart, the two CTAs of a cluster.
// What bounds it (clocks inside the kernel, 12 entries of 128 x 256, 1560 tokens, 96 CTAs): 3600 until the first products, then 1720 per tile
// (first stage 750 with its waits, epilogue 1080, second stage 700, the reload of v 760: v's ring of two is what 227 KB leave), 5000 for
// the momentum state and the stores, which run once and wait for their instructions.  Slices of 64, whose planes are 48 KB, left two
// stages for k and v and took 3300 a tile on half the CTAs.  An update of these sizes: pointwise stage 17 us and contraction 17 us, now
// 24 in one launch (video clip 1420 -> 1278 us).
#pragma once
#include "ops.cuh"

namespace lact {

struct GradFusedArgs {
  CUtensorMap k, v;     // box [128 tokens][64]
  CUtensorMap w02, w1;  // box [32 rows][64]; [128 rows][32], 64-byte swizzle
  EpiFwGrad lr;
  EpiDW e[2];           // [dw0; dw2] and dw1 (`partial`: as OpDW<128> leaves it)
  int32_t start, len, H;
  int32_t* status;
};

constexpr int kGradD = 128, kGradSlice = 32, kGradThreads = kGemmThreadsV2 + 32;
struct GradSmem {
  static constexpr uint32_t kBox = 128 * 128, kHalfBox = 128 * 64;   // [128][64] and [128][32] bf16
  static constexpr uint32_t kW = 0, kW1 = kBox, kK = kW1 + kHalfBox, kV = kK + 6 * kBox, kDy = kV + 4 * kBox, kHid = kDy + kBox,
                            kBars = kHid + kHalfBox;   // three tiles of k, two of v
  static constexpr uint32_t kSums = kBars + 256, kBytes = kSums + 12 * 32 * 4 + 1024;   // squares per lane: eight blocks of [dw0; dw2], the peer's four of dw1
};
static_assert(GradSmem::kK % 1024 == 0 && GradSmem::kDy % 1024 == 0 && GradSmem::kHid % 1024 == 0, "swizzled tiles");
static_assert(kEpiWarps * 32 * 144 <= 6 * GradSmem::kBox, "the gradient's epilogue works in the memory of k");

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGradThreads, 1) grad_gemm_kernel(const __grid_constant__ GradFusedArgs a) {
  using SM = GradSmem;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + SM::kBars);
  uint64_t* w_full = bars;
  uint64_t* k_full = bars + 1;        // [3]
  uint64_t* k_empty = bars + 4;       // [3]
  uint64_t* v_full = bars + 7;        // [2]
  uint64_t* v_empty = bars + 9;       // [2]
  uint64_t* y_full = bars + 11;       // [2]
  uint64_t* y_empty = bars + 13;      // [2], 8 arrivals
  uint64_t* planes_full = bars + 15;  // 8 arrivals
  uint64_t* planes_empty = bars + 16;
  uint64_t* acc_full = bars + 17;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* sums = reinterpret_cast<float*>(aligned + SM::kSums);

  const uint32_t window = base & 0x3FFFFu;   // as descriptors have it (in a cluster the address holds the CTA's rank above)

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&y_full[s], 1);
      mbar_init(&y_empty[s], kEpiWarps);
    }
    mbar_init(planes_full, kEpiWarps);
    mbar_init(planes_empty, 1);
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&a.k);
    tma_prefetch_desc(&a.v);
    tma_prefetch_desc(&a.w02);
    tma_prefetch_desc(&a.w1);
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync();   // (both CTAs run: one stores into the other's shared memory at the end)
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);   // y of stage s: columns 96 s to 96 s + 95; [dw0; dw2]^T: 192 to 255; dw1: 256 to 287
  griddep_launch_dependents();
  griddep_wait();

  const int slices = a.H / kGradSlice;
  // cluster c of an entry: slices 4 (c / 2) + c % 2 and the one two on
  const int batch = blockIdx.x / slices, at = blockIdx.x % slices, slice = (at & ~3) + ((at >> 1) & 1) + (at & 1) * 2;
  const int tiles = (a.len + 127) / 128;
  auto load = [&](uint32_t leader, const CUtensorMap* map, uint64_t* full, uint32_t at, int i) {
    mbar_expect_tx_if(leader, full, 2 * SM::kBox);
    for (int j = 0; j < 2; ++j) tma_load_3d_if(leader, at + j * SM::kBox, map, smem_u32(full), 64 * j, a.start + i * 128, batch);
  };
  if (warp == 0) {   // the first tile and the weights are on their way while the status word is read
    const uint32_t leader = elect_leader();
    load(leader, &a.k, &k_full[0], base + SM::kK, 0);
    mbar_expect_tx_if(leader, w_full, SM::kBox + SM::kHalfBox);
    for (int j = 0; j < 2; ++j) {
      tma_load_3d_if(leader, base + SM::kW + j * SM::kHalfBox, &a.w02, smem_u32(w_full), 64 * j, slice * kGradSlice, batch);
      tma_load_3d_if(leader, base + SM::kW + j * SM::kHalfBox + SM::kHalfBox / 2, &a.w02, smem_u32(w_full), 64 * j,
                     a.H + slice * kGradSlice, batch);
    }
    tma_load_3d_if(leader, base + SM::kW1, &a.w1, smem_u32(w_full), slice * kGradSlice, 0, batch);
    load(leader, &a.v, &v_full[0], base + SM::kV, 0);
  }
  // (the second issuing warp waits at mbarriers alone and reads the word by itself)
  bool failed = warp < 2 + kEpiWarps ? earlier_launch_failed(a.status)
                                     : uniform(static_cast<uint32_t>(*reinterpret_cast<volatile int32_t*>(a.status))) != kStatusOk;
  const bool skip = failed;
  const uint32_t rank = cluster_rank();
  float own1 = 0.f;   // this lane's share of the squares of dw1

  if (skip) {
    // (shared memory stays until the copies have landed)
    if (warp == 0 && !(mbar_wait_warp(w_full, 0, abort_flag) && mbar_wait_warp(&k_full[0], 0, abort_flag) && mbar_wait_warp(&v_full[0], 0, abort_flag)))
      *abort_flag = 1;
  } else if (warp == 0) {
    const uint32_t leader = elect_leader();
    uint32_t ks = 1, kph = 1;   // stage of k in turn, parity of its release
    for (int i = 1; i < tiles; ++i) {
      const uint32_t s = i & 1;
      if (!mbar_wait_warp(&k_empty[ks], kph, abort_flag)) { failed = true; break; }
      load(leader, &a.k, &k_full[ks], base + SM::kK + ks * 2 * SM::kBox, i);
      if (++ks == 3) { ks = 0; kph ^= 1; }
      if (!mbar_wait_warp(&v_empty[s], ((i >> 1) & 1) ^ 1, abort_flag)) { failed = true; break; }
      load(leader, &a.v, &v_full[s], base + SM::kV + s * 2 * SM::kBox, i);
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_leader();
    const uint32_t id_y = make_idesc_bf16(128, 64, 0, 0), id_h = make_idesc_bf16(128, 32, 0, 1);
    const SmemDescBase desc(0), narrow = SmemDescBase::half_atom();
    constexpr uint32_t kB16 = SM::kBox >> 4, kHB16 = SM::kHalfBox >> 4;
    const uint32_t w = (window + SM::kW) >> 4, w1 = (window + SM::kW1) >> 4, k0 = (window + SM::kK) >> 4, v0 = (window + SM::kV) >> 4;
    uint32_t ks = 0, kph = 0;
    failed = !mbar_wait_warp(w_full, 0, abort_flag);
    for (int i = 0; i < tiles && !failed; ++i) {
      const uint32_t s = i & 1, ph = (i >> 1) & 1, kt = k0 + ks * 2 * kB16, vt = v0 + s * 2 * kB16;
      if (!mbar_wait_warp(&y_empty[s], ph ^ 1, abort_flag) || !mbar_wait_warp(&k_full[ks], kph, abort_flag)) { failed = true; break; }
      if (++ks == 3) { ks = 0; kph ^= 1; }
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16_if(leader, tmem + s * 96, desc.at(kt + (kk >> 2) * kB16 + (kk & 3) * 2), desc.at(w + (kk >> 2) * kHB16 + (kk & 3) * 2), id_y,
                     kk != 0);
      if (!mbar_wait_warp(&v_full[s], ph, abort_flag)) { failed = true; break; }
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16_if(leader, tmem + s * 96 + 64, desc.at(vt + (kk >> 2) * kB16 + (kk & 3) * 2), narrow.at(w1 + kk * 64), id_h, kk != 0);
      umma_commit_if(leader, &y_full[s]);
    }
  } else if (warp == 2 + kEpiWarps) {
    const uint32_t leader = elect_leader();
    const uint32_t id_02 = make_idesc_bf16(128, 64, 1, 1), id_1 = make_idesc_bf16(128, 32, 1, 1);
    const SmemDescBase desc(SM::kBox), narrow = SmemDescBase::half_atom();   // (atoms of 64 features are boxes apart)
    constexpr uint32_t kB16 = SM::kBox >> 4;
    const uint32_t k0 = (window + SM::kK) >> 4, v0 = (window + SM::kV) >> 4, dy = (window + SM::kDy) >> 4, hid = (window + SM::kHid) >> 4;
    uint32_t ks = 0;
    for (int i = 0; i < tiles; ++i) {
      const uint32_t s = i & 1, kt = k0 + ks * 2 * kB16, vt = v0 + s * 2 * kB16;
      // (the planes were made from this tile's k and v: both have landed)
      if (!mbar_wait_warp(planes_full, i & 1, abort_flag)) { failed = true; break; }
      tc_fence_after();
      // (v first: its ring is the shorter one)
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) umma_bf16_if(leader, tmem + 256, desc.at(vt + kk * 128), narrow.at(hid + kk * 64), id_1, (i | kk) != 0);
      umma_commit_if(leader, &v_empty[s]);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) umma_bf16_if(leader, tmem + 192, desc.at(kt + kk * 128), desc.at(dy + kk * 128), id_02, (i | kk) != 0);
      umma_commit_if(leader, &k_empty[ks]);
      umma_commit_if(leader, planes_empty);
      if (++ks == 3) ks = 0;
    }
    if (!failed) umma_commit_if(leader, acc_full);
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2, r = quarter * 32 + lane;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    using Op = OpFwGradPointwise;
    typename Op::Prefetch pf, pf_next;
    Op::prefetch(a.lr, batch, r, 0, 0, a.len, 0, pf_next);
    for (int i = 0; i < tiles; ++i) {
      const uint32_t s = i & 1, ph = (i >> 1) & 1;
      pf = pf_next;
      if (i + 1 < tiles) Op::prefetch(a.lr, batch, (i + 1) * 128 + r, 0, 0, a.len, 0, pf_next);
      if (!mbar_wait_warp(&y_full[s], ph, abort_flag)) { failed = true; break; }
      tc_fence_after();
      float v[3][16], o[3][16];
      {
        uint32_t bits[3][16];
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_ld16(lanes + s * 96 + p * 32 + half * 16, bits[p]);
        tmem_ld_wait();
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int j = 0; j < 16; ++j) v[p][j] = __uint_as_float(bits[p][j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&y_empty[s]);
      Op::pointwise<16>(a.lr, v, o, pf);
      // rows past the end are zeros in both contractions (0 times a weight that is not finite is none)
      if (__builtin_expect(i * 128 + r >= a.len, 0)) {
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int j = 0; j < 16; ++j) o[p][j] = 0.f;
      }
      if (i > 0 && !mbar_wait_warp(planes_empty, (i - 1) & 1, abort_flag)) { failed = true; break; }
      // dy0, dy2: halves of rows of 128 bytes; hidden: rows of 64 bytes
      const uint32_t dy = base + SM::kDy + r * 128, hid = base + SM::kHid + r * 64;
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const uint32_t at = p < 2 ? dy + (((p * 4 + half * 2 + g) ^ (r & 7)) << 4) : hid + (((half * 2 + g) ^ ((r >> 1) & 3)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(pack_bf16x2(o[p][g * 8], o[p][g * 8 + 1])),
                       "r"(pack_bf16x2(o[p][g * 8 + 2], o[p][g * 8 + 3])), "r"(pack_bf16x2(o[p][g * 8 + 4], o[p][g * 8 + 5])),
                       "r"(pack_bf16x2(o[p][g * 8 + 6], o[p][g * 8 + 7]))
                       : "memory");
        }
      fence_async_proxy();
      __syncwarp();
      if (lane == 0) mbar_arrive(planes_full);
    }
    // A 32 x 32 block of the transposed [dw0; dw2] per warp (`half`: of w0 or of w2), one of dw1 per warp of the first half.  The state they
    // are added to is read while the last products run.
    const int row02 = half * a.H + slice * kGradSlice, col1 = slice * kGradSlice;
    float4 old[8], old1[8] = {};
    float bt = a.e[0].load_state(batch, row02, quarter * 32, 2 * a.H, kGradD, lane, old), bt1 = 0.f;
    if (half == 0) bt1 = a.e[1].load_state(batch, quarter * 32, col1, kGradD, a.H, lane, old1);
    if (!failed && !mbar_wait_warp(acc_full, 0, abort_flag)) failed = true;
    if (failed) *abort_flag = 1;
    // (the memory of k is all the warps' scratch now, and they give up together)
    failed = named_barrier_any(1, kEpiWarps * 32, failed);
    if (!failed) {
      tc_fence_after();
      const uint32_t scratch = base + SM::kK + (warp - 2) * (32 * 144);
      const bool want = a.e[0].partial != nullptr;
      // (a loop: this code runs once per launch and waits for its instructions)
#pragma unroll 1
      for (int n = 0; n < 2 - half; ++n) {
        const EpiDW& e = a.e[n];
        uint32_t x[32];
        float v[32];
        tmem_ld32(lanes + (n == 0 ? 192 + half * 32 : 256), x);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(x[j]);
        if (n == 0) e.put_block<true>(v, scratch, lane);
        else e.put_block<false>(v, scratch, lane);
        const float squares = e.add_block(batch, n == 0 ? row02 : quarter * 32, n == 0 ? quarter * 32 : col1, n == 0 ? 2 * a.H : kGradD,
                                          n == 0 ? kGradD : a.H, scratch, lane, want, old, bt);
        if (n == 0) sums[(half * 4 + quarter) * 32 + lane] = squares;
        else if (rank == 0) own1 = squares;
        else st_shared_cluster(leader_address(sums + (8 + quarter) * 32 + lane), squares);
#pragma unroll
        for (int i = 0; i < 8; ++i) old[i] = old1[i];
        bt = bt1;
      }
      tc_fence_before();
    }
  }
  if (failed && !skip) {
    *abort_flag = 1;
    report_timeout(a.status);
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync();   // (every thread of both CTAs comes here, whatever its waits returned)
  if (!failed && warp >= 2 && warp < 2 + kEpiWarps && a.e[0].partial != nullptr) {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    if (quarter < 2) {   // rows of w0 or w2 by `half`; columns 32 quarter to 32 quarter + 31 and 64 on
      const float x = warp_sum(sums[(half * 4 + quarter) * 32 + lane] + sums[(half * 4 + quarter + 2) * 32 + lane]);
      const int row = half * a.H + slice * kGradSlice;
      if (lane == 0) a.e[0].partial[(static_cast<int64_t>(batch) * (2 * a.H / kBM) + row / kBM) * kEpiWarps + ((row / 32 + 2) & 3) + quarter * 4] = x;
    }
    if (half == 0 && rank == 0) {
      const float x = warp_sum(own1 + sums[(8 + quarter) * 32 + lane]);
      if (lane == 0)
        a.e[1].partial[(static_cast<int64_t>(batch) * (a.H / kBM) + slice / 4) * kEpiWarps + ((quarter + 2) & 3) + (slice & 1) * 4] = x;
    }
  }
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 256; ++i) __nanosleep(1000);  // bulk copies still in flight land before shared memory goes
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

}  // namespace lact
