// fp32 mode (fp32 activations) on the tensor cores.  tcgen05 multiplies no fp32 by fp32, so every operand is kept as three bf16
// matrices ("pieces"), x = hi + mid + lo, each the rounding of what the ones before it leave (8 + 8 + 8 bits), and six products
// stand for the one: hi hi, hi mid, mid hi, mid mid, hi lo, lo hi.  What is left out (mid lo, lo mid, lo lo) is below 2^-23 of a
// term at worst, about 2^-27 in the mean, and of either sign.  Each product of two pieces is exact.  The tensor core adds 64 of
// them (four steps of 16) to accumulators that start at zero, hi hi in one and the small five in another; the epilogue warps add
// the accumulators of all 64-wide slabs of k to fp32 registers with rounding, so its truncating additions never see more than
// four steps.  An infinity or NaN is its own hi with zeros behind it; where the hi hi sum is not finite it stands alone (infinity
// times a zero piece would make a NaN of it).
// A bf16 value is a multiple of 2^-133, a float of 2^-149: mid is kept times 2^7 and lo times 2^14, so that nothing is lost down to
// 2^-124 and at most 2^-148 below (as they are, values under 2^-110 would keep fewer bits).  The products of one order carry one
// factor: mid mid, hi lo and lo hi are added first, and hi mid, mid hi onto their sum divided by 2^7, which tcgen05.mma does on the
// way.  With 7 the sum of the small products stays below 1.01 times the sum of the terms' magnitudes; with 8 it could be twice that,
// and infinite where the result is not.  (Error of results near 1e-36, as pieces are / kept this way: 2e-5 to 6e-4 / 3e-7.)
// Error against 64 bits of a whole call (update and apply, Muon off; relative 2-norm, FFMA contractions / these), x 1e-7:
// 4 entries of 192, 4096 tokens 6.0 / 3.3; 4 of 192, 8192 7.3 / 3.6; 16 of 256, 2048 6.2 / 3.1; 8 of 128, 1000 4.3 / 3.0; 2 of
// 64 x 128, 256 3.4 / 2.8; 2 of 256, 333 5.3 / 2.7.
//
//   cut_planes_kernel   pieces of q, k, v and the weights
//   cut_gemm_kernel     gate (64 + 64 columns), gradient planes, plain products (token contractions, down projection); the
//                       recurrence's pointwise stages in the epilogue, which writes the next operand's pieces
//
// One persistent CTA per SM: warp 0 loads (TMA; the pieces of one matrix are entries `piece * batch + entry` of one map), warp 1
// issues, sixteen warps drain and finish.  Accumulators of a slab are double-buffered.  A slab of 128 x 128 is 1536 clocks of
// products and 96 KB of operands at 64 bytes a clock; what is left above that is the finish of short sums (a gradient-plane tile
// of three slabs twice; 18 warps leave 96 registers a thread: the gradient planes spill 78 bytes, 128-wide plain products 40).  4
// entries of 192, 4096 tokens, us per launch, FFMA / these: gradient planes 138 / 51, gate 83 / 27, token contractions 2 x 48 / 36, down
// 48 / 17, the cuts - / 18; the call with Muon 434 / 192.
#pragma once
#include "f32_gemm.cuh"

namespace lact {

// The middle piece is kept times 2^kCutShift, the last one times 2^(2 kCutShift).
constexpr int kCutShift = 7;

// The three pieces of eight values, packed.  A finite value that would round to infinity is truncated instead.
__device__ __forceinline__ void cut8(const float (&x)[8], uint32_t (&hi)[4], uint32_t (&mid)[4], uint32_t (&lo)[4]) {
  constexpr float kUp = 1 << kCutShift;
  float r[8];
  uint32_t special = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    hi[j] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
    special |= (hi[j] & 0x7F807F80u) + 0x00800080u;
  }
  if (special & 0x80008000u) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t h = 0;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t b = hi[j] >> (16 * e) & 0xFFFFu;
        const bool finite = fabsf(x[2 * j + e]) <= 3.402823466e38f;
        if ((b & 0x7F80u) == 0x7F80u && finite) b = __float_as_uint(x[2 * j + e]) >> 16;
        h |= b << (16 * e);
        r[2 * j + e] = finite ? x[2 * j + e] - __uint_as_float(b << 16) : 0.f;
      }
      hi[j] = h;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      r[2 * j] = x[2 * j] - __uint_as_float(hi[j] << 16);
      r[2 * j + 1] = x[2 * j + 1] - __uint_as_float(hi[j] & 0xFFFF0000u);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float r0 = r[2 * j] * kUp, r1 = r[2 * j + 1] * kUp;
    mid[j] = pack_bf16x2(r0, r1);
    lo[j] = pack_bf16x2((r0 - __uint_as_float(mid[j] << 16)) * kUp, (r1 - __uint_as_float(mid[j] & 0xFFFF0000u)) * kUp);
  }
}

// Eight values of a row as pieces, `plane` elements apart.
__device__ __forceinline__ void store_pieces8(bf16* p, int64_t plane, const float (&x)[8]) {
  uint32_t w[3][4];
  cut8(x, w[0], w[1], w[2]);
#pragma unroll
  for (int q = 0; q < 3; ++q) st_global_16(p + q * plane, w[q][0], w[q][1], w[q][2], w[q][3]);
}

// fp32 matrices [batch][rows][cols] (any strides and alignment) into pieces [3][batch][rows][ld], ld = cols rounded up to 8.
struct CutSource {
  const float* src;
  int64_t src_ld, src_bs;
  bf16* dst;
  int32_t rows, cols, ld, vec;  // vec: rows start on 16 bytes
};
struct CutPlanesArgs {
  CutSource s[4];
  int64_t first[5];  // units of eight values before source i; [n]: all of them
  int32_t n, batch;
};
__global__ void __launch_bounds__(256) cut_planes_kernel(const __grid_constant__ CutPlanesArgs a) {
  griddep_launch_dependents();
  griddep_wait();
  const int64_t unit = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (unit >= a.first[a.n]) return;
  int i = 0;
  while (unit >= a.first[i + 1]) ++i;
  const CutSource& s = a.s[i];
  const int64_t u = unit - a.first[i];
  const int per_row = s.ld / 8, c = static_cast<int>(u % per_row) * 8;
  const int64_t line = u / per_row, b = line / s.rows, r = line - b * s.rows;
  const float* const p = s.src + b * s.src_bs + r * s.src_ld + c;
  const int n = s.cols - c;
  float x[8];
  if (s.vec && n >= 8) {
    const float4 v0 = *reinterpret_cast<const float4*>(p), v1 = *reinterpret_cast<const float4*>(p + 4);
    x[0] = v0.x; x[1] = v0.y; x[2] = v0.z; x[3] = v0.w;
    x[4] = v1.x; x[5] = v1.y; x[6] = v1.z; x[7] = v1.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = j < n ? p[j] : 0.f;
  }
  store_pieces8(s.dst + line * s.ld + c, static_cast<int64_t>(a.batch) * s.rows * s.ld, x);
}

enum CutMode : int { kCutStore = 0, kCutGate = 1, kCutGrad = 2 };

// c[m][n] = sum_k a(m, k) b(n, k), all of them pieces.  Gate / gradient planes: b holds rows n and N + n for hidden column n.
struct CutProblem {
  CUtensorMap a, b;     // entry `piece * batch + entry`; box 64 x 128 (K-major a), 64 x 64 (K-major b, MN-major a and b)
  int32_t a_mn, b_mn;
  int32_t M, N, K, batch;
  int32_t splits, kper;  // kCutStore: split s covers k in [s * kper, (s + 1) * kper), its sums go to c + s * batch * c_bs
  float* c;
  int64_t c_ld, c_bs;
  int32_t c_vec;         // rows of c start on 16 bytes, or (2) on 32
};
struct CutArgs {
  CutProblem prob[2];    // (the second one: kCutStore only)
  int32_t nprob;
  // kCutGrad: dh[m][n] = sum_k a2(m, k) b2(n, k), same M, N, K
  CUtensorMap a2, b2;    // a2 K-major, b2 MN-major
  bf16* hidden;          // pieces [3][batch][M][N] of the hidden activations (kCutGrad: times lr1)
  bf16* dy;              // kCutGrad: pieces [3][batch][M][2N] of dy0 | dy2
  const void *lr0, *lr1, *lr2;
  int32_t lr_f32;
  int64_t lr_bs;
  float w_scale;
  int32_t* status;
};

// Sixteen epilogue warps: what a tile takes beside its products is the arithmetic of the pointwise stage and of the cuts, and two
// warps per scheduler leave most of its latencies open.
constexpr int kCutEpiWarps = 16;
constexpr int kCutThreads = 64 + 32 * kCutEpiWarps;

// columns of b per tile and plane
template <int MODE, int BT>
struct CutTile {
  static_assert(BT == 64 || BT == 128, "tile widths");
  static constexpr int kOut = MODE == kCutStore ? BT : BT / 2;  // output columns
  static constexpr uint32_t kPlaneA = kBM * 128, kPlaneB = BT * 128;
  static constexpr uint32_t kStage = 3 * (kPlaneA + kPlaneB);
  static constexpr int kRing = BT == 64 ? 3 : 2;
  static constexpr uint32_t kScratch = MODE == kCutStore ? 0 : kCutEpiWarps * 32 * 48;  // 32 rows of 32 bytes (padded) per epilogue warp
  static constexpr uint32_t kSmem = kRing * kStage + kScratch + 1024 + 256;
};

template <int MODE, int BT>
__global__ void __launch_bounds__(kCutThreads, 1) cut_gemm_kernel(const __grid_constant__ CutArgs a) {
  using T = CutTile<MODE, BT>;
  constexpr int RING = T::kRing, OUT = T::kOut;
  constexpr uint32_t kTmemCols = 4 * BT;  // two buffers of hi hi | the rest
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem_raw + (base - smem_u32(smem_raw)) + RING * T::kStage + T::kScratch);
  uint64_t* const full = bars;             // [RING]
  uint64_t* const empty = full + RING;     // [RING]
  uint64_t* const acc_full = empty + RING;    // [2]
  uint64_t* const acc_empty = acc_full + 2;   // [2]
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* const abort_flag = tmem_slot + 1;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < RING; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], kCutEpiWarps); }
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
  bool failed = __syncthreads_or(*reinterpret_cast<volatile int32_t*>(a.status) != kStatusOk) != 0;  // an earlier launch gave up
  const bool work = !failed;

  // units: the tiles of a batch entry and split are consecutive (column tiles fastest), so that they share operands in L2
  int units[2] = {0, 0}, tn[2] = {1, 1}, tm[2] = {1, 1};
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    if (p < a.nprob) {
      tn[p] = (a.prob[p].N + OUT - 1) / OUT;
      tm[p] = (a.prob[p].M + kBM - 1) / kBM;
      units[p] = tn[p] * tm[p] * a.prob[p].batch * a.prob[p].splits;
    }
  }
  const int total = units[0] + units[1];
  struct Unit { int prob, b, split, m0, n0, k_lo, slabs; };
  auto locate = [&](int u) {
    Unit r;
    r.prob = u >= units[0] ? 1 : 0;
    if (r.prob) u -= units[0];
    const CutProblem& P = a.prob[r.prob];
    const int per = tn[r.prob] * tm[r.prob], e = u / per;
    u -= e * per;
    r.split = e % P.splits;
    r.b = e / P.splits;
    r.m0 = (u / tn[r.prob]) * kBM;
    r.n0 = (u % tn[r.prob]) * OUT;
    r.k_lo = r.split * P.kper;
    r.slabs = (min(P.K, r.k_lo + P.kper) - r.k_lo + kBK - 1) / kBK;
    return r;
  };

  if (warp == 0) {
    const uint32_t leader = elect_leader();
    int s = 0;
    uint32_t ph = 0;
    for (int u = blockIdx.x; u < total && !failed; u += gridDim.x) {
      const Unit r = locate(u);
      const CutProblem& P = a.prob[r.prob];
      const int passes = MODE == kCutGrad ? 2 : 1;
      for (int i = 0; i < passes * r.slabs; ++i) {
        const bool second = i >= r.slabs;  // dh
        const int k = r.k_lo + (second ? i - r.slabs : i) * kBK;
        if (!mbar_wait_warp(&empty[s], ph ^ 1, abort_flag)) { failed = true; break; }
        const uint32_t bar = smem_u32(&full[s]), st = base + s * T::kStage, sb = st + 3 * T::kPlaneA;
        mbar_expect_tx_if(leader, bar, second ? 3 * (T::kPlaneA + T::kPlaneB / 2) : T::kStage);
        const CUtensorMap* const ma = second ? &a.a2 : &P.a;
        const bool a_mn = !second && P.a_mn != 0, b_mn = second || P.b_mn != 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int e = q * P.batch + r.b;
          if (!a_mn) tma_load_3d_if(leader, st + q * T::kPlaneA, ma, bar, k, r.m0, e);
          else {
            tma_load_3d_if(leader, st + q * T::kPlaneA, ma, bar, r.m0, k, e);
            tma_load_3d_if(leader, st + q * T::kPlaneA + kAtomBytes, ma, bar, r.m0 + 64, k, e);
          }
          if (MODE == kCutGrad && second) {
            tma_load_3d_if(leader, sb + q * (T::kPlaneB / 2), &a.b2, bar, r.n0, k, e);
          } else {
#pragma unroll
            for (int j = 0; j < BT / 64; ++j) {
              const int n = MODE == kCutStore ? r.n0 + 64 * j : r.n0 + j * P.N;
              if (!b_mn) tma_load_3d_if(leader, sb + q * T::kPlaneB + j * kAtomBytes, &P.b, bar, k, n, e);
              else tma_load_3d_if(leader, sb + q * T::kPlaneB + j * kAtomBytes, &P.b, bar, n, k, e);
            }
          }
        }
        if (++s == RING) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_leader();
    int s = 0;
    uint32_t ph = 0, n = 0;
    const SmemDescBase desc(kAtomBytes);  // (MN-major: 64-wide atoms follow one another; K-major descriptors ignore it)
    for (int u = blockIdx.x; u < total && !failed; u += gridDim.x) {
      const Unit r = locate(u);
      const CutProblem& P = a.prob[r.prob];
      const int passes = MODE == kCutGrad ? 2 : 1;
      for (int i = 0; i < passes * r.slabs; ++i, ++n) {
        const bool second = i >= r.slabs;
        const uint32_t buf = n & 1;
        if (!mbar_wait_warp(&acc_empty[buf], ((n >> 1) & 1) ^ 1, abort_flag) || !mbar_wait_warp(&full[s], ph, abort_flag)) {
          failed = true;
          break;
        }
        tc_fence_after();
        const uint32_t st = base + s * T::kStage, sb = st + 3 * T::kPlaneA, acc = tmem + buf * (2 * BT);
        const uint32_t a_mn = !second && P.a_mn != 0, b_mn = second || P.b_mn != 0;
        const uint32_t step_a = a_mn ? 128 : 2, step_b = b_mn ? 128 : 2, plane_b = second ? T::kPlaneB / 2 : T::kPlaneB;
        const uint32_t nb = second ? BT / 2 : BT;  // columns of this product
        const uint32_t one = make_idesc_bf16(kBM, nb, a_mn, b_mn), two = make_idesc_bf16(kBM, 2 * nb, a_mn, b_mn);
        // steps [from, 4) of piece pa of A times piece pb of B, onto what the columns hold or (fresh) in its place
        auto product = [&](int pa, int pb, uint32_t col, uint32_t idesc, bool fresh, int from) {
          const uint32_t at = (st + pa * T::kPlaneA) >> 4, bt = (sb + pb * plane_b) >> 4;
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4)
            if (k4 >= from)
              umma_bf16_if(leader, acc + col, desc.at(at + k4 * step_a), desc.at(bt + k4 * step_b), idesc, (k4 != from || !fresh) ? 1u : 0u);
        };
        // hi hi into columns [0, nb), the rest into [nb, 2 nb).  The rest: the three products of the order of mid mid, which are
        // 2^(2 kCutShift) times too large; onto their sum, scaled down by 2^kCutShift, those of the order of hi mid.  B's hi and mid
        // lie next to each other: from the second step on one product for hi hi and hi mid.
        product(1, 1, nb, one, true, 0);
        product(0, 2, nb, one, false, 0);
        product(2, 0, nb, one, false, 0);
        umma_bf16_onto_scaled_if<kCutShift>(leader, acc + nb, desc.at((st + T::kPlaneA) >> 4), desc.at(sb >> 4), one);
        product(1, 0, nb, one, false, 1);
        umma_bf16_if(leader, acc, desc.at(st >> 4), desc.at(sb >> 4), one, 0);
        umma_bf16_if(leader, acc + nb, desc.at(st >> 4), desc.at((sb + plane_b) >> 4), one, 1);
        product(0, 0, 0, two, false, 1);
        umma_commit_if(leader, &empty[s]);
        umma_commit_if(leader, &acc_full[buf]);
        if (++s == RING) { s = 0; ph ^= 1; }
      }
    }
  } else if (work) {
    // the four warps of a lane quarter take the quarters of every accumulator: SUMS columns of c, or HC hidden columns
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    uint32_t n = 0;
    constexpr int SUMS = BT / 4;          // per thread: BT / 4 columns of c, or HC of the gate and as many of the up projection
    constexpr int HC = BT / 8;            // hidden columns per thread (gate, gradient planes)
    for (int u = blockIdx.x; u < total && !failed; u += gridDim.x) {
      const Unit r = locate(u);
      const CutProblem& P = a.prob[r.prob];
      const int row = r.m0 + quarter * 32 + lane;
      float l0 = 1.f, l1 = 1.f, l2 = 1.f;
      if constexpr (MODE == kCutGrad) {
        if (row < P.M) {
          const int64_t li = r.b * a.lr_bs + row;
          l0 = load_scalar(a.lr0, a.lr_f32, li) * a.w_scale;
          l1 = load_scalar(a.lr1, a.lr_f32, li) * a.w_scale;
          l2 = load_scalar(a.lr2, a.lr_f32, li) * a.w_scale;
        }
      }
      float sum[SUMS], dh[MODE == kCutGrad ? HC : 1];
#pragma unroll
      for (int j = 0; j < SUMS; ++j) sum[j] = 0.f;
      if constexpr (MODE == kCutGrad) {
#pragma unroll
        for (int j = 0; j < HC; ++j) dh[j] = 0.f;
      }
      // x[0..16) += hi hi + rest of 16 columns
      auto take = [&](uint32_t at, uint32_t rest, float* x) {
        uint32_t big[16], small[16];
        tmem_ld16(at, big);
        tmem_ld16(at + rest, small);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float v = __uint_as_float(big[j]);
          x[j] += fabsf(v) <= 3.402823466e38f ? fmaf(__uint_as_float(small[j]), 1.f / (1 << kCutShift), v) : v;
        }
      };
      const int passes = MODE == kCutGrad ? 2 : 1;
      for (int i = 0; i < passes * r.slabs; ++i, ++n) {
        const uint32_t buf = n & 1;
        if (!__all_sync(0xFFFFFFFFu, mbar_wait(&acc_full[buf], (n >> 1) & 1, abort_flag))) { failed = true; break; }
        tc_fence_after();
        const uint32_t acc = tmem + buf * (2 * BT) + lanes;
        if (MODE == kCutGrad && i >= r.slabs) {
          if constexpr (MODE == kCutGrad) {
#pragma unroll
            for (int c = 0; c < HC; c += 16) take(acc + part * HC + c, BT / 2, dh + c);
          }
        } else {
#pragma unroll
          for (int c = 0; c < SUMS; c += 16) {
            // gate columns [part HC, + HC), then the same of the up projection, BT / 2 columns on
            const int col = MODE == kCutStore ? part * SUMS + c : (c < HC ? part * HC + c : BT / 2 + part * HC + c - HC);
            take(acc + col, BT, sum + c);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
      if (failed) break;
      if constexpr (MODE == kCutStore) {
        if (row < P.M) {
          float* const C = P.c + (static_cast<int64_t>(r.split) * P.batch + r.b) * P.c_bs + static_cast<int64_t>(row) * P.c_ld + r.n0 + part * SUMS;
          const int left = P.N - r.n0 - part * SUMS;
#pragma unroll
          for (int j = 0; j < SUMS; j += 8) {
            if (j + 8 <= left && P.c_vec == 2) {
              uint32_t w[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(sum[j + e]);
              st_global_32(C + j, w);
            } else {
#pragma unroll
              for (int e = 0; e < 8; e += 4) {
                if (j + e + 4 <= left && P.c_vec) {
                  *reinterpret_cast<float4*>(C + j + e) = make_float4(sum[j + e], sum[j + e + 1], sum[j + e + 2], sum[j + e + 3]);
                } else {
#pragma unroll
                  for (int f = e; f < e + 4; ++f)
                    if (j + f < left) C[j + f] = sum[j + f];
                }
              }
            }
          }
        }
        __syncwarp();  // (the next unit's tensor-memory loads want the warp together)
      } else {
        // h, dy0 and dy2 take the places of y0, y2 and dh
#pragma unroll
        for (int j = 0; j < HC; ++j) {
          const float y0 = sum[j], y2 = sum[HC + j];
          const float sg = 1.0f / (1.0f + expf(-y0)), sw = sg * y0;
          sum[j] = sw * y2 * l1;
          if constexpr (MODE == kCutGrad) {
            sum[HC + j] = sg * y2 * dh[j] * (1.0f + y0 * (1.0f - sg)) * l0;
            dh[j] = sw * dh[j] * l2;
          }
        }
        // 16 columns of a warp's 32 rows as pieces, each through the warp's scratch so that two lanes cover 32 bytes of a row (32 lanes
        // on 32 rows, 16 bytes each, took 9200 clocks of the store path per tile, twice the products)
        static_assert(HC == 16, "one block per thread");
        const uint32_t scratch = base + RING * T::kStage + (warp - 2) * (32 * 48);
        const int col = r.n0 + part * HC, u2 = lane & 1, first = r.m0 + quarter * 32 + (lane >> 1);
        auto put = [&](const float* x, bf16* dst, int64_t ld, int64_t plane) {
          uint32_t w[2][3][4];
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = x[g * 8 + j];
            cut8(v, w[g][0], w[g][1], w[g][2]);
          }
          bf16* const out = dst + (static_cast<int64_t>(r.b) * P.M + first) * ld + col + u2 * 8;
#pragma unroll
          for (int q = 0; q < 3; ++q) {
#pragma unroll
            for (int g = 0; g < 2; ++g)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(scratch + lane * 48 + g * 16), "r"(w[g][q][0]),
                           "r"(w[g][q][1]), "r"(w[g][q][2]), "r"(w[g][q][3])
                           : "memory");
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint32_t y[4];
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(y[0]), "=r"(y[1]), "=r"(y[2]), "=r"(y[3])
                           : "r"(scratch + (i * 16 + (lane >> 1)) * 48 + u2 * 16)
                           : "memory");
              if (first + i * 16 < P.M && col + u2 * 8 < P.N)  // N is a multiple of 8
                st_global_16(out + q * plane + i * 16 * ld, y[0], y[1], y[2], y[3]);
            }
            __syncwarp();
          }
        };
        const int64_t plane = static_cast<int64_t>(P.batch) * P.M * P.N;
        put(sum, a.hidden, P.N, plane);
        if constexpr (MODE == kCutGrad) {
          put(sum + HC, a.dy, 2 * P.N, 2 * plane);
          put(dh, a.dy + P.N, 2 * P.N, 2 * plane);
        }
      }
    }
  }
  if (failed && work) {
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

// Sum of the split partials in split order (deterministic), plus beta[batch] * c when accumulating; up to two arrays
// (the two gradients of an update) in one launch.  n: elements per batch entry, a multiple of 4.
struct F32ReduceArgs {
  const float* part[2];
  float* c[2];
  int64_t n[2];
  int32_t splits[2];
  int32_t batch, accumulate;
  int32_t fresh;  // accumulate: c counts as zeros and is not read
  const float* beta;
};
__global__ void __launch_bounds__(256) f32_reduce_kernel(const F32ReduceArgs a) {
  griddep_launch_dependents();
  griddep_wait();
  const int64_t q0 = a.n[0] * a.batch / 4, q1 = a.n[1] * a.batch / 4;
  int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= q0 + q1) return;
  const int w = i >= q0 ? 1 : 0;
  if (w) i -= q0;
  const int64_t stride = (w ? q1 : q0) * 4;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = 0; k < a.splits[w]; ++k) {
    const float4 p = *reinterpret_cast<const float4*>(a.part[w] + k * stride + i * 4);
    s.x += p.x; s.y += p.y; s.z += p.z; s.w += p.w;
  }
  float4* o = reinterpret_cast<float4*>(a.c[w] + i * 4);
  if (a.accumulate) {
    const float bt = a.beta != nullptr ? a.beta[i * 4 / a.n[w]] : 1.f;
    const float4 old = a.fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *o;
    s = make_float4(fmaf(old.x, bt, s.x), fmaf(old.y, bt, s.y), fmaf(old.z, bt, s.z), fmaf(old.w, bt, s.w));
  }
  *o = s;
}

}  // namespace lact
