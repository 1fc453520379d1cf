// Newton-Schulz on matrices that fit one SM: a whole Muon orthogonalisation -- normalisation and all iterations -- by one
// CTA per matrix, iterate and Gram matrix in shared memory, accumulators in tensor memory.
//
// The dataflow kernel (ns_fused.cuh) sends every product through global memory: 15 dependent phases of about 5.5 us each
// (counter, TMA load, store, publication) however small the matrix.  With both operands resident a phase is its MMAs plus
// one pass of the epilogue warps, which write the rounded result straight into the swizzled layout the next product reads:
//   iterate X   [R][C]: panels of 64 columns, [R rows][128 bytes], 128-byte swizzle.  Read K-major (columns = k) or MN-major
//               (rows = k) from the same bytes, so neither product needs a transpose;
//   S, then P   [m][m]: the same panels; P overwrites S once the MMAs that read S have completed, X' overwrites X likewise.
// Same products, k order and rounding points as the dataflow kernel (values are bit-identical).  M = 128 tiles whose rows
// run past the matrix read whatever follows in shared memory (inside the allocation) into accumulator rows nobody reads.
// Bound by the chain of MMA and epilogue latencies of one SM; taken whenever X, S and the reach of the last tile fit.
#pragma once
#include "ns_fused.cuh"

namespace lact {

struct NsChipGroup {
  CUtensorMap x_in;    // first iterate when `load` (unscaled bf16 gradient), [nmat][R][C]
  CUtensorMap x_out;   // result; with `keep`: all iterates, batch = iteration * nmat + matrix
  CUtensorMap s_out, p_out;  // keep: shifted Gram matrices and polynomials, batch = iteration * nmat + matrix
  const void* src;     // gradient [nmat][R][C], fp32 or bf16 (read when not `load`)
  const float* partial;  // [nmat][nparts] sums of squares of bf16(G), or nullptr: computed here
  int32_t src_f32, nparts;
  int32_t nmat, R, C, m, n, tall;
  int32_t box_rows;    // rows of an x_in / x_out box (R or a divisor)
};

struct NsChipArgs {
  NsChipGroup grp[2];
  int32_t ngroups, steps;
  int32_t load;        // 1: start from bf16(G) as it is, normalisation folded into the first iteration
  int32_t keep;        // 1: every iterate, S and P goes to global memory (training)
  float coef[16][3];
  int32_t* status;
};

constexpr int kNsChipThreads = 320;
constexpr uint32_t kNsChipSmem = 232448;
constexpr uint32_t kNsChipTail = 1024 + 1024;  // alignment slack, barriers and norm partials

// Whether a matrix fits: X and S, plus what the last M = 128 tile of each operand may reach beyond its own rows.
inline bool ns_chip_fits(int64_t R, int64_t C, int tall) {
  const int64_t m = std::min(R, C), n = std::max(R, C);
  if (R % 64 != 0 || C % 64 != 0 || m > 192) return false;
  if (n > 512 || (!tall && ((m + 127) / 128) * n > 512)) return false;
  const int64_t x = R * C * 2, s = m * m * 2, pad = ((m + 127) / 128) * 128 - m;
  // MN-major X tiles reach `pad` / 64 further panels of R rows behind X; K-major ones at most 64 rows behind X or S
  const int64_t reach = std::max<int64_t>(tall ? (pad / 64) * R * 128 - s : 0, 8192);
  return x + s + reach + static_cast<int64_t>(kNsChipTail) <= static_cast<int64_t>(kNsChipSmem);
}

// One M = 128 x N x K product from shared memory, N <= 256, operands as described by (base, major, panel stride).
struct ChipOperand {
  uint32_t base;    // first byte of the tile (row offset included for K-major, panel offset for MN-major)
  uint32_t panel;   // bytes between 64-column panels
  int32_t mn_major;
  // descriptor of the 16-element k-slice `ks`
  __device__ __forceinline__ uint64_t desc(int ks) const {
    return mn_major ? make_smem_desc(base + ks * 2048, panel, 1024)
                    : make_smem_desc(base + (ks >> 2) * panel + (ks & 3) * 32, 0, 1024);
  }
};
__device__ __forceinline__ void chip_product(uint32_t acc, const ChipOperand& a, const ChipOperand& b, int n, int k) {
  const uint32_t idesc = make_idesc_bf16(kBM, n, a.mn_major, b.mn_major);
  for (int ks = 0; ks < k / kUmmaK; ++ks) umma_bf16(acc, a.desc(ks), b.desc(ks), idesc, ks > 0);
}

// X0 = bf16(bf16(G) / den) (or, load mode, only the scale 1 / den), with the norm from given partials or from G itself
// in the order ns_sumsq_kernel uses.  Runs on the eight epilogue warps; returns the scale.
__device__ __forceinline__ float chip_prepare(const NsChipGroup& G, int mat, int load, uint32_t xs, float* red) {
  const int t = threadIdx.x - 64, warp = t >> 5, lane = t & 31;
  const int64_t base = static_cast<int64_t>(mat) * G.R * G.C;
  if (load) {  // fixed order of ns_den_kernel
    float tot = 0.f;
    for (int i = lane; i < G.nparts; i += 32) tot += G.partial[static_cast<int64_t>(mat) * G.nparts + i];
    return 1.0f / bf16_round(bf16_round(sqrtf(warp_sum(tot))) + 1e-7f);
  }
  float tot = 0.f;
  if (G.partial != nullptr) {
    for (int i = 0; i < G.nparts; ++i) tot += G.partial[static_cast<int64_t>(mat) * G.nparts + i];
  } else {
    const int per = (G.R + kNsSlabs - 1) / kNsSlabs;
    for (int slab = 0; slab < kNsSlabs; ++slab) {
      const int r1 = min(G.R, slab * per + per);
      float ss = 0.f;
      for (int r = slab * per + warp; r < r1; r += 8)
        for (int c0 = lane; c0 < G.C; c0 += 256) {
          float xv[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            xv[i] = c0 + 32 * i < G.C ? load_scalar(G.src, G.src_f32, base + static_cast<int64_t>(r) * G.C + c0 + 32 * i) : 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float x = bf16_round(xv[i]);
            ss += x * x;
          }
        }
      ss = warp_sum(ss);
      if (lane == 0) red[slab * 8 + warp] = ss;
    }
    named_barrier_sync(1, 256);
    for (int slab = 0; slab < kNsSlabs; ++slab) tot += warp_sum(lane < 8 ? red[slab * 8 + lane] : 0.f);
  }
  const float den = bf16_round(bf16_round(sqrtf(tot)) + 1e-7f);
  const int units = G.C / 8;  // 16-byte units of a row
  for (int i = t; i < G.R * units; i += 256) {
    const int r = i / units, u = i - r * units;
    float v[8];
    if (G.src_f32) {
      const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(G.src) + base + static_cast<int64_t>(r) * G.C + u * 8);
      const float4 a = p[0], b = p[1];
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
      load8_bf16(static_cast<const bf16*>(G.src) + base + static_cast<int64_t>(r) * G.C + u * 8, v);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = bf16_round(v[j]) / den;
    const uint32_t addr = xs + (u >> 3) * (G.R * 128) + r * 128 + (((u & 7) ^ (r & 7)) << 4);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(pack_bf16x2(v[0], v[1])), "r"(pack_bf16x2(v[2], v[3])),
                 "r"(pack_bf16x2(v[4], v[5])), "r"(pack_bf16x2(v[6], v[7]))
                 : "memory");
  }
  return 1.f;
}

__global__ void __launch_bounds__(kNsChipThreads, 1) ns_chip_kernel(const __grid_constant__ NsChipArgs args) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  int mat = blockIdx.x, gi = 0;
  if (mat >= args.grp[0].nmat) { mat -= args.grp[0].nmat; gi = 1; }
  const NsChipGroup& G = args.grp[gi];
  // barriers and norm partials sit at the end of the allocation
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + kNsChipSmem - kNsChipTail);
  uint64_t* loaded = bars;        // [1] TMA load of X
  uint64_t* ready = bars + 1;     // [1] eight epilogue warps: operands of the next pass are in shared memory
  uint64_t* full = bars + 2;      // [1] the pass's accumulators are complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* red = reinterpret_cast<float*>(bars + 8);  // [16][8]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(loaded, 1);
    mbar_init(ready, kEpiWarps);
    mbar_init(full, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  griddep_launch_dependents();
  griddep_wait();
  // an earlier launch gave up: decided once per CTA, so that all its threads meet the same named barriers
  if (threadIdx.x == 0) abort_flag[1] = *reinterpret_cast<volatile int32_t*>(args.status) != kStatusOk ? 1u : 0u;
  __syncthreads();
  bool failed = abort_flag[1] != 0;

  const uint32_t xs = base, ss = base + G.R * G.C * 2;
  const uint32_t xpanel = G.R * 128, spanel = G.m * 128;
  const int mt = (G.m + kBM - 1) / kBM;                  // M tiles of the Gram matrix and the polynomial
  // update X': passes of at most 512 accumulator columns.  Tall: M tiles over the rows, N = m; wide: all M tiles, N = n.
  const int ut = (G.R + kBM - 1) / kBM;
  const int per_pass = G.tall ? 512 / G.m : mt;          // M tiles per pass
  const int upasses = G.tall ? (ut + per_pass - 1) / per_pass : 1;

  if (warp == 0) {
    if (lane == 0 && !failed && args.load) {
      mbar_expect_tx(loaded, G.R * G.C * 2);
      for (int p = 0; p < G.C / 64; ++p)
        for (int r = 0; r < G.R; r += G.box_rows)
          tma_load_3d(xs + p * xpanel + r * 128, &G.x_in, loaded, p * 64, r, mat);
    }
  } else if (warp == 1) {
    if (lane == 0 && !failed) {
      if (args.load && !mbar_wait(loaded, 0, abort_flag)) failed = true;
      uint32_t pass = 0;
      auto begin = [&]() -> bool {  // operands ready (for the first pass: X prepared)
        if (!mbar_wait(ready, pass & 1, abort_flag)) { failed = true; return false; }
        tc_fence_after();
        ++pass;
        return true;
      };
      for (int it = 0; it < args.steps && !failed; ++it) {
        if (!begin()) break;
        for (int t = 0; t < mt; ++t) {
          const uint32_t off = G.tall ? t * 2 * xpanel : t * (kBM * 128);
          chip_product(tmem + t * G.m, ChipOperand{xs + off, xpanel, G.tall}, ChipOperand{xs, xpanel, G.tall}, G.m, G.n);
        }
        umma_commit(full);
        if (!begin()) break;
        for (int t = 0; t < mt; ++t)
          chip_product(tmem + t * G.m, ChipOperand{ss + t * (kBM * 128), spanel, 0}, ChipOperand{ss, spanel, 0}, G.m, G.m);
        umma_commit(full);
        for (int up = 0; up < upasses && !failed; ++up) {
          if (!begin()) break;
          if (G.tall) {
            for (int t = up * per_pass; t < min(ut, (up + 1) * per_pass); ++t)
              chip_product(tmem + (t - up * per_pass) * G.m, ChipOperand{xs + t * (kBM * 128), xpanel, 0}, ChipOperand{ss, spanel, 0},
                           G.m, G.m);
          } else {
            for (int t = 0; t < mt; ++t)
              for (int c = 0; c < G.n; c += 256)
                chip_product(tmem + t * G.n + c, ChipOperand{ss + t * (kBM * 128), spanel, 0},
                             ChipOperand{xs + (c / 64) * xpanel, xpanel, 1}, min(256, G.n - c), G.m);
          }
          umma_commit(full);
        }
      }
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const bool storer = threadIdx.x == 64;
    float scale = 1.f;
    if (!failed) scale = chip_prepare(G, mat, args.load, xs, red);
    fence_async_proxy();
    __syncwarp();
    if (lane == 0) mbar_arrive(ready);
    uint32_t pass = 0;
    // keep: the whole buffer just completed goes to global memory (all warps have written it: named barrier)
    auto keep_buffer = [&](const CUtensorMap* map, uint32_t buf, uint32_t panel, int rows, int cols, int box, int slot) {
      named_barrier_sync(1, 256);
      if (storer) {
        for (int p = 0; p < cols / 64; ++p)
          for (int r = 0; r < rows; r += box) tma_store_3d(map, buf + p * panel + r * 128, p * 64, r, slot * G.nmat + mat);
        bulk_commit_group();
      }
    };
    // before a buffer is overwritten its stores must have read it (only one thread stores)
    auto stores_read = [&]() {
      if (args.keep) {
        if (storer) bulk_wait_read_all();
        named_barrier_sync(2, 256);
      }
    };
    // one pass: accumulator tiles [t0, t1) of width n (TMEM columns (t - t0) * n), rows < rows, into `dst`
    auto drain = [&](int t0, int t1, int n, int rows, uint32_t dst, uint32_t panel, float sc, float diag) {
      if (!failed && !mbar_wait(full, pass & 1, abort_flag)) failed = true;
      ++pass;
      tc_fence_after();
      stores_read();
      if (!failed) {
        for (int t = t0; t < t1; ++t) {
          const int row = t * kBM + quarter * 32 + lane;
          if (t * kBM + quarter * 32 >= rows) continue;  // warp-uniform: rows is a multiple of 64
          for (int c = half * 32; c < n; c += 64) {
            uint32_t bits[32];
            tmem_ld32(tmem + lanes + (t - t0) * n + c, bits);
            tmem_ld_wait();
            float o[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = bf16_round(__uint_as_float(bits[j]) * sc + (row == c + j ? diag : 0.f));
            const uint32_t addr = dst + (c >> 6) * panel + row * 128;
#pragma unroll
            for (int g = 0; g < 4; ++g)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr + (((((c & 63) >> 3) + g) ^ (row & 7)) << 4)),
                           "r"(pack_bf16x2(o[g * 8], o[g * 8 + 1])), "r"(pack_bf16x2(o[g * 8 + 2], o[g * 8 + 3])),
                           "r"(pack_bf16x2(o[g * 8 + 4], o[g * 8 + 5])), "r"(pack_bf16x2(o[g * 8 + 6], o[g * 8 + 7]))
                           : "memory");
          }
        }
      }
      tc_fence_before();
      fence_async_proxy();
      __syncwarp();
    };
    auto hand_over = [&]() {
      if (lane == 0) mbar_arrive(ready);
    };
    if (args.keep) keep_buffer(&G.x_out, xs, xpanel, G.R, G.C, G.box_rows, 0);
    for (int it = 0; it < args.steps; ++it) {
      const float a = args.coef[it][0], b = args.coef[it][1], c = args.coef[it][2];
      const bool fold = it == 0 && args.load;
      drain(0, mt, G.m, G.m, ss, spanel, fold ? scale * scale : 1.f, b / (2.f * c));
      hand_over();
      if (args.keep) keep_buffer(&G.s_out, ss, spanel, G.m, G.m, G.m, it);
      drain(0, mt, G.m, G.m, ss, spanel, c, a - b * b / (4.f * c));
      hand_over();
      if (args.keep) keep_buffer(&G.p_out, ss, spanel, G.m, G.m, G.m, it);
      for (int up = 0; up < upasses; ++up) {
        if (G.tall) drain(up * per_pass, min(ut, (up + 1) * per_pass), G.m, G.R, xs, xpanel, fold ? scale : 1.f, 0.f);
        else drain(0, mt, G.n, G.R, xs, xpanel, fold ? scale : 1.f, 0.f);
        if (it + 1 < args.steps || up + 1 < upasses) hand_over();
      }
      if (args.keep || it + 1 == args.steps) keep_buffer(&G.x_out, xs, xpanel, G.R, G.C, G.box_rows, args.keep ? it + 1 : 0);
    }
    if (storer) bulk_wait_all();
  }
  if (failed && *reinterpret_cast<volatile int32_t*>(args.status) == kStatusOk) {
    *abort_flag = 1;
    report_timeout(args.status);
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 256; ++i) __nanosleep(1000);  // a bulk load still in flight lands before shared memory goes
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

}  // namespace lact
