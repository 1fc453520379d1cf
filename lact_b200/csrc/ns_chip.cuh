// Newton-Schulz on matrices that fit one SM: a whole Muon orthogonalisation -- normalisation and all iterations -- by one
// CTA per matrix, iterate and Gram matrix in shared memory, accumulators in tensor memory.
//
// The dataflow kernel (ns_fused.cuh) sends every product through global memory: 15 dependent phases of about 5.5 us each
// (counter, TMA load, store, publication) however small the matrix.  With both operands resident a phase is its MMAs plus
// one pass of the epilogue warps, which write the rounded result straight into the swizzled layout the next product reads:
//   iterate X   [R][C]: panels of 64 columns, [R rows][128 bytes], 128-byte swizzle.  Read K-major (columns = k) or MN-major
//               (rows = k) from the same bytes, so neither product needs a transpose;
//   S, P        [m][m]: the same panels; where shared memory is too small for both, P overwrites S once the MMAs that read S
//               have completed.  X' overwrites X likewise (tall: tile by tile, a tile reads only its own rows).
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
  int32_t two;         // 1: P has a buffer of its own, so its tiles are written while later tiles are still multiplied
};

struct NsChipDims {
  int R, C, m, n, tall, two, box_rows, nmat;
  __device__ __forceinline__ explicit NsChipDims(const NsChipGroup& g)
      : R(g.R), C(g.C), m(g.m), n(g.n), tall(g.tall), two(g.two), box_rows(g.box_rows), nmat(g.nmat) {}
};

struct NsChipArgs {
  NsChipGroup grp[2];
  int32_t ngroups, steps;
  int32_t load;        // 1: start from bf16(G) as it is, normalisation folded into the first iteration
  int32_t keep;        // 1: every iterate, S and P goes to global memory (training)
  float coef[16][3];
  int32_t* status;
};

constexpr int kChipEpi = 16;                       // epilogue warps: four per tensor-memory lane quarter
constexpr int kNsChipThreads = 64 + 32 * kChipEpi;
constexpr uint32_t kNsChipSmem = 232448;
constexpr uint32_t kNsChipTail = 1024 + 256;  // alignment slack, barriers

// Whether a matrix fits: X and S (with `two`, also a buffer of its own for P), plus what the last M = 128 tile of each
// operand may reach beyond its own rows.
inline bool ns_chip_fits(int64_t R, int64_t C, int tall, bool two = false) {
  const int64_t m = std::min(R, C), n = std::max(R, C);
  if (R % 64 != 0 || C % 64 != 0 || m > 192) return false;
  if (n > 512 || (!tall && ((m + 127) / 128) * n > 512)) return false;
  const int64_t x = R * C * 2, s = m * m * 2, pad = ((m + 127) / 128) * 128 - m;
  // MN-major X tiles reach `pad` / 64 further panels of R rows behind X; K-major ones at most 64 rows behind X or S
  const int64_t reach = std::max<int64_t>(tall ? (pad / 64) * R * 128 - s : 0, 8192);
  return x + (two ? 2 : 1) * s + reach + static_cast<int64_t>(kNsChipTail) <= static_cast<int64_t>(kNsChipSmem);
}

// Operand tile of an M = 128 x N x K product in shared memory: `base` = first byte (row offset included for K-major, panel
// offset for MN-major), `panel` = bytes between 64-column panels.  Descriptors of consecutive 16-element k-slices are 2048
// bytes apart (MN-major: 16 k-rows), or 32 bytes inside a panel and `panel` bytes from one panel to the next (K-major).
struct ChipOperand {
  SmemDescBase d;
  uint32_t addr, step, jump;  // 16-byte units
  int32_t mn_major;
  __device__ __forceinline__ ChipOperand(uint32_t base, uint32_t panel, int32_t mn)
      : d(panel), addr(base >> 4), step(mn ? 128 : 2), jump(mn ? 512 : panel >> 4), mn_major(mn) {}
};
__device__ __forceinline__ void chip_product(uint32_t leader, uint32_t acc, ChipOperand a, ChipOperand b, int n, int k) {
  const uint32_t idesc = make_idesc_bf16(kBM, n, a.mn_major, b.mn_major);
  for (int kb = 0; kb < k / 64; ++kb) {
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4)
      umma_bf16_if(leader, acc, a.d.at(a.addr + k4 * a.step), b.d.at(b.addr + k4 * b.step), idesc, (kb | k4) != 0);
    a.addr += a.jump;
    b.addr += b.jump;
  }
}

// X0 = bf16(bf16(G) / den) in shared memory (or, load mode, only the scale 1 / den; the TMA load brings X), with the norm
// from given partial sums or from G itself.  Runs on the epilogue warps; returns the scale.  G is read once: its bf16
// rounding goes to the panels, is summed on the way (in a fixed order) and normalised in place.  `red`: 512 floats of scratch.
__device__ __forceinline__ float chip_prepare(const NsChipGroup& G, int mat, int load, uint32_t xs, float* red) {
  constexpr int kThreads = 32 * kChipEpi, kAhead = 6;  // kAhead: 16-byte units of X in flight per thread
  const int t = threadIdx.x - 64, warp = t >> 5, lane = t & 31;
  const int64_t base = static_cast<int64_t>(mat) * G.R * G.C;
  if (load) {  // fixed order of ns_den_kernel
    float tot = 0.f;
    for (int i = lane; i < G.nparts; i += 32) tot += G.partial[static_cast<int64_t>(mat) * G.nparts + i];
    return 1.0f / bf16_round(bf16_round(sqrtf(warp_sum(tot))) + 1e-7f);
  }
  const int R = G.R, f32 = G.src_f32;
  const int units = G.C / 8, total = R * units;  // 16-byte units of a row, of the matrix
  const int dr = kThreads / units, du = kThreads - dr * units, r_first = t / units, u_first = t - r_first * units;
  int r_at = r_first, u_at = u_first;  // row and unit of this thread's next unit
  auto next_addr = [&]() {
    const uint32_t a = xs + (u_at >> 3) * (R * 128) + r_at * 128 + (((u_at & 7) ^ (r_at & 7)) << 4);
    r_at += dr; u_at += du;
    if (u_at >= units) { u_at -= units; ++r_at; }
    return a;
  };
  const bool given = G.partial != nullptr;
  if (given && t < G.nparts) red[t] = G.partial[static_cast<int64_t>(mat) * G.nparts + t];  // (at most 512)
  float ss = 0.f;
  for (int i0 = t; i0 < total; i0 += kAhead * kThreads) {
    uint4 w[kAhead];
    if (f32) {
      float4 v[kAhead][2];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const int i = i0 + j * kThreads;
        if (i < total) {
          const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(G.src) + base + static_cast<int64_t>(i) * 8);
          v[j][0] = p[0];
          v[j][1] = p[1];
        }
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j)
        w[j] = make_uint4(pack_bf16x2(v[j][0].x, v[j][0].y), pack_bf16x2(v[j][0].z, v[j][0].w), pack_bf16x2(v[j][1].x, v[j][1].y),
                          pack_bf16x2(v[j][1].z, v[j][1].w));
    } else {
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const int i = i0 + j * kThreads;
        if (i < total) w[j] = *reinterpret_cast<const uint4*>(static_cast<const bf16*>(G.src) + base + static_cast<int64_t>(i) * 8);
      }
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (i0 + j * kThreads >= total) break;
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(next_addr()), "r"(w[j].x), "r"(w[j].y), "r"(w[j].z), "r"(w[j].w)
                   : "memory");
      const uint32_t x[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float lo = __uint_as_float(x[q] << 16), hi = __uint_as_float(x[q] & 0xFFFF0000u);
        ss += lo * lo + hi * hi;
      }
    }
  }
  if (!given) {
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
  }
  named_barrier_sync(1, kThreads);
  float tot = 0.f;
  const int parts = given ? G.nparts : kChipEpi;
  for (int i = 0; i < parts; ++i) tot += red[i];
  const float den = bf16_round(bf16_round(sqrtf(tot)) + 1e-7f);
  r_at = r_first; u_at = u_first;
  for (int i = t; i < total; i += kThreads) {  // (a thread's own units)
    const uint32_t addr = next_addr();
    uint32_t w[4];
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = pack_bf16x2(__uint_as_float(w[j] << 16) / den, __uint_as_float(w[j] & 0xFFFF0000u) / den);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
  }
  return 1.f;
}

// 32 accumulator columns of one row, scaled and rounded, as four swizzled 16-byte stores; on the diagonal block lane l's
// l-th value gets `diag` added before the rounding and is stored once more.
__device__ __forceinline__ void chip_store32(const uint32_t (&bits)[32], uint32_t row_addr, int c, int row, float sc, float diag,
                                             bool on_diag) {
  const uint32_t unit0 = (c & 63) >> 3;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = pack_bf16x2(__uint_as_float(bits[g * 8 + 2 * j]) * sc, __uint_as_float(bits[g * 8 + 2 * j + 1]) * sc);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + (((unit0 + g) ^ (row & 7)) << 4)), "r"(w[0]), "r"(w[1]),
                 "r"(w[2]), "r"(w[3])
                 : "memory");
  }
  if (on_diag) {  // warp-uniform
    const int lane = row & 31;
    uint32_t mine = bits[0];
#pragma unroll
    for (int j = 1; j < 32; ++j) mine = lane == j ? bits[j] : mine;
    const __nv_bfloat16 h = __float2bfloat16_rn(fmaf(__uint_as_float(mine), sc, diag));
    asm volatile("st.shared.b16 [%0], %1;" ::"r"(row_addr + (((unit0 + (lane >> 3)) ^ (row & 7)) << 4) + (lane & 7) * 2),
                 "h"(*reinterpret_cast<const uint16_t*>(&h))
                 : "memory");
  }
}

__global__ void __launch_bounds__(kNsChipThreads, 1) ns_chip_kernel(const __grid_constant__ NsChipArgs args) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  int mat = blockIdx.x, gi = 0;
  if (mat >= args.grp[0].nmat) { mat -= args.grp[0].nmat; gi = 1; }
  const NsChipGroup& P = args.grp[gi];
  const NsChipDims G(P);  // (scalars in registers: indexed parameter loads cost about 40 clocks each time)
  // barriers sit at the end of the allocation
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + kNsChipSmem - kNsChipTail);
  uint64_t* loaded = bars;        // [1] TMA load of X
  uint64_t* ready = bars + 1;     // [1] every epilogue warp: operands of the next pass are in shared memory
  uint64_t* full = bars + 2;      // [4] accumulator tile t of the pass is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(loaded, 1);
    mbar_init(ready, kChipEpi);
    for (int t = 0; t < 4; ++t) mbar_init(&full[t], 1);
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
  const uint32_t tmem = uniform(*tmem_slot);
  griddep_launch_dependents();
  griddep_wait();
  // an earlier launch gave up: decided once per CTA, so that all its threads meet the same named barriers
  if (threadIdx.x == 0) abort_flag[1] = *reinterpret_cast<volatile int32_t*>(args.status) != kStatusOk ? 1u : 0u;
  __syncthreads();
  bool failed = abort_flag[1] != 0;

  const uint32_t xs = base, ss = base + G.R * G.C * 2, ps = G.two ? ss + G.m * G.m * 2 : ss;
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
          tma_load_3d(xs + p * xpanel + r * 128, &P.x_in, loaded, p * 64, r, mat);
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_leader();
    if (!failed) {
      if (args.load && !mbar_wait_warp(loaded, 0, abort_flag)) failed = true;
      uint32_t pass = 0;
      auto begin = [&]() -> bool {  // operands ready (for the first pass: X prepared)
        if (!mbar_wait_warp(ready, pass & 1, abort_flag)) { failed = true; return false; }
        tc_fence_after();
        ++pass;
        return true;
      };
      for (int it = 0; it < args.steps && !failed; ++it) {
        if (!begin()) break;
        for (int t = 0; t < mt; ++t) {
          const uint32_t off = G.tall ? t * 2 * xpanel : t * (kBM * 128);
          chip_product(leader, tmem + t * G.m, ChipOperand(xs + off, xpanel, G.tall), ChipOperand(xs, xpanel, G.tall), G.m, G.n);
          umma_commit_if(leader, &full[t]);
        }
        if (!begin()) break;
        for (int t = 0; t < mt; ++t) {
          chip_product(leader, tmem + t * G.m, ChipOperand(ss + t * (kBM * 128), spanel, 0), ChipOperand(ss, spanel, 0), G.m, G.m);
          if (G.two || t + 1 == mt) umma_commit_if(leader, &full[G.two ? t : 0]);  // P over S: nothing is written before all is read
        }
        for (int up = 0; up < upasses && !failed; ++up) {
          if (!begin()) break;
          if (G.tall) {
            for (int t = up * per_pass; t < min(ut, (up + 1) * per_pass); ++t) {
              chip_product(leader, tmem + (t - up * per_pass) * G.m, ChipOperand(xs + t * (kBM * 128), xpanel, 0), ChipOperand(ps, spanel, 0),
                           G.m, G.m);
              umma_commit_if(leader, &full[t - up * per_pass]);  // (a tile reads only its own rows of X)
            }
          } else {
            for (int t = 0; t < mt; ++t)
              for (int c = 0; c < G.n; c += 256)
                chip_product(leader, tmem + t * G.n + c, ChipOperand(ps + t * (kBM * 128), spanel, 0),
                             ChipOperand(xs + (c / 64) * xpanel, xpanel, 1), min(256, G.n - c), G.m);
            umma_commit_if(leader, &full[0]);
          }
        }
      }
    }
  } else {
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const bool storer = threadIdx.x == 64;
    float scale = 1.f;
    if (!failed) scale = chip_prepare(P, mat, args.load, xs, reinterpret_cast<float*>(aligned + (ss - base)));
    fence_async_proxy();
    __syncwarp();
    if (lane == 0) mbar_arrive(ready);
    uint32_t phases = 0;  // parity of each accumulator barrier
    // keep: the whole buffer just completed goes to global memory (all warps have written it: named barrier)
    auto keep_buffer = [&](const CUtensorMap* map, uint32_t buf, uint32_t panel, int rows, int cols, int box, int slot) {
      named_barrier_sync(1, 32 * kChipEpi);
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
        named_barrier_sync(2, 32 * kChipEpi);
      }
    };
    // one pass: accumulator tiles [t0, t1) of width n (TMEM columns (t - t0) * n), rows < rows, into `dst`; `each`: a
    // barrier per tile, else one for the pass
    auto drain = [&](int t0, int t1, bool each, int n, int rows, uint32_t dst, uint32_t panel, float sc, float diag) {
      stores_read();
      for (int t = t0; t < t1; ++t) {
        if (each || t == t0) {
          const int f = t - t0;
          if (!failed && !mbar_wait(&full[f], (phases >> f) & 1, abort_flag)) failed = true;
          phases ^= 1u << f;
          tc_fence_after();
        }
        const int row0 = t * kBM + quarter * 32, row = row0 + lane;
        if (failed || row0 >= rows) continue;  // warp-uniform: rows is a multiple of 64
        const uint32_t acc = tmem + lanes + (t - t0) * n;
        for (int c = part * 32; c < n; c += 128) {  // this warp's 32-column blocks
          uint32_t v[32];
          tmem_ld32(acc + c, v);
          tmem_ld_wait();
          chip_store32(v, dst + (c >> 6) * panel + row * 128, c, row, sc, diag, diag != 0.f && row0 == c);
        }
      }
      tc_fence_before();
      fence_async_proxy();
      __syncwarp();
    };
    auto hand_over = [&]() {
      if (lane == 0) mbar_arrive(ready);
    };
    if (args.keep) keep_buffer(&P.x_out, xs, xpanel, G.R, G.C, G.box_rows, 0);
    for (int it = 0; it < args.steps; ++it) {
      const float a = args.coef[it][0], b = args.coef[it][1], c = args.coef[it][2];
      const bool fold = it == 0 && args.load;
      drain(0, mt, true, G.m, G.m, ss, spanel, fold ? scale * scale : 1.f, b / (2.f * c));
      hand_over();
      if (args.keep) keep_buffer(&P.s_out, ss, spanel, G.m, G.m, G.m, it);
      drain(0, mt, G.two, G.m, G.m, ps, spanel, c, a - b * b / (4.f * c));
      hand_over();
      if (args.keep) keep_buffer(&P.p_out, ps, spanel, G.m, G.m, G.m, it);
      for (int up = 0; up < upasses; ++up) {
        if (G.tall) drain(up * per_pass, min(ut, (up + 1) * per_pass), true, G.m, G.R, xs, xpanel, fold ? scale : 1.f, 0.f);
        else drain(0, mt, false, G.n, G.R, xs, xpanel, fold ? scale : 1.f, 0.f);
        if (it + 1 < args.steps || up + 1 < upasses) hand_over();
      }
      if (args.keep || it + 1 == args.steps) keep_buffer(&P.x_out, xs, xpanel, G.R, G.C, G.box_rows, args.keep ? it + 1 : 0);
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
