// fp32 mode (fp32 activations): FFMA contractions with the recurrence's pointwise stages in their epilogues.
// tcgen05 has no fp32 x fp32 MMA, so these run on the FP32 pipes (128 FMA per clock and SM, about 72 TFLOP/s at
// 1.9 GHz); what bounds them is FFMA issue.  One CTA = 128 threads = a 128 x 64 output tile, 8 x 8 values per thread:
// per k a thread reads 16 values as four 16-byte shared loads (each one wavefront per warp) for 64 FMAs, so the shared
// memory pipe is a quarter busy; four CTAs share an SM.  The k-slabs of 16 are double-buffered through registers.
// Measured over the whole call at 4 entries x 4096 tokens x 192 x 192, Muon on: 30 TFLOP/s.  (A 64 x 64 tile with 4 x 4 values
// per thread reads 8 scalars for 16 FMAs, and unsplit token contractions have 12 - 24 CTAs for 148 SMs: 5.5 TFLOP/s.)
#pragma once
#include "ops.cuh"

namespace lact {

constexpr int kFM = 128, kFN = 64, kFK = 16, kFThreads = 128;
constexpr int kFSA = kFM + 4, kFSB = kFN + 4;  // shared row strides (16-byte aligned)

// element (r, k) of batch entry b: p[b * bs + (t ? k * ld + r : r * ld + k)]
struct F32Mat {
  const float* p;
  int64_t ld, bs;
  int32_t t;
  int32_t vec;  // 16-byte loads allowed: base, ld, bs and the contiguous extent are multiples of 4 elements
};

enum F32Mode : int { kF32Store = 0, kF32Gate = 1, kF32Grad = 2 };

struct F32Args {
  F32Mat a, b;          // c[m][n] = sum_k a(m, k) b(n, k)
  F32Mat a2, b2;        // kF32Grad: dh[m][n] = sum_k a2(m, k) b2(n, k)
  int32_t M, N, K;      // kF32Gate / kF32Grad: N = H hidden columns; b rows n and N + n are the two projections
  int32_t batch, splits, kper;  // split s covers k in [s * kper, min(K, (s + 1) * kper)); partial s at c + s * batch * c_bs
  float* c;
  int64_t c_ld, c_bs;
  int32_t c_vec;        // kF32Store: rows of c start on 16 bytes (set by the launch)
  int32_t accumulate;   // kF32Store, splits = 1: c = acc + beta[batch] * c (beta nullptr: 1)
  const float* beta;
  // kF32Grad
  float* c2;            // [batch][M][2N]: dy0 | dy2 (c: hidden * lr1)
  int64_t c2_ld, c2_bs;
  const void *lr0, *lr1, *lr2;
  int32_t lr_f32;
  int64_t lr_bs;
  float w_scale;
};

// One k-slab of ROWS x 16 into registers: 16-byte loads along the contiguous axis (zero outside), or scalars.
template <int ROWS, bool SPLITROWS>
struct F32Slab {
  static constexpr int kN = ROWS * kFK / (4 * kFThreads);  // float4 per thread
  float4 v[kN];
  // SPLITROWS: rows [0, 32) come from row0 + r, rows [32, 64) from row0 + n_split + (r - 32)
  __device__ __forceinline__ int row_of(int r, int row0, int split_off) const {
    if constexpr (SPLITROWS) return r < 32 ? row0 + r : row0 + split_off + r - 32;
    else return row0 + r;
  }
  __device__ __forceinline__ bool row_ok(int r, int row0, int rows) const {
    if constexpr (SPLITROWS) return row0 + (r & 31) < rows;
    else return row0 + r < rows;
  }
  __device__ __forceinline__ void load(const F32Mat& m, const float* base, int row0, int rows, int split_off, int k0, int k1) {
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      const int id = i * kFThreads + threadIdx.x;
      const int r = m.t ? (id % (ROWS / 4)) * 4 : id / 4, k = k0 + (m.t ? id / (ROWS / 4) : (id & 3) * 4);
      float x[4] = {0.f, 0.f, 0.f, 0.f};
      if (m.vec) {
        if (k < k1 && row_ok(r, row0, rows)) {
          const int64_t off = m.t ? static_cast<int64_t>(k) * m.ld + row_of(r, row0, split_off)
                                  : static_cast<int64_t>(row_of(r, row0, split_off)) * m.ld + k;
          v[i] = __ldg(reinterpret_cast<const float4*>(base + off));
          continue;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int rr = m.t ? r + j : r, kk = m.t ? k : k + j;
          if (kk < k1 && row_ok(rr, row0, rows))
            x[j] = base[m.t ? static_cast<int64_t>(kk) * m.ld + row_of(rr, row0, split_off)
                            : static_cast<int64_t>(row_of(rr, row0, split_off)) * m.ld + kk];
        }
      }
      v[i] = make_float4(x[0], x[1], x[2], x[3]);
    }
  }
  __device__ __forceinline__ void store(const F32Mat& m, float* s, int stride) const {
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      const int id = i * kFThreads + threadIdx.x;
      if (m.t) {
        *reinterpret_cast<float4*>(s + (id / (ROWS / 4)) * stride + (id % (ROWS / 4)) * 4) = v[i];
      } else {
        const int r = id / 4, k = (id & 3) * 4;
        s[(k + 0) * stride + r] = v[i].x; s[(k + 1) * stride + r] = v[i].y;
        s[(k + 2) * stride + r] = v[i].z; s[(k + 3) * stride + r] = v[i].w;
      }
    }
  }
};

// acc[8][NG * 4] += tile product over k in [k_lo, k_hi); thread (tx, ty): rows 4 ty + {0..3} and 64 + 4 ty + {0..3},
// columns 4 tx + {0..3} of every 32-wide group.  BROWS = 32 * NG rows of b.
template <int NG, bool SPLITROWS>
__device__ __forceinline__ void f32_mainloop(const F32Mat& am, const F32Mat& bm, const float* A, const float* B, int m0,
                                             int M, int n0, int N, int split_off, int k_lo, int k_hi, float* As, float* Bs,
                                             float (&acc)[8][NG * 4]) {
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  F32Slab<kFM, false> sa;
  F32Slab<32 * NG, SPLITROWS> sb;
  sa.load(am, A, m0, M, 0, k_lo, k_hi);
  sb.load(bm, B, n0, N, split_off, k_lo, k_hi);
  sa.store(am, As, kFSA);
  sb.store(bm, Bs, kFSB);
  __syncthreads();
  int buf = 0;
  for (int k0 = k_lo; k0 < k_hi; k0 += kFK) {
    const bool more = k0 + kFK < k_hi;
    if (more) {
      sa.load(am, A, m0, M, 0, k0 + kFK, k_hi);
      sb.load(bm, B, n0, N, split_off, k0 + kFK, k_hi);
    }
    const float* as = As + buf * (kFK * kFSA);
    const float* bs = Bs + buf * (kFK * kFSB);
#pragma unroll
    for (int kk = 0; kk < kFK; ++kk) {
      float a[8], b[NG * 4];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(as + kk * kFSA + ty * 4);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(as + kk * kFSA + 64 + ty * 4);
#pragma unroll
      for (int g = 0; g < NG; ++g)
        *reinterpret_cast<float4*>(b + g * 4) = *reinterpret_cast<const float4*>(bs + kk * kFSB + g * 32 + tx * 4);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < NG * 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (more) {
      buf ^= 1;
      sa.store(am, As + buf * (kFK * kFSA), kFSA);
      sb.store(bm, Bs + buf * (kFK * kFSB), kFSB);
    }
    __syncthreads();
  }
}

template <int MODE>
__global__ void __launch_bounds__(kFThreads, MODE == kF32Grad ? 3 : 4) f32_gemm_kernel(const F32Args a) {
  __shared__ __align__(16) float As[2 * kFK * kFSA];
  __shared__ __align__(16) float Bs[2 * kFK * kFSB];
  griddep_launch_dependents();
  griddep_wait();
  constexpr int kCols = MODE == kF32Store ? kFN : 32;  // output columns of the tile
  const int n0 = blockIdx.x * kCols, m0 = blockIdx.y * kFM;
  const int b = blockIdx.z % a.batch, split = blockIdx.z / a.batch;
  const int k_lo = split * a.kper, k_hi = min(a.K, k_lo + a.kper);
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  float acc[8][8] = {};
  f32_mainloop<2, MODE != kF32Store>(a.a, a.b, a.a.p + b * a.a.bs, a.b.p + b * a.b.bs, m0, a.M, n0, a.N, a.N, k_lo, k_hi, As,
                                     Bs, acc);
  if constexpr (MODE == kF32Store) {
    float* C = a.c + (static_cast<int64_t>(split) * a.batch + b) * a.c_bs;
    const float cb = a.accumulate ? (a.beta != nullptr ? a.beta[b] : 1.f) : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + (i < 4 ? 0 : 64) + ty * 4 + (i & 3);
      if (m >= a.M) continue;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int n = n0 + g * 32 + tx * 4;
        float* o = C + static_cast<int64_t>(m) * a.c_ld + n;
        if (n + 4 <= a.N && a.c_vec) {
          float4 r = make_float4(acc[i][g * 4], acc[i][g * 4 + 1], acc[i][g * 4 + 2], acc[i][g * 4 + 3]);
          if (a.accumulate) {
            const float4 old = *reinterpret_cast<const float4*>(o);
            r = make_float4(fmaf(old.x, cb, r.x), fmaf(old.y, cb, r.y), fmaf(old.z, cb, r.z), fmaf(old.w, cb, r.w));
          }
          *reinterpret_cast<float4*>(o) = r;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < a.N) o[j] = a.accumulate ? fmaf(o[j], cb, acc[i][g * 4 + j]) : acc[i][g * 4 + j];
        }
      }
    }
  } else {
    float dh[8][4] = {};
    if constexpr (MODE == kF32Grad)
      f32_mainloop<1, false>(a.a2, a.b2, a.a2.p + b * a.a2.bs, a.b2.p + b * a.b2.bs, m0, a.M, n0, a.N, 0, 0, a.K, As, Bs, dh);
    const int n = n0 + tx * 4;
    if (n >= a.N) return;  // N is a multiple of 4
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + (i < 4 ? 0 : 64) + ty * 4 + (i & 3);
      if (m >= a.M) continue;
      float l0 = 1.f, l1 = 1.f, l2 = 1.f;
      if constexpr (MODE == kF32Grad) {
        const int64_t li = b * a.lr_bs + m;
        l0 = load_scalar(a.lr0, a.lr_f32, li) * a.w_scale;
        l1 = load_scalar(a.lr1, a.lr_f32, li) * a.w_scale;
        l2 = load_scalar(a.lr2, a.lr_f32, li) * a.w_scale;
      }
      float h[4], d0[4], d2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float y0 = acc[i][j], y2 = acc[i][4 + j];
        const float sg = 1.0f / (1.0f + expf(-y0)), sw = sg * y0;
        h[j] = sw * y2 * l1;
        if constexpr (MODE == kF32Grad) {
          d0[j] = sg * y2 * dh[i][j] * (1.0f + y0 * (1.0f - sg)) * l0;
          d2[j] = sw * dh[i][j] * l2;
        }
      }
      *reinterpret_cast<float4*>(a.c + b * a.c_bs + static_cast<int64_t>(m) * a.c_ld + n) = make_float4(h[0], h[1], h[2], h[3]);
      if constexpr (MODE == kF32Grad) {
        float* o = a.c2 + b * a.c2_bs + static_cast<int64_t>(m) * a.c2_ld + n;
        *reinterpret_cast<float4*>(o) = make_float4(d0[0], d0[1], d0[2], d0[3]);
        *reinterpret_cast<float4*>(o + a.N) = make_float4(d2[0], d2[1], d2[2], d2[3]);
      }
    }
  }
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
