// fp32 product on the FP32 pipes (the recurrence's own contractions run on the tensor cores, f32_split.cuh; this one is for the
// entry point that has no status word for a wait that ran out).  One CTA = 128 threads = a 128 x 64 output tile, 8 x 8 values per
// thread: per k a thread reads 16 values as four 16-byte shared loads (each one wavefront per warp) for 64 FMAs; four CTAs share
// an SM.  The k-slabs of 16 are double-buffered through registers.  Bound by FFMA issue.
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

struct F32Args {
  F32Mat a, b;          // c[m][n] = sum_k a(m, k) b(n, k)
  int32_t M, N, K;
  int32_t batch;
  float* c;
  int64_t c_ld, c_bs;
  int32_t c_vec;        // rows of c start on 16 bytes (set by the launch)
  int32_t accumulate;   // c = acc + beta[batch] * c (beta nullptr: 1)
  const float* beta;
};

// One k-slab of ROWS x 16 into registers: 16-byte loads along the contiguous axis (zero outside), or scalars.
template <int ROWS>
struct F32Slab {
  static constexpr int kN = ROWS * kFK / (4 * kFThreads);  // float4 per thread
  float4 v[kN];
  __device__ __forceinline__ void load(const F32Mat& m, const float* base, int row0, int rows, int k0, int k1) {
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      const int id = i * kFThreads + threadIdx.x;
      const int r = m.t ? (id % (ROWS / 4)) * 4 : id / 4, k = k0 + (m.t ? id / (ROWS / 4) : (id & 3) * 4);
      float x[4] = {0.f, 0.f, 0.f, 0.f};
      if (m.vec) {
        if (k < k1 && row0 + r < rows) {
          const int64_t off = m.t ? static_cast<int64_t>(k) * m.ld + (row0 + r)
                                  : static_cast<int64_t>((row0 + r)) * m.ld + k;
          v[i] = __ldg(reinterpret_cast<const float4*>(base + off));
          continue;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int rr = m.t ? r + j : r, kk = m.t ? k : k + j;
          if (kk < k1 && row0 + rr < rows)
            x[j] = base[m.t ? static_cast<int64_t>(kk) * m.ld + (row0 + rr)
                            : static_cast<int64_t>((row0 + rr)) * m.ld + kk];
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

// acc[8][8] += tile product over all k; thread (tx, ty): rows 4 ty + {0..3} and 64 + 4 ty + {0..3}, columns 4 tx + {0..3} of
// both 32-wide groups.
__device__ __forceinline__ void f32_mainloop(const F32Mat& am, const F32Mat& bm, const float* A, const float* B, int m0, int M, int n0,
                                             int N, int K, float* As, float* Bs, float (&acc)[8][8]) {
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  F32Slab<kFM> sa;
  F32Slab<kFN> sb;
  sa.load(am, A, m0, M, 0, K);
  sb.load(bm, B, n0, N, 0, K);
  sa.store(am, As, kFSA);
  sb.store(bm, Bs, kFSB);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += kFK) {
    const bool more = k0 + kFK < K;
    if (more) {
      sa.load(am, A, m0, M, k0 + kFK, K);
      sb.load(bm, B, n0, N, k0 + kFK, K);
    }
    const float* as = As + buf * (kFK * kFSA);
    const float* bs = Bs + buf * (kFK * kFSB);
#pragma unroll
    for (int kk = 0; kk < kFK; ++kk) {
      float a[8], b[8];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(as + kk * kFSA + ty * 4);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(as + kk * kFSA + 64 + ty * 4);
#pragma unroll
      for (int g = 0; g < 2; ++g)
        *reinterpret_cast<float4*>(b + g * 4) = *reinterpret_cast<const float4*>(bs + kk * kFSB + g * 32 + tx * 4);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (more) {
      buf ^= 1;
      sa.store(am, As + buf * (kFK * kFSA), kFSA);
      sb.store(bm, Bs + buf * (kFK * kFSB), kFSB);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kFThreads, 4) f32_gemm_kernel(const F32Args a) {
  __shared__ __align__(16) float As[2 * kFK * kFSA];
  __shared__ __align__(16) float Bs[2 * kFK * kFSB];
  griddep_launch_dependents();
  griddep_wait();
  const int n0 = blockIdx.x * kFN, m0 = blockIdx.y * kFM, b = blockIdx.z;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  float acc[8][8] = {};
  f32_mainloop(a.a, a.b, a.a.p + b * a.a.bs, a.b.p + b * a.b.bs, m0, a.M, n0, a.N, a.K, As, Bs, acc);
  float* C = a.c + b * a.c_bs;
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
}

}  // namespace lact
