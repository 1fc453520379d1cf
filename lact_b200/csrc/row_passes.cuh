// Row-wise passes of the layer for the usual head sizes: LPR lanes share one (batch, token, head) row of d = 8 * LPR * V
// features, V 16-byte units per lane (unit u = lane + LPR * i), so no lane idles and a lane has all its loads in flight.
// Grid (token blocks, heads [x tensors], batch entries): no index divisions, and a block's rows are consecutive tokens.
// What bounds them is HBM and the instructions between the loads: 2 batches x 8192 tokens x 4 heads of 384 take 83 us in the
// prologue forward (302 MB: 3.6 TB/s) and 107 backward (125 with the sigmoid worked out again behind the row sums: two of the
// special-function unit's operations per feature, which it takes half of that time for; keeping it spills 12 bytes at the 80
// registers of three blocks per SM), 40 and 52 in the epilogue.  Persistent
// blocks with the next row's loads in flight take 12 to 20 % longer (fewer warps).  (A warp per row leaves a quarter of the
// lanes without a unit at that size and the loads of too few warps in flight: 144, 324, 59 and 111 us.)  Head sizes without a
// (LPR, V) of this table take the warp-per-row kernels of ops.cuh.
#pragma once
#include "swa_bwd.cuh"

namespace lact {

template <int LPR>
__device__ __forceinline__ float group_sum(float x) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
  return x;
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ uint4 load_unit(const bf16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ float silu_bf16(float x) { return bf16_round(x * sigmoidf_fast(x)); }

// The rotation partner of unit u sits hd / 16 units away inside its attention head (hd a power of two): another lane of
// the row's group, or another unit of the same lane.
template <int LPR, int V>
__device__ __forceinline__ void rope_partner(const uint4 (&y)[V], int half_units, uint4 (&other)[V]) {
  if (half_units < LPR) {
#pragma unroll
    for (int i = 0; i < V; ++i)
      other[i] = make_uint4(__shfl_xor_sync(0xFFFFFFFFu, y[i].x, half_units), __shfl_xor_sync(0xFFFFFFFFu, y[i].y, half_units),
                            __shfl_xor_sync(0xFFFFFFFFu, y[i].z, half_units), __shfl_xor_sync(0xFFFFFFFFu, y[i].w, half_units));
    return;
  }
  // (indices known to the compiler: an array indexed at run time would live in local memory)
#pragma unroll
  for (int i = 0; i < V; ++i) other[i] = half_units == LPR ? y[(i ^ 1) < V ? (i ^ 1) : i] : y[(i ^ 2) < V ? (i ^ 2) : i];
}

template <int LPR, int V, bool ROPE>
__global__ void __launch_bounds__(256, V <= 3 ? 4 : 2) qkv_rows_kernel(const PrologueArgs a) {
  griddep_launch_dependents();
  griddep_wait();
  const int lane = threadIdx.x % LPR, t = blockIdx.y / a.n_h, h = blockIdx.y - t * a.n_h, bi = blockIdx.z;
  const int tok = blockIdx.x * (256 / LPR) + threadIdx.x / LPR;
  const bool live = tok < a.s;  // (every lane takes part in the shuffles)
  const bf16* src = a.x[t] + bi * a.bs[t] + static_cast<int64_t>(live ? tok : 0) * a.ld[t] + static_cast<int64_t>(h) * a.d;
  uint4 raw[V];
#pragma unroll
  for (int i = 0; i < V; ++i) raw[i] = load_unit(src + (lane + LPR * i) * 8);
  float y[V][8], ss = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    unpack8(raw[i], y[i]);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (a.silu[t]) y[i][e] = silu_bf16(y[i][e]);
      ss += y[i][e] * y[i][e];
    }
  }
  if (a.l2norm[t]) {
    const float inv = 1.f / bf16_round(bf16_round(sqrtf(group_sum<LPR>(ss))) + 1e-5f);
#pragma unroll
    for (int i = 0; i < V; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e) y[i][e] *= inv;
  }
  bf16* dst = a.out[t] + ((static_cast<int64_t>(bi) * a.n_h + h) * a.s + tok) * a.d;
  if (ROPE && t < 2) {
    const int half = a.rope_hd >> 1;
    const int64_t trow = static_cast<int64_t>(a.pos0 + (live ? tok - (a.seq_start != nullptr ? a.seq_start[tok] : 0) : 0)) * half;
    uint4 own[V], other[V];  // the normalised row, rounded to bf16 as the reference's l2_norm returns it
#pragma unroll
    for (int i = 0; i < V; ++i) own[i] = pack8(y[i]);
    rope_partner<LPR, V>(own, half >> 3, other);
    const bool single = ((LPR * 8) & (a.rope_hd - 1)) == 0;  // every unit of a lane sits at the same place of its head
    float cs[8], sn[8];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int j = ((lane + LPR * i) * 8) & (a.rope_hd - 1);
      const bool first = j < half;
      if (i == 0 || !single) {
        unpack8(load_unit(a.cos + trow + (first ? j : j - half)), cs);
        unpack8(load_unit(a.sin + trow + (first ? j : j - half)), sn);
      }
      float x[8], o[8], r[8];
      unpack8(own[i], x);
      unpack8(other[i], o);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float xc = __fmul_rn(x[e], cs[e]), ps = __fmul_rn(o[e], sn[e]);
        r[e] = first ? __fsub_rn(xc, ps) : __fadd_rn(ps, xc);
      }
      if (live) *reinterpret_cast<uint4*>(dst + (lane + LPR * i) * 8) = pack8(r);
    }
    return;
  }
  if (!live) return;
#pragma unroll
  for (int i = 0; i < V; ++i) *reinterpret_cast<uint4*>(dst + (lane + LPR * i) * 8) = pack8(y[i]);
}

template <int LPR, int V, bool ROPE>
__global__ void __launch_bounds__(256, V <= 3 ? 3 : 2) qkv_rows_bwd_kernel(const PrologueBwdArgs a) {
  griddep_launch_dependents();
  griddep_wait();
  const int lane = threadIdx.x % LPR, t = blockIdx.y / a.n_h, h = blockIdx.y - t * a.n_h, bi = blockIdx.z;
  const int tok = blockIdx.x * (256 / LPR) + threadIdx.x / LPR;
  const bool live = tok < a.s;
  const int64_t at = live ? tok : 0;
  const bf16* src = a.x[t] + bi * a.bs[t] + at * a.ld[t] + static_cast<int64_t>(h) * a.d;
  const bf16* gz = a.dz[t] != nullptr ? a.dz[t] + ((static_cast<int64_t>(bi) * a.n_h + h) * a.s + at) * a.d : nullptr;
  uint4 rx[V], rg[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    rx[i] = load_unit(src + (lane + LPR * i) * 8);
    rg[i] = gz != nullptr ? load_unit(gz + (lane + LPR * i) * 8) : make_uint4(0, 0, 0, 0);
  }
  float g[V][8];
  if (ROPE && t < 2) {  // dy = R^T dz: first half dz cos + partner sin, second half dz cos - partner sin
    const int half = a.rope_hd >> 1;
    const int64_t trow = static_cast<int64_t>(a.pos0 + (live ? tok - (a.seq_start != nullptr ? a.seq_start[tok] : 0) : 0)) * half;
    uint4 other[V];
    rope_partner<LPR, V>(rg, half >> 3, other);
    const bool single = ((LPR * 8) & (a.rope_hd - 1)) == 0;
    float cs[8], sn[8];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int j = ((lane + LPR * i) * 8) & (a.rope_hd - 1);
      const bool first = j < half;
      if (i == 0 || !single) {
        unpack8(load_unit(a.cos + trow + (first ? j : j - half)), cs);
        unpack8(load_unit(a.sin + trow + (first ? j : j - half)), sn);
#pragma unroll
        for (int e = 0; e < 8; ++e) sn[e] = first ? sn[e] : -sn[e];
      }
      float z[8], o[8];
      unpack8(rg[i], z);
      unpack8(other[i], o);
#pragma unroll
      for (int e = 0; e < 8; ++e) g[i][e] = z[e] * cs[e] + o[e] * sn[e];
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) unpack8(rg[i], g[i]);
  }
  const bool silu = a.silu[t] != 0;
  if (a.l2norm[t]) {
    float ss = 0.f, dot = 0.f, sgm[V][8];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float x[8];
      unpack8(rx[i], x);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        sgm[i][e] = sigmoidf_fast(x[e]);
        const float u = silu ? bf16_round(x[e] * sgm[i][e]) : x[e];
        ss += u * u;
        dot += g[i][e] * u;
      }
    }
    ss = group_sum<LPR>(ss);
    dot = group_sum<LPR>(dot);
    const float nrm = sqrtf(ss), den = nrm + 1e-5f;
    const float inv = 1.f / den, coef = dot / (den * den * fmaxf(nrm, 1e-30f));
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float x[8];
      unpack8(rx[i], x);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float sg = sgm[i][e];
        const float u = silu ? bf16_round(x[e] * sg) : x[e];
        const float d = g[i][e] * inv - u * coef;
        g[i][e] = silu ? d * (sg * (1.f + x[e] * (1.f - sg))) : d;
      }
    }
  } else if (silu) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float x[8];
      unpack8(rx[i], x);
#pragma unroll
      for (int e = 0; e < 8; ++e) g[i][e] *= silu_grad(x[e]);
    }
  }
  if (!live) return;
  bf16* dst = a.dx[t] + (static_cast<int64_t>(bi) * a.s + tok) * (static_cast<int64_t>(a.n_h) * a.d) + static_cast<int64_t>(h) * a.d;
#pragma unroll
  for (int i = 0; i < V; ++i) *reinterpret_cast<uint4*>(dst + (lane + LPR * i) * 8) = pack8(g[i]);
}

template <int LPR, int V>
__global__ void __launch_bounds__(256) out_rows_kernel(const EpilogueArgs a) {
  griddep_launch_dependents();
  griddep_wait();
  const int lane = threadIdx.x % LPR, h = blockIdx.y, bi = blockIdx.z;
  const int tok = blockIdx.x * (256 / LPR) + threadIdx.x / LPR;
  const bool live = tok < a.s;
  const int64_t at = live ? tok : 0, row = static_cast<int64_t>(bi) * a.s + at, off = static_cast<int64_t>(h) * a.d;
  const bf16* src = a.x + ((static_cast<int64_t>(bi) * a.n_h + h) * a.s + at) * a.d;
  uint4 rx[V], rg[V], rr[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = (lane + LPR * i) * 8;
    rx[i] = load_unit(src + c);
    if (a.gate != nullptr) rg[i] = load_unit(a.gate + row * a.gate_ld + off + c);
    if (a.resid != nullptr) rr[i] = load_unit(a.resid + row * a.resid_ld + off + c);
  }
  float v[V][8], ss = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    unpack8(rx[i], v[i]);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += v[i][e] * v[i][e];
  }
  const float rstd = 1.f / sqrtf(group_sum<LPR>(ss) / static_cast<float>(a.d) + a.eps);
  if (!live) return;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = (lane + LPR * i) * 8;
    const float4 w0 = *reinterpret_cast<const float4*>(a.weight + c), w1 = *reinterpret_cast<const float4*>(a.weight + c + 4);
    const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
    float y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = bf16_round(v[i][e] * rstd * w[e]);
    if (a.gate != nullptr) {
      float gt[8];
      unpack8(rg[i], gt);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = bf16_round(y[e] * silu_bf16(gt[e]));
    }
    if (a.resid != nullptr) {
      float r[8];
      unpack8(rr[i], r);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] += r[e];
    }
    *reinterpret_cast<uint4*>(a.out + row * a.out_ld + off + c) = pack8(y);
  }
}

// Persistent: a group of LPR lanes walks rows (tokens of one head and batch entry after the other) in a fixed order and
// keeps its share of the norm weight's gradient in registers; the block's shares are added in shared memory.
template <int LPR, int V>
__global__ void __launch_bounds__(256, 2) out_rows_bwd_kernel(const EpilogueBwdArgs a) {
  griddep_launch_dependents();
  griddep_wait();
  constexpr int kGroups = 256 / LPR, D = 8 * LPR * V;
  __shared__ float red[8][D];
  const int lane = threadIdx.x % LPR, grp = threadIdx.x / LPR;
  float dw[V][8] = {}, w[V][8];
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int e = 0; e < 8; ++e) w[i][e] = a.weight[(lane + LPR * i) * 8 + e];
  const int tiles = (a.s + kGroups - 1) / kGroups;  // blocks of kGroups tokens
  const int64_t work = static_cast<int64_t>(tiles) * a.n_h * a.b;
  for (int64_t job = blockIdx.x; job < work; job += gridDim.x) {
    // heads fastest: the blocks that run together read whole token rows
    const int64_t rest = job / a.n_h;
    const int h = static_cast<int>(job - rest * a.n_h), bi = static_cast<int>(rest / tiles);
    const int tok = static_cast<int>(rest - static_cast<int64_t>(bi) * tiles) * kGroups + grp;
    const bool live = tok < a.s;
    const int64_t at = live ? tok : 0, row = static_cast<int64_t>(bi) * a.s + at, off = static_cast<int64_t>(h) * D;
    const int64_t x_off = ((static_cast<int64_t>(bi) * a.n_h + h) * a.s + at) * D;
    uint4 rx[V], rd[V], rg[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (lane + LPR * i) * 8;
      rx[i] = load_unit(a.x + x_off + c);
      rd[i] = load_unit(a.dout + row * a.dout_ld + off + c);
      if (a.gate != nullptr) rg[i] = load_unit(a.gate + row * a.gate_ld + off + c);
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float v[8];
      unpack8(rx[i], v);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += v[e] * v[e];
    }
    const float rstd = 1.f / sqrtf(group_sum<LPR>(ss) / static_cast<float>(D) + a.eps);
    float dn[V][8], dot = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float v[8];
      unpack8(rx[i], v);
      unpack8(rd[i], dn[i]);
      if (a.gate != nullptr) {
        float gt[8], dg[8];
        unpack8(rg[i], gt);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float sg = sigmoidf_fast(gt[e]);
          dg[e] = dn[i][e] * (v[e] * rstd * w[i][e]) * (sg * (1.f + gt[e] * (1.f - sg)));
          dn[i][e] *= gt[e] * sg;
        }
        if (a.dgate != nullptr && live)
          *reinterpret_cast<uint4*>(a.dgate + row * (static_cast<int64_t>(a.n_h) * D) + off + (lane + LPR * i) * 8) = pack8(dg);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (live) dw[i][e] += dn[i][e] * v[e] * rstd;
        dot += dn[i][e] * w[i][e] * v[e];
      }
    }
    const float k3 = rstd * rstd * rstd * group_sum<LPR>(dot) / static_cast<float>(D);
    if (live) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float v[8], o[8];
        unpack8(rx[i], v);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = rstd * w[i][e] * dn[i][e] - v[e] * k3;
        *reinterpret_cast<uint4*>(a.dx + x_off + (lane + LPR * i) * 8) = pack8(o);
      }
    }
  }
  // groups of a warp, then the eight warps, in a fixed order
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
#pragma unroll
      for (int o = LPR; o < 32; o <<= 1) dw[i][e] += __shfl_xor_sync(0xFFFFFFFFu, dw[i][e], o);
      if ((threadIdx.x & 31) < LPR) red[threadIdx.x >> 5][(lane + LPR * i) * 8 + e] = dw[i][e];
    }
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += 256) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += red[k][c];
    a.dw_partial[static_cast<int64_t>(blockIdx.x) * D + c] = t;
  }
}

// Delta of the attention backward: row sums of dO * O, LPR lanes per (batch, token, head) row; rows of a token's heads are
// adjacent, so a block reads whole token rows.
template <int LPR>
__global__ void __launch_bounds__(256) swa_delta_rows_kernel(const SwaDeltaArgs a) {
  constexpr int D = 16 * LPR;  // two units per lane
  const int lane = threadIdx.x % LPR, bi = blockIdx.y;
  const int64_t r = static_cast<int64_t>(blockIdx.x) * (256 / LPR) + threadIdx.x / LPR;  // token * heads + head
  const bool live = r < static_cast<int64_t>(a.L) * a.heads;
  const uint32_t rr = live ? static_cast<uint32_t>(r) : 0;
  const uint32_t tok = rr / static_cast<uint32_t>(a.heads), h = rr - tok * static_cast<uint32_t>(a.heads);
  const bf16* o = a.o + bi * a.o_bs + static_cast<int64_t>(tok) * a.o_ts + h * D;
  const bf16* d = a.dout + bi * a.d_bs + static_cast<int64_t>(tok) * a.d_ts + h * D;
  uint4 ro[2], rd[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    ro[i] = load_unit(o + (lane + LPR * i) * 8);
    rd[i] = load_unit(d + (lane + LPR * i) * 8);
  }
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float x[8], y[8];
    unpack8(ro[i], x);
    unpack8(rd[i], y);
#pragma unroll
    for (int e = 0; e < 8; ++e) s += x[e] * y[e];
  }
  s = group_sum<LPR>(s);
  if (live && lane == 0) a.delta[(static_cast<int64_t>(bi) * a.heads + h) * a.L + tok] = s;
}

// Calls `f` with the (LPR, V) that covers head size d exactly; false if there is none.
template <class F>
bool with_row_shape(int64_t d, F&& f) {
  if (d % 8 != 0) return false;
  const int64_t u = d / 8;
#define LACT_ROW_SHAPE(LPRV, VV) \
  if (u == LPRV * VV) { f(std::integral_constant<int, LPRV>{}, std::integral_constant<int, VV>{}); return true; }
  LACT_ROW_SHAPE(8, 1)    // 64
  LACT_ROW_SHAPE(8, 2)    // 128
  LACT_ROW_SHAPE(8, 3)    // 192
  LACT_ROW_SHAPE(16, 2)   // 256
  LACT_ROW_SHAPE(16, 3)   // 384
  LACT_ROW_SHAPE(32, 2)   // 512
  LACT_ROW_SHAPE(32, 3)   // 768
  LACT_ROW_SHAPE(32, 4)   // 1024
#undef LACT_ROW_SHAPE
  return false;
}

}  // namespace lact
