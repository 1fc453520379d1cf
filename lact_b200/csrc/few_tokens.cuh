// SwiGLU apply on a few tokens in one launch: out = (silu(x W0^T) * (x W2^T)) W1^T for up to 64 tokens per entry, what generation
// asks for between two updates of the weights.
//
// The token x weight products of the GEMM engine would be two dependent launches whose 128-row tiles are nearly empty; the whole
// call is latency (0.6 us of memory traffic for 4 entries of 384 and 16 tokens).  Here the weights are the M side of the
// products and the tokens the N side, and a cluster of H / 64 CTAs works on one entry:
//   - CTA r holds 64 rows each of W0 and W2 (one 128-row operand) and its D / C rows of W1, all of them on their way from the start;
//   - [y0 ; y2]^T of its 64 hidden features comes out of one accumulator, the product of the gate is rounded to bf16 and written
//     into the shared memory of all CTAs of the cluster as k-block r of the second product's token operand;
//   - after a cluster barrier every CTA computes its own features of the output from all hidden features.
// Same products, k order and roundings as the two launches, whose bits it reproduces.  Calls one after another, us, two launches /
// this: 4 entries of 384, 16 tokens 12.4 / 8.8 (the host's share of a call, one launch and one allocation fewer); 16 of 512, 16
// tokens 14.4 / 11.7.
#pragma once
#include "ops.cuh"

namespace lact {

constexpr int kFewThreads = 64 + 128;  // loading warp, MMA warp, four epilogue warps
constexpr int kFewMaxTokens = 64;

struct FewArgs {
  CUtensorMap w02, w1, x;  // boxes of 64 columns and 64, 64 and `nt` rows
  bf16* out;
  int64_t o_bs, o_ts;
  int32_t D, H, tokens, nt;  // nt: tokens rounded up to 16
  int32_t rows1;             // output features per CTA
  int32_t* status;
};

__host__ __device__ constexpr uint32_t few_w1_bytes(int H) { return (H / 64) * 8192u; }
__host__ __device__ constexpr uint32_t few_w02_bytes(int D) { return (D / 64) * 16384u; }
inline uint32_t few_smem_bytes(int D, int H, int nt) {
  return few_w1_bytes(H) + few_w02_bytes(D) + static_cast<uint32_t>(nt * 2 * (D + H)) + 1024 + 256;
}
inline bool few_fits(int64_t D, int64_t H, int64_t tokens) {
  if (tokens < 1 || tokens > kFewMaxTokens || D % 64 != 0 || H % 64 != 0 || H > 512 || D > H) return false;
  return few_smem_bytes(static_cast<int>(D), static_cast<int>(H), static_cast<int>((tokens + 15) / 16 * 16)) <= 232448;
}

__device__ __forceinline__ uint32_t cluster_address(uint32_t smem, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem), "r"(rank));
  return a;
}

__global__ void __launch_bounds__(kFewThreads, 1) few_tokens_kernel(const __grid_constant__ FewArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int kb_d = a.D / 64, ranks = a.H / 64, nt = a.nt;
  // W1 rows (64 per k-block; the product's M = 128 reads 64 more, into what follows) | W0, W2 rows | tokens | hidden activations
  const uint32_t w1_s = base, w02_s = w1_s + few_w1_bytes(a.H), x_s = w02_s + few_w02_bytes(a.D), h_s = x_s + kb_d * nt * 128;
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem_raw + (h_s - smem_u32(smem_raw)) + ranks * nt * 128);
  uint64_t* const full = bars;        // [8] k-blocks of the first product
  uint64_t* const w1_full = bars + 8;
  uint64_t* const done = bars + 9;    // [2] accumulator of each product
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  volatile uint32_t* const abort_flag = tmem_slot + 1;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  if (threadIdx.x == 0) {
    for (int i = 0; i < 11; ++i) mbar_init(&bars[i], 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot);
  cluster_arrive();  // (waited for below, before the first write into another CTA's shared memory: all of them have started)
  griddep_launch_dependents();
  griddep_wait();
  const bool work = __syncthreads_or(*reinterpret_cast<volatile int32_t*>(a.status) != kStatusOk) == 0;  // (no earlier launch gave up)
  const int entry = blockIdx.x / ranks, h0 = static_cast<int>(rank) * 64, d0 = static_cast<int>(rank) * a.rows1;
  const uint32_t idesc = make_idesc_bf16(kBM, nt, 0, 0);
  bool failed = false;

  if (warp == 0 && work) {
    const uint32_t leader = elect_leader();
    for (int kb = 0; kb < kb_d; ++kb) {
      const uint32_t bar = smem_u32(&full[kb]), w = w02_s + kb * 16384;
      mbar_expect_tx_if(leader, bar, 16384 + nt * 128);
      tma_load_3d_if(leader, w, &a.w02, bar, kb * 64, h0, entry);
      tma_load_3d_if(leader, w + 8192, &a.w02, bar, kb * 64, a.H + h0, entry);
      tma_load_3d_if(leader, x_s + kb * nt * 128, &a.x, bar, kb * 64, 0, entry);
    }
    mbar_expect_tx_if(leader, w1_full, few_w1_bytes(a.H));
    for (int kb = 0; kb < ranks; ++kb) tma_load_3d_if(leader, w1_s + kb * 8192, &a.w1, smem_u32(w1_full), kb * 64, d0, entry);
  } else if (warp == 1 && work) {
    const uint32_t leader = elect_leader();
    const SmemDescBase desc(0);
    for (int kb = 0; kb < kb_d && !failed; ++kb) {
      failed = !mbar_wait_warp(&full[kb], 0, abort_flag);
      tc_fence_after();
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4)
        umma_bf16_if(leader, tmem, desc.at(((w02_s + kb * 16384) >> 4) + k4 * 2), desc.at(((x_s + kb * nt * 128) >> 4) + k4 * 2), idesc,
                     (kb | k4) != 0);
    }
    if (!failed) umma_commit_if(leader, &done[0]);
  }
  // ---------------- gate: lanes 0-63 of the accumulator hold y0 of this CTA's features, lanes 64-127 y2 of the same
  const int quarter = warp & 3, row = quarter * 32 + lane;
  const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
  const uint32_t mine = h_s + rank * nt * 128;  // this CTA's k-block of the hidden activations: [token][64 features], swizzled
  const uint32_t xch = w02_s;                   // y2, [token][64] fp32: the first product has read these bytes
  if (warp >= 2) {
    failed = work && !mbar_wait_warp(&done[0], 0, abort_flag);
    tc_fence_after();
    for (int n0 = 0; n0 < nt; n0 += 16) {
      uint32_t v[16];
      if (quarter >= 2) {
        tmem_ld16(tmem + lanes + n0, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(xch + ((n0 + j) * 64 + row - 64) * 4), "r"(v[j]) : "memory");
      }
    }
    named_barrier_sync(1, 128);
    if (quarter < 2) {
      for (int n0 = 0; n0 < nt; n0 += 16) {
        uint32_t v[16];
        tmem_ld16(tmem + lanes + n0, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          uint32_t y2;
          const int n = n0 + j;
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(y2) : "r"(xch + (n * 64 + row) * 4) : "memory");
          const float y0 = __uint_as_float(v[j]);
          const __nv_bfloat16 h = __float2bfloat16_rn(__uint_as_float(y2) * (y0 * sigmoidf_fast(y0)));
          asm volatile("st.shared.b16 [%0], %1;" ::"r"(mine + n * 128 + (((row >> 3) ^ (n & 7)) << 4) + (row & 7) * 2),
                       "h"(*reinterpret_cast<const uint16_t*>(&h))
                       : "memory");
        }
      }
    }
    tc_fence_before();
    named_barrier_sync(1, 128);
    cluster_wait();
    for (int u = threadIdx.x - 64; u < nt * 8; u += 128) {
      uint32_t w[4];
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(mine + u * 16) : "memory");
      for (int p = 1; p < ranks; ++p) {
        const uint32_t to = rank + p >= static_cast<uint32_t>(ranks) ? rank + p - ranks : rank + p;
        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_address(mine + u * 16, to)), "r"(w[0]), "r"(w[1]),
                     "r"(w[2]), "r"(w[3])
                     : "memory");
      }
    }
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  __syncwarp();
  if (warp < 2) cluster_wait();
  cluster_sync();  // (every thread arrives, whatever its waits returned)
  if (warp == 1 && work) {
    const uint32_t leader = elect_leader();
    const SmemDescBase desc(0);
    failed = failed || !mbar_wait_warp(w1_full, 0, abort_flag);
    asm volatile("fence.proxy.async;" ::: "memory");
    tc_fence_after();
    for (int kb = 0; kb < ranks && !failed; ++kb) {
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4)
        umma_bf16_if(leader, tmem + 64, desc.at(((w1_s + kb * 8192) >> 4) + k4 * 2), desc.at(((h_s + kb * nt * 128) >> 4) + k4 * 2), idesc,
                     (kb | k4) != 0);
    }
    if (!failed) umma_commit_if(leader, &done[1]);
  } else if (warp >= 2 && work && !failed && quarter < 2) {
    failed = !mbar_wait_warp(&done[1], 0, abort_flag);
    tc_fence_after();
    const int d = d0 + row;
    bf16* const out = a.out + entry * a.o_bs + d;
    for (int n0 = 0; n0 < nt; n0 += 16) {
      uint32_t v[16];
      tmem_ld16(tmem + lanes + 64 + n0, v);
      tmem_ld_wait();
      if (!failed && row < a.rows1 && d < a.D) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (n0 + j < a.tokens) out[(n0 + j) * a.o_ts] = __float2bfloat16_rn(__uint_as_float(v[j]));
      }
      __syncwarp();  // (the next load of tensor memory wants the warp together; rows1 may end inside it)
    }
    tc_fence_before();
  }
  if (failed) {
    *abort_flag = 1;
    report_timeout(a.status);
  }
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 256; ++i) __nanosleep(1000);  // bulk copies still in flight land before shared memory goes
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 128);
}

}  // namespace lact
