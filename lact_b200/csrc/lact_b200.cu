// Host side of liblact_b200: argument validation, TMA tensor-map construction, workspace
// planning, the chunk-recurrence driver and the extern "C" entry points declared in
// include/lact_b200.h.  No device memory is allocated here: all scratch is carved out of the
// caller's workspace.
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/lact_b200.h"
#include "f32_split.cuh"
#include "ns_bwd_fused.cuh"
#include "ns_chip.cuh"
#include "few_tokens.cuh"
#include "pair_gemm.cuh"
#include "row_passes.cuh"
#include "grad_fused.cuh"
#include "swa_bwd.cuh"
#include "swa_pairs.cuh"

namespace lact {
namespace {

// ------------------------------------------------------------------------------------------
// tensor maps
// ------------------------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn get_encode_fn() {
  static EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
    return reinterpret_cast<EncodeFn>(p);
  }();
  return fn;
}

// A batched row-major bf16 matrix in global memory: [batch][rows][cols], cols contiguous.
struct Mat {
  const void* ptr;
  int64_t rows, cols, ld, batch, bs;  // ld / bs: row / batch stride in elements
  int64_t segs = 1, ss = 0;           // segments (ops with `kSegments`) and their stride
};

// Encodes a 3-D map (cols, rows, batch) with a {64, box_rows, 1} box and 128-byte swizzle, or a {32, box_rows, 1} box and
// 64-byte swizzle.
int encode_map(CUtensorMap* map, const Mat& m, uint32_t box_rows, uint32_t box_cols = 64) {
  EncodeFn fn = get_encode_fn();
  if (fn == nullptr) return LACT_ERR_CUDA;
  if ((reinterpret_cast<uintptr_t>(m.ptr) & 15) != 0 || (m.ld % 8) != 0 || (m.batch > 1 && (m.bs % 8) != 0))
    return LACT_ERR_SHAPE;
  if (m.rows < 1 || m.cols < 1 || m.batch < 1 || box_rows > 256) return LACT_ERR_SHAPE;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(m.cols), static_cast<cuuint64_t>(m.rows),
                        static_cast<cuuint64_t>(m.batch)};
  const int64_t bs = m.batch > 1 ? m.bs : m.ld * m.rows;
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(m.ld) * 2, static_cast<cuuint64_t>(bs) * 2};
  cuuint32_t box[3] = {box_cols, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(m.ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? LACT_OK : LACT_ERR_CUDA;
}

// As encode_map with a fourth axis, the segments (ops with `kSegments`).
int encode_map_segments(CUtensorMap* map, const Mat& m, uint32_t box_rows) {
  EncodeFn fn = get_encode_fn();
  if (fn == nullptr) return LACT_ERR_CUDA;
  if ((reinterpret_cast<uintptr_t>(m.ptr) & 15) != 0 || (m.ld % 8) != 0 || (m.batch > 1 && (m.bs % 8) != 0) ||
      (m.segs > 1 && (m.ss % 8) != 0))
    return LACT_ERR_SHAPE;
  if (m.rows < 1 || m.cols < 1 || m.batch < 1 || m.segs < 1 || box_rows > 256) return LACT_ERR_SHAPE;
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(m.cols), static_cast<cuuint64_t>(m.rows), static_cast<cuuint64_t>(m.batch),
                        static_cast<cuuint64_t>(m.segs)};
  const int64_t bs = m.batch > 1 ? m.bs : m.ld * m.rows, ss = m.segs > 1 ? m.ss : bs;
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(m.ld) * 2, static_cast<cuuint64_t>(bs) * 2, static_cast<cuuint64_t>(ss) * 2};
  cuuint32_t box[4] = {64, box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(m.ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? LACT_OK : LACT_ERR_CUDA;
}

// What the maps of a problem's operands depend on: whether there is a segment axis.
struct OperandForm {
  bool segments;
};
template <class Op>
constexpr OperandForm form_of(const GemmProblem<Op>&) {
  return OperandForm{op_segments<Op>::value};
}

// Operand of a GEMM: `m` used K-major (mn = rows, k = cols; boxes of `tile_rows`) or MN-major (k = rows, mn = cols; boxes of 64 k
// rows and 64 columns).
int make_operand(OperandForm form, CUtensorMap* map, OperandInfo* info, const Mat& m, int mn_major, int tile_rows, int mn_off,
                 int k_off, int batch_off = 0) {
  info->mn_major = mn_major;
  info->mn_off = mn_off;
  info->k_off = k_off;
  info->batch_off = batch_off;
  if (((mn_major ? mn_off : k_off) % 8) != 0) return LACT_ERR_SHAPE;  // innermost TMA coordinate: 16-byte rule
  if (form.segments) return encode_map_segments(map, m, static_cast<uint32_t>(mn_major ? kBK : tile_rows));
  return encode_map(map, m, static_cast<uint32_t>(mn_major ? kBK : tile_rows));
}

// Output of a staged epilogue: bf16 matrix `m` whose extents clip the stored tiles.
int make_output(OperandForm form, CUtensorMap* map, OutInfo* info, const Mat& m, int row_off, int col_off, int batch_off = 0) {
  info->row_off = row_off;
  info->col_off = col_off;
  info->batch_off = batch_off;
  info->enabled = 1;
  info->ptr = const_cast<bf16*>(static_cast<const bf16*>(m.ptr) + batch_off * m.bs + row_off * m.ld + col_off);
  info->bs = m.bs;
  info->ld = static_cast<int32_t>(m.ld);
  info->wide = (reinterpret_cast<uintptr_t>(info->ptr) & 31) == 0 && m.ld % 16 == 0 && m.bs % 16 == 0;
  if (m.ld > 0x7FFFFFFF) return LACT_ERR_SHAPE;
  if ((col_off % 8) != 0 || row_off < 0 || col_off < 0) return LACT_ERR_SHAPE;
  return form.segments ? encode_map_segments(map, m, kBM) : encode_map(map, m, kBM);
}

// ------------------------------------------------------------------------------------------
// launch accounting and optional per-kernel-class timing
// ------------------------------------------------------------------------------------------
enum KernelClass : int {
  kClsPrepare = 0, kClsGate, kClsDown, kClsGradPointwise, kClsGradContract, kClsMomentumMean, kClsNsPrepare,
  kClsNsGram, kClsNsPoly, kClsNsUpdate, kClsRenorm, kClsNsFused, kClsOther, kNumClasses
};
const char* const kClassNames[kNumClasses] = {
    "prepare_weights", "gemm_swiglu_gate", "gemm_down_proj", "gemm_fwgrad_pointwise", "gemm_fwgrad_contract",
    "momentum_mean", "ns_prepare", "gemm_ns_gram", "gemm_ns_poly", "gemm_ns_update", "add_renorm", "ns_fused", "other"};

struct Profiler {
  std::mutex mu;
  std::atomic<bool> enabled{false};
  std::atomic<int64_t> launches{0};
  struct Rec { cudaEvent_t a, b; int cls; };
  std::vector<Rec> recs;
  std::vector<cudaEvent_t> pool;
  cudaEvent_t get() {
    std::lock_guard<std::mutex> lock(mu);
    if (!pool.empty()) { cudaEvent_t e = pool.back(); pool.pop_back(); return e; }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
  }
};
Profiler g_prof;
std::atomic<int64_t> g_stream_syncs{0};  // cudaStreamSynchronize calls made by the library

// Counts one kernel launch; when timing is enabled, brackets it with two events on its stream.
std::atomic<bool> g_nvtx{false};  // NVTX range around every launch, named after its kernel class

struct KernelScope {
  int cls;
  cudaStream_t stream;
  cudaEvent_t a = nullptr, b = nullptr;
  bool range = false;
  KernelScope(int cls_, cudaStream_t s) : cls(cls_), stream(s) {
    g_prof.launches.fetch_add(1, std::memory_order_relaxed);
    if (g_nvtx.load(std::memory_order_relaxed)) {
      nvtxRangePushA(kClassNames[cls]);
      range = true;
    }
    if (g_prof.enabled.load(std::memory_order_relaxed)) {
      a = g_prof.get();
      b = g_prof.get();
      if (a) cudaEventRecord(a, stream);
    }
  }
  ~KernelScope() {
    if (a && b) {
      cudaEventRecord(b, stream);
      std::lock_guard<std::mutex> lock(g_prof.mu);
      g_prof.recs.push_back({a, b, cls});
    }
    if (range) nvtxRangePop();
  }
};

// ------------------------------------------------------------------------------------------
// launch helpers
// ------------------------------------------------------------------------------------------
#define LACT_TRY(expr)                   \
  do {                                   \
    int _rc = (expr);                    \
    if (_rc != LACT_OK) return _rc;      \
  } while (0)

#define LACT_CUDA(expr)                               \
  do {                                                \
    if ((expr) != cudaSuccess) return LACT_ERR_CUDA;  \
  } while (0)

int check_device() {
  static std::mutex mu;
  static int ok_dev[64] = {0};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (dev < 64 && ok_dev[dev] == 1) return LACT_OK;
  int major = 0;
  LACT_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  if (major != 10) return LACT_ERR_DEVICE;
  if (dev < 64) ok_dev[dev] = 1;
  return LACT_OK;
}

// Launch with programmatic stream serialization: the kernel's prologue may overlap the tail of the
// previous kernel in the stream; every kernel waits (griddepcontrol.wait) before it touches global memory.
template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                       Args&&... args) {
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  // Measured (10 forward steps of the benchmark shape, same GPU, back to back): 8.16 -> 8.05 ms at 32 (batch x head)
  // units, 3.58 -> 3.39 ms at 8 units, 2.94 -> 2.74 ms at 4 units: the fewer units, the larger the share of the
  // launch gaps that the overlap hides.
  // The layer's row passes, forward and backward, gain 4 % (302 -> 290 us for ten launches), the attention forward and
  // a program's first kernels 1 to 3 us a call.  Plain launches are the row kernels of the recurrence's reverse sweep and
  // the attention backward: a training step of 32 entries took 2.5 % longer with them, 8 entries of 192 718 -> 729 us.
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

inline int ceil_div(int64_t a, int64_t b) { return static_cast<int>((a + b - 1) / b); }

// Launches the first `nprob` problems of `args` as one persistent grid (one CTA per SM at most).
template <class Op, int NPROB>
int launch_gemm(const GemmArgs<Op, NPROB>& args, cudaStream_t stream, int cls, int nprob = NPROB) {
  auto kernel = umma_gemm_kernel<Op, NPROB>;
  constexpr uint32_t smem = gemm_smem_bytes<Op>();
  static_assert(smem <= 232448, "shared memory budget exceeded");
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (dev < 64) configured[dev] = true;
    }
  }
  int64_t tiles = 0;
  for (int p = 0; p < nprob; ++p) {
    const auto& P = args.prob[p];
    if (P.M < 1 || P.N < 1 || P.batch < 1 || P.K < 1) return LACT_ERR_SHAPE;
    tiles += static_cast<int64_t>((P.M + kBM - 1) / kBM) * ((P.N + Op::BT - 1) / Op::BT) * P.batch * std::max(1, P.splits);
  }
  if (tiles > (1ll << 30)) return LACT_ERR_SHAPE;
  const int grid = static_cast<int>(std::min<int64_t>(tiles, sm_count()));
  KernelScope scope(cls, stream);
  LACT_CUDA(launch_pdl(kernel, dim3(grid), dim3(kGemmThreadsV2), smem, stream, args, nprob));
  return LACT_OK;
}

// Whether a product of `batch` x `M` tokens and N columns goes to pairs of SMs (pair_gemm.cuh).  All sides measured as us of the
// call with pairs / with single SMs, pointwise stage and apply, 2 to 16 tiles of 256 tokens per pair:
//   - a ring of three stages has to fit beside the weights: at K = 512 the pointwise stage has two and takes 1.14 to 1.74 times as
//     long (18 entries of 512, 4096 tokens: 193 / 154); at 384, three: 0.89 to 0.95;
//   - six of seven pairs have to find work: a team of pairs has one for every column tile, so that 25 tiles (H = 1600) leave 24 of
//     74 pairs idle (98.7 / 83.1), 40 (H = 2560) leave 34 (116 / 81); 16 leave 10 (55.1 / 63.5);
//   - rows are computed in halves of 256: entries of 16 or 128 tokens waste a half or more (394 of 384, 128 tokens: 119 / 90; apply
//     of 592 entries of 192, 16 tokens: 51 / 32), 384 tokens a quarter (119 / 110).  A tenth may be wasted;
//   - a set of weights has to serve enough products, or loading the next one shows: 49152 columns x k per 128 rows, 65536 where
//     tiles are narrow.  At one tile per set 256 or more wide features reach that (197 entries of 384, 256 tokens: 73.9 / 78.1, apply
//     60.7 / 63.6), 192 do not (apply 76.0 / 64.1), with two the pointwise stage alone (70.2 / 72.1; the gate's 64-wide tiles
//     51.1 / 43.0), with three all (65.7 / 69.0, apply 57.4 / 58.3);
//   - six tiles per pair in all, for a launch of clusters costs about 2 us more than a plain one: 1.3 tiles (4 entries of 384, 2048
//     tokens) gate 16.2 / 14.7, down 12.7 / 10.7; 7 to 10.7 (32 of 384) pointwise 96 / 99, gate 43 / 48, down 28.8 / 31.5.
template <class Op>
bool pair_pays(int64_t batch, int64_t M, int64_t N, int64_t K) {
  if (K > kPairMaxKb * kBK || pair_ring<Op>(ceil_div(K, kBK)) < 3) return false;
  const int64_t pairs = sm_count() / 2, tn = ceil_div(N, Op::BT), cols = Op::NACC * Op::BT, per_set = ceil_div(M, kPairRows);
  return tn <= pairs && 7 * (pairs / tn * tn) >= 6 * pairs && 20 * per_set <= 11 * ceil_div(M, kBM) &&
         per_set * cols * K >= (cols > 128 ? 49152 : 65536) && per_set * batch * tn >= 6 * pairs;
}

// The same launch on pairs of SMs with the weights kept in shared memory.
template <class Op>
int launch_pair(const GemmArgs<Op, 1>& args, cudaStream_t stream, int cls) {
  auto kernel = pair_gemm_kernel<Op>;
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
      if (dev < 64) configured[dev] = true;
    }
  }
  const auto& P = args.prob[0];
  if (P.M < 1 || P.N < 1 || P.batch < 1 || P.K < 1) return LACT_ERR_SHAPE;
  const int64_t tiles = static_cast<int64_t>(ceil_div(P.M, kPairRows)) * P.batch;
  const int tn = ceil_div(P.N, Op::BT), teams = static_cast<int>(std::min<int64_t>(tiles, sm_count() / 2 / tn));
  if (tiles > (1ll << 30) || teams < 1) return LACT_ERR_SHAPE;
  const int num_kb = ceil_div(P.K, kBK), ring = pair_ring<Op>(num_kb);
  if (num_kb > kPairMaxKb || ring < 2) return LACT_ERR_CONFIG;
  const size_t smem = 1024 + kPairBars + pair_panels<Op>() * kPairPanel + pair_b_bytes<Op>(num_kb) + ring * pair_stage_bytes<Op>();
  KernelScope scope(cls, stream);
  LACT_CUDA(launch_pdl(kernel, dim3(2 * teams * tn), dim3(kGemmThreadsV2), smem, stream, args, ring));
  return LACT_OK;
}
// c = a b^T in bf16 tiles of Op::BT columns; `fill` as for launch_op, with B boxes of half a tile.
template <class Op, class Fill>
int launch_pair_store(Fill&& fill, cudaStream_t stream, int cls) {
  GemmArgs<Op, 1> g;
  std::memset(&g, 0, sizeof(g));
  LACT_TRY(fill(g, Op::BT / 2));
  return launch_pair(g, stream, cls);
}

// Output-tile width for a single-accumulator GEMM: the candidate with the least padded work over
// the problems of the launch (ties go to the wider tile, whose MMA shape is more efficient).
struct NW { int64_t n, weight; };
int choose_bt(std::initializer_list<NW> probs) {
  const int cands[4] = {256, 192, 128, 64};
  int best = 128;
  int64_t best_cost = -1;
  for (int bt : cands) {
    int64_t cost = 0;
    for (const NW& q : probs) cost += ((q.n + bt - 1) / bt) * bt * q.weight;
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = bt; }
  }
  return best;
}

// Split of a long contraction: into how many units each output tile is cut.  Few entries or small heads have few output
// tiles (16 heads of 192: 80 on 148 SMs), and a tile of 49152 tokens is 768 k-blocks of serial work; shorter units fill the
// SMs and even out the last round.  The rule looks at the length of the sum alone, never at the number of entries: an
// entry's result is the same bits in any batch.  From 96 k-blocks up three units per tile, from 192 five (both odd, so that
// tile counts just above half the SMs do not double their rounds): 16 entries of 192 and 768 k-blocks 315 -> 270 us (twelve
// units take longer: their partial sums cost more than the rounds they even out), 8 entries of 256 and 192 k-blocks 126 -> 93,
// 37 of 192 and 128 k-blocks 142 -> 130.  Below 96 nothing is gained: at 32 k-blocks (4 entries of 384) 25 us either way, at
// 25 (12 of 128 x 256) 19 -> 23.  Where the tiles fill the chip anyway the partial sums cost what they are: nothing at 64
// entries of 192 (204 us either way), 345 -> 378 at 128 of them, 255 -> 288 at 96 of 128 x 256; entries of 384 gain alone
// (49 -> 33 at 128 k-blocks) and in fours (60 -> 58), and lose in eights (70 -> 82) and beyond (32: 219 -> 256; 64 at 96
// k-blocks: 365 -> 485).  (A unit's k-blocks are rounded up to an even number: where the cuts lie decides an entry's bits, and they
// stay where they have been.)
struct Split {
  int splits, kb_per_split;
};
Split choose_split(int64_t num_kb) {
  if (num_kb < 96) return Split{1, static_cast<int>(num_kb)};
  const int64_t want = num_kb < 192 ? 3 : 5;
  const int64_t per = ((num_kb + want - 1) / want + 1) & ~1ll;
  return Split{static_cast<int>((num_kb + per - 1) / per), static_cast<int>(per)};
}
inline int64_t output_tiles(int64_t M, int64_t N, int64_t batch, int bt) {
  return static_cast<int64_t>(ceil_div(M, kBM)) * ceil_div(N, bt) * batch;
}
struct SplitScratch {
  float* part = nullptr;      // fp32 sums of all units: tiles x splits x 128 x bt
  uint32_t* count = nullptr;  // a word per tile, zero
};
template <class P>
void set_split(P& prob, const Split& sp, const SplitScratch& ws) {
  prob.splits = sp.splits;
  prob.kb_per_split = sp.kb_per_split;
  prob.part = ws.part;
  prob.count = ws.count;
}

// Instantiates OpT<BT> for the chosen tile width; `fill(args, bt)` populates the problems.
template <template <int> class OpT, int NPROB, class Fill>
int launch_op(int bt, Fill&& fill, cudaStream_t stream, int cls, int nprob) {
#define LACT_OP_CASE(BTV)                                    \
  case BTV: {                                                \
    GemmArgs<OpT<BTV>, NPROB> g;                             \
    std::memset(&g, 0, sizeof(g));                           \
    LACT_TRY(fill(g, BTV));                                  \
    return launch_gemm(g, stream, cls, nprob);               \
  }
  switch (bt) {
    LACT_OP_CASE(64)
    LACT_OP_CASE(128)
    LACT_OP_CASE(192)
    LACT_OP_CASE(256)
    default: return LACT_ERR_CONFIG;
  }
#undef LACT_OP_CASE
}
template <int BT> using OpStoreDirectT = OpBmm<EpiStore, BT>;
template <int BT> using OpStore2T = OpBmm2<EpiStore, BT>;

// ------------------------------------------------------------------------------------------
// building blocks (device pointers in, kernels enqueued)
// ------------------------------------------------------------------------------------------
struct ApplyArgs {
  const bf16* w02b;  // [B][2H][D]
  const bf16* w1b;   // [B][D][H]
  const void* x;     // activations [B][*][D], bf16
  int64_t x_bs, x_ts;
  int64_t start, end;  // token range
  void* out;           // [B][*][D] bf16
  int64_t o_bs, o_ts;
  int64_t out_start;
  bf16* hidden;  // scratch [segments][B][end-start][H]
  int64_t B, D, H;
  // Several ranges of one length at once ("segments"), each with its own weights: segment i reads tokens from start + i x_step,
  // writes from out_start + i o_step and takes its weights w_step elements on.
  int64_t segs = 1, x_step = 0, o_step = 0, w_step = 0;
};

template <int BT>
int launch_gate(const ApplyArgs& a, const Mat& x, const Mat& w02, int64_t len, int32_t* status, cudaStream_t stream) {
  GemmArgs<OpSwigluGate<BT>, 1> g;
  std::memset(&g, 0, sizeof(g));
  auto& P = g.prob[0];
  LACT_TRY(make_operand(form_of(P), &P.a[0], &P.ai[0], x, 0, kBM, 0, 0));
  LACT_TRY(make_operand(form_of(P), &P.b[0], &P.bi[0], w02, 0, BT, 0, 0));
  LACT_TRY(make_operand(form_of(P), &P.b[1], &P.bi[1], w02, 0, BT, static_cast<int>(a.H), 0));
  const Mat hid{a.hidden, len, a.H, a.H, a.B, len * a.H, a.segs, a.B * len * a.H};
  LACT_TRY(make_output(form_of(P), &P.out[0], &P.oi[0], hid, 0, 0));
  P.M = static_cast<int>(len); P.N = static_cast<int>(a.H); P.K = static_cast<int>(a.D);
  P.batch = static_cast<int>(a.segs * a.B);
  P.entries = static_cast<int>(a.B);
  g.status = status;
  if (pair_pays<OpSwigluGate<BT>>(P.batch, len, a.H, a.D)) return launch_pair(g, stream, kClsGate);
  return launch_gemm(g, stream, kClsGate);
}

// Whether apply on `tokens` tokens of `B` entries goes to one cluster per entry (few_tokens.cuh): where the
// clusters of all entries run at once.  us per call, two launches / one cluster per entry: up to there 12.3 / 8.6 at 256, 192 and 128 x
// 256 (64 entries of 256, 16 tokens, two CTAs per SM: 12.6 / 10.9), 12.4 / 8.8 at 384, 14.3 / 8.6 at 512; past it 12.7 / 14.2 (32
// of 384, 32 tokens), 12.3 / 16.6 (64 of 192, 64 tokens), 14.7 / 18.1 (32 of 512, 16 tokens).
bool few_pays(int64_t B, int64_t tokens, int64_t D, int64_t H) {
  if (!few_fits(D, H, tokens)) return false;
  const int64_t nt = (tokens + 15) / 16 * 16;
  const int64_t per_sm = 233472 / (few_smem_bytes(static_cast<int>(D), static_cast<int>(H), static_cast<int>(nt)) + 1024);
  return B * (H / 64) <= per_sm * sm_count();
}
int launch_few(const ApplyArgs& a, const Mat& x, const Mat& w02, const Mat& w1, const Mat& om, int32_t* status, cudaStream_t stream) {
  // (outputs that the two launches' maps do not take are refused here too: stores of single values want 2 bytes all the same)
  if ((reinterpret_cast<uintptr_t>(om.ptr) & 15) != 0 || om.ld % 8 != 0 || (om.batch > 1 && om.bs % 8 != 0)) return LACT_ERR_SHAPE;
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(few_tokens_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
      if (dev < 64) configured[dev] = true;
    }
  }
  FewArgs f;
  std::memset(&f, 0, sizeof(f));
  f.D = static_cast<int32_t>(a.D); f.H = static_cast<int32_t>(a.H);
  f.tokens = static_cast<int32_t>(a.end - a.start);
  f.nt = (f.tokens + 15) / 16 * 16;
  const int ranks = f.H / 64;
  f.rows1 = ceil_div(f.D, ranks);
  f.out = static_cast<bf16*>(a.out) + a.out_start * a.o_ts;
  f.o_bs = a.o_bs; f.o_ts = a.o_ts;
  f.status = status;
  LACT_TRY(encode_map(&f.w02, w02, 64));
  LACT_TRY(encode_map(&f.w1, w1, 64));
  LACT_TRY(encode_map(&f.x, x, static_cast<uint32_t>(f.nt)));
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(static_cast<unsigned>(a.B * ranks));
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = few_smem_bytes(f.D, f.H, f.nt);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(ranks);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  KernelScope scope(kClsGate, stream);
  LACT_CUDA(cudaLaunchKernelEx(&cfg, few_tokens_kernel, f));
  return LACT_OK;
}

int run_apply(const ApplyArgs& a, int32_t* status, cudaStream_t stream) {
  const int64_t len = a.end - a.start;
  if (len <= 0) return LACT_OK;
  const Mat w02{a.w02b, 2 * a.H, a.D, a.D, a.B, 2 * a.H * a.D, a.segs, a.w_step};
  const Mat w1{a.w1b, a.D, a.H, a.H, a.B, a.D * a.H, a.segs, a.w_step};
  // (token strides are multiples of 16 bytes, so a range may start at any token; the maps end with it: nothing is written
  // beyond the range)
  const Mat x{static_cast<const bf16*>(a.x) + a.start * a.x_ts, len, a.D, a.x_ts, a.B, a.x_bs, a.segs, a.x_step * a.x_ts};
  const Mat om{static_cast<bf16*>(a.out) + a.out_start * a.o_ts, len, a.D, a.o_ts, a.B, a.o_bs, a.segs, a.o_step * a.o_ts};
  const Mat hid{a.hidden, len, a.H, a.H, a.B, len * a.H, a.segs, a.B * len * a.H};
  const int64_t batch = a.segs * a.B;
  if (a.segs == 1 && few_pays(a.B, len, a.D, a.H)) return launch_few(a, x, w02, w1, om, status, stream);
  if (a.H % 128 == 0) LACT_TRY(launch_gate<128>(a, x, w02, len, status, stream));
  else LACT_TRY(launch_gate<64>(a, x, w02, len, status, stream));
  const int bt = choose_bt({{a.D, 1}});
  auto fill = [&](auto& g, int btv) -> int {
    auto& P = g.prob[0];
    LACT_TRY(make_operand(form_of(P), &P.a[0], &P.ai[0], hid, 0, kBM, 0, 0));
    LACT_TRY(make_operand(form_of(P), &P.b[0], &P.bi[0], w1, 0, btv, 0, 0));
    LACT_TRY(make_output(form_of(P), &P.out[0], &P.oi[0], om, 0, 0));
    P.M = static_cast<int>(len); P.N = static_cast<int>(a.D); P.K = static_cast<int>(a.H);
    P.batch = static_cast<int>(batch);
    P.entries = static_cast<int>(a.B);
    g.status = status;
    return LACT_OK;
  };
  if (bt == 256 && pair_pays<OpBmmStore<256>>(batch, len, a.D, a.H)) return launch_pair_store<OpBmmStore<256>>(fill, stream, kClsDown);
  if (bt == 192 && pair_pays<OpBmmStore<192>>(batch, len, a.D, a.H)) return launch_pair_store<OpBmmStore<192>>(fill, stream, kClsDown);
  if (bt == 128 && pair_pays<OpBmmStore<128>>(batch, len, a.D, a.H)) return launch_pair_store<OpBmmStore<128>>(fill, stream, kClsDown);
  return launch_op<OpBmmStore, 1>(bt, fill, stream, kClsDown, 1);
}

struct GradArgs {
  const bf16* w02b;
  const bf16* w1b;
  const void *k, *v;
  int64_t k_bs, k_ts, v_bs, v_ts;
  int64_t start, end;
  const void *lr0, *lr1, *lr2;
  int32_t lr_f32;
  int64_t lr_bs;
  float w_scale;
  bf16* dy02;  // scratch [B][len][2H]
  bf16* hid;   // scratch [B][len][H]
  void* g02;   // [B][2H][D] fp32 (state) or bf16
  void* g1;    // [B][D][H]
  int32_t g_f32;
  const float* beta;  // [B] or nullptr
  int64_t B, D, H;
  float* partial02 = nullptr;  // optional per-tile sums of squares of the two outputs
  float* partial1 = nullptr;
  bf16* gb02 = nullptr;        // optional bf16 copies of the two outputs (Newton-Schulz input)
  bf16* gb1 = nullptr;
  const float* g02_prev = nullptr;  // optional: momentum state read from here instead of g02 / g1 (fp32)
  const float* g1_prev = nullptr;
  int32_t fresh = 0;                // 1: the momentum state is still zero
  SplitScratch split;               // optional: scratch for a split contraction
};

inline int contract_bt(int64_t D, int64_t H) { return choose_bt({{D, 2 * H}, {H, D}}); }
inline int64_t contract_tiles(int64_t B, int64_t D, int64_t H) {
  const int bt = contract_bt(D, H);
  return output_tiles(2 * H, D, B, bt) + output_tiles(D, H, B, bt);
}

// Pointwise stage: dy02 = [dy0 | dy2] ([B][len][2H]) and hid = hidden * lr1 ([B][len][H]) for tokens [start, end).
int run_grad_pointwise(const GradArgs& a, int32_t* status, cudaStream_t stream) {
  const int64_t len = a.end - a.start;
  if (len <= 0) return LACT_ERR_STEPS;
  const Mat w02{a.w02b, 2 * a.H, a.D, a.D, a.B, 2 * a.H * a.D};
  const Mat w1{a.w1b, a.D, a.H, a.H, a.B, a.D * a.H};
  const Mat km{a.k, a.end, a.D, a.k_ts, a.B, a.k_bs};
  const Mat vm{a.v, a.end, a.D, a.v_ts, a.B, a.v_bs};
  const Mat hid{a.hid, len, a.H, a.H, a.B, len * a.H};
  GemmArgs<OpFwGradPointwise, 1> g;
  std::memset(&g, 0, sizeof(g));
  auto& P = g.prob[0];
  constexpr int BT = OpFwGradPointwise::BT;
  LACT_TRY(make_operand(form_of(P), &P.a[0], &P.ai[0], km, 0, kBM, static_cast<int>(a.start), 0));
  LACT_TRY(make_operand(form_of(P), &P.a[1], &P.ai[1], vm, 0, kBM, static_cast<int>(a.start), 0));
  LACT_TRY(make_operand(form_of(P), &P.b[0], &P.bi[0], w02, 0, BT, 0, 0));
  LACT_TRY(make_operand(form_of(P), &P.b[1], &P.bi[1], w02, 0, BT, static_cast<int>(a.H), 0));
  // dh = v w1: w1 is [D][H], i.e. k (= D) rows with the n (= H) axis contiguous
  LACT_TRY(make_operand(form_of(P), &P.b[2], &P.bi[2], w1, 1, BT, 0, 0));
  P.M = static_cast<int>(len); P.N = static_cast<int>(a.H); P.K = static_cast<int>(a.D);
  P.batch = static_cast<int>(a.B);
  P.ep = EpiFwGrad{a.lr0, a.lr1, a.lr2, a.lr_f32, static_cast<int32_t>(a.start), a.lr_bs, a.w_scale};
  // dy0 and dy2 share the [len][2H] plane: two maps of H columns each, so neither can spill
  const Mat dy0m{a.dy02, len, a.H, 2 * a.H, a.B, len * 2 * a.H};
  const Mat dy2m{a.dy02 + a.H, len, a.H, 2 * a.H, a.B, len * 2 * a.H};
  LACT_TRY(make_output(form_of(P), &P.out[0], &P.oi[0], dy0m, 0, 0));
  LACT_TRY(make_output(form_of(P), &P.out[1], &P.oi[1], dy2m, 0, 0));
  LACT_TRY(make_output(form_of(P), &P.out[2], &P.oi[2], hid, 0, 0));
  g.status = status;
  if (pair_pays<OpFwGradPointwise>(a.B, len, a.H, a.D)) {
    LACT_TRY(encode_map(&P.b[2], w1, 64, 32));  // a CTA's half of these columns: atoms of 32
    return launch_pair(g, stream, kClsGradPointwise);
  }
  return launch_gemm(g, stream, kClsGradPointwise);
}

// Whether an update of `len` tokens runs as one launch (grad_fused.cuh): by an estimate of both in us (they give the same bits; sums that
// choose_split cuts stay cut).  One launch: rounds of CTAs, two per pair of SMs, each with its chain of tiles; a last round of few CTAs takes as
// long as a full one.  Two: tiles of both over the SMs and what the planes between them cost in memory.  Fitted to 645 gradients and 436
// whole updates (1 to 96 entries, h = 128 to 512, 16 to 5632 tokens) timed both ways: in 26 the chosen way is more than 3 % slower, at most
// 7 %.  Measured, us per gradient, two launches / one: 12 entries of 128 x 256, 384 tokens 17.1 / 12.6, 1560 30 / 23; 32 entries, 2048 70 / 48;
// 16 entries, 4096 69 / 41.  Chains of few CTAs lose: one entry, 2048 tokens 21 / 25; so does a short last round: 20 entries, 780
// tokens 26 / 29, 40 entries, 16 tokens 21 / 25.
bool grad_in_one_launch(int64_t B, int64_t D, int64_t H, int64_t len) {
  if (D != kGradD || H % kBM != 0 || len < 1 || choose_split(ceil_div(len, kBK)).splits > 1) return false;
  const int64_t sms = sm_count(), tiles = ceil_div(len, 128);
  const double one = 4.0 + ceil_div(B * (H / kGradSlice), sms) * (0.97 * tiles + 5.9);
  const double two = 11.8 + 1.03 * ceil_div(B * tiles * (H / 64), sms) + ceil_div(B * (3 * H / kBM), sms) * (0.27 * tiles + 1.9) +
                     2.03 * (B * tiles * (H / 64)) / sms;
  return one < two;
}

int run_grad_fused(const GradArgs& a, int32_t* status, cudaStream_t stream) {
  GradFusedArgs g;
  std::memset(&g, 0, sizeof(g));
  LACT_TRY(encode_map(&g.k, Mat{a.k, a.end, a.D, a.k_ts, a.B, a.k_bs}, 128));
  LACT_TRY(encode_map(&g.v, Mat{a.v, a.end, a.D, a.v_ts, a.B, a.v_bs}, 128));
  LACT_TRY(encode_map(&g.w02, Mat{a.w02b, 2 * a.H, a.D, a.D, a.B, 2 * a.H * a.D}, kGradSlice));
  LACT_TRY(encode_map(&g.w1, Mat{a.w1b, a.D, a.H, a.H, a.B, a.D * a.H}, 128, kGradSlice));
  g.lr = EpiFwGrad{a.lr0, a.lr1, a.lr2, a.lr_f32, static_cast<int32_t>(a.start), a.lr_bs, a.w_scale};
  g.e[0] = EpiDW{a.g02, 2 * a.H * a.D, a.D, a.beta, 1, a.g_f32, a.partial02, 0, 0, a.gb02, a.g02_prev, a.fresh};
  g.e[1] = EpiDW{a.g1, a.D * a.H, a.H, a.beta, 1, a.g_f32, a.partial1, 0, 0, a.gb1, a.g1_prev, a.fresh};
  g.start = static_cast<int32_t>(a.start);
  g.len = static_cast<int32_t>(a.end - a.start);
  g.H = static_cast<int32_t>(a.H);
  g.status = status;
  const int64_t ctas = a.B * (a.H / kGradSlice);
  if (ctas > 0x7FFFFFFFll) return LACT_ERR_SHAPE;
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(grad_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GradSmem::kBytes));
      if (dev < 64) configured[dev] = true;
    }
  }
  KernelScope scope(kClsGradContract, stream);
  LACT_CUDA(launch_pdl(grad_gemm_kernel, dim3(static_cast<unsigned>(ctas)), dim3(kGradThreads), GradSmem::kBytes, stream, g));
  return LACT_OK;
}

int run_grad(const GradArgs& a, int32_t* status, cudaStream_t stream) {
  const int64_t len = a.end - a.start;
  if (grad_in_one_launch(a.B, a.D, a.H, len)) return run_grad_fused(a, status, stream);
  LACT_TRY(run_grad_pointwise(a, status, stream));
  const Mat km{a.k, a.end, a.D, a.k_ts, a.B, a.k_bs};
  const Mat vm{a.v, a.end, a.D, a.v_ts, a.B, a.v_bs};
  const Mat dy{a.dy02, len, 2 * a.H, 2 * a.H, a.B, len * 2 * a.H};
  const Mat hid{a.hid, len, a.H, a.H, a.B, len * a.H};
  // token contraction: [dw0; dw2] = dy02^T k  and  dw1 = v^T hidden
  const int bt = contract_bt(a.D, a.H);
  const Split split = a.split.part != nullptr ? choose_split(ceil_div(len, kBK)) : Split{1, 0};
  auto fill = [&](auto& g, int btv) -> int {
    auto& P0 = g.prob[0];
    LACT_TRY(make_operand(form_of(P0), &P0.a[0], &P0.ai[0], dy, 1, kBM, 0, 0));
    LACT_TRY(make_operand(form_of(P0), &P0.b[0], &P0.bi[0], km, 1, btv, 0, static_cast<int>(a.start)));
    P0.M = static_cast<int>(2 * a.H); P0.N = static_cast<int>(a.D); P0.K = static_cast<int>(len);
    P0.batch = static_cast<int>(a.B);
    P0.ep = EpiDW{a.g02, 2 * a.H * a.D, a.D, a.beta, 1, a.g_f32, a.partial02, ceil_div(2 * a.H, kBM),
                  ceil_div(a.D, btv), a.gb02, a.g02_prev, a.fresh};
    auto& P1 = g.prob[1];
    LACT_TRY(make_operand(form_of(P1), &P1.a[0], &P1.ai[0], vm, 1, kBM, 0, static_cast<int>(a.start)));
    LACT_TRY(make_operand(form_of(P1), &P1.b[0], &P1.bi[0], hid, 1, btv, 0, 0));
    P1.M = static_cast<int>(a.D); P1.N = static_cast<int>(a.H); P1.K = static_cast<int>(len);
    P1.batch = static_cast<int>(a.B);
    P1.ep = EpiDW{a.g1, a.D * a.H, a.H, a.beta, 1, a.g_f32, a.partial1, ceil_div(a.D, kBM), ceil_div(a.H, btv),
                  a.gb1, a.g1_prev, a.fresh};
    set_split(P0, split, a.split);
    set_split(P1, split, a.split);
    g.status = status;
    return LACT_OK;
  };
  return launch_op<OpDW, 2>(bt, fill, stream, kClsGradContract, 2);
}

// Newton-Schulz coefficient schedules.
const float kNsTuned[5][3] = {{4.0848f, -6.8946f, 2.9270f},
                              {3.9505f, -6.3029f, 2.6377f},
                              {3.7418f, -5.5913f, 2.3037f},
                              {2.8769f, -3.1427f, 1.2046f},
                              {2.8366f, -3.0525f, 1.2012f}};
const float kNsConst[3] = {3.4445f, -4.7750f, 2.0315f};

constexpr int kNsMaxParts = 512;

// One group of equally shaped gradient matrices [R][C] under iteration.  The iterate X keeps the
// gradient's own [R][C] layout.  With m = min(R, C), n = max(R, C) the Gram matrix is m x m:
//   wide (R <= C):               A = X X^T   (operands K-major),       X' = P X    (X read MN-major)
//   tall (R > C, `transposed`):  A = X^T X   (operands MN-major),      X' = X P^T  (P's rows as K-major B operand)
// which is the reference's "transpose, iterate, transpose back" without moving data.
struct NsGroup {
  int32_t nmat, R, C, m, n, transposed;
  bf16 *xa, *xb;              // ping-pong iterates, nmat * R * C each
  bf16 *gram, *poly;  // [nmat][m][m]: shifted Gram matrix S = A + (b / 2c) I and polynomial P
  float* partial;             // [nmat][<= kNsMaxParts] partial sums of squares
  float* scale;               // [nmat] 1 / (||G||_F + 1e-7) when the first iterate is the unscaled bf16(G)
  uint32_t* done;             // [nmat] tile completion counters of the fused kernel
};

inline size_t ns_group_bytes(int64_t nmat, int64_t m, int64_t n) {
  return static_cast<size_t>(nmat) * (2 * m * n + 3 * m * m) * 2 + static_cast<size_t>(nmat) * kNsMaxParts * 4 +
         static_cast<size_t>(nmat) * 8 + 8 * 256;
}

void ns_group_init(NsGroup& g, int64_t nmat, int64_t R, int64_t C, int gram_right) {
  g.nmat = static_cast<int32_t>(nmat);
  g.R = static_cast<int32_t>(R);
  g.C = static_cast<int32_t>(C);
  g.m = static_cast<int32_t>(std::min(R, C));
  g.n = static_cast<int32_t>(std::max(R, C));
  g.transposed = (R > C) || (R == C && gram_right);
}

// columns of the update product's output: X' is [R][C] = [m][n] (wide) or [n][m] (tall)
inline int ns_upd_cols(const NsGroup& g) { return g.transposed ? g.m : g.n; }
inline int ns_upd_rows(const NsGroup& g) { return g.transposed ? g.n : g.m; }

// Start of the iteration for one or two groups (src[g]: [nmat][R][C], contiguous).
//   scaled = 1: the first iterate X0 = bf16(bf16(G) / (||G|| + 1e-7)) is written to grp[g].xa
//               (norm partials from `fused_parts`, or computed here);
//   scaled = 0: the first iterate is bf16(G), already in grp[g].xa with `fused_parts` partial sums
//               per matrix; only the scale factors 1 / (||G|| + 1e-7) are computed.
int launch_ns_prepare(const NsGroup* grp, int ngroups, const void* const* src, int src_f32, int scaled,
                      cudaStream_t stream, const int* fused_parts = nullptr) {
  NsPrepArgs pa;
  std::memset(&pa, 0, sizeof(pa));
  pa.ngroups = ngroups;
  int nmat = 0, tiles = 0;
  bool need_sumsq = false;
  for (int g = 0; g < ngroups; ++g) {
    const NsGroup& G = grp[g];
    const int parts = (fused_parts != nullptr && fused_parts[g] > 0) ? fused_parts[g] : kNsSlabs;
    if (fused_parts == nullptr || fused_parts[g] <= 0) need_sumsq = true;
    pa.grp[g] = NsPrepGroup{src[g], src_f32, G.nmat, G.R, G.C, G.xa, G.partial, parts, G.scale, G.done};
    nmat += G.nmat;
    tiles = std::max(tiles, ceil_div(G.R, 64) * ceil_div(G.C, 64));
  }
  if (need_sumsq) {
    if (fused_parts != nullptr) return LACT_ERR_CONFIG;  // all groups or none
    KernelScope scope(kClsNsPrepare, stream);
    LACT_CUDA(launch_pdl(ns_sumsq_kernel, dim3(nmat, kNsSlabs), dim3(256), 0, stream, pa));
  }
  KernelScope scope(kClsNsPrepare, stream);
  if (scaled) LACT_CUDA(launch_pdl(ns_scale_kernel, dim3(nmat, tiles), dim3(256), 0, stream, pa));
  else LACT_CUDA(launch_pdl(ns_den_kernel, dim3(ceil_div(nmat, 4)), dim3(128), 0, stream, pa));
  return LACT_OK;
}

// Fills the three contractions of one iteration of group G, reading the iterate `cur` and writing
// `nxt` (both [nmat][R][C]).  PG / PP / PU: GemmProblem<OpNs<..>> of the gram, poly and update phase.
template <class PG, class PP, class PU>
int wire_ns_group(const NsGroup& G, bf16* cur, bf16* nxt, int bt_mm, int bt_mn, PG& gram, PP& poly, PU& upd) {
  const int64_t mm = static_cast<int64_t>(G.m) * G.m, rc = static_cast<int64_t>(G.R) * G.C;
  const Mat X{cur, G.R, G.C, G.C, G.nmat, rc};
  const Mat XN{nxt, G.R, G.C, G.C, G.nmat, rc};
  const Mat S{G.gram, G.m, G.m, G.m, G.nmat, mm};
  const Mat PB{G.poly, G.m, G.m, G.m, G.nmat, mm};
  const int tall = G.transposed;
  // gram: S = X X^T (wide) / X^T X (tall) + (b / 2c) I
  LACT_TRY(make_operand(form_of(gram), &gram.a[0], &gram.ai[0], X, tall, kBM, 0, 0));
  LACT_TRY(make_operand(form_of(gram), &gram.b[0], &gram.bi[0], X, tall, bt_mm, 0, 0));
  gram.M = G.m; gram.N = G.m; gram.K = G.n; gram.batch = G.nmat;
  LACT_TRY(make_output(form_of(gram), &gram.out[0], &gram.oi[0], S, 0, 0));
  // poly: P = c S S + (a - b^2 / 4c) I   (S is exactly symmetric: its rows serve as the K-major B operand too)
  LACT_TRY(make_operand(form_of(poly), &poly.a[0], &poly.ai[0], S, 0, kBM, 0, 0));
  LACT_TRY(make_operand(form_of(poly), &poly.b[0], &poly.bi[0], S, 0, bt_mm, 0, 0));
  poly.M = G.m; poly.N = G.m; poly.K = G.m; poly.batch = G.nmat;
  LACT_TRY(make_output(form_of(poly), &poly.out[0], &poly.oi[0], PB, 0, 0));
  // update: X' = poly X (wide; X is [k][n]: MN-major B operand) / X' = X poly^T (tall)
  if (!tall) {
    LACT_TRY(make_operand(form_of(upd), &upd.a[0], &upd.ai[0], PB, 0, kBM, 0, 0));
    LACT_TRY(make_operand(form_of(upd), &upd.b[0], &upd.bi[0], X, 1, bt_mn, 0, 0));
  } else {
    LACT_TRY(make_operand(form_of(upd), &upd.a[0], &upd.ai[0], X, 0, kBM, 0, 0));
    LACT_TRY(make_operand(form_of(upd), &upd.b[0], &upd.bi[0], PB, 0, bt_mn, 0, 0));
  }
  upd.M = ns_upd_rows(G); upd.N = ns_upd_cols(G); upd.K = G.m; upd.batch = G.nmat;
  LACT_TRY(make_output(form_of(upd), &upd.out[0], &upd.oi[0], XN, 0, 0));
  return LACT_OK;
}

inline void ns_tile_widths(const NsGroup* grp, int ngroups, int* bt_mm, int* bt_mn) {
  const NsGroup& G0 = grp[0];
  const NsGroup& G1 = grp[ngroups - 1];
  *bt_mm = choose_bt({{G0.m, static_cast<int64_t>(G0.nmat) * G0.m}, {G1.m, static_cast<int64_t>(G1.nmat) * G1.m}});
  *bt_mn = choose_bt({{ns_upd_cols(G0), static_cast<int64_t>(G0.nmat) * ns_upd_rows(G0)},
                      {ns_upd_cols(G1), static_cast<int64_t>(G1.nmat) * ns_upd_rows(G1)}});
}

// Runs `steps` iterations on one or two groups, one launch per contraction (every launch covers
// all groups).  The first iterate is grp[g].xa (scaled unless `unscaled_first`, in which case the
// scale factors grp[g].scale are folded into the first iteration).
// result[g] = buffer holding the final iterate of group g.
int run_ns_iterations(const NsGroup* grp, int ngroups, int steps, int const_coeffs, const bf16** result,
                      int32_t* status, cudaStream_t stream, int unscaled_first = 0, int coef_offset = 0) {
  // `steps` iterations of the schedule starting at iteration `coef_offset` (the tuned table has five
  // entries; the public entry points insist on all five)
  if (ngroups < 1 || ngroups > 2) return LACT_ERR_CONFIG;
  if (!const_coeffs && steps + coef_offset > 5) return LACT_ERR_CONFIG;
  bf16* cur[2];
  bf16* nxt[2];
  for (int g = 0; g < ngroups; ++g) { cur[g] = grp[g].xa; nxt[g] = grp[g].xb; }
  int bt_mm = 0, bt_mn = 0;
  ns_tile_widths(grp, ngroups, &bt_mm, &bt_mn);
  for (int it = 0; it < steps; ++it) {
    const float* co = const_coeffs ? kNsConst : kNsTuned[it + coef_offset];
    const int fold = (it == 0 && unscaled_first) ? 1 : 0;
    // which = 0 gram, 1 poly, 2 update: every fill wires all three and keeps the one it launches
    auto fill = [&](auto& ga, int btv, int which) -> int {
      using Prob = std::remove_reference_t<decltype(ga.prob[0])>;
      for (int g = 0; g < ngroups; ++g) {
        Prob pg, pp, pu;
        std::memset(&pg, 0, sizeof(Prob)); std::memset(&pp, 0, sizeof(Prob)); std::memset(&pu, 0, sizeof(Prob));
        LACT_TRY(wire_ns_group(grp[g], cur[g], nxt[g], btv, btv, pg, pp, pu));
        const float* sc = fold ? grp[g].scale : nullptr;
        if (which == 0) { ga.prob[g] = pg; ga.prob[g].ep = EpiNs{co[1] / (2.f * co[2]), 1.f, sc, fold ? 2 : 0}; }
        if (which == 1) {
          ga.prob[g] = pp;
          ga.prob[g].ep = EpiNs{co[0] - co[1] * co[1] / (4.f * co[2]), co[2], nullptr, 0};
        }
        if (which == 2) { ga.prob[g] = pu; ga.prob[g].ep = EpiNs{0.f, 1.f, sc, fold ? 1 : 0}; }
      }
      ga.status = status;
      return LACT_OK;
    };
    LACT_TRY((launch_op<OpNs, 2>(bt_mm, [&](auto& ga, int btv) { return fill(ga, btv, 0); }, stream, kClsNsGram, ngroups)));
    LACT_TRY((launch_op<OpNs, 2>(bt_mm, [&](auto& ga, int btv) { return fill(ga, btv, 1); }, stream, kClsNsPoly, ngroups)));
    LACT_TRY((launch_op<OpNs, 2>(bt_mn, [&](auto& ga, int btv) { return fill(ga, btv, 2); }, stream, kClsNsUpdate, ngroups)));
    for (int g = 0; g < ngroups; ++g) std::swap(cur[g], nxt[g]);
  }
  for (int g = 0; g < ngroups; ++g) result[g] = cur[g];
  return LACT_OK;
}

// Fused path: all iterations in one cooperative launch.  launch_ns_prepare must have run on the same groups
// just before: it leaves the first iterates in grp[g].xa and clears the completion counters grp[g].done.
// NITER = 2: iterates ping-pong between grp[g].xa / xb, one Gram / polynomial buffer.  NITER > 2 (steps <= NITER):
// every iteration has its own buffers, `keep[g]` = {iterates (steps + 1) x [nmat][R][C] starting with the first
// iterate, shifted Gram matrices steps x [nmat][m][m], polynomials likewise}.
struct NsKeep {
  bf16 *X, *A, *P;
};
template <int BT_MM, int BT_MN, int NITER, bool SYM = false>
int launch_ns_fused(const NsGroup* grp, int ngroups, int steps, int const_coeffs, int32_t* status,
                    cudaStream_t stream, int unscaled_first, const NsKeep* keep = nullptr, int coef_offset = 0) {
  using Args = NsFusedArgs<BT_MM, BT_MN, NITER, SYM>;
  auto kernel = ns_fused_kernel<BT_MM, BT_MN, NITER, SYM>;
  constexpr uint32_t smem = ns_fused_smem_bytes<BT_MM, BT_MN, SYM>();
  static_assert(smem <= 232448, "shared memory budget exceeded");
  static_assert(ns_fused_ring<BT_MM, BT_MN, SYM>() >= 2, "ring too shallow");
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (dev < 64) configured[dev] = true;
    }
  }
  if (NITER > 2 && (keep == nullptr || steps > NITER)) return LACT_ERR_CONFIG;
  // the argument block (a few KB per problem set) lives on the heap: it is copied at launch
  std::vector<uint8_t> storage(sizeof(Args));
  Args& args = *reinterpret_cast<Args*>(storage.data());
  std::memset(&args, 0, sizeof(args));
  int64_t max_tiles = 1;
  for (int g = 0; g < ngroups; ++g) {
    const NsGroup& G = grp[g];
    const int64_t rc = static_cast<int64_t>(G.nmat) * G.R * G.C, mm = static_cast<int64_t>(G.nmat) * G.m * G.m;
    for (int par = 0; par < NITER; ++par) {
      NsGroup Gi = G;
      bf16 *cur, *nxt;
      if (NITER == 2) {
        cur = par == 0 ? G.xa : G.xb;
        nxt = par == 0 ? G.xb : G.xa;
      } else {
        cur = keep[g].X + rc * par;
        nxt = keep[g].X + rc * (par + 1);
        Gi.gram = keep[g].A + mm * par;
        Gi.poly = keep[g].P + mm * par;
      }
      LACT_TRY(wire_ns_group(Gi, cur, nxt, BT_MM, BT_MN, args.gram[par][g], args.poly[par][g], args.upd[par][g]));
    }
    args.scale[g] = unscaled_first ? G.scale : nullptr;
    max_tiles = std::max<int64_t>(max_tiles, static_cast<int64_t>(G.nmat) * ceil_div(ns_upd_rows(G), kBM) *
                                                 ceil_div(ns_upd_cols(G), BT_MN) * ngroups);
  }
  for (int it = 0; it < steps; ++it) {
    const float* co = const_coeffs ? kNsConst : kNsTuned[it + coef_offset];
    args.coef[it][0] = co[0]; args.coef[it][1] = co[1]; args.coef[it][2] = co[2];
  }
  args.steps = steps;
  args.ngroups = ngroups;
  args.status = status;
  for (int g = 0; g < ngroups; ++g) args.done[g] = grp[g].done;  // cleared by launch_ns_prepare
  const int grid = static_cast<int>(std::min<int64_t>(sm_count(), std::max<int64_t>(max_tiles, 8)));
  void* kargs[] = {&args};
  KernelScope scope(kClsNsFused, stream);
  LACT_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kernel), dim3(grid), dim3(kGemmThreadsFlow), kargs, smem,
                                        stream));
  return LACT_OK;
}

// Picks the fused kernel instantiated for the tile widths this problem wants; returns
// LACT_ERR_CONFIG when there is none (the caller then runs the multi-launch path).
int try_ns_fused(const NsGroup* grp, int ngroups, int steps, int const_coeffs, int32_t* status,
                 cudaStream_t stream, const bf16** result, int unscaled_first = 0, const NsKeep* keep = nullptr) {
  if (steps < 1 || steps > kNsFusedMaxSteps) return LACT_ERR_CONFIG;
  if (!const_coeffs && steps != 5) return LACT_ERR_CONFIG;
  if (keep != nullptr && steps > 5) return LACT_ERR_CONFIG;
  int bt_mm = 0, bt_mn = 0;
  ns_tile_widths(grp, ngroups, &bt_mm, &bt_mn);
  for (int g = 0; g < ngroups; ++g) {
    if (keep != nullptr) result[g] = keep[g].X + static_cast<int64_t>(grp[g].nmat) * grp[g].R * grp[g].C * steps;
    else result[g] = (steps % 2 == 0) ? grp[g].xa : grp[g].xb;
  }
  // Few matrices per launch (a small (batch x head) shard): the kernel is bound by the 15-phase chain of each
  // matrix, not by throughput, so narrower tiles that spread every phase over more SMs (and shorten the serial
  // work per tile) win.  Tiles of the Gram phase at width bt over all groups:
  auto gram_tiles = [&](int bt) {
    int64_t t = 0;
    for (int g = 0; g < ngroups; ++g) t += static_cast<int64_t>(grp[g].nmat) * ceil_div(grp[g].m, kBM) * ceil_div(grp[g].m, bt);
    return t;
  };
  // keep == nullptr: iterates ping-pong (two problem sets); else every iteration keeps its buffers (five sets)
#define LACT_NS_FUSED(BTV)                                                                                          \
  (keep == nullptr ? launch_ns_fused<BTV, BTV, 2>(grp, ngroups, steps, const_coeffs, status, stream, unscaled_first) \
                   : launch_ns_fused<BTV, BTV, 5>(grp, ngroups, steps, const_coeffs, status, stream, unscaled_first, keep))
  const int64_t want = static_cast<int64_t>(sm_count()) * 3 / 4;
  // Gram side a multiple of 128 in every group and plenty of matrices: the symmetric phases (Gram matrix, polynomial)
  // run on 128 x 128 tiles on and above the diagonal only, the update keeps its 192-wide tiles.  With fewer matrices
  // (measured at D = H = 384: 16 and 12 units, i.e. under 1.5 Gram tiles of width 192 per SM) the symmetric phases
  // leave a second, nearly empty round of tiles and plain 128-wide tiles are 4-5 % faster; from 20 units up the
  // symmetric variant wins.
  // Gram sides that 256 divides run on the same tiles; the training forward (`keep`) refuses them as it always has.  Five iterations on
  // 3, 24, 48 and 96 square matrices by themselves, us, one launch per product / this kernel: side 256 125, 128, 134, 189 / 76, 86, 99,
  // 140; side 512 150, 221, 319, 613 / 94, 154, 233, 469; side 768 195, 422, 855, 1680 / 145, 320, 655, 1357.  (Three tiles of four are
  // no gain: 256 stays plain.)
  const bool by256 = keep == nullptr && bt_mm == 256 && bt_mn != 64;
  const bool wide = bt_mm == 192 && bt_mn == 192;
  bool symmable = wide || by256;
  for (int g = 0; g < ngroups; ++g) symmable = symmable && grp[g].m % kBM == 0 && grp[g].m >= 3 * kBM;
  if (symmable && gram_tiles(192) >= static_cast<int64_t>(sm_count()) * 3 / 2)
    return keep == nullptr
               ? launch_ns_fused<128, 192, 2, true>(grp, ngroups, steps, const_coeffs, status, stream, unscaled_first)
               : launch_ns_fused<128, 192, 5, true>(grp, ngroups, steps, const_coeffs, status, stream, unscaled_first, keep);
  if (wide && !symmable && gram_tiles(192) >= want) return LACT_NS_FUSED(192);
  // (256-wide update tiles would leave a ring of four stages: 128 is used)
  const bool ok128 = wide || by256 || (bt_mm == 128 && (bt_mn == 128 || bt_mn == 256));
  if (ok128 && (gram_tiles(128) >= want || gram_tiles(64) == gram_tiles(128))) return LACT_NS_FUSED(128);
  if (ok128 || (bt_mm == 64 && bt_mn == 64)) return LACT_NS_FUSED(64);
#undef LACT_NS_FUSED
  return LACT_ERR_CONFIG;
}

// All of Newton-Schulz, normalisation included, by one CTA per matrix (ns_chip.cuh); every group must fit an SM.
// src[g]: gradients (read unless `unscaled`, when the bf16 gradient is already in grp[g].xa); parts[g]: partial sums of
// squares per matrix in grp[g].partial, or 0 / nullptr: the kernel adds them up itself.
int launch_ns_chip(const NsGroup* grp, int ngroups, const void* const* src, int src_f32, const int* parts, int unscaled,
                   int steps, int const_coeffs, int32_t* status, cudaStream_t stream, const bf16** result, const NsKeep* keep) {
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(ns_chip_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNsChipSmem));
      if (dev < 64) configured[dev] = true;
    }
  }
  NsChipArgs a;
  std::memset(&a, 0, sizeof(a));
  int64_t ctas = 0;
  for (int g = 0; g < ngroups; ++g) {
    const NsGroup& G = grp[g];
    NsChipGroup& K = a.grp[g];
    const int64_t rc = static_cast<int64_t>(G.R) * G.C, mm = static_cast<int64_t>(G.m) * G.m;
    K.nmat = G.nmat; K.R = G.R; K.C = G.C; K.m = G.m; K.n = G.n; K.tall = G.transposed;
    K.box_rows = G.R <= 256 ? G.R : G.R / 2;
    K.two = ns_chip_fits(G.R, G.C, G.transposed, true);
    K.src = src[g]; K.src_f32 = src_f32;
    K.nparts = parts != nullptr ? parts[g] : 0;
    K.partial = K.nparts > 0 ? G.partial : nullptr;
    if (unscaled) LACT_TRY(encode_map(&K.x_in, Mat{G.xa, G.R, G.C, G.C, G.nmat, rc}, static_cast<uint32_t>(K.box_rows)));
    bf16* out = keep != nullptr ? keep[g].X : G.xb;
    LACT_TRY(encode_map(&K.x_out, Mat{out, G.R, G.C, G.C, keep != nullptr ? static_cast<int64_t>(steps + 1) * G.nmat : G.nmat, rc},
                        static_cast<uint32_t>(K.box_rows)));
    result[g] = keep != nullptr ? keep[g].X + rc * G.nmat * steps : G.xb;
    if (keep != nullptr) {
      const int64_t all = static_cast<int64_t>(steps) * G.nmat;
      LACT_TRY(encode_map(&K.s_out, Mat{keep[g].A, G.m, G.m, G.m, all, mm}, static_cast<uint32_t>(G.m)));
      LACT_TRY(encode_map(&K.p_out, Mat{keep[g].P, G.m, G.m, G.m, all, mm}, static_cast<uint32_t>(G.m)));
    }
    ctas += G.nmat;
  }
  for (int it = 0; it < steps; ++it) {
    const float* co = const_coeffs ? kNsConst : kNsTuned[it];
    a.coef[it][0] = co[0]; a.coef[it][1] = co[1]; a.coef[it][2] = co[2];
  }
  a.ngroups = ngroups;
  a.steps = steps;
  a.load = unscaled;
  a.keep = keep != nullptr;
  a.status = status;
  KernelScope scope(kClsNsFused, stream);
  LACT_CUDA(launch_pdl(ns_chip_kernel, dim3(static_cast<unsigned>(ctas)), dim3(kNsChipThreads), kNsChipSmem, stream, a));
  return LACT_OK;
}

// Newton-Schulz of one or two groups by the best path: one CTA per matrix where the matrices fit an SM, however many there
// are, else the preparation kernels and the dataflow kernel, else one launch per product.  (The whole call, one CTA per matrix
// against preparation and dataflow, us: 64 x 128, 1 / 32 / 192 / 1200 matrices 25 / 27 / 43 / 153 against 86 / 87 / 111 / 260;
// 128 x 256 39 / 39 / 72 / 299 against 99 / 104 / 135 / 545; 192 x 192 53 / 55 / 104 / 442 against 104 / 119 / 172 / 901.)  `unscaled`: grp[g].xa holds bf16(G) and
// the normalisation is folded into the first iteration.
int run_newton_schulz(NsGroup* grp, int ngroups, const void* const* src, int src_f32, const int* parts, int unscaled, int steps,
                      int const_coeffs, int32_t* status, cudaStream_t stream, const bf16** result, const NsKeep* keep = nullptr) {
  bool chip = steps >= 1 && steps <= 16 && (const_coeffs || steps == 5);
  for (int g = 0; g < ngroups; ++g)  // (that kernel reads 16 bytes of the gradients at a time, the others half of that in bf16)
    chip = chip && ns_chip_fits(grp[g].R, grp[g].C, grp[g].transposed) && (reinterpret_cast<uintptr_t>(src[g]) & 15) == 0;
  const bool given = parts != nullptr && parts[0] > 0;
  if (chip) return launch_ns_chip(grp, ngroups, src, src_f32, given ? parts : nullptr, unscaled, steps, const_coeffs, status, stream,
                                  result, keep);
  LACT_TRY(launch_ns_prepare(grp, ngroups, src, src_f32, !unscaled, stream, given ? parts : nullptr));
  const int rc = try_ns_fused(grp, ngroups, steps, const_coeffs, status, stream, result, unscaled, keep);
  if (rc != LACT_ERR_CONFIG || keep != nullptr) return rc;
  return run_ns_iterations(grp, ngroups, steps, const_coeffs, result, status, stream, unscaled);
}

// ------------------------------------------------------------------------------------------
// workspace planning
// ------------------------------------------------------------------------------------------
struct Carver {
  uint8_t* base;
  size_t off = 0;
  explicit Carver(void* b) : base(static_cast<uint8_t*>(b)) {}
  template <class T>
  T* take(size_t count) {
    off = (off + 255) & ~static_cast<size_t>(255);
    T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
    off += count * sizeof(T);
    return p;
  }
};

struct NsPlan {
  int ngroups;
  NsGroup grp[2];
};

void carve_ns_group(Carver& c, NsGroup& g) {
  const size_t mn = static_cast<size_t>(g.nmat) * g.m * g.n, mm = static_cast<size_t>(g.nmat) * g.m * g.m;
  g.xa = c.take<bf16>(mn);
  g.xb = c.take<bf16>(mn);
  g.gram = c.take<bf16>(mm);
  g.poly = c.take<bf16>(mm);
  g.partial = c.take<float>(static_cast<size_t>(g.nmat) * kNsMaxParts);
  g.scale = c.take<float>(static_cast<size_t>(g.nmat));
  g.done = c.take<uint32_t>(static_cast<size_t>(g.nmat));
}

// Group 0 orthogonalises the [w0; w2] gradient (concat: B matrices [2H][D]; separate: 2B matrices
// [H][D], w0 and w2 of batch b at 2b, 2b+1), group 1 the w1 gradient (B matrices [D][H]).
void plan_ns(Carver& c, int64_t B, int64_t D, int64_t H, int concat, int gram_right, NsPlan* plan) {
  plan->ngroups = 2;
  if (concat) ns_group_init(plan->grp[0], B, 2 * H, D, gram_right);
  else ns_group_init(plan->grp[0], 2 * B, H, D, gram_right);
  ns_group_init(plan->grp[1], B, D, H, gram_right);
  carve_ns_group(c, plan->grp[0]);
  carve_ns_group(c, plan->grp[1]);
}

// Trace layout in the caller's buffer (bf16 unless noted): group scratch (norm partials,
// scale factors); X[0..steps] ([B][R][C] each); shifted Gram matrix A + (b/2c) I and polynomial P per iteration
// ([B][m][m]); then the backward's temporaries: c A + (b/2) I, Q, S ([B][m][m]) and two [B][R][C] gradient buffers.
struct NsTrace {
  NsGroup grp;
  bf16* X;   // (steps + 1) iterates
  bf16 *A, *P;  // steps matrices each (A: the shifted Gram matrix)
  bf16 *CB, *Q, *S, *dXa, *dXb;
  size_t bytes;
};

int plan_ns_trace(void* base, int64_t B, int64_t R, int64_t C, int steps, int gram_right, NsTrace* t) {
  if (B < 1 || B > 65535 || R < 8 || C < 8 || (R % 8) || (C % 8) || steps < 1 || steps > 16) return LACT_ERR_SHAPE;
  Carver cv(base);
  ns_group_init(t->grp, B, R, C, gram_right);
  const size_t rc = static_cast<size_t>(B) * R * C, mm = static_cast<size_t>(B) * t->grp.m * t->grp.m;
  t->grp.partial = cv.take<float>(static_cast<size_t>(B) * kNsMaxParts);
  t->grp.scale = cv.take<float>(B);
  t->grp.done = cv.take<uint32_t>(static_cast<size_t>(B) + 64);
  t->X = cv.take<bf16>(rc * (steps + 1));
  t->A = cv.take<bf16>(mm * steps);
  t->P = cv.take<bf16>(mm * steps);
  t->CB = cv.take<bf16>(mm);
  t->Q = cv.take<bf16>(mm);
  t->S = cv.take<bf16>(mm);
  t->dXa = cv.take<bf16>(rc);
  t->dXb = cv.take<bf16>(rc);
  t->bytes = cv.off + 256;
  return LACT_OK;
}


static int ns_norm_bwd_launch(const float* g, const void* dx0, int dx_bf16, float* dg, float* partials, int64_t nmat,
                              int64_t elems, cudaStream_t s) {
  if (nmat < 1 || nmat > 65535 * 16 || elems < 4 || (elems % 4) != 0) return LACT_ERR_SHAPE;
  if (((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(dx0) | reinterpret_cast<uintptr_t>(dg)) & 15) != 0)
    return LACT_ERR_SHAPE;
  const dim3 grid(static_cast<unsigned>(nmat), kNormBwdSlices);
  {
    KernelScope scope(kClsOther, s);
    ns_norm_bwd_partial_kernel<<<grid, 512, 0, s>>>(g, dx0, dx_bf16, partials, elems);
    LACT_CUDA(cudaGetLastError());
  }
  KernelScope scope(kClsOther, s);
  ns_norm_bwd_apply_kernel<<<grid, 512, 0, s>>>(g, dx0, dx_bf16, dg, partials, elems);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

// ---- all iterations of the Newton-Schulz backward of one or two groups in one cooperative launch
template <int BT_MM, int BT, bool SYM>
static int launch_ns_bwd_fused(const NsTrace* tr, const bf16* const* du, int ngroups, int steps, int const_coeffs,
                               int32_t* status, cudaStream_t stream) {
  constexpr int NITER = 5;
  using Args = NsBwdFusedArgs<BT_MM, BT, NITER, SYM>;
  auto kernel = ns_bwd_fused_kernel<BT_MM, BT, NITER, SYM>;
  constexpr uint32_t smem = ns_bwd_smem_bytes<BT_MM, BT, SYM>();
  static_assert(smem <= 232448, "shared memory budget exceeded");
  static_assert(ns_bwd_ring<BT_MM, BT, SYM>() >= 2, "ring too shallow");
  static_assert(sizeof(Args) <= 32000, "kernel parameter block too large");
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (dev < 64) configured[dev] = true;
    }
  }
  std::vector<uint8_t> storage(sizeof(Args));
  Args& args = *reinterpret_cast<Args*>(storage.data());
  std::memset(&args, 0, sizeof(args));
  int64_t max_tiles = 1;
  for (int g = 0; g < ngroups; ++g) {
    const NsTrace& t = tr[g];
    const NsGroup& G = t.grp;
    const int64_t rc1 = static_cast<int64_t>(G.R) * G.C, mm1 = static_cast<int64_t>(G.m) * G.m;
    const int64_t rc = rc1 * G.nmat, mm = mm1 * G.nmat;
    const int tall = G.transposed;
    const Mat Q{t.Q, G.m, G.m, G.m, G.nmat, mm1};
    const Mat T{t.S, G.m, G.m, G.m, G.nmat, mm1};
    const bf16* dX = du[g];
    for (int it = steps - 1; it >= 0; --it) {
      bf16* out = (it & 1) ? t.dXa : t.dXb;
      const Mat X{t.X + rc * it, G.R, G.C, G.C, G.nmat, rc1};
      const Mat D{dX, G.R, G.C, G.C, G.nmat, rc1};
      const Mat O{out, G.R, G.C, G.C, G.nmat, rc1};
      const Mat S{t.A + mm * it, G.m, G.m, G.m, G.nmat, mm1};
      const Mat PB{t.P + mm * it, G.m, G.m, G.m, G.nmat, mm1};
      auto& pq = args.q[it][g];
      auto& pt = args.t[it][g];
      auto& px = args.dx[it][g];
      // Q = dX X^T + X dX^T (wide; the iterate's rows are K-major operands) / dX^T X + X^T dX (tall; MN-major)
      LACT_TRY(make_operand(OperandForm{false}, &pq.a[0], &pq.ai[0], D, tall, kBM, 0, 0));
      LACT_TRY(make_operand(OperandForm{false}, &pq.b[0], &pq.bi[0], X, tall, BT_MM, 0, 0));
      LACT_TRY(make_operand(OperandForm{false}, &pq.a[1], &pq.ai[1], X, tall, kBM, 0, 0));
      LACT_TRY(make_operand(OperandForm{false}, &pq.b[1], &pq.bi[1], D, tall, BT_MM, 0, 0));
      pq.M = G.m; pq.N = G.m; pq.K = G.n; pq.batch = G.nmat;
      LACT_TRY(make_output(form_of(pq), &pq.out[0], &pq.oi[0], Q, 0, 0));
      // T = c (S Q + Q S): all three symmetric, rows serve as K-major operands on either side
      LACT_TRY(make_operand(OperandForm{false}, &pt.a[0], &pt.ai[0], S, 0, kBM, 0, 0));
      LACT_TRY(make_operand(OperandForm{false}, &pt.b[0], &pt.bi[0], Q, 0, BT_MM, 0, 0));
      LACT_TRY(make_operand(OperandForm{false}, &pt.a[1], &pt.ai[1], Q, 0, kBM, 0, 0));
      LACT_TRY(make_operand(OperandForm{false}, &pt.b[1], &pt.bi[1], S, 0, BT_MM, 0, 0));
      pt.M = G.m; pt.N = G.m; pt.K = G.m; pt.batch = G.nmat;
      LACT_TRY(make_output(form_of(pt), &pt.out[0], &pt.oi[0], T, 0, 0));
      // dX_i = P dX + T X (wide: the [k][n] iterates are MN-major B operands) / dX P + X T (tall)
      if (!tall) {
        LACT_TRY(make_operand(OperandForm{false}, &px.a[0], &px.ai[0], PB, 0, kBM, 0, 0));
        LACT_TRY(make_operand(OperandForm{false}, &px.b[0], &px.bi[0], D, 1, BT, 0, 0));
        LACT_TRY(make_operand(OperandForm{false}, &px.a[1], &px.ai[1], T, 0, kBM, 0, 0));
        LACT_TRY(make_operand(OperandForm{false}, &px.b[1], &px.bi[1], X, 1, BT, 0, 0));
      } else {
        LACT_TRY(make_operand(OperandForm{false}, &px.a[0], &px.ai[0], D, 0, kBM, 0, 0));
        LACT_TRY(make_operand(OperandForm{false}, &px.b[0], &px.bi[0], PB, 0, BT, 0, 0));
        LACT_TRY(make_operand(OperandForm{false}, &px.a[1], &px.ai[1], X, 0, kBM, 0, 0));
        LACT_TRY(make_operand(OperandForm{false}, &px.b[1], &px.bi[1], T, 0, BT, 0, 0));
      }
      px.M = ns_upd_rows(G); px.N = ns_upd_cols(G); px.K = G.m; px.batch = G.nmat;
      LACT_TRY(make_output(form_of(px), &px.out[0], &px.oi[0], O, 0, 0));
      dX = out;
    }
    args.done[g] = G.done;
    LACT_CUDA(cudaMemsetAsync(G.done, 0, sizeof(uint32_t) * G.nmat, stream));
    max_tiles = std::max<int64_t>(max_tiles, static_cast<int64_t>(G.nmat) * ceil_div(ns_upd_rows(G), kBM) *
                                                 ceil_div(ns_upd_cols(G), BT) * ngroups);
  }
  for (int it = 0; it < steps; ++it) args.coef_c[it] = (const_coeffs ? kNsConst : kNsTuned[it])[2];
  args.steps = steps;
  args.ngroups = ngroups;
  args.status = status;
  const int grid = static_cast<int>(std::min<int64_t>(sm_count(), std::max<int64_t>(max_tiles, 8)));
  void* kargs[] = {&args};
  KernelScope scope(kClsOther, stream);
  LACT_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kernel), dim3(grid), dim3(kGemmThreadsFlow), kargs, smem,
                                        stream));
  return LACT_OK;
}


// 4-D map (feature, token, head, batch) of a [b][l][h][d] bf16 activation whose token / batch strides are free
// (views of a fused projection) and whose heads are adjacent; box {64, 128, 1, 1}, 128-byte swizzle.
int encode_map_heads(CUtensorMap* map, const void* ptr, int64_t b, int64_t l, int64_t h, int64_t d, int64_t ts,
                     int64_t bs, uint32_t box_rows = 128) {
  EncodeFn fn = get_encode_fn();
  if (fn == nullptr) return LACT_ERR_CUDA;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || (ts % 8) != 0 || (bs % 8) != 0 || ts < h * d) return LACT_ERR_SHAPE;
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(d), static_cast<cuuint64_t>(l), static_cast<cuuint64_t>(h),
                        static_cast<cuuint64_t>(b)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(ts) * 2, static_cast<cuuint64_t>(d) * 2,
                           static_cast<cuuint64_t>(b > 1 ? bs : ts * l) * 2};
  cuuint32_t box[4] = {64, box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? LACT_OK : LACT_ERR_CUDA;
}

template <int HD>
int launch_swa(const SwaArgs& a, int64_t ctas, cudaStream_t stream) {
  auto kernel = swa_fwd_kernel<HD>;
  constexpr uint32_t smem = SwaSmem<HD>::kBytes;
  static_assert(smem <= 232448, "shared memory budget exceeded");
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (dev < 64) configured[dev] = true;
    }
  }
  KernelScope scope(kClsOther, stream);
  LACT_CUDA(launch_pdl(kernel, dim3(static_cast<unsigned>(ctas)), dim3(320), smem, stream, a));
  return LACT_OK;
}

template <int HD>
int launch_swa_pairs(const SwaPairArgs& a, int64_t ctas, cudaStream_t stream) {
  auto kernel = swa_pairs_kernel<HD>;
  constexpr uint32_t smem = SwaPairSmem<HD>::kBytes;
  static_assert(smem <= 232448, "shared memory budget exceeded");
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (dev < 64) configured[dev] = true;
    }
  }
  KernelScope scope(kClsOther, stream);
  LACT_CUDA(launch_pdl(kernel, dim3(static_cast<unsigned>(ctas)), dim3(kSwaPairThreads), smem, stream, a));
  if (a.cutters > 0) LACT_CUDA(launch_pdl(swa_combine_kernel<HD>, dim3(static_cast<unsigned>(a.rest) * 32), dim3(256), 0, stream, a));
  return LACT_OK;
}

template <int HD, int MODE>
int launch_swa_bwd(const SwaBwdArgs& a, int64_t ctas, cudaStream_t stream) {
  auto kernel = swa_bwd_kernel<HD, MODE>;
  constexpr uint32_t smem = SwaBwdSmem<HD>::kBytes;
  static_assert(smem <= 232448, "shared memory budget exceeded");
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (dev < 64) configured[dev] = true;
    }
  }
  KernelScope scope(kClsOther, stream);
  kernel<<<static_cast<unsigned>(ctas), kSwaBwdThreads, smem, stream>>>(a);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

struct ScanPlan {
  int32_t* status;
  float *W02, *W1, *W02c, *W1c, *n02, *n1, *G02, *G1, *beta;
  bf16 *Wb, *hidden, *dy02, *hid;  // Wb: `w_slots` times [W0W2 | W1]
  int32_t w_slots;
  SplitScratch split;
  int32_t split_tiles;
  NsPlan ns;
  size_t bytes;
};

// How many APPLY steps from step `i` on are left to the last of them, which then runs all in one launch (ApplyArgs::segs): steps
// of one length, evenly spaced, with one UPDATE between each two (so that their weights lie in consecutive slots), whose outputs
// do not overlap.  A step of few tiles costs its launches' fill and drain, in series with the chain of updates.  Steps are collected
// until they have kApplyRounds tiles of 128 tokens and hidden features per SM, which bounds the memory of their hidden activations to
// 58 MB beside one step's, and as long as their weights take no more than kRunWeightBytes: short steps of many weights would fill
// hundreds of slots.  us per call:
//   12 entries of 128 x 256, 21 steps of 1560 tokens: single steps 1674, six tiles per SM 1510, twelve 1473, twenty-four 1466; 4 entries of
//   384, 16 steps of 512 tokens 1795 / 1611 / 1602 / 1617
//   4 entries of 384, 255 steps of 128 tokens: single steps 10035, weights of 16 MB 7008, 64 MB 6310, 128 MB 6255, no bound 6167 (524 MB);
//   16 entries of 512, 16 steps of 512 tokens 1833 / 1837 / 1782 / 1740 / 1710
// `free_slots`: how many weight slots there are from the one of step `i` on.
constexpr int64_t kApplyRounds = 12, kRunWeightBytes = 128 << 20;
// The most steps of `len` tokens that share a launch.
int64_t longest_run(const lact_scan_config& c, int64_t len) {
  const int64_t tiles = c.B * ceil_div(len, kBM) * ceil_div(c.H, kBM);
  return std::max<int64_t>(1, std::min((kApplyRounds * sm_count() + tiles - 1) / tiles, kRunWeightBytes / (c.B * 3 * c.H * c.D * 2)));
}
// Whether APPLY step `i` and the one two steps on may be neighbours in a run.
bool run_goes_on(int32_t n_steps, const int32_t* kind, const int64_t* start, const int64_t* end, int32_t i) {
  const int64_t len = end[i] - start[i];
  return i + 2 < n_steps && kind[i + 1] == LACT_STEP_UPDATE && kind[i + 2] == LACT_STEP_APPLY && len > 0 &&
         end[i + 2] - start[i + 2] == len && start[i + 2] > start[i];
}
struct ApplyRun {
  int64_t steps, x_step, o_step;
};
ApplyRun apply_run(const lact_scan_config& c, int32_t n_steps, const int32_t* kind, const int64_t* start, const int64_t* end,
                   const int64_t* out_start, int32_t i, int64_t free_slots) {
  ApplyRun r{1, 0, 0};
  const int64_t len = end[i] - start[i];
  if (len <= 0) return r;
  const int64_t most = std::min(longest_run(c, len), free_slots);
  for (int32_t at = i; r.steps < most && run_goes_on(n_steps, kind, start, end, at); at += 2) {
    const int64_t dx = start[at + 2] - start[at], dout = out_start[at + 2] - out_start[at];
    if (dout < len) break;
    if (r.steps == 1) {
      r.x_step = dx;
      r.o_step = dout;
    } else if (dx != r.x_step || dout != r.o_step) {
      break;
    }
    ++r.steps;
  }
  return r;
}

int plan_scan(const lact_scan_config& c, int32_t n_steps, const int32_t* kind, const int64_t* start,
              const int64_t* end, void* base, ScanPlan* p) {
  int64_t max_apply = 0, max_update = 0, slots = 1;
  for (int i = 0; i < n_steps; ++i) {
    if (start[i] < 0 || end[i] > c.L || end[i] < start[i]) return LACT_ERR_STEPS;
    const int64_t len = end[i] - start[i];
    if (kind[i] == LACT_STEP_APPLY) {
      max_apply = std::max(max_apply, len);
    } else if (kind[i] == LACT_STEP_UPDATE) {
      if (len <= 0) return LACT_ERR_STEPS;
      max_update = std::max(max_update, len);
    } else return LACT_ERR_STEPS;
  }
  // As many slots as the longest run of evenly spaced steps, wherever it begins (which runs there are also depends on the outputs'
  // places).  A run that does not begin in slot 0 may find fewer and ends earlier.  `even[i & 1]`: steps of the evenly spaced stretch
  // that ends with step i.
  int64_t even[2] = {1, 1};
  for (int i = 0; i < n_steps; ++i) {
    int64_t& n = even[i & 1];
    if (i < 2 || kind[i - 2] != LACT_STEP_APPLY || !run_goes_on(n_steps, kind, start, end, i - 2)) n = 1;
    else n = n > 1 && start[i] - start[i - 2] != start[i - 2] - start[i - 4] ? 2 : n + 1;
    if (kind[i] != LACT_STEP_APPLY || end[i] == start[i]) continue;
    const int64_t len = end[i] - start[i], steps = std::min(n, longest_run(c, len));
    slots = std::max(slots, steps);
    max_apply = std::max(max_apply, steps * len);
  }
  Carver cv(base);
  const size_t B = c.B, D = c.D, H = c.H;
  p->status = cv.take<int32_t>(64);  // device status word
  p->W02 = cv.take<float>(B * 2 * H * D);
  p->W1 = cv.take<float>(B * D * H);
  p->W02c = cv.take<float>(B * 2 * H * D);
  p->W1c = cv.take<float>(B * D * H);
  p->n02 = cv.take<float>(B * 2 * H);
  p->n1 = cv.take<float>(B * D);
  p->G02 = cv.take<float>(B * 2 * H * D);
  p->G1 = cv.take<float>(B * D * H);
  p->beta = cv.take<float>(B * static_cast<size_t>(std::max(1, n_steps)));
  p->w_slots = static_cast<int32_t>(slots);
  p->Wb = cv.take<bf16>(B * 3 * H * D * static_cast<size_t>(slots));
  p->hidden = cv.take<bf16>(B * static_cast<size_t>(max_apply) * H);
  p->dy02 = cv.take<bf16>(B * static_cast<size_t>(max_update) * 2 * H);
  p->hid = cv.take<bf16>(B * static_cast<size_t>(max_update) * H);
  p->split = SplitScratch{};
  const int splits = choose_split(ceil_div(max_update, kBK)).splits;  // (the longest update is cut into the most units)
  p->split_tiles = splits > 1 ? static_cast<int32_t>(contract_tiles(c.B, c.D, c.H)) : 0;
  if (splits > 1) {
    p->split.count = cv.take<uint32_t>(p->split_tiles);
    p->split.part = cv.take<float>(static_cast<size_t>(p->split_tiles) * splits * kBM * contract_bt(c.D, c.H));
  }
  p->ns.ngroups = 0;
  if (c.use_muon && max_update > 0) plan_ns(cv, c.B, c.D, c.H, c.ns_concat, c.ns_gram_right, &p->ns);
  p->bytes = cv.off + 256;
  return LACT_OK;
}

// add + renormalise of one or two weight arrays (a1.B = 0: one); rows of up to 1024 elements
int launch_add_renorm(const RenormArgs& a0, const RenormArgs& a1, cudaStream_t stream) {
  const int64_t rows = static_cast<int64_t>(a0.B) * a0.R + static_cast<int64_t>(a1.B) * a1.R;
  const int nv = ceil_div(std::max(a0.C, a1.B > 0 ? a1.C : 0), 128);
  if (rows < 1 || nv > 8) return LACT_ERR_SHAPE;
  const dim3 grid(ceil_div(rows, 8)), block(256);
  KernelScope scope(kClsRenorm, stream);
  switch (nv) {
    case 1: LACT_CUDA(launch_pdl(add_renorm_kernel<1>, grid, block, 0, stream, a0, a1)); break;
    case 2: LACT_CUDA(launch_pdl(add_renorm_kernel<2>, grid, block, 0, stream, a0, a1)); break;
    case 3: LACT_CUDA(launch_pdl(add_renorm_kernel<3>, grid, block, 0, stream, a0, a1)); break;
    case 4: LACT_CUDA(launch_pdl(add_renorm_kernel<4>, grid, block, 0, stream, a0, a1)); break;
    default: LACT_CUDA(launch_pdl(add_renorm_kernel<8>, grid, block, 0, stream, a0, a1)); break;
  }
  return LACT_OK;
}

int validate_scan_config(const lact_scan_config& c) {
  if (c.B < 1 || c.L < 1 || c.D < 16 || c.H < 16 || c.out_len < 0) return LACT_ERR_SHAPE;
  if ((c.D % 16) != 0 || (c.H % 16) != 0) return LACT_ERR_SHAPE;
  if (c.B > 65535 / 3 || c.L > (1ll << 30)) return LACT_ERR_SHAPE;
  if (c.act_dtype != LACT_BF16) return LACT_ERR_DTYPE;
  if (c.use_muon) {
    if (c.ns_steps < 0 || c.ns_steps > 64) return LACT_ERR_CONFIG;
    if (!c.ns_const_coeffs && c.ns_steps != 5) return LACT_ERR_CONFIG;
  }
  if (c.renorm < 0 || c.renorm > 2) return LACT_ERR_CONFIG;
  if (c.prenorm && c.overwrite_quirk) return LACT_ERR_CONFIG;
  return LACT_OK;
}

// True if an UPDATE step follows step i (then the fp32 copy of the normalised weights, which only
// the final export reads in post-norm mode, need not be written).
bool has_later_update(const int32_t* kind, int n_steps, int i) {
  for (int j = i + 1; j < n_steps; ++j)
    if (kind[j] == LACT_STEP_UPDATE) return true;
  return false;
}

// Bytes of Newton-Schulz trace one UPDATE step keeps in training (both groups, 256-byte aligned), and the offset of
// the second group's trace; LACT_ERR_CONFIG if this configuration keeps none (Muon off, more than five steps).
int scan_ns_trace_layout(const lact_scan_config& c, size_t* stride, size_t* g0_bytes) {
  if (!c.use_muon || c.ns_steps < 1 || c.ns_steps > 5) return LACT_ERR_CONFIG;
  NsGroup g0, g1;
  if (c.ns_concat) ns_group_init(g0, c.B, 2 * c.H, c.D, c.ns_gram_right);
  else ns_group_init(g0, 2 * c.B, c.H, c.D, c.ns_gram_right);
  ns_group_init(g1, c.B, c.D, c.H, c.ns_gram_right);
  NsTrace t0, t1;
  LACT_TRY(plan_ns_trace(nullptr, g0.nmat, g0.R, g0.C, c.ns_steps, c.ns_gram_right, &t0));
  LACT_TRY(plan_ns_trace(nullptr, g1.nmat, g1.R, g1.C, c.ns_steps, c.ns_gram_right, &t1));
  const size_t a = (t0.bytes + 255) & ~static_cast<size_t>(255), b = (t1.bytes + 255) & ~static_cast<size_t>(255);
  *g0_bytes = a;
  *stride = a + b;
  return LACT_OK;
}

struct StateCopy {
  StateCopyArgs a;
  int64_t longest = 0;
  cudaStream_t stream;
  StateCopy(int64_t batch, cudaStream_t s) : stream(s) {
    std::memset(&a, 0, sizeof(a));
    a.batch = static_cast<int32_t>(batch);
  }
  int add(const float* src, int64_t src_bs, void* dst, int64_t dst_bs, int64_t n) {
    if (dst == nullptr || src == dst) return LACT_OK;
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 3) != 0) {  // (an array packed behind bytes)
      LACT_CUDA(cudaMemcpy2DAsync(dst, dst_bs * 4, src, src_bs * 4, n * 4, a.batch, cudaMemcpyDeviceToDevice, stream));
      return LACT_OK;
    }
    const int i = a.copies++;
    a.src[i] = src;
    a.dst[i] = static_cast<float*>(dst);
    a.src_bs[i] = src_bs; a.dst_bs[i] = dst_bs; a.n[i] = n;
    a.vec[i] = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 && (src_bs | dst_bs | n) % 4 == 0;
    longest = std::max(longest, n);
    return LACT_OK;
  }
  int launch() {
    if (a.copies == 0) return LACT_OK;
    KernelScope scope(kClsOther, stream);
    LACT_CUDA(launch_pdl(state_copy_kernel, dim3(ceil_div(longest, 2048), a.copies, a.batch), dim3(256), 0, stream, a));
    return LACT_OK;
  }
};

// Momentum state the program starts from: the caller's.  Without one the first update adds its factor times zero without
// reading it, and zeros are written only for a program that hands the state back untouched.
inline bool has_initial_momentum(const lact_scan_io& io) { return io.m0_in && io.m1_in && io.m2_in; }
int load_momentum_state(const lact_scan_config& c, const lact_scan_io& io, float* G02, float* G1, cudaStream_t stream) {
  const size_t B = c.B, D = c.D, H = c.H;
  if (has_initial_momentum(io)) {
    const int64_t n = static_cast<int64_t>(H * D);
    StateCopy copy(c.B, stream);
    LACT_TRY(copy.add(static_cast<const float*>(io.m0_in), n, G02, 2 * n, n));
    LACT_TRY(copy.add(static_cast<const float*>(io.m2_in), n, G02 + n, 2 * n, n));
    LACT_TRY(copy.add(static_cast<const float*>(io.m1_in), n, G1, n, n));
    LACT_TRY(copy.launch());
  } else {
    LACT_CUDA(cudaMemsetAsync(G02, 0, B * 2 * H * D * 4, stream));
    LACT_CUDA(cudaMemsetAsync(G1, 0, B * D * H * 4, stream));
  }
  return LACT_OK;
}

// Per-update momentum factors beta[u][b], all UPDATE steps at once.
int launch_momentum_means(const lact_scan_config& c, const lact_scan_io& io, int32_t n_steps, const int32_t* kind,
                          const int64_t* start, const int64_t* end, float* beta, cudaStream_t stream) {
  MeanArgs ma;
  std::memset(&ma, 0, sizeof(ma));
  int u = 0, first_u = 0;
  auto flush = [&]() -> int {
    if (ma.n == 0) return LACT_OK;
    KernelScope scope(kClsMomentumMean, stream);
    LACT_CUDA(launch_pdl(momentum_mean_kernel, dim3(static_cast<unsigned>(c.B), ma.n), dim3(256), 0, stream, io.momentum,
                         c.mom_dtype == LACT_F32, c.L, ma, beta + first_u * c.B, static_cast<int>(c.B)));
    LACT_CUDA(cudaGetLastError());
    first_u = u;
    ma.n = 0;
    return LACT_OK;
  };
  for (int i = 0; i < n_steps; ++i) {
    if (kind[i] != LACT_STEP_UPDATE) continue;
    ma.s[ma.n] = static_cast<int32_t>(start[i]);
    ma.e[ma.n] = static_cast<int32_t>(end[i]);
    ++ma.n; ++u;
    if (ma.n == kMeanBatch) LACT_TRY(flush());
  }
  return flush();
}

// Final fast weights and momentum state into the caller's arrays (those that are given).
int store_state(const lact_scan_config& c, const lact_scan_io& io, const float* W02, const float* W1, const float* G02,
                const float* G1, cudaStream_t stream) {
  const int64_t n = c.D * c.H;
  StateCopy copy(c.B, stream);
  LACT_TRY(copy.add(W02, 2 * n, io.w0_out, n, n));
  LACT_TRY(copy.add(W02 + n, 2 * n, io.w2_out, n, n));
  LACT_TRY(copy.add(W1, n, io.w1_out, n, n));
  LACT_TRY(copy.add(G02, 2 * n, io.m0_out, n, n));
  LACT_TRY(copy.add(G02 + n, 2 * n, io.m2_out, n, n));
  LACT_TRY(copy.add(G1, n, io.m1_out, n, n));
  return copy.launch();
}

int scan_fwd(const lact_scan_config& c, const lact_scan_io& io, int32_t n_steps, const int32_t* kind,
             const int64_t* start, const int64_t* end, const int64_t* out_start, void* workspace, size_t ws_bytes,
             cudaStream_t stream) {
  LACT_TRY(check_device());
  LACT_TRY(validate_scan_config(c));
  if (!io.w0 || !io.w1 || !io.w2 || !io.q || !io.k || !io.v || !io.lr0 || !io.lr1 || !io.lr2 || !io.o)
    return LACT_ERR_NULL;
  if (c.use_momentum && !io.momentum) return LACT_ERR_NULL;
  if (!workspace) return LACT_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return LACT_ERR_WORKSPACE;
  ScanPlan p;
  LACT_TRY(plan_scan(c, n_steps, kind, start, end, workspace, &p));
  if (p.bytes > ws_bytes) return LACT_ERR_WORKSPACE;
  for (int i = 0; i < n_steps; ++i)
    if (kind[i] == LACT_STEP_APPLY && (out_start[i] < 0 || out_start[i] + (end[i] - start[i]) > c.out_len))
      return LACT_ERR_STEPS;

  const int64_t B = c.B, D = c.D, H = c.H;
  // Training (post-norm): the per-update state the backward needs is not copied out, it LIVES in the caller's dump:
  // update u reads its master weights from slot u and writes the new ones into slot u + 1 (the last update into the
  // workspace), and the gradient / momentum state of update u is written into slot u while slot u - 1 is read.
  const size_t n02 = static_cast<size_t>(B) * 2 * H * D, n1 = static_cast<size_t>(B) * D * H;
  int n_updates = 0;
  for (int i = 0; i < n_steps; ++i) n_updates += kind[i] == LACT_STEP_UPDATE;
  const bool dump_in_place = io.state_dump != nullptr && !c.prenorm && n_updates > 0;
  auto slot = [&](int u) { return static_cast<float*>(io.state_dump) + static_cast<size_t>(u) * 2 * (n02 + n1); };
  float* W02cur = dump_in_place ? slot(0) : p.W02;   // master weights in force
  float* W1cur = dump_in_place ? slot(0) + n02 : p.W1;
  // bf16 copies of the weights in force (MMA operands), [W0W2 | W1] per slot; training keeps those of every update in the
  // caller's buffer, else there are as many slots as one run of APPLY steps needs, used in turn
  bf16* const Wb = io.shadow_dump != nullptr ? static_cast<bf16*>(io.shadow_dump) : p.Wb;
  int w_slot = 0;
  bf16 *W02b = Wb, *W1b = Wb + n02;
  float* G02cur = p.G02;                              // gradient / momentum state after the latest update
  float* G1cur = p.G1;
  {
    const int64_t rows = B * (2 * H + D);
    KernelScope scope(kClsPrepare, stream);
    LACT_CUDA(launch_pdl(prepare_weights_kernel, dim3(ceil_div(rows, 8)), dim3(256), 0, stream, io.w0, io.w1, io.w2,
                         c.w_dtype == LACT_F32, static_cast<int>(B), static_cast<int>(H), static_cast<int>(D), W02cur, W1cur, p.W02c,
                         p.W1c, p.n02, p.n1, W02b, W1b, p.status, p.split.count, p.split_tiles));
    LACT_CUDA(cudaGetLastError());
  }
  if (has_initial_momentum(io) || n_updates == 0) LACT_TRY(load_momentum_state(c, io, p.G02, p.G1, stream));
  if (c.use_momentum) LACT_TRY(launch_momentum_means(c, io, n_steps, kind, start, end, p.beta, stream));

  // training with Muon: per-update Newton-Schulz traces in the caller's buffer (see lact_scan_ns_trace_bytes)
  size_t ns_trace_stride = 0, ns_trace_g0 = 0;
  const bool ns_keep = io.ns_trace != nullptr && c.use_muon && scan_ns_trace_layout(c, &ns_trace_stride, &ns_trace_g0) == LACT_OK;
  if (io.ns_trace != nullptr && !ns_keep) return LACT_ERR_CONFIG;
  if (ns_keep && (reinterpret_cast<uintptr_t>(io.ns_trace) & 255) != 0) return LACT_ERR_WORKSPACE;

  int update_idx = 0;
  ApplyArgs pending{};     // the run of APPLY steps being collected, none if `missing` is 0
  int64_t missing = 0;     // how many of its steps are still to come
  for (int i = 0; i < n_steps; ++i) {
    if (kind[i] == LACT_STEP_APPLY) {
      if (missing == 0) {
        const int64_t free_slots = io.shadow_dump != nullptr ? n_steps : p.w_slots - w_slot;
        const ApplyRun run = apply_run(c, n_steps, kind, start, end, out_start, i, free_slots);
        pending = ApplyArgs{W02b, W1b, io.q, c.q_bs, c.q_ts, start[i], end[i], io.o, c.o_bs, c.o_ts, out_start[i],
                            p.hidden, B, D, H};
        pending.segs = missing = run.steps;
        pending.x_step = run.x_step;
        pending.o_step = run.o_step;
        pending.w_step = static_cast<int64_t>(n02 + n1);
      }
      if (--missing == 0) LACT_TRY(run_apply(pending, p.status, stream));
      continue;
    }
    const float* beta = c.use_momentum ? p.beta + static_cast<int64_t>(update_idx) * B : nullptr;
    const bool fresh = update_idx == 0 && !has_initial_momentum(io);
    float* dump = nullptr;
    if (io.state_dump != nullptr && !dump_in_place) {
      // training (pre-norm): the weights this update computed with and (below) its gradient after momentum are copied
      dump = slot(update_idx);
      LACT_CUDA(cudaMemcpyAsync(dump, c.prenorm ? p.W02c : p.W02, n02 * 4, cudaMemcpyDeviceToDevice, stream));
      LACT_CUDA(cudaMemcpyAsync(dump + n02, c.prenorm ? p.W1c : p.W1, n1 * 4, cudaMemcpyDeviceToDevice, stream));
    }
    const float* G02prev = nullptr;
    const float* G1prev = nullptr;
    if (dump_in_place) {
      G02prev = G02cur;
      G1prev = G1cur;
      G02cur = slot(update_idx) + n02 + n1;
      G1cur = slot(update_idx) + 2 * n02 + n1;
    }
    ++update_idx;
    GradArgs g{W02b, W1b, io.k, io.v, c.k_bs, c.k_ts, c.v_bs, c.v_ts, start[i], end[i], io.lr0, io.lr1, io.lr2,
               c.lr_dtype == LACT_F32, c.L, c.w_scale, p.dy02, p.hid, G02cur, G1cur, 1, beta, B, D, H};
    g.g02_prev = G02prev;
    g.g1_prev = G1prev;
    g.fresh = fresh;
    g.split = p.split;
    // The Frobenius norms Newton-Schulz needs are gathered per output tile by the contraction when a
    // tile never straddles two matrices (concatenated [2H, D], or H a multiple of the 128-row tile).
    int fused_parts[2] = {0, 0};
    if (c.use_muon && (c.ns_concat || H % kBM == 0)) {
      const int bt = contract_bt(D, H);
      const int tn0 = ceil_div(D, bt), tn1 = ceil_div(H, bt);
      fused_parts[0] = (c.ns_concat ? ceil_div(2 * H, kBM) : static_cast<int>(H / kBM)) * tn0 * kEpiWarps;
      fused_parts[1] = ceil_div(D, kBM) * tn1 * kEpiWarps;
      if (fused_parts[0] <= kNsMaxParts && fused_parts[1] <= kNsMaxParts) {
        g.partial02 = p.ns.grp[0].partial;
        g.partial1 = p.ns.grp[1].partial;
        if (c.ns_steps > 0 && !ns_keep) {  // the iteration starts from bf16(G) itself, normalisation folded in
          g.gb02 = p.ns.grp[0].xa;
          g.gb1 = p.ns.grp[1].xa;
        }
      } else {
        fused_parts[0] = fused_parts[1] = 0;
      }
    }
    LACT_TRY(run_grad(g, p.status, stream));
    if (dump != nullptr) {
      LACT_CUDA(cudaMemcpyAsync(dump + n02 + n1, p.G02, n02 * 4, cudaMemcpyDeviceToDevice, stream));
      LACT_CUDA(cudaMemcpyAsync(dump + 2 * n02 + n1, p.G1, n1 * 4, cudaMemcpyDeviceToDevice, stream));
    }

    // add + renormalise arguments (the update is the Newton-Schulz result when Muon is on)
    // (the fp32 copy of the normalised weights is what pre-norm computes with and what the final export reads)
    const bool want_compute = c.prenorm || ((io.w0_out || io.w1_out || io.w2_out) && !has_later_update(kind, n_steps, i));
    // (the weights of steps still to run are not overwritten: a run takes the slots from the one on that the weights are in, and no
    // more than there are)
    const int next_slot = io.shadow_dump != nullptr ? update_idx : (missing > 0 ? w_slot + 1 : 0);
    RenormArgs rn[2];
    for (int w = 0; w < 2; ++w) {
      RenormArgs& r = rn[w];
      std::memset(&r, 0, sizeof(r));
      const int R = static_cast<int>(w == 0 ? 2 * H : D), C = static_cast<int>(w == 0 ? D : H);
      if (C > kRenormMaxCols) return LACT_ERR_SHAPE;
      r.master = w == 0 ? p.W02 : p.W1;
      if (dump_in_place) {  // read slot u, write slot u + 1 (the last update writes the workspace copy)
        r.master_in = w == 0 ? W02cur : W1cur;
        if (update_idx < n_updates) r.master = w == 0 ? slot(update_idx) : slot(update_idx) + n02;
      }
      r.compute = want_compute ? (w == 0 ? p.W02c : p.W1c) : nullptr;
      r.shadow = Wb + static_cast<size_t>(next_slot) * (n02 + n1) + (w == 0 ? 0 : n02);
      r.n0 = w == 0 ? p.n02 : p.n1;
      r.g = w == 0 ? G02cur : G1cur;
      r.x = nullptr;
      r.x_bs = static_cast<int64_t>(R) * C;
      r.B = static_cast<int>(B); r.R = R; r.C = C;
      r.mode = c.renorm; r.prenorm = c.prenorm; r.prenorm_bf16 = c.prenorm_bf16; r.quirk = c.overwrite_quirk;
    }
    if (c.use_muon && ns_keep) {
      // training: every iterate, shifted Gram matrix and polynomial of this update stays in the caller's trace
      // buffers (the layout lact_ns_trace_bwd reads); the first iterate is the explicitly normalised gradient
      NsPlan& ns = p.ns;
      const bf16* xres[2] = {nullptr, nullptr};
      const void* srcs[2] = {G02cur, G1cur};
      NsGroup tg[2];
      NsKeep keep[2];
      uint8_t* tb = static_cast<uint8_t*>(io.ns_trace) + static_cast<size_t>(update_idx - 1) * ns_trace_stride;
      for (int gi = 0; gi < 2; ++gi) {
        NsTrace t;
        LACT_TRY(plan_ns_trace(tb + (gi == 0 ? 0 : ns_trace_g0), ns.grp[gi].nmat, ns.grp[gi].R, ns.grp[gi].C, c.ns_steps,
                               c.ns_gram_right, &t));
        tg[gi] = ns.grp[gi];
        tg[gi].xa = t.X;
        keep[gi] = NsKeep{t.X, t.A, t.P};
      }
      LACT_TRY(run_newton_schulz(tg, 2, srcs, 1, fused_parts, 0, c.ns_steps, c.ns_const_coeffs, p.status, stream, xres, keep));
      rn[0].x = xres[0];
      rn[1].x = xres[1];
    } else if (c.use_muon) {
      NsPlan& ns = p.ns;
      const bf16* xres[2] = {nullptr, nullptr};
      const void* srcs[2] = {G02cur, G1cur};
      const int unscaled = g.gb02 != nullptr ? 1 : 0;
      LACT_TRY(run_newton_schulz(ns.grp, ns.ngroups, srcs, 1, fused_parts, unscaled, c.ns_steps, c.ns_const_coeffs, p.status,
                                 stream, xres));
      rn[0].x = xres[0];
      rn[1].x = xres[1];
    }
    LACT_TRY(launch_add_renorm(rn[0], rn[1], stream));
    w_slot = next_slot;
    W02b = Wb + static_cast<size_t>(w_slot) * (n02 + n1);
    W1b = W02b + n02;
    if (dump_in_place) {
      W02cur = rn[0].master;
      W1cur = rn[1].master;
    }
  }
  return store_state(c, io, p.W02c, p.W1c, G02cur, G1cur, stream);
}

// ------------------------------------------------------------------------------------------
// fp32 mode: the same step programs on fp32 activations (contractions in bf16 pieces, f32_split.cuh)
// ------------------------------------------------------------------------------------------
F32Mat f32_mat(const float* p, int64_t ld, int64_t bs, int t, int64_t rows, int64_t k) {
  const int64_t contiguous = t ? rows : k;
  const bool vec = (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (ld % 4) == 0 && (bs % 4) == 0 && (contiguous % 4) == 0;
  return F32Mat{p, ld, bs, t, vec ? 1 : 0};
}

template <int MODE, int BT>
int launch_cut_gemm(CutArgs& a, cudaStream_t stream) {
  auto kernel = cut_gemm_kernel<MODE, BT>;
  constexpr uint32_t smem = CutTile<MODE, BT>::kSmem;
  static_assert(smem <= 232448, "shared memory budget exceeded");
  static std::mutex mu;
  static bool configured[64] = {false};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !configured[dev]) {
      LACT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (dev < 64) configured[dev] = true;
    }
  }
  int64_t units = 0;
  for (int i = 0; i < a.nprob; ++i) {
    CutProblem& P = a.prob[i];
    if (P.M < 1 || P.N < 1 || P.K < 1 || ceil_div(P.M, kBM) > 65535 || static_cast<int64_t>(P.batch) * P.splits > 65535)
      return LACT_ERR_SHAPE;
    auto starts_on = [&](int bytes) {
      return reinterpret_cast<uintptr_t>(P.c) % bytes == 0 && P.c_ld % (bytes / 4) == 0 && P.c_bs % (bytes / 4) == 0;
    };
    P.c_vec = starts_on(32) ? 2 : starts_on(16) ? 1 : 0;
    units += static_cast<int64_t>(ceil_div(P.M, kBM)) * ceil_div(P.N, CutTile<MODE, BT>::kOut) * P.batch * P.splits;
  }
  if (units > (1ll << 30)) return LACT_ERR_SHAPE;
  KernelScope scope(kClsOther, stream);
  LACT_CUDA(launch_pdl(kernel, dim3(static_cast<unsigned>(std::min<int64_t>(units, sm_count()))), dim3(kCutThreads), smem, stream, a));
  return LACT_OK;
}
// (128-wide tiles move half as many bytes per product, 64-wide ones waste less of other sizes)
int launch_cut_store(CutArgs& a, int bt, cudaStream_t stream) {
  return bt == 128 ? launch_cut_gemm<kCutStore, 128>(a, stream) : launch_cut_gemm<kCutStore, 64>(a, stream);
}

// Pieces of an fp32 matrix: [3][batch][rows][ld].
struct Pieces {
  bf16* p;
  int64_t rows, cols, ld;
};
inline int64_t piece_ld(int64_t cols) { return (cols + 7) & ~7ll; }
inline Mat piece_mat(const Pieces& x, int64_t batch) { return Mat{x.p, x.rows, x.cols, x.ld, 3 * batch, x.rows * x.ld}; }

struct CutPlanes {
  CutPlanesArgs a;
  explicit CutPlanes(int64_t batch) {
    std::memset(&a, 0, sizeof(a));
    a.batch = static_cast<int32_t>(batch);
  }
  void add(const float* src, int64_t ld, int64_t bs, const Pieces& x) {
    const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && ld % 4 == 0 && bs % 4 == 0;
    a.s[a.n] = CutSource{src, ld, bs, x.p, static_cast<int32_t>(x.rows), static_cast<int32_t>(x.cols), static_cast<int32_t>(x.ld), vec};
    a.first[a.n + 1] = a.first[a.n] + a.batch * x.rows * (x.ld / 8);
    ++a.n;
  }
  int launch(cudaStream_t stream) {
    const int64_t blocks = (a.first[a.n] + 255) / 256;
    if (blocks < 1 || blocks > 0x7FFFFFFF) return LACT_ERR_SHAPE;
    KernelScope scope(kClsOther, stream);
    LACT_CUDA(launch_pdl(cut_planes_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, stream, a));
    return LACT_OK;
  }
};

// Splits of the two token contractions of an update ([2H x D] and [D x H] per entry, `len` tokens): two units per SM, at least 64
// tokens each, and no more than 65535 partial results.  At 4 entries of 192 x 192 and 4096 tokens one split would be 60 units of
// 64 slabs on 148 SMs.
inline int cut_bt(int64_t D, int64_t H) { return D % 128 == 0 && H % 128 == 0 ? 128 : 64; }
int f32_splits(int64_t B, int64_t D, int64_t H, int64_t len) {
  const int bt = cut_bt(D, H);
  const int64_t tiles = output_tiles(2 * H, D, B, bt) + output_tiles(D, H, B, bt);
  return static_cast<int>(
      std::max<int64_t>(1, std::min<int64_t>({2 * static_cast<int64_t>(sm_count()) / tiles, (len + kBK - 1) / kBK, 64, 65535 / B})));
}

struct ScanF32Plan {
  int32_t* status;
  float *W02, *W1, *W02c, *W1c, *n02, *n1, *G02, *G1, *beta, *part02, *part1;
  bf16 *w02, *w1, *x, *v, *hidden, *dy02;  // pieces of the weights, of q or k, of v, of the hidden activations, of dy0 | dy2
  bool updates;  // some update has tokens
  NsPlan ns;
  size_t bytes;
};

int plan_scan_f32(const lact_scan_config& c, int32_t n_steps, const int32_t* kind, const int64_t* start, const int64_t* end,
                  void* base, ScanF32Plan* p) {
  int64_t max_apply = 0, max_update = 0;
  for (int i = 0; i < n_steps; ++i) {
    if (start[i] < 0 || end[i] > c.L || end[i] < start[i]) return LACT_ERR_STEPS;
    const int64_t len = end[i] - start[i];
    if (kind[i] == LACT_STEP_APPLY) max_apply = std::max(max_apply, len);
    else if (kind[i] == LACT_STEP_UPDATE) max_update = std::max(max_update, len);
    else return LACT_ERR_STEPS;
  }
  Carver cv(base);
  const size_t B = c.B, D = c.D, H = c.H;
  p->status = cv.take<int32_t>(64);
  p->W02 = cv.take<float>(B * 2 * H * D);
  p->W1 = cv.take<float>(B * D * H);
  p->W02c = cv.take<float>(B * 2 * H * D);
  p->W1c = cv.take<float>(B * D * H);
  p->n02 = cv.take<float>(B * 2 * H);
  p->n1 = cv.take<float>(B * D);
  p->G02 = cv.take<float>(B * 2 * H * D);
  p->G1 = cv.take<float>(B * D * H);
  p->beta = cv.take<float>(B * static_cast<size_t>(std::max(1, n_steps)));
  const size_t any = static_cast<size_t>(std::max(max_apply, max_update)), upd = static_cast<size_t>(max_update), Dp = piece_ld(c.D);
  p->w02 = cv.take<bf16>(3 * B * 2 * H * Dp);
  p->w1 = cv.take<bf16>(3 * B * D * H);
  p->x = cv.take<bf16>(3 * B * any * Dp);
  p->v = cv.take<bf16>(3 * B * upd * Dp);
  p->hidden = cv.take<bf16>(3 * B * any * H);
  p->dy02 = cv.take<bf16>(3 * B * upd * 2 * H);
  p->updates = max_update > 0;
  // (splits grow with the token count: the longest update needs the most)
  const size_t splits = max_update > 0 ? static_cast<size_t>(f32_splits(c.B, c.D, c.H, max_update)) : 0;
  p->part02 = cv.take<float>(splits * B * 2 * H * D);
  p->part1 = cv.take<float>(splits * B * D * H);
  p->ns.ngroups = 0;
  if (c.use_muon && max_update > 0) plan_ns(cv, c.B, c.D, c.H, c.ns_concat, c.ns_gram_right, &p->ns);
  p->bytes = cv.off + 256;
  return LACT_OK;
}

int validate_scan_f32(const lact_scan_config& c) {
  if (c.B < 1 || c.L < 1 || c.D < 4 || c.H < 8 || c.out_len < 0 || (c.D % 4) != 0 || (c.H % 8) != 0) return LACT_ERR_SHAPE;
  if (c.B > 65535 || c.L > (1ll << 30)) return LACT_ERR_SHAPE;
  if (c.act_dtype != LACT_F32) return LACT_ERR_DTYPE;
  if (c.use_muon) {
    if (c.ns_steps < 0 || c.ns_steps > 64 || (c.D % 8) != 0) return LACT_ERR_CONFIG;
    if (!c.ns_const_coeffs && c.ns_steps != 5) return LACT_ERR_CONFIG;
  }
  if (c.renorm < 0 || c.renorm > 2) return LACT_ERR_CONFIG;
  return LACT_OK;
}

int scan_fwd_f32(const lact_scan_config& c, const lact_scan_io& io, int32_t n_steps, const int32_t* kind, const int64_t* start,
                 const int64_t* end, const int64_t* out_start, void* workspace, size_t ws_bytes, cudaStream_t stream) {
  LACT_TRY(check_device());
  LACT_TRY(validate_scan_f32(c));
  if (!io.w0 || !io.w1 || !io.w2 || !io.q || !io.k || !io.v || !io.lr0 || !io.lr1 || !io.lr2 || !io.o) return LACT_ERR_NULL;
  if (c.use_momentum && !io.momentum) return LACT_ERR_NULL;
  if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return LACT_ERR_WORKSPACE;
  ScanF32Plan p;
  LACT_TRY(plan_scan_f32(c, n_steps, kind, start, end, workspace, &p));
  if (p.bytes > ws_bytes) return LACT_ERR_WORKSPACE;
  for (int i = 0; i < n_steps; ++i)
    if (kind[i] == LACT_STEP_APPLY && (out_start[i] < 0 || out_start[i] + (end[i] - start[i]) > c.out_len)) return LACT_ERR_STEPS;
  const int64_t B = c.B, D = c.D, H = c.H;
  if (p.updates && (D > kRenormMaxCols || H > kRenormMaxCols)) return LACT_ERR_SHAPE;  // (rows of an update's renormalisation)
  {
    KernelScope scope(kClsPrepare, stream);
    LACT_CUDA(launch_pdl(prepare_weights_kernel, dim3(ceil_div(B * (2 * H + D), 8)), dim3(256), 0, stream, io.w0, io.w1, io.w2,
                         c.w_dtype == LACT_F32, static_cast<int>(B), static_cast<int>(H), static_cast<int>(D), p.W02, p.W1, p.W02c,
                         p.W1c, p.n02, p.n1, nullptr, nullptr, p.status, nullptr, 0));
    LACT_CUDA(cudaGetLastError());
  }
  if (has_initial_momentum(io) || io.m0_out || io.m1_out || io.m2_out) LACT_TRY(load_momentum_state(c, io, p.G02, p.G1, stream));
  if (c.use_momentum) LACT_TRY(launch_momentum_means(c, io, n_steps, kind, start, end, p.beta, stream));
  const float* W02 = c.prenorm ? p.W02c : p.W02;  // the weights the steps compute with
  const float* W1 = c.prenorm ? p.W1c : p.W1;
  const float *q = static_cast<const float*>(io.q), *k = static_cast<const float*>(io.k), *v = static_cast<const float*>(io.v);
  int update_idx = 0;
  bool weights_cut = false;                       // the pieces are those of W02 and W1 as they are
  bool state_written = has_initial_momentum(io);  // by the caller, or by an update that had tokens
  for (int i = 0; i < n_steps; ++i) {
    const int64_t len = end[i] - start[i];
    if (len <= 0) {
      update_idx += kind[i] == LACT_STEP_UPDATE;
      continue;
    }
    const int64_t Dp = piece_ld(D);
    const Pieces w02{p.w02, 2 * H, D, Dp}, w1{p.w1, D, H, H}, x{p.x, len, D, Dp}, hidden{p.hidden, len, H, H};
    CutPlanes cut(B);
    if (!weights_cut) {
      cut.add(W02, D, 2 * H * D, w02);
      cut.add(W1, H, D * H, w1);
      weights_cut = true;
    }
    CutArgs a;
    std::memset(&a, 0, sizeof(a));
    a.status = p.status;
    a.nprob = 1;
    a.hidden = p.hidden;
    {
      CutProblem& P = a.prob[0];
      LACT_TRY(encode_map(&P.a, piece_mat(x, B), kBM));
      LACT_TRY(encode_map(&P.b, piece_mat(w02, B), 64));
      P.M = static_cast<int32_t>(len); P.N = static_cast<int32_t>(H); P.K = P.kper = static_cast<int32_t>(D);
      P.batch = static_cast<int32_t>(B);
      P.splits = 1;
    }
    if (kind[i] == LACT_STEP_APPLY) {
      cut.add(q + start[i] * c.q_ts, c.q_ts, c.q_bs, x);
      LACT_TRY(cut.launch(stream));
      LACT_TRY((launch_cut_gemm<kCutGate, 128>(a, stream)));
      CutProblem& P = a.prob[0];
      LACT_TRY(encode_map(&P.a, piece_mat(hidden, B), kBM));
      LACT_TRY(encode_map(&P.b, piece_mat(w1, B), 64));
      P.N = static_cast<int32_t>(D); P.K = P.kper = static_cast<int32_t>(H);
      P.c = static_cast<float*>(io.o) + out_start[i] * c.o_ts; P.c_ld = c.o_ts; P.c_bs = c.o_bs;
      LACT_TRY(launch_cut_store(a, D % 128 == 0 ? 128 : 64, stream));
      continue;
    }
    const Pieces v_pieces{p.v, len, D, Dp}, dy{p.dy02, len, 2 * H, 2 * H};
    cut.add(k + start[i] * c.k_ts, c.k_ts, c.k_bs, x);
    cut.add(v + start[i] * c.v_ts, c.v_ts, c.v_bs, v_pieces);
    LACT_TRY(cut.launch(stream));
    LACT_TRY(encode_map(&a.a2, piece_mat(v_pieces, B), kBM));
    LACT_TRY(encode_map(&a.b2, piece_mat(w1, B), 64));  // dh = v w1: w1 is [D][H], k = D rows
    a.dy = p.dy02;
    const int u = update_idx++;
    const int64_t esz = c.lr_dtype == LACT_F32 ? 4 : 2;
    auto at = [&](const void* t) { return static_cast<const uint8_t*>(t) + start[i] * esz; };
    a.lr0 = at(io.lr0); a.lr1 = at(io.lr1); a.lr2 = at(io.lr2);
    a.lr_f32 = c.lr_dtype == LACT_F32;
    a.lr_bs = c.L;
    a.w_scale = c.w_scale;
    LACT_TRY((launch_cut_gemm<kCutGrad, 128>(a, stream)));
    F32ReduceArgs red;
    std::memset(&red, 0, sizeof(red));
    red.batch = static_cast<int32_t>(B);
    red.accumulate = c.use_momentum;
    red.fresh = !state_written;
    red.beta = c.use_momentum ? p.beta + static_cast<int64_t>(u) * B : nullptr;
    state_written = true;
    // [dw0; dw2] = dy^T k, dw1 = v^T hidden
    const int splits = f32_splits(B, D, H, len);
    for (int w = 0; w < 2; ++w) {
      CutProblem& P = a.prob[w];
      LACT_TRY(encode_map(&P.a, piece_mat(w == 0 ? dy : v_pieces, B), 64));
      LACT_TRY(encode_map(&P.b, piece_mat(w == 0 ? x : hidden, B), 64));
      P.a_mn = P.b_mn = 1;
      P.M = static_cast<int32_t>(w == 0 ? 2 * H : D); P.N = static_cast<int32_t>(w == 0 ? D : H); P.K = static_cast<int32_t>(len);
      P.batch = static_cast<int32_t>(B);
      P.kper = ceil_div(ceil_div(len, splits), kBK) * kBK;
      P.splits = ceil_div(len, P.kper);
      P.c = w == 0 ? p.part02 : p.part1;
      P.c_ld = P.N; P.c_bs = static_cast<int64_t>(P.M) * P.N;
      red.part[w] = P.c;
      red.c[w] = w == 0 ? p.G02 : p.G1;
      red.n[w] = P.c_bs;
      red.splits[w] = P.splits;
    }
    a.nprob = 2;
    LACT_TRY(launch_cut_store(a, cut_bt(D, H), stream));
    {
      KernelScope scope(kClsOther, stream);
      LACT_CUDA(launch_pdl(f32_reduce_kernel, dim3(ceil_div((red.n[0] + red.n[1]) * B / 4, 256)), dim3(256), 0, stream, red));
    }
    const bf16* xres[2] = {nullptr, nullptr};
    if (c.use_muon) {
      const void* srcs[2] = {p.G02, p.G1};
      LACT_TRY(run_newton_schulz(p.ns.grp, 2, srcs, 1, nullptr, 0, c.ns_steps, c.ns_const_coeffs, p.status, stream, xres));
    }
    RenormArgs rn[2];
    for (int w = 0; w < 2; ++w) {
      RenormArgs& r = rn[w];
      std::memset(&r, 0, sizeof(r));
      r.R = static_cast<int>(w == 0 ? 2 * H : D); r.C = static_cast<int>(w == 0 ? D : H);
      r.B = static_cast<int>(B);
      r.master = w == 0 ? p.W02 : p.W1;
      r.compute = !c.prenorm ? nullptr : (w == 0 ? p.W02c : p.W1c);
      r.n0 = w == 0 ? p.n02 : p.n1;
      r.g = w == 0 ? p.G02 : p.G1;
      r.x = xres[w];
      r.x_bs = static_cast<int64_t>(r.R) * r.C;
      r.mode = c.renorm; r.prenorm = c.prenorm; r.prenorm_bf16 = c.prenorm_bf16; r.quirk = c.overwrite_quirk;
    }
    LACT_TRY(launch_add_renorm(rn[0], rn[1], stream));
    weights_cut = false;
  }
  return store_state(c, io, W02, W1, p.G02, p.G1, stream);
}

}  // namespace
}  // namespace lact

// ==========================================================================================
// extern "C" entry points
// ==========================================================================================
using namespace lact;

extern "C" {

int lact_version(void) { return 1002; }

const char* lact_error_string(int code) {
  switch (code) {
    case LACT_OK: return "ok";
    case LACT_ERR_NULL: return "a required pointer is NULL";
    case LACT_ERR_SHAPE: return "unsupported or inconsistent sizes, strides or alignment";
    case LACT_ERR_DTYPE: return "unsupported dtype combination";
    case LACT_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
    case LACT_ERR_CONFIG: return "inconsistent configuration flags";
    case LACT_ERR_STEPS: return "malformed step list";
    case LACT_ERR_CUDA: return "a CUDA runtime or driver call failed";
    case LACT_ERR_DEVICE: return "device is not compute capability 10.x (B200)";
    case LACT_ERR_STATIC_LIMIT:
      return "problem needs more scratch than the library's built-in static buffer holds (16 MiB): "
             "use the workspace variant or a smaller B * N * H";
    case kStatusWaitTimeout: return "device: a bounded barrier wait timed out";
    default: return "unknown code";
  }
}

int64_t lact_launch_count(void) { return g_prof.launches.load(); }

int lact_profile_enable(int enable) {
  g_prof.enabled.store(enable != 0);
  return LACT_OK;
}

int lact_nvtx_enable(int enable) {
  g_nvtx.store(enable != 0);
  return LACT_OK;
}

int lact_profile_num_classes(void) { return kNumClasses; }

const char* lact_profile_class_name(int cls) { return (cls >= 0 && cls < kNumClasses) ? kClassNames[cls] : "?"; }

int lact_profile_read(double* ms, int64_t* launches) {
  if (!ms || !launches) return LACT_ERR_NULL;
  std::vector<Profiler::Rec> recs;
  {
    std::lock_guard<std::mutex> lock(g_prof.mu);
    recs.swap(g_prof.recs);
  }
  for (int i = 0; i < kNumClasses; ++i) { ms[i] = 0.0; launches[i] = 0; }
  int rc = LACT_OK;
  for (auto& r : recs) {
    float t = 0.f;
    if (cudaEventSynchronize(r.b) != cudaSuccess || cudaEventElapsedTime(&t, r.a, r.b) != cudaSuccess) rc = LACT_ERR_CUDA;
    ms[r.cls] += t;
    launches[r.cls] += 1;
  }
  std::lock_guard<std::mutex> lock(g_prof.mu);
  for (auto& r : recs) { g_prof.pool.push_back(r.a); g_prof.pool.push_back(r.b); }
  return rc;
}

// Copies one status word to the host; the only place where the library waits for a stream.
static int read_status_word(const void* device_word, cudaStream_t stream) {
  int32_t st = 0;
  g_stream_syncs.fetch_add(1, std::memory_order_relaxed);
  if (cudaMemcpyAsync(&st, device_word, 4, cudaMemcpyDeviceToHost, stream) != cudaSuccess) return LACT_ERR_CUDA;
  if (cudaStreamSynchronize(stream) != cudaSuccess) return LACT_ERR_CUDA;
  return st;
}

int lact_read_status(const void* workspace, void* stream) {
  if (!workspace) return LACT_ERR_NULL;
  return read_status_word(workspace, static_cast<cudaStream_t>(stream));
}

int64_t lact_stream_sync_count(void) { return g_stream_syncs.load(); }

// Makes a device's word of mapped host memory and tells its kernels where it is.  The call that needs it first may be inside
// a stream capture, which forbids this thread allocations and stream 0: the relaxed mode and a stream of its own keep the
// capture out of it.
static int make_status_host_word(int32_t** word) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  LACT_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
  auto make = [&]() -> int {
    void *h = nullptr, *d = nullptr;
    LACT_CUDA(cudaHostAlloc(&h, sizeof(int32_t), cudaHostAllocMapped | cudaHostAllocPortable));
    *static_cast<int32_t*>(h) = 0;
    cudaStream_t s = nullptr;
    cudaError_t e = cudaHostGetDevicePointer(&d, h, 0);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(g_host_status, &d, sizeof(d), 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (s != nullptr) cudaStreamDestroy(s);
    if (e != cudaSuccess) {
      cudaFreeHost(h);
      return LACT_ERR_CUDA;
    }
    *word = static_cast<int32_t*>(h);
    return LACT_OK;
  };
  const int rc = make();
  LACT_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
  return rc;
}

int lact_status_host_word(int32_t** word_out) {
  if (!word_out) return LACT_ERR_NULL;
  static std::mutex mu;
  static int32_t* words[64] = {nullptr};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return LACT_ERR_DEVICE;
  std::lock_guard<std::mutex> lock(mu);
  if (words[dev] == nullptr) LACT_TRY(make_status_host_word(&words[dev]));
  *word_out = words[dev];
  return LACT_OK;
}

int lact_set_wait_limit_ns(uint64_t limit_ns) {
  if (limit_ns == 0) limit_ns = kDefaultWaitLimitNs;
  LACT_CUDA(cudaMemcpyToSymbol(g_wait_limit_ns, &limit_ns, sizeof(limit_ns)));
  return LACT_OK;
}

// One CTA whose single waiting thread sits on an mbarrier that nobody arrives on: the bounded
// wait runs out and the kernel records kStatusWaitTimeout, exactly as the GEMM kernels do.
__global__ void wait_timeout_probe_kernel(int32_t* status) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    if (!mbar_wait(&bar, 0)) report_timeout(status);
  }
}

int lact_debug_wait_timeout(int32_t* status_word, void* stream) {
  if (!status_word) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  wait_timeout_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(status_word);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_scan_workspace_bytes(const lact_scan_config* cfg, int32_t n_steps, const int32_t* kind,
                              const int64_t* start, const int64_t* end, size_t* bytes_out) {
  if (!cfg || !bytes_out || (n_steps > 0 && (!kind || !start || !end))) return LACT_ERR_NULL;
  LACT_TRY(validate_scan_config(*cfg));
  ScanPlan p;
  LACT_TRY(plan_scan(*cfg, n_steps, kind, start, end, nullptr, &p));
  *bytes_out = p.bytes;
  return LACT_OK;
}

int lact_scan_ns_trace_bytes(const lact_scan_config* cfg, size_t* bytes_per_update, size_t* second_group_offset) {
  if (!cfg || !bytes_per_update || !second_group_offset) return LACT_ERR_NULL;
  LACT_TRY(validate_scan_config(*cfg));
  return scan_ns_trace_layout(*cfg, bytes_per_update, second_group_offset);
}

int lact_scan_fwd(const lact_scan_config* cfg, const lact_scan_io* io, int32_t n_steps, const int32_t* kind,
                  const int64_t* start, const int64_t* end, const int64_t* out_start, void* workspace,
                  size_t workspace_bytes, void* stream) {
  if (!cfg || !io || (n_steps > 0 && (!kind || !start || !end || !out_start))) return LACT_ERR_NULL;
  return scan_fwd(*cfg, *io, n_steps, kind, start, end, out_start, workspace, workspace_bytes,
                  static_cast<cudaStream_t>(stream));
}

int lact_scan_f32_workspace_bytes(const lact_scan_config* cfg, int32_t n_steps, const int32_t* kind, const int64_t* start,
                                  const int64_t* end, size_t* bytes_out) {
  if (!cfg || !bytes_out || (n_steps > 0 && (!kind || !start || !end))) return LACT_ERR_NULL;
  LACT_TRY(validate_scan_f32(*cfg));
  ScanF32Plan p;
  LACT_TRY(plan_scan_f32(*cfg, n_steps, kind, start, end, nullptr, &p));
  *bytes_out = p.bytes;
  return LACT_OK;
}

int lact_scan_f32_fwd(const lact_scan_config* cfg, const lact_scan_io* io, int32_t n_steps, const int32_t* kind,
                      const int64_t* start, const int64_t* end, const int64_t* out_start, void* workspace,
                      size_t workspace_bytes, void* stream) {
  if (!cfg || !io || (n_steps > 0 && (!kind || !start || !end || !out_start))) return LACT_ERR_NULL;
  return scan_fwd_f32(*cfg, *io, n_steps, kind, start, end, out_start, workspace, workspace_bytes,
                      static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------- sub-ops
static int check_dims(int64_t B, int64_t N, int64_t D, int64_t H) {
  if (B < 1 || N < 1 || D < 16 || H < 16 || (D % 16) || (H % 16) || B > 65535 || N > (1ll << 30))
    return LACT_ERR_SHAPE;
  return LACT_OK;
}

int lact_swiglu_ffn_workspace_bytes(int64_t B, int64_t N, int64_t D, int64_t H, size_t* bytes_out) {
  if (!bytes_out) return LACT_ERR_NULL;
  LACT_TRY(check_dims(B, N, D, H));
  *bytes_out = 512 + static_cast<size_t>(B) * N * H * 2;
  return LACT_OK;
}

int lact_swiglu_ffn_fwd(const void* w0w2, const void* w1, const void* x, void* out, int64_t B, int64_t N, int64_t D,
                        int64_t H, void* workspace, size_t workspace_bytes, void* stream) {
  if (!w0w2 || !w1 || !x || !out) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  size_t need = 0;
  LACT_TRY(lact_swiglu_ffn_workspace_bytes(B, N, D, H, &need));
  if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255)) return LACT_ERR_WORKSPACE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  LACT_CUDA(cudaMemsetAsync(workspace, 0, 256, s));
  ApplyArgs a{static_cast<const bf16*>(w0w2), static_cast<const bf16*>(w1), x, N * D, D, 0, N, out, N * D, D, 0,
              reinterpret_cast<bf16*>(static_cast<uint8_t*>(workspace) + 256), B, D, H};
  return run_apply(a, static_cast<int32_t*>(workspace), s);
}

int lact_swiglu_ffn_hidden_bytes(int64_t B, int64_t N, int64_t D, int64_t H, size_t* bytes_out) {
  if (!bytes_out) return LACT_ERR_NULL;
  LACT_TRY(check_dims(B, N, D, H));
  *bytes_out = few_pays(B, N, D, H) ? 0 : static_cast<size_t>(B) * N * H * 2;
  return LACT_OK;
}

int lact_swiglu_ffn_apply(const void* w0w2, const void* w1, const void* x, void* out, void* hidden, int64_t B, int64_t N,
                          int64_t D, int64_t H, int32_t* status_word, void* stream) {
  if (!w0w2 || !w1 || !x || !out || !status_word) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  LACT_TRY(check_dims(B, N, D, H));
  if (!hidden && !few_pays(B, N, D, H)) return LACT_ERR_NULL;
  const ApplyArgs a{static_cast<const bf16*>(w0w2), static_cast<const bf16*>(w1), x, N * D, D, 0, N, out, N * D, D, 0,
                    static_cast<bf16*>(hidden), B, D, H};
  return run_apply(a, status_word, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------- allocation-free variant
// Scratch for lact_swiglu_ffn_fwd_static.  It lives in the library image: every GPU that loads
// the library holds these bytes until the process exits.
#define LACT_STATIC_SCRATCH_BYTES (16u << 20)
static __device__ __align__(256) unsigned char g_static_scratch[LACT_STATIC_SCRATCH_BYTES];

// Device address of g_static_scratch on the current device, resolved once per device.  In host
// code the array's name is only a handle for the runtime, never a pointer a kernel may use, so
// the address is asked for with cudaGetSymbolAddress and that result is what kernels receive.
static int static_scratch_address(void** out) {
  static std::mutex mu;
  static void* addr[64] = {nullptr};
  int dev = 0;
  LACT_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return LACT_ERR_DEVICE;
  std::lock_guard<std::mutex> lock(mu);
  if (addr[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_static_scratch) != cudaSuccess || p == nullptr)
      return LACT_ERR_CUDA;
    addr[dev] = p;
  }
  *out = addr[dev];
  return LACT_OK;
}

size_t lact_static_scratch_bytes(void) { return LACT_STATIC_SCRATCH_BYTES; }

int lact_swiglu_ffn_fwd_static(const void* w0w2, const void* w1, const void* x, void* out, int64_t B, int64_t N,
                               int64_t D, int64_t H, void* stream) {
  if (!w0w2 || !w1 || !x || !out) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  LACT_TRY(check_dims(B, N, D, H));
  // status word (256 bytes reserved) + hidden activations [B, N, H] bf16
  const unsigned long long hidden_bytes = static_cast<unsigned long long>(B) * static_cast<unsigned long long>(N) *
                                          static_cast<unsigned long long>(H) * 2ull;
  if (hidden_bytes > LACT_STATIC_SCRATCH_BYTES - 256ull) return LACT_ERR_STATIC_LIMIT;
  void* scratch = nullptr;
  LACT_TRY(static_scratch_address(&scratch));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the array keeps whatever the previous call left: the status word must start at zero; the
  // hidden activations behind it are fully overwritten before they are read
  LACT_CUDA(cudaMemsetAsync(scratch, 0, 256, s));
  ApplyArgs a{static_cast<const bf16*>(w0w2), static_cast<const bf16*>(w1), x, N * D, D, 0, N, out, N * D, D, 0,
              reinterpret_cast<bf16*>(static_cast<uint8_t*>(scratch) + 256), B, D, H};
  return run_apply(a, static_cast<int32_t*>(scratch), s);
}

int lact_static_status(void* stream) {
  LACT_TRY(check_device());
  void* scratch = nullptr;
  LACT_TRY(static_scratch_address(&scratch));
  return read_status_word(scratch, static_cast<cudaStream_t>(stream));
}

int lact_fw_grad_workspace_bytes(int64_t B, int64_t N, int64_t D, int64_t H, size_t* bytes_out) {
  if (!bytes_out) return LACT_ERR_NULL;
  LACT_TRY(check_dims(B, N, D, H));
  *bytes_out = 1024 + static_cast<size_t>(B) * N * 3 * H * 2;
  return LACT_OK;
}

int lact_fw_grad(const void* w0w2, const void* w1, const void* k, const void* v, const void* lr0, const void* lr1,
                 const void* lr2, int32_t lr_dtype, void* dw0w2, void* dw1, int64_t B, int64_t N, int64_t D, int64_t H,
                 void* workspace, size_t workspace_bytes, void* stream) {
  if (!w0w2 || !w1 || !k || !v || !lr0 || !lr1 || !lr2 || !dw0w2 || !dw1) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  size_t need = 0;
  LACT_TRY(lact_fw_grad_workspace_bytes(B, N, D, H, &need));
  if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255)) return LACT_ERR_WORKSPACE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  LACT_CUDA(cudaMemsetAsync(workspace, 0, 256, s));
  Carver cv(workspace);
  int32_t* status = cv.take<int32_t>(64);
  bf16* dy02 = cv.take<bf16>(static_cast<size_t>(B) * N * 2 * H);
  bf16* hid = cv.take<bf16>(static_cast<size_t>(B) * N * H);
  GradArgs g{static_cast<const bf16*>(w0w2), static_cast<const bf16*>(w1), k, v, N * D, D, N * D, D, 0, N, lr0, lr1,
             lr2, lr_dtype == LACT_F32, N, 1.0f, dy02, hid, dw0w2, dw1, 0, nullptr, B, D, H};
  return run_grad(g, status, s);
}

int lact_newton_schulz_workspace_bytes(int64_t B, int64_t R, int64_t C, size_t* bytes_out) {
  if (!bytes_out) return LACT_ERR_NULL;
  if (B < 1 || B > 65535 || R < 8 || C < 8 || (R % 8) || (C % 8)) return LACT_ERR_SHAPE;
  *bytes_out = 2048 + ns_group_bytes(B, std::min(R, C), std::max(R, C));
  return LACT_OK;
}

// The gradients are read four at a time.
static bool ns_source_aligned(const void* g, int32_t g_dtype) {
  return (reinterpret_cast<uintptr_t>(g) & (g_dtype == LACT_F32 ? 15 : 7)) == 0;
}

int lact_newton_schulz(const void* g, int32_t g_dtype, void* x, int64_t B, int64_t R, int64_t C, int32_t steps,
                       int32_t const_coeffs, void* workspace, size_t workspace_bytes, void* stream) {
  if (!g || !x) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  size_t need = 0;
  LACT_TRY(lact_newton_schulz_workspace_bytes(B, R, C, &need));
  if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255)) return LACT_ERR_WORKSPACE;
  if (steps < 0 || steps > 64 || (!const_coeffs && steps != 5)) return LACT_ERR_CONFIG;
  if (!ns_source_aligned(g, g_dtype)) return LACT_ERR_SHAPE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  LACT_CUDA(cudaMemsetAsync(workspace, 0, 256, s));
  Carver cv(workspace);
  int32_t* status = cv.take<int32_t>(64);
  NsGroup grp;
  ns_group_init(grp, B, R, C, 0);
  carve_ns_group(cv, grp);
  const bf16* res = nullptr;
  const void* srcs[2] = {g, g};
  LACT_TRY(run_newton_schulz(&grp, 1, srcs, g_dtype == LACT_F32, nullptr, 0, steps, const_coeffs, status, s, &res));
  LACT_CUDA(cudaMemcpyAsync(x, res, static_cast<size_t>(B) * R * C * 2, cudaMemcpyDeviceToDevice, s));
  return LACT_OK;
}

// ---------------------------------------------------------------- Newton-Schulz with saved iterates, and its backward
int lact_ns_trace_bytes(int64_t B, int64_t R, int64_t C, int32_t steps, size_t* bytes_out) {
  if (!bytes_out) return LACT_ERR_NULL;
  NsTrace t;
  LACT_TRY(plan_ns_trace(nullptr, B, R, C, steps, 0, &t));
  *bytes_out = t.bytes;
  return LACT_OK;
}

int lact_ns_trace_result_offset(int64_t B, int64_t R, int64_t C, int32_t steps, size_t* offset_out) {
  if (!offset_out) return LACT_ERR_NULL;
  NsTrace t;
  // carve from a fake, never dereferenced base (a null base yields null pointers) and subtract it again
  uint8_t* const fake = reinterpret_cast<uint8_t*>(static_cast<uintptr_t>(1) << 40);
  LACT_TRY(plan_ns_trace(fake, B, R, C, steps, 0, &t));
  *offset_out = static_cast<size_t>(reinterpret_cast<uint8_t*>(t.X) - fake) +
                static_cast<size_t>(B) * R * C * steps * sizeof(bf16);
  return LACT_OK;
}

int lact_ns_trace_fwd(const void* g, int32_t g_dtype, void* x_out, int64_t B, int64_t R, int64_t C, int32_t steps,
                      int32_t const_coeffs, int32_t gram_right, void* trace, size_t trace_bytes, int32_t* status_word,
                      void* stream) {
  if (!g || !x_out || !trace || !status_word) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  if ((reinterpret_cast<uintptr_t>(trace) & 255) != 0) return LACT_ERR_WORKSPACE;
  if (!const_coeffs && steps != 5) return LACT_ERR_CONFIG;
  if (!ns_source_aligned(g, g_dtype)) return LACT_ERR_SHAPE;
  NsTrace t;
  LACT_TRY(plan_ns_trace(trace, B, R, C, steps, gram_right, &t));
  if (t.bytes > trace_bytes) return LACT_ERR_WORKSPACE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t rc = static_cast<size_t>(B) * R * C, mm = static_cast<size_t>(B) * t.grp.m * t.grp.m;
  t.grp.xa = t.X;
  const void* srcs[2] = {g, g};
  // all iterations in one launch that keeps every iterate (up to five: both coefficient schedules of the reference's
  // drivers); longer constant-coefficient runs go iteration by iteration
  int rc_f = LACT_ERR_CONFIG;
  if (steps <= 5) {
    const NsKeep keep{t.X, t.A, t.P};
    const bf16* res = nullptr;
    rc_f = run_newton_schulz(&t.grp, 1, srcs, g_dtype == LACT_F32, nullptr, 0, steps, const_coeffs, status_word, s, &res, &keep);
  } else {
    LACT_TRY(launch_ns_prepare(&t.grp, 1, srcs, g_dtype == LACT_F32, 1, s));  // X[0] = normalised bf16(g)
  }
  if (rc_f == LACT_ERR_CONFIG) {
    for (int it = 0; it < steps; ++it) {
      NsGroup gi = t.grp;
      gi.xa = t.X + rc * it;
      gi.xb = t.X + rc * (it + 1);
      gi.gram = t.A + mm * it;
      gi.poly = t.P + mm * it;
      const bf16* res = nullptr;
      LACT_TRY(run_ns_iterations(&gi, 1, 1, const_coeffs, &res, status_word, s, 0, const_coeffs ? 0 : it));
    }
  } else {
    LACT_TRY(rc_f);
  }
  LACT_CUDA(cudaMemcpyAsync(x_out, t.X + rc * steps, rc * 2, cudaMemcpyDeviceToDevice, s));
  return LACT_OK;
}

static int bmm2_scaled(const void* a0, int32_t a0_mn, const void* b0, int32_t b0_mn, const void* a1, int32_t a1_mn,
                       const void* b1, int32_t b1_mn, void* c, int32_t c_dtype, int64_t batch, int64_t M, int64_t N,
                       int64_t K, int32_t* status_word, void* stream, float alpha);

// dx0 (fp32) = gradient w.r.t. the normalised first iterate X[0], given du = bf16 gradient w.r.t. the
// result X[steps]; roundings are treated as identities and every operand is bf16 (the reference
// differentiates its bf16 iteration the same way).  With Q = dP + dP^T (dP = dX' X^T) and
// CB = c A + (b/2) I the three products per iteration are, for a wide iterate ([m][n], A = X X^T):
//   Q = dX' X^T + X dX'^T,   S = CB Q + Q CB,   dX = P dX' + S X,
// and for a tall one ([n][m], A = X^T X, X' = X P^T):  Q = dX'^T X + X^T dX',  dX = dX' P + X S.
int lact_ns_trace_bwd(const void* du, void* dx0, int64_t B, int64_t R, int64_t C, int32_t steps, int32_t const_coeffs,
                      int32_t gram_right, void* trace, size_t trace_bytes, int32_t* status_word, void* stream) {
  if (!du || !dx0 || !trace || !status_word) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  NsTrace t;
  LACT_TRY(plan_ns_trace(trace, B, R, C, steps, gram_right, &t));
  if (t.bytes > trace_bytes) return LACT_ERR_WORKSPACE;
  const int64_t m = t.grp.m, n = t.grp.n;
  const size_t rc = static_cast<size_t>(B) * R * C, mm = static_cast<size_t>(B) * m * m;
  const int tall = t.grp.transposed;
  const bf16* dX = static_cast<const bf16*>(du);
  for (int it = steps - 1; it >= 0; --it) {
    const float* co = const_coeffs ? kNsConst : kNsTuned[it];
    const bf16* X = t.X + rc * it;
    const bf16* P = t.P + mm * it;
    // Q [m][m]: contraction over the long side n
    LACT_TRY(lact_bmm2_bf16(dX, tall, X, tall, X, tall, dX, tall, t.Q, LACT_BF16, 0, B, m, m, n, status_word, stream));
    // S = CB Q + Q CB with CB = c A + (b/2) I = c (A + (b/2c) I): the kept shifted Gram matrix, scaled in the epilogue
    const bf16* As = t.A + mm * it;
    LACT_TRY(bmm2_scaled(As, 0, t.Q, 0, t.Q, 0, As, 0, t.S, LACT_BF16, B, m, m, m, status_word, stream, co[2]));
    void* out = it == 0 ? dx0 : static_cast<void*>((it & 1) ? t.dXa : t.dXb);
    const int out_dt = it == 0 ? LACT_F32 : LACT_BF16;
    if (!tall) LACT_TRY(lact_bmm2_bf16(P, 0, dX, 1, t.S, 0, X, 1, out, out_dt, 0, B, m, n, m, status_word, stream));
    else LACT_TRY(lact_bmm2_bf16(dX, 0, P, 1, X, 0, t.S, 0, out, out_dt, 0, B, n, m, m, status_word, stream));
    dX = static_cast<const bf16*>(out);
  }
  return LACT_OK;
}

static int qkv_prologue_impl(const void* xq, const void* xk, const void* xv, int64_t ld_q, int64_t ld_k, int64_t ld_v,
                             int64_t bs_q, int64_t bs_k, int64_t bs_v, void* q, void* k, void* v, int64_t b, int64_t s,
                             int64_t n_heads, int64_t d, int32_t qkv_silu, int32_t v_silu, const void* cos,
                             const void* sin, int64_t rope_head_dim, int64_t n_positions, int64_t seqlen_offset,
                             const int32_t* seq_start, void* stream) {
  if (!xq || !xk || !xv || !q || !k || !v) return LACT_ERR_NULL;
  if (seq_start != nullptr && (b != 1 || rope_head_dim == 0)) return LACT_ERR_CONFIG;
  LACT_TRY(check_device());
  if (b < 1 || s < 1 || n_heads < 1 || d < 8 || d > 1024 || (d % 8) != 0) return LACT_ERR_SHAPE;
  if (b * s * n_heads > (1ll << 40) || b > 65535 || s > (1ll << 30)) return LACT_ERR_SHAPE;
  const void* xs[3] = {xq, xk, xv};
  void* outs[3] = {q, k, v};
  const int64_t lds[3] = {ld_q, ld_k, ld_v}, bss[3] = {bs_q, bs_k, bs_v};
  PrologueArgs a;
  std::memset(&a, 0, sizeof(a));
  for (int t = 0; t < 3; ++t) {
    // rows move as 16-byte vectors
    if ((reinterpret_cast<uintptr_t>(xs[t]) & 15) != 0 || (reinterpret_cast<uintptr_t>(outs[t]) & 15) != 0 ||
        lds[t] < n_heads * d || (lds[t] % 8) != 0 || (bss[t] % 8) != 0)
      return LACT_ERR_SHAPE;
    a.x[t] = static_cast<const bf16*>(xs[t]);
    a.out[t] = static_cast<bf16*>(outs[t]);
    a.ld[t] = lds[t];
    a.bs[t] = bss[t];
  }
  a.b = static_cast<int32_t>(b); a.s = static_cast<int32_t>(s);
  a.n_h = static_cast<int32_t>(n_heads); a.d = static_cast<int32_t>(d);
  a.silu[0] = a.silu[1] = qkv_silu ? 1 : 0;
  a.silu[2] = (qkv_silu && v_silu) ? 1 : 0;
  a.l2norm[0] = a.l2norm[1] = 1;
  a.l2norm[2] = 0;
  if (rope_head_dim != 0) {
    if (!cos || !sin) return LACT_ERR_NULL;
    // attention heads of a power-of-two size that tile every fast-weight head; positions inside the tables
    if (rope_head_dim < 32 || rope_head_dim > 1024 || (rope_head_dim & (rope_head_dim - 1)) != 0 ||
        (d % rope_head_dim) != 0 || seqlen_offset < 0 || seqlen_offset + s > n_positions)
      return LACT_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(cos) & 15) != 0 || (reinterpret_cast<uintptr_t>(sin) & 15) != 0) return LACT_ERR_SHAPE;
    a.cos = static_cast<const bf16*>(cos);
    a.sin = static_cast<const bf16*>(sin);
    a.rope_hd = static_cast<int32_t>(rope_head_dim);
    a.pos0 = static_cast<int32_t>(seqlen_offset);
    a.seq_start = seq_start;
  }
  const int64_t rows = b * s * n_heads;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  const unsigned grid = static_cast<unsigned>(ceil_div(rows, 8));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool exact = n_heads <= 65535 / 3 && with_row_shape(d, [&](auto lpr, auto v) {
    const dim3 g(ceil_div(s, 256 / lpr.value), static_cast<unsigned>(3 * n_heads), static_cast<unsigned>(b));
    if (a.rope_hd != 0) (void)launch_pdl(qkv_rows_kernel<lpr.value, v.value, true>, g, dim3(256), 0, st, a);
    else (void)launch_pdl(qkv_rows_kernel<lpr.value, v.value, false>, g, dim3(256), 0, st, a);
  });
  if (exact) {
  } else if (a.rope_hd != 0) {
    switch (ceil_div(d, 256)) {
      case 1: qkv_prologue_kernel<1, true><<<grid, 256, 0, st>>>(a); break;
      case 2: qkv_prologue_kernel<2, true><<<grid, 256, 0, st>>>(a); break;
      case 3: qkv_prologue_kernel<3, true><<<grid, 256, 0, st>>>(a); break;
      default: qkv_prologue_kernel<4, true><<<grid, 256, 0, st>>>(a); break;
    }
  } else {
    switch (ceil_div(d, 256)) {
      case 1: qkv_prologue_kernel<1, false><<<grid, 256, 0, st>>>(a); break;
      case 2: qkv_prologue_kernel<2, false><<<grid, 256, 0, st>>>(a); break;
      case 3: qkv_prologue_kernel<3, false><<<grid, 256, 0, st>>>(a); break;
      default: qkv_prologue_kernel<4, false><<<grid, 256, 0, st>>>(a); break;
    }
  }
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_qkv_prologue_bwd(const void* xq, const void* xk, const void* xv, int64_t ld_q, int64_t ld_k, int64_t ld_v,
                          int64_t bs_q, int64_t bs_k, int64_t bs_v, const void* dq, const void* dk, const void* dv,
                          void* dxq, void* dxk, void* dxv, int64_t b, int64_t s, int64_t n_heads, int64_t d,
                          int32_t qkv_silu, int32_t v_silu, const void* cos, const void* sin, int64_t rope_head_dim,
                          int64_t n_positions, int64_t seqlen_offset, const int32_t* seq_start, void* stream) {
  if (!xq || !xk || !xv || !dxq || !dxk || !dxv) return LACT_ERR_NULL;
  if (seq_start != nullptr && (b != 1 || rope_head_dim == 0)) return LACT_ERR_CONFIG;
  LACT_TRY(check_device());
  if (b < 1 || s < 1 || n_heads < 1 || d < 8 || d > 1024 || (d % 8) != 0) return LACT_ERR_SHAPE;
  if (b * s * n_heads > (1ll << 40) || b > 65535 || s > (1ll << 30)) return LACT_ERR_SHAPE;
  const void* xs[3] = {xq, xk, xv};
  const void* dzs[3] = {dq, dk, dv};
  void* outs[3] = {dxq, dxk, dxv};
  const int64_t lds[3] = {ld_q, ld_k, ld_v}, bss[3] = {bs_q, bs_k, bs_v};
  PrologueBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  for (int t = 0; t < 3; ++t) {
    if ((reinterpret_cast<uintptr_t>(xs[t]) & 15) != 0 || (reinterpret_cast<uintptr_t>(outs[t]) & 15) != 0 ||
        (reinterpret_cast<uintptr_t>(dzs[t]) & 15) != 0 || lds[t] < n_heads * d || (lds[t] % 8) != 0 || (bss[t] % 8) != 0)
      return LACT_ERR_SHAPE;
    a.x[t] = static_cast<const bf16*>(xs[t]);
    a.dz[t] = static_cast<const bf16*>(dzs[t]);
    a.dx[t] = static_cast<bf16*>(outs[t]);
    a.ld[t] = lds[t];
    a.bs[t] = bss[t];
  }
  a.b = static_cast<int32_t>(b); a.s = static_cast<int32_t>(s);
  a.n_h = static_cast<int32_t>(n_heads); a.d = static_cast<int32_t>(d);
  a.silu[0] = a.silu[1] = qkv_silu ? 1 : 0;
  a.silu[2] = (qkv_silu && v_silu) ? 1 : 0;
  a.l2norm[0] = a.l2norm[1] = 1;
  a.l2norm[2] = 0;
  if (rope_head_dim != 0) {
    if (!cos || !sin) return LACT_ERR_NULL;
    if (rope_head_dim < 32 || rope_head_dim > 1024 || (rope_head_dim & (rope_head_dim - 1)) != 0 ||
        (d % rope_head_dim) != 0 || seqlen_offset < 0 || seqlen_offset + s > n_positions)
      return LACT_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(cos) & 15) != 0 || (reinterpret_cast<uintptr_t>(sin) & 15) != 0) return LACT_ERR_SHAPE;
    a.cos = static_cast<const bf16*>(cos);
    a.sin = static_cast<const bf16*>(sin);
    a.rope_hd = static_cast<int32_t>(rope_head_dim);
    a.pos0 = static_cast<int32_t>(seqlen_offset);
    a.seq_start = seq_start;
  }
  const int64_t rows = b * s * n_heads;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  const unsigned grid = static_cast<unsigned>(ceil_div(rows, 8));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool exact = n_heads <= 65535 / 3 && with_row_shape(d, [&](auto lpr, auto v) {
    const dim3 g(ceil_div(s, 256 / lpr.value), static_cast<unsigned>(3 * n_heads), static_cast<unsigned>(b));
    if (a.rope_hd != 0) (void)launch_pdl(qkv_rows_bwd_kernel<lpr.value, v.value, true>, g, dim3(256), 0, st, a);
    else (void)launch_pdl(qkv_rows_bwd_kernel<lpr.value, v.value, false>, g, dim3(256), 0, st, a);
  });
  if (exact) {
  } else if (a.rope_hd != 0) {
    switch (ceil_div(d, 256)) {
      case 1: qkv_prologue_bwd_kernel<1, true><<<grid, 256, 0, st>>>(a); break;
      case 2: qkv_prologue_bwd_kernel<2, true><<<grid, 256, 0, st>>>(a); break;
      case 3: qkv_prologue_bwd_kernel<3, true><<<grid, 256, 0, st>>>(a); break;
      default: qkv_prologue_bwd_kernel<4, true><<<grid, 256, 0, st>>>(a); break;
    }
  } else {
    switch (ceil_div(d, 256)) {
      case 1: qkv_prologue_bwd_kernel<1, false><<<grid, 256, 0, st>>>(a); break;
      case 2: qkv_prologue_bwd_kernel<2, false><<<grid, 256, 0, st>>>(a); break;
      case 3: qkv_prologue_bwd_kernel<3, false><<<grid, 256, 0, st>>>(a); break;
      default: qkv_prologue_bwd_kernel<4, false><<<grid, 256, 0, st>>>(a); break;
    }
  }
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

// Two blocks per SM: what an SM holds of out_rows_bwd_kernel, and the better number for the general kernel too (2 batches x
// 8192 tokens x 4 heads of 72 / 320 / 640 / 896: 71 / 118 / 169 / 255 us; with four per SM 75 / 122 / 177 / 263).
int lact_out_epilogue_bwd_blocks(void) { return sm_count() * 2; }

int lact_out_epilogue_bwd(const void* fw_x, const void* weight, const void* gate_proj, int64_t gate_ld, const void* dout,
                          int64_t dout_ld, void* dx, void* dgate, void* dw_partial, int64_t b, int64_t s, int64_t n_heads,
                          int64_t d, float eps, void* stream) {
  if (!fw_x || !weight || !dout || !dx || !dw_partial) return LACT_ERR_NULL;
  if ((gate_proj == nullptr) != (dgate == nullptr)) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  if (b < 1 || s < 1 || n_heads < 1 || d < 8 || d > 1024 || (d % 8) != 0 || b > 65535 || s > (1ll << 30))
    return LACT_ERR_SHAPE;
  auto bad = [&](const void* p, int64_t ld) {
    return p != nullptr && ((reinterpret_cast<uintptr_t>(p) & 15) != 0 || ld < n_heads * d || (ld % 8) != 0);
  };
  if ((reinterpret_cast<uintptr_t>(fw_x) & 15) != 0 || (reinterpret_cast<uintptr_t>(weight) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(dx) & 15) != 0 || (reinterpret_cast<uintptr_t>(dgate) & 15) != 0 ||
      bad(gate_proj, gate_ld) || bad(dout, dout_ld))
    return LACT_ERR_SHAPE;
  EpilogueBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  a.x = static_cast<const bf16*>(fw_x);
  a.weight = static_cast<const float*>(weight);
  a.gate = static_cast<const bf16*>(gate_proj);
  a.dout = static_cast<const bf16*>(dout);
  a.gate_ld = gate_ld; a.dout_ld = dout_ld;
  a.dx = static_cast<bf16*>(dx);
  a.dgate = static_cast<bf16*>(dgate);
  a.dw_partial = static_cast<float*>(dw_partial);
  a.b = static_cast<int32_t>(b); a.s = static_cast<int32_t>(s);
  a.n_h = static_cast<int32_t>(n_heads); a.d = static_cast<int32_t>(d);
  a.eps = eps;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  const unsigned grid = static_cast<unsigned>(lact_out_epilogue_bwd_blocks());
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool exact = with_row_shape(
      d, [&](auto lpr, auto v) { (void)launch_pdl(out_rows_bwd_kernel<lpr.value, v.value>, grid, dim3(256), 0, st, a); });
  if (!exact) switch (ceil_div(d, 256)) {
    case 1: out_epilogue_bwd_kernel<1><<<grid, 256, 0, st>>>(a); break;
    case 2: out_epilogue_bwd_kernel<2><<<grid, 256, 0, st>>>(a); break;
    case 3: out_epilogue_bwd_kernel<3><<<grid, 256, 0, st>>>(a); break;
    default: out_epilogue_bwd_kernel<4><<<grid, 256, 0, st>>>(a); break;
  }
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_qkv_prologue(const void* xq, const void* xk, const void* xv, int64_t ld_q, int64_t ld_k, int64_t ld_v,
                      int64_t bs_q, int64_t bs_k, int64_t bs_v, void* q, void* k, void* v, int64_t b, int64_t s,
                      int64_t n_heads, int64_t d, int32_t qkv_silu, int32_t v_silu, void* stream) {
  return qkv_prologue_impl(xq, xk, xv, ld_q, ld_k, ld_v, bs_q, bs_k, bs_v, q, k, v, b, s, n_heads, d, qkv_silu, v_silu,
                           nullptr, nullptr, 0, 0, 0, nullptr, stream);
}

int lact_qkv_prologue_rope(const void* xq, const void* xk, const void* xv, int64_t ld_q, int64_t ld_k, int64_t ld_v,
                           int64_t bs_q, int64_t bs_k, int64_t bs_v, void* q, void* k, void* v, int64_t b, int64_t s,
                           int64_t n_heads, int64_t d, int32_t qkv_silu, int32_t v_silu, const void* cos, const void* sin,
                           int64_t rope_head_dim, int64_t n_positions, int64_t seqlen_offset, const int32_t* seq_start,
                           void* stream) {
  if (rope_head_dim == 0) return LACT_ERR_SHAPE;
  return qkv_prologue_impl(xq, xk, xv, ld_q, ld_k, ld_v, bs_q, bs_k, bs_v, q, k, v, b, s, n_heads, d, qkv_silu, v_silu,
                           cos, sin, rope_head_dim, n_positions, seqlen_offset, seq_start, stream);
}

int lact_lr_prologue(const void* lr_proj, int32_t proj_dtype, int64_t proj_ld, float base_lr_inv, const void* mom_logits,
                     int32_t logits_dtype, int64_t logits_ld, void* lr0, void* lr1, void* lr2, void* momentum, int64_t b,
                     int64_t s, int64_t n_heads, void* stream) {
  if (!lr_proj || !lr0 || !lr1 || !lr2 || ((mom_logits == nullptr) != (momentum == nullptr))) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  if (b < 1 || s < 1 || n_heads < 1 || b > 65535 || s > (1ll << 30) || n_heads > 4096) return LACT_ERR_SHAPE;
  if (proj_ld < 3 * n_heads || (mom_logits && logits_ld < n_heads)) return LACT_ERR_SHAPE;
  if ((proj_dtype != LACT_F32 && proj_dtype != LACT_BF16) ||
      (mom_logits && logits_dtype != LACT_F32 && logits_dtype != LACT_BF16))
    return LACT_ERR_DTYPE;
  LrPrologueArgs a;
  std::memset(&a, 0, sizeof(a));
  a.proj = lr_proj; a.logits = mom_logits;
  a.proj_f32 = proj_dtype == LACT_F32; a.logits_f32 = logits_dtype == LACT_F32;
  a.proj_ld = proj_ld; a.logits_ld = logits_ld;
  a.base_lr_inv = base_lr_inv;
  a.lr[0] = static_cast<float*>(lr0); a.lr[1] = static_cast<float*>(lr1); a.lr[2] = static_cast<float*>(lr2);
  a.mom = static_cast<float*>(momentum);
  a.b = static_cast<int32_t>(b); a.s = static_cast<int32_t>(s); a.n_h = static_cast<int32_t>(n_heads);
  const int64_t total = b * s * n_heads;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  LACT_CUDA(launch_pdl(lr_prologue_kernel, dim3(static_cast<unsigned>(ceil_div(total, 256))), dim3(256), 0,
                       static_cast<cudaStream_t>(stream), a));
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_lr_prologue_bwd(const void* lr_proj, int32_t proj_dtype, int64_t proj_ld, float base_lr_inv, const void* mom_logits,
                         int32_t logits_dtype, int64_t logits_ld, const void* g0, const void* g1, const void* g2, const void* gm,
                         void* dproj, void* dlogits, int64_t b, int64_t s, int64_t n_heads, void* stream) {
  if (!lr_proj || !dproj || ((mom_logits == nullptr) != (dlogits == nullptr))) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  if (b < 1 || s < 1 || n_heads < 1 || b > 65535 || s > (1ll << 30) || n_heads > 4096) return LACT_ERR_SHAPE;
  if (proj_ld < 3 * n_heads || (mom_logits && logits_ld < n_heads)) return LACT_ERR_SHAPE;
  LrPrologueBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  a.proj = lr_proj; a.logits = mom_logits;
  a.proj_f32 = proj_dtype == LACT_F32; a.logits_f32 = logits_dtype == LACT_F32;
  a.proj_ld = proj_ld; a.logits_ld = logits_ld;
  a.base_lr_inv = base_lr_inv;
  a.g[0] = static_cast<const float*>(g0); a.g[1] = static_cast<const float*>(g1); a.g[2] = static_cast<const float*>(g2);
  a.gm = static_cast<const float*>(gm);
  a.dproj = dproj; a.dlogits = dlogits;
  a.b = static_cast<int32_t>(b); a.s = static_cast<int32_t>(s); a.n_h = static_cast<int32_t>(n_heads);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  KernelScope scope(kClsOther, st);
  LACT_CUDA(launch_pdl(lr_prologue_bwd_kernel, dim3(static_cast<unsigned>(ceil_div(b * s * n_heads, 256))), dim3(256), 0, st, a));
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_column_sums(const float* x, float* out, int64_t rows, int64_t cols, void* stream) {
  if (!x || !out) return LACT_ERR_NULL;
  if (rows < 1 || cols < 1 || cols > (1ll << 30)) return LACT_ERR_SHAPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  KernelScope scope(kClsOther, st);
  LACT_CUDA(launch_pdl(column_sums_kernel, dim3(static_cast<unsigned>(ceil_div(cols, 32))), dim3(256), 0, st, x, out, rows, cols));
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_seq_start(const int32_t* cu_seqlens, int64_t n_sequences, int64_t n_tokens, int32_t* out, void* stream) {
  if (!cu_seqlens || !out) return LACT_ERR_NULL;
  if (n_sequences < 1 || n_tokens < 1 || n_tokens > (1ll << 30)) return LACT_ERR_SHAPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  KernelScope scope(kClsOther, st);
  seq_start_kernel<<<static_cast<unsigned>(ceil_div(n_tokens, 256)), 256, 0, st>>>(cu_seqlens, n_sequences, n_tokens, out);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_out_epilogue(const void* fw_x, const void* weight, const void* gate_proj, int64_t gate_ld, const void* resid,
                      int64_t resid_ld, void* out, int64_t out_ld, int64_t b, int64_t s, int64_t n_heads, int64_t d,
                      float eps, void* stream) {
  if (!fw_x || !weight || !out) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  if (b < 1 || s < 1 || n_heads < 1 || d < 8 || d > 1024 || (d % 8) != 0 || b > 65535 || s > (1ll << 30))
    return LACT_ERR_SHAPE;
  auto bad = [&](const void* p, int64_t ld) {
    return p != nullptr && ((reinterpret_cast<uintptr_t>(p) & 15) != 0 || ld < n_heads * d || (ld % 8) != 0);
  };
  if ((reinterpret_cast<uintptr_t>(fw_x) & 15) != 0 || (reinterpret_cast<uintptr_t>(weight) & 15) != 0 ||
      bad(gate_proj, gate_ld) || bad(resid, resid_ld) || bad(out, out_ld))
    return LACT_ERR_SHAPE;
  EpilogueArgs a;
  std::memset(&a, 0, sizeof(a));
  a.x = static_cast<const bf16*>(fw_x);
  a.weight = static_cast<const float*>(weight);
  a.gate = static_cast<const bf16*>(gate_proj);
  a.resid = static_cast<const bf16*>(resid);
  a.out = static_cast<bf16*>(out);
  a.gate_ld = gate_ld; a.resid_ld = resid_ld; a.out_ld = out_ld;
  a.b = static_cast<int32_t>(b); a.s = static_cast<int32_t>(s);
  a.n_h = static_cast<int32_t>(n_heads); a.d = static_cast<int32_t>(d);
  a.eps = eps;
  const int64_t rows = b * s * n_heads;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  const unsigned grid = static_cast<unsigned>(ceil_div(rows, 8));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool exact = n_heads <= 65535 && with_row_shape(d, [&](auto lpr, auto v) {
    const dim3 g(ceil_div(s, 256 / lpr.value), static_cast<unsigned>(n_heads), static_cast<unsigned>(b));
    (void)launch_pdl(out_rows_kernel<lpr.value, v.value>, g, dim3(256), 0, st, a);
  });
  if (!exact) switch (ceil_div(d, 256)) {
    case 1: out_epilogue_kernel<1><<<grid, 256, 0, st>>>(a); break;
    case 2: out_epilogue_kernel<2><<<grid, 256, 0, st>>>(a); break;
    case 3: out_epilogue_kernel<3><<<grid, 256, 0, st>>>(a); break;
    default: out_epilogue_kernel<4><<<grid, 256, 0, st>>>(a); break;
  }
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

// Which query tiles of an attention launch are cut over their keys, and into how many CTAs.  Whole tiles fill whole rounds
// of the SMs (a CTA takes an SM's shared memory); the rest, all tiles where there are fewer than SMs, are cut so that the
// launch ends sooner: a CTA takes about 4 us plus 1.5 us per 128 keys (1.2 at d = 64), combining about 0.6 us per share.
// Measured: 1560 queries over 4680 keys, 12 heads of 128 (156 tiles on 148 SMs, the last 8 cut in 8) 110 -> 80 us.
struct SwaSplit {
  int64_t whole;
  int splits;
  double us;
};
// Estimates of both attention forwards, which swa_takes_pairs compares.  An SM spends `tile` us per key tile and `item` per query tile or
// pair, a launch `launch`: fitted to 1722 random shapes (1 to 16 entries, 1 to 32 heads of 64 and 128, 32 to 16384 queries, windows of any
// share, caches and blocks up to 16384 keys), each timed on single tiles, on pairs whole and on pairs cut in three ways, in replayed graphs, so that
// small calls show what the device takes.  What is chosen is more than 5 % slower than the fastest way in 92, than single tiles in 9.
struct SwaCost {
  double tile, item, launch;
};
static SwaCost swa_single_cost(int64_t d) { return d == 64 ? SwaCost{1.19, 5.1, 1.05} : SwaCost{1.12, 6.4, 1.05}; }
static SwaCost swa_pair_cost(int64_t d) { return d == 64 ? SwaCost{1.62, 1.63, 4.5} : SwaCost{1.87, 2.23, 4.5}; }
// Causal attention: the first key tile that query tile i meets is i - swa_behind, or 0.
static int64_t swa_band(int64_t l, int64_t window) { return window > 0 && window < l ? window : l; }
static int64_t swa_behind(int64_t l, int64_t window) { return ceil_div(swa_band(l, window) - 1, 128); }

static SwaSplit swa_split(int64_t b, int64_t l, int64_t lk, int64_t heads, int64_t d, int64_t window, bool may_cut) {
  const int64_t sms = sm_count(), n = ceil_div(l, 128), tiles = b * heads * n;
  const int64_t span = window < 0 ? (lk > 0 ? lk : l) : window > 0 && window < l ? std::min(l, window + 127) : l;
  const int64_t T = ceil_div(span, 128), rest = tiles % sms;
  const double per_tile = d == 64 ? 1.2 : 1.5, round = T * per_tile + 4.0;
  // Whole tiles: rounds of equal ones; causal ones differ in length, are taken as SMs come free, and the last of them are the long ones of
  // a head: an equal share of the work and 0.45 of the longest; where the rest is cut, 0.57 of one of its pieces.
  const SwaCost cost = swa_single_cost(d);
  const double longest = T * cost.tile + cost.item;
  double share = 0.0;
  if (window >= 0) {
    const int64_t c = swa_behind(l, window), keys = n * (n + 1) / 2 - (n > c ? (n - c) * (n - c - 1) / 2 : 0);
    share = static_cast<double>(b * heads) * (keys * cost.tile + n * cost.item) / sms;
  }
  SwaSplit best{tiles, 1, cost.launch + (window < 0 || tiles <= sms ? ((tiles + sms - 1) / sms) * longest : std::max(longest, share + 0.45 * longest))};
  if (!may_cut || rest == 0 || tiles > 64 * sms) return best;
  double end = round;   // of the rest
  for (int s = 2; s <= 16 && s <= T; ++s) {
    const int64_t turns = (rest * s + sms - 1) / sms, keys = (T + s - 1) / s;
    const double c = turns * (keys * per_tile + 4.0) + 2.0 + 0.6 * s;
    if (c < 0.9 * end) {
      end = c;
      const double piece = keys * cost.tile + cost.item, put = 2.4 + 0.57 * s;   // (and the pieces put together)
      const double us = window < 0 || tiles < sms ? (tiles / sms) * longest + turns * piece + put
                                                  : std::max(longest, share + rest * (s - 1) * cost.item / sms + 0.57 * piece + put);
      best = SwaSplit{tiles - rest, s, cost.launch + us};
    }
  }
  return best;
}

// The same launch on pairs of query tiles (see SwaPairArgs).  Whole pairs fill whole rounds of the SMs; the rest, all pairs where there are
// fewer than SMs, are cut over their keys if the longest CTA then ends sooner.  A second launch puts the pieces together: it, what it
// waits for and the pieces' rows take 6.9 us and 0.05 per piece.  Measured: 1560 queries over 4680 keys, 12
// heads of 128 (84 pairs on 148 SMs, 38 key tiles each) whole 86, cut 73 us.  Pairs of causal attention without a window differ in length and
// are dealt the long ones first: 8 heads of 8192 queries (256 pairs) are left whole, 134 us, 221 with the 108 shortest cut.
struct SwaPairSplit {
  int64_t whole, rest, cutters, span;   // cutters = 0: nothing is cut (and rest = 0)
  double us;
};
static SwaPairSplit swa_pair_split(int64_t b, int64_t l, int64_t lk, int64_t heads, int64_t d, int64_t window, bool may_cut) {
  const int64_t sms = sm_count(), bh = b * heads, pairs = ceil_div(l, 256), items = bh * pairs;
  const bool causal = window >= 0;
  const int64_t behind = swa_behind(l, window);
  // key tiles of an item, at most (what is cut is laid out by it: none may have more)
  const int64_t span = causal ? std::min<int64_t>(ceil_div(l, 128), behind + 2) : ceil_div(lk > 0 ? lk : l, 128);
  const SwaCost cost = swa_pair_cost(d);
  const double longest = span * cost.tile + cost.item;
  // key tiles of pair p and of all pairs before it (of the last pair's second tile there may be no rows)
  auto keys = [&](int64_t p) { return 2 * (p + 1) - std::max<int64_t>(0, 2 * p - behind) - (p + 1 == pairs ? ceil_div(l, 128) % 2 : 0); };
  auto keys_before = [&](int64_t p) {
    const int64_t m = (behind + 1) / 2;
    return p * (p + 1) - (p > m ? (p - m) * (p + m - 1 - behind) : 0);
  };
  // The longest CTA's time for the first n items.  Where their lengths differ: up to eight rounds by those of five CTAs (the call waits for
  // this), beyond by an equal share of the work and 0.27 of the longest item.
  auto dealt = [&](int64_t n) -> double {
    const int64_t rounds = (n + sms - 1) / sms;
    if (!causal || n <= sms) return rounds * longest;
    if (rounds > 8) {
      const int64_t full = n / bh, part = n % bh;
      const int64_t all = bh * (keys_before(pairs) - ceil_div(l, 128) % 2 - keys_before(pairs - full)) + (part > 0 ? part * keys(pairs - 1 - full) : 0);
      return (all * cost.tile + n * cost.item) / sms + 0.27 * longest;
    }
    double worst = 0.0;
    for (int64_t i = 0; i <= 4; ++i) {
      const int64_t c = i * (sms - 1) / 4;
      double t = 0.0;
      for (int64_t r = 0; r < rounds; ++r) {
        const int64_t item = r * sms + ((r & 1) ? sms - 1 - c : c);
        if (item < n) t += keys(pairs - 1 - item / bh) * cost.tile + cost.item;
      }
      worst = std::max(worst, t);
    }
    return worst;
  };
  SwaPairSplit best{items, 0, 0, 0, dealt(items) + cost.launch};
  const int64_t rest = items % sms;
  if (!may_cut || rest == 0 || items > 64 * sms) return best;
  const double before = dealt(items - rest) + cost.launch + 6.9;
  for (int64_t s = 2, last = 0; s <= 16; s += 1 + s / 4) {
    const int64_t cutters = std::min(rest * std::min(s, span), sms);
    if (cutters == last) break;
    last = cutters;
    const double us = before + ceil_div(rest * span, cutters) * cost.tile + 0.05 * (cutters + rest);
    if (us < best.us) best = SwaPairSplit{items - rest, rest, cutters, span, us};
  }
  return best;
}
// Scratch of a cut launch: fewer pieces than cutters and items together, 256 rows each, from the caller's next multiple of 32 bytes on
// (the caller's own has 16, rows are stored 32 bytes at a time).
static size_t swa_pair_scratch(const SwaPairSplit& sp, int64_t d) {
  return sp.cutters > 0 ? static_cast<size_t>(sp.cutters + sp.rest) * 256 * (d * sizeof(float) + sizeof(float2)) + 16 : 0;
}
// Whether a launch runs on pairs: by the estimates of both.  Measured (us, single tiles / pairs; heads of 128 unless stated): 4 x 8192 queries,
// 12 heads, no window 1084 / 769; 16 x 2048 392 / 246, of 64 325 / 184; 12 heads, 32768 queries of packed sequences of 256 under a window of
// 2048 182 / 75, of 2048 387 / 317; 128 entries of 256 queries 176 / 73; 4096 queries, window 1024 57 / 46.  Few or uneven items lose: 12
// heads of 1024 queries, window 256 12.6 / 15.8; 24 of 64 with 121 queries 7.8 / 8.7; 24 with 768 over 132 keys 12 / 17; 8 heads of 2305, window 2048 32 / 46; 4 heads of 8192 121 / 134; 8 of 64 with 777 queries
// over 2777 keys 28 / 30.  What a launch would not meet (sequences packed into its entry) is not looked at.
static bool swa_takes_pairs(int64_t b, int64_t l, int64_t lk, int64_t heads, int64_t d, int64_t window, bool may_cut, SwaPairSplit* pairs) {
  *pairs = swa_pair_split(b, l, lk, heads, d, window, may_cut);
  return pairs->us < swa_split(b, l, lk, heads, d, window, may_cut).us;
}

int lact_swa_fwd_split_bytes(int64_t b, int64_t l, int64_t lk, int64_t n_heads, int64_t d, int64_t window, size_t* bytes,
                             int64_t* counters) {
  if (!bytes || !counters) return LACT_ERR_NULL;
  if ((d != 64 && d != 128) || b < 1 || l < 1 || n_heads < 1 || b > 65535 || n_heads > 65535 || l > (1ll << 30) || lk > (1ll << 30))
    return LACT_ERR_SHAPE;
  SwaPairSplit pairs;
  if (swa_takes_pairs(b, l, lk, n_heads, d, window, true, &pairs)) {
    *counters = 0;
    *bytes = swa_pair_scratch(pairs, d);
    return LACT_OK;
  }
  const SwaSplit sp = swa_split(b, l, lk, n_heads, d, window, true);
  *counters = sp.splits > 1 ? b * n_heads * ceil_div(l, 128) - sp.whole : 0;
  *bytes = static_cast<size_t>(*counters) * sp.splits * (128 * d * sizeof(float) + 256 * sizeof(float2));
  return LACT_OK;
}

int lact_swa_fwd(const void* q, const void* k, const void* v, void* o, int64_t b, int64_t l, int64_t lk, int64_t n_heads,
                 int64_t d, int64_t q_ts, int64_t q_bs, int64_t k_ts, int64_t k_bs, int64_t v_ts, int64_t v_bs, int64_t o_ts,
                 int64_t o_bs, int64_t window, float softmax_scale, const int32_t* seq_start, void* lse, int32_t* status_word,
                 void* stream) {
  return lact_swa_fwd_split(q, k, v, o, b, l, lk, n_heads, d, q_ts, q_bs, k_ts, k_bs, v_ts, v_bs, o_ts, o_bs, window, softmax_scale,
                            seq_start, lse, nullptr, nullptr, 0, status_word, stream);
}

// Keys of two runs as the kernel counts them: the second begins at the next whole tile.
static int64_t swa_two_runs(int64_t lk1, int64_t lk2) { return static_cast<int64_t>(ceil_div(lk1, 128)) * 128 + lk2; }

// A second run of keys and values (block attention), or k = nullptr.
struct SwaSecond {
  const void *k, *v;
  int64_t lk, k_ts, k_bs, v_ts, v_bs;
};
static int swa_fwd_impl(const void* q, const void* k, const void* v, const SwaSecond& two, void* o, int64_t b, int64_t l, int64_t lk,
                        int64_t n_heads, int64_t d, int64_t q_ts, int64_t q_bs, int64_t k_ts, int64_t k_bs, int64_t v_ts,
                        int64_t v_bs, int64_t o_ts, int64_t o_bs, int64_t window, float softmax_scale, const int32_t* seq_start,
                        void* lse, void* counters, void* scratch, size_t scratch_bytes, int32_t* status_word, void* stream) {
  if (!q || !k || !v || !o || !status_word) return LACT_ERR_NULL;
  if (seq_start != nullptr && b != 1) return LACT_ERR_CONFIG;   // packed sequences live in one batch entry
  const bool causal = window >= 0;
  if (lk <= 0) lk = l;
  if (causal ? lk != l : seq_start != nullptr) return LACT_ERR_CONFIG;   // causal: keys = queries; block: no packing
  LACT_TRY(check_device());
  if (d != 64 && d != 128) return LACT_ERR_SHAPE;
  if (b < 1 || l < 1 || n_heads < 1 || b > 65535 || n_heads > 65535 || l > (1ll << 30) || lk > (1ll << 30)) return LACT_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(o) & 15) != 0 || o_ts < n_heads * d || (o_ts % 8) != 0 || (o_bs % 8) != 0)
    return LACT_ERR_SHAPE;
  if (!(softmax_scale > 0.f)) return LACT_ERR_CONFIG;
  SwaArgs a;
  std::memset(&a, 0, sizeof(a));
  LACT_TRY(encode_map_heads(&a.q, q, b, l, n_heads, d, q_ts, q_bs));
  LACT_TRY(encode_map_heads(&a.k, k, b, lk, n_heads, d, k_ts, k_bs));
  LACT_TRY(encode_map_heads(&a.v, v, b, lk, n_heads, d, v_ts, v_bs));
  if (two.k != nullptr) {
    LACT_TRY(encode_map_heads(&a.k2, two.k, b, two.lk, n_heads, d, two.k_ts, two.k_bs));
    LACT_TRY(encode_map_heads(&a.v2, two.v, b, two.lk, n_heads, d, two.v_ts, two.v_bs));
    a.Lk1 = static_cast<int32_t>(lk);
    lk = swa_two_runs(lk, two.lk);
  }
  a.Lk = static_cast<int32_t>(lk);
  a.causal = causal ? 1 : 0;
  a.o = static_cast<bf16*>(o);
  a.o_bs = o_bs; a.o_ts = o_ts; a.o_hs = d;
  a.L = static_cast<int32_t>(l);
  a.window = window > 0 && window < l ? static_cast<int32_t>(window) : 0;
  a.heads = static_cast<int32_t>(n_heads);
  a.q_tiles = ceil_div(l, 128);
  a.scale_log2 = softmax_scale * 1.4426950408889634f;
  a.lse = static_cast<float*>(lse);
  a.seq_start = seq_start;
  a.status = status_word;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int64_t ctas = b * n_heads * a.q_tiles;
  if (ctas > 0x7FFFFFFFll) return LACT_ERR_SHAPE;
  SwaPairSplit sp2;
  if (swa_takes_pairs(b, l, lk, n_heads, d, window, scratch != nullptr && counters != nullptr, &sp2)) {
    SwaPairArgs p;
    std::memset(&p, 0, sizeof(p));
    p.q = a.q; p.k = a.k; p.v = a.v; p.k2 = a.k2; p.v2 = a.v2;
    p.o = a.o; p.o_bs = a.o_bs; p.o_ts = a.o_ts; p.o_hs = a.o_hs;
    p.L = a.L; p.window = a.window; p.Lk = a.Lk; p.causal = a.causal; p.Lk1 = a.Lk1;
    p.heads = a.heads;
    p.entries = static_cast<int32_t>(b);
    p.pairs = ceil_div(l, 256);
    p.scale_log2 = a.scale_log2; p.seq_start = a.seq_start; p.lse = a.lse; p.status = a.status;
    p.whole = static_cast<int32_t>(sp2.whole);
    if (sp2.cutters > 0) {
      if (scratch_bytes < swa_pair_scratch(sp2, d) || (reinterpret_cast<uintptr_t>(scratch) & 15) != 0) return LACT_ERR_WORKSPACE;
      p.rest = static_cast<int32_t>(sp2.rest);
      p.cutters = static_cast<int32_t>(sp2.cutters);
      p.span = static_cast<int32_t>(sp2.span);
      p.share = static_cast<int32_t>(sp2.rest * sp2.span / sp2.cutters);
      p.longer = static_cast<int32_t>(sp2.rest * sp2.span % sp2.cutters);
      p.part = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(scratch) + 31) & ~static_cast<uintptr_t>(31));
      p.ml = reinterpret_cast<float2*>(p.part + (sp2.cutters + sp2.rest) * 256 * d);
    }
    ctas = std::max<int64_t>(p.cutters, std::min<int64_t>(p.whole, sm_count()));
    p.rounds = ceil_div(p.whole, ctas);
    return d == 64 ? launch_swa_pairs<64>(p, ctas, st) : launch_swa_pairs<128>(p, ctas, st);
  }
  a.whole = static_cast<int32_t>(ctas);
  a.splits = 1;
  if (scratch != nullptr && counters != nullptr) {
    const SwaSplit sp = swa_split(b, l, lk, n_heads, d, window, true);
    const int64_t rest = ctas - sp.whole;
    const size_t rows = static_cast<size_t>(rest) * sp.splits;
    if (sp.splits > 1) {
      if (scratch_bytes < rows * (128 * d * sizeof(float) + 256 * sizeof(float2)) || (reinterpret_cast<uintptr_t>(scratch) & 15) != 0)
        return LACT_ERR_WORKSPACE;
      a.whole = static_cast<int32_t>(sp.whole);
      a.splits = sp.splits;
      a.part = static_cast<float4*>(scratch);
      a.ml = reinterpret_cast<float2*>(static_cast<uint8_t*>(scratch) + rows * 128 * d * sizeof(float));
      a.count = static_cast<uint32_t*>(counters);
      ctas = sp.whole + rest * sp.splits;
    }
  }
  return d == 64 ? launch_swa<64>(a, ctas, st) : launch_swa<128>(a, ctas, st);
}

int lact_swa_fwd_split(const void* q, const void* k, const void* v, void* o, int64_t b, int64_t l, int64_t lk, int64_t n_heads,
                       int64_t d, int64_t q_ts, int64_t q_bs, int64_t k_ts, int64_t k_bs, int64_t v_ts, int64_t v_bs, int64_t o_ts,
                       int64_t o_bs, int64_t window, float softmax_scale, const int32_t* seq_start, void* lse, void* counters,
                       void* scratch, size_t scratch_bytes, int32_t* status_word, void* stream) {
  return swa_fwd_impl(q, k, v, SwaSecond{}, o, b, l, lk, n_heads, d, q_ts, q_bs, k_ts, k_bs, v_ts, v_bs, o_ts, o_bs, window,
                      softmax_scale, seq_start, lse, counters, scratch, scratch_bytes, status_word, stream);
}

int lact_swa_fwd_cache_bytes(int64_t b, int64_t l, int64_t l_cache, int64_t l_new, int64_t n_heads, int64_t d, size_t* bytes,
                             int64_t* counters) {
  if (l_cache < 1 || l_new < 1 || l_cache > (1ll << 29) || l_new > (1ll << 29)) return LACT_ERR_SHAPE;
  return lact_swa_fwd_split_bytes(b, l, swa_two_runs(l_cache, l_new), n_heads, d, -1, bytes, counters);
}

int lact_swa_fwd_cache(const void* q, const void* k_cache, const void* v_cache, const void* k, const void* v, void* o, int64_t b,
                       int64_t l, int64_t l_cache, int64_t l_new, int64_t n_heads, int64_t d, const int64_t* strides,
                       float softmax_scale, void* counters, void* scratch, size_t scratch_bytes, int32_t* status_word, void* stream) {
  if (!k || !v || !strides) return LACT_ERR_NULL;
  if (l_cache < 1 || l_new < 1 || l_cache > (1ll << 29) || l_new > (1ll << 29)) return LACT_ERR_SHAPE;
  const int64_t* s = strides;
  return swa_fwd_impl(q, k_cache, v_cache, SwaSecond{k, v, l_new, s[6], s[7], s[8], s[9]}, o, b, l, l_cache, n_heads, d, s[0], s[1], s[2],
                      s[3], s[4], s[5], s[10], s[11], -1, softmax_scale, nullptr, nullptr, counters, scratch, scratch_bytes, status_word,
                      stream);
}

int lact_swa_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout, const void* lse, void* dq,
                 void* dk, void* dv, void* delta, int64_t b, int64_t l, int64_t lk, int64_t n_heads, int64_t d, int64_t q_ts,
                 int64_t q_bs, int64_t k_ts, int64_t k_bs, int64_t v_ts, int64_t v_bs, int64_t o_ts, int64_t o_bs,
                 int64_t do_ts, int64_t do_bs, int64_t window, float softmax_scale, const int32_t* seq_start,
                 int32_t* status_word, void* stream) {
  if (!q || !k || !v || !o || !dout || !lse || !dq || !dk || !dv || !delta || !status_word) return LACT_ERR_NULL;
  if (seq_start != nullptr && b != 1) return LACT_ERR_CONFIG;
  const bool causal = window >= 0;
  if (lk <= 0) lk = l;
  if (causal ? lk != l : seq_start != nullptr) return LACT_ERR_CONFIG;
  LACT_TRY(check_device());
  if (d != 64 && d != 128) return LACT_ERR_SHAPE;
  if (b < 1 || l < 1 || n_heads < 1 || b > 65535 || n_heads > 65535 || l > (1ll << 30) || lk > (1ll << 30)) return LACT_ERR_SHAPE;
  if (!(softmax_scale > 0.f)) return LACT_ERR_CONFIG;
  for (const void* p : {static_cast<const void*>(dq), static_cast<const void*>(dk), static_cast<const void*>(dv), o, dout})
    if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return LACT_ERR_SHAPE;
  if (o_ts < n_heads * d || do_ts < n_heads * d || (o_ts % 8) || (o_bs % 8) || (do_ts % 8) || (do_bs % 8)) return LACT_ERR_SHAPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  {
    SwaDeltaArgs da;
    std::memset(&da, 0, sizeof(da));
    da.o = static_cast<const bf16*>(o);
    da.dout = static_cast<const bf16*>(dout);
    da.o_ts = o_ts; da.o_bs = o_bs; da.d_ts = do_ts; da.d_bs = do_bs;
    da.delta = static_cast<float*>(delta);
    da.b = static_cast<int32_t>(b); da.L = static_cast<int32_t>(l);
    da.heads = static_cast<int32_t>(n_heads); da.d = static_cast<int32_t>(d);
    const int64_t rows = l * n_heads;
    KernelScope scope(kClsOther, st);
    if (d == 64) swa_delta_rows_kernel<4><<<dim3(ceil_div(rows, 64), static_cast<unsigned>(b)), 256, 0, st>>>(da);
    else swa_delta_rows_kernel<8><<<dim3(ceil_div(rows, 32), static_cast<unsigned>(b)), 256, 0, st>>>(da);
    LACT_CUDA(cudaGetLastError());
  }
  SwaBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  LACT_TRY(encode_map_heads(&a.q, q, b, l, n_heads, d, q_ts, q_bs));
  LACT_TRY(encode_map_heads(&a.k, k, b, lk, n_heads, d, k_ts, k_bs));
  LACT_TRY(encode_map_heads(&a.v, v, b, lk, n_heads, d, v_ts, v_bs));
  LACT_TRY(encode_map_heads(&a.dout, dout, b, l, n_heads, d, do_ts, do_bs));
  LACT_TRY(encode_map_heads(&a.q16, q, b, l, n_heads, d, q_ts, q_bs, 16));
  LACT_TRY(encode_map_heads(&a.k16, k, b, lk, n_heads, d, k_ts, k_bs, 16));
  LACT_TRY(encode_map_heads(&a.v16, v, b, lk, n_heads, d, v_ts, v_bs, 16));
  LACT_TRY(encode_map_heads(&a.dout16, dout, b, l, n_heads, d, do_ts, do_bs, 16));
  a.lse = static_cast<const float*>(lse);
  a.delta = static_cast<const float*>(delta);
  a.seq_start = seq_start;
  a.o_ts = n_heads * d; a.o_hs = d;   // gradients are written contiguous [b][l or lk][h][d]
  a.L = static_cast<int32_t>(l);
  a.Lk = static_cast<int32_t>(lk);
  a.causal = causal ? 1 : 0;
  a.window = window > 0 && window < l ? static_cast<int32_t>(window) : 0;
  a.heads = static_cast<int32_t>(n_heads);
  a.scale_log2 = softmax_scale * 1.4426950408889634f;
  a.scale = softmax_scale;
  a.status = status_word;
  const int64_t k_tiles = ceil_div(lk, 128), q_tiles = ceil_div(l, 128);
  if (b * n_heads * std::max(k_tiles, q_tiles) > 0x7FFFFFFFll) return LACT_ERR_SHAPE;
  // keys' side (dK, dV): one CTA per key tile; then queries' side (dQ): one CTA per query tile
  a.out0 = static_cast<bf16*>(dk);
  a.out1 = static_cast<bf16*>(dv);
  a.tiles = static_cast<int32_t>(k_tiles);
  a.o_bs = lk * n_heads * d;
  LACT_TRY((d == 64 ? launch_swa_bwd<64, 0>(a, b * n_heads * k_tiles, st) : launch_swa_bwd<128, 0>(a, b * n_heads * k_tiles, st)));
  a.out0 = static_cast<bf16*>(dq);
  a.out1 = nullptr;
  a.tiles = static_cast<int32_t>(q_tiles);
  a.o_bs = l * n_heads * d;
  const int64_t ctas = b * n_heads * q_tiles;
  return d == 64 ? launch_swa_bwd<64, 1>(a, ctas, st) : launch_swa_bwd<128, 1>(a, ctas, st);
}

int lact_l2_norm_add(const void* x, int32_t x_dtype, const void* x_add, int32_t add_dtype, const void* scale, void* y,
                     int32_t y_dtype, int64_t B, int64_t T, int64_t D, float eps, void* stream) {
  if (!x || !x_add || !scale || !y) return LACT_ERR_NULL;
  if (B < 1 || T < 1 || D < 1) return LACT_ERR_SHAPE;
  const int64_t rows = B * T;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  l2_norm_add_kernel<<<ceil_div(rows, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      x, x_dtype == LACT_F32, x_add, add_dtype == LACT_F32, static_cast<const float*>(scale), y, y_dtype == LACT_F32,
      rows, static_cast<int>(D), eps);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_prenorm_momentum_l2norm(const void* x, const void* dx, const void* m, const void* mu, const void* scale,
                                 void* x_out, void* m_out, void* y_out, int64_t B, int64_t T, int64_t D, float eps,
                                 void* stream) {
  if (!x || !dx || !m || !mu || !scale || !x_out || !m_out || !y_out) return LACT_ERR_NULL;
  if (B < 1 || T < 1 || D < 1) return LACT_ERR_SHAPE;
  const int64_t rows = B * T;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  prenorm_momentum_kernel<<<ceil_div(rows, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(x), static_cast<const bf16*>(dx), static_cast<const float*>(m),
      static_cast<const float*>(mu), static_cast<const float*>(scale), static_cast<float*>(x_out),
      static_cast<float*>(m_out), static_cast<bf16*>(y_out), rows, static_cast<int>(T), static_cast<int>(D), eps);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

// One or two independent problems c (+)= alpha (a0 b0^T [+ a1 b1^T]) in one persistent launch (both single-product
// or both two-product; one tile width for the launch).
static int group_bt(const lact_bmm_desc* d, int n) {
  const lact_bmm_desc& l = d[n - 1];
  const int bt = choose_bt({{d[0].N, d[0].M * d[0].batch}, {l.N, n > 1 ? l.M * l.batch : 0}});
  return d[0].a1 != nullptr ? std::min(bt, 192) : bt;
}
// Split of a group whose problems are one long contraction each (single products of one K), else one unit per tile.
static Split group_split(const lact_bmm_desc* d, int n) {
  for (int p = 0; p < n; ++p)
    if (d[p].a1 != nullptr || d[p].K != d[0].K) return Split{1, 0};
  return choose_split(ceil_div(d[0].K, kBK));
}

static int bmm_group(const lact_bmm_desc* d, int n, int32_t* status_word, void* stream, float alpha,
                     const SplitScratch& scratch = SplitScratch{}) {
  if (!d || !status_word) return LACT_ERR_NULL;
  if (n < 1 || n > 2) return LACT_ERR_CONFIG;
  LACT_TRY(check_device());
  const bool two = d[0].a1 != nullptr;
  for (int p = 0; p < n; ++p) {
    const lact_bmm_desc& q = d[p];
    if (!q.a0 || !q.b0 || !q.c || ((q.a1 == nullptr) != (q.b1 == nullptr))) return LACT_ERR_NULL;
    if ((q.a1 != nullptr) != two) return LACT_ERR_CONFIG;
    if (q.batch < 1 || q.batch > 65535 || q.M < 1 || q.N < 8 || q.K < 1 || (q.N % 8)) return LACT_ERR_SHAPE;
    // the contiguous axis of every operand must be a multiple of 8 elements (16-byte TMA strides)
    if (((q.a0_mn || (q.a1 && q.a1_mn)) && (q.M % 8)) ||
        ((!q.a0_mn || (q.a1 && !q.a1_mn) || !q.b0_mn || (q.b1 && !q.b1_mn)) && (q.K % 8)))
      return LACT_ERR_SHAPE;
    if (q.accumulate && q.c_dtype != LACT_F32) return LACT_ERR_DTYPE;
    // c is written in 16-byte (fp32) / 8-byte (bf16) units
    if ((reinterpret_cast<uintptr_t>(q.c) & 15) != 0 || q.c_ld < q.N || (q.c_ld % 8) != 0 ||
        (q.batch > 1 && (q.c_bs % 8) != 0))
      return LACT_ERR_SHAPE;
    auto bad = [&](int mn, int64_t rows, int64_t ld) { return ld < (mn ? rows : q.K); };
    if (bad(q.a0_mn, q.M, q.a0_ld) || bad(q.b0_mn, q.N, q.b0_ld) ||
        (q.a1 && (bad(q.a1_mn, q.M, q.a1_ld) || bad(q.b1_mn, q.N, q.b1_ld))))
      return LACT_ERR_SHAPE;
  }
  // operand as a matrix of `rows` = M or N: [rows][K] with row stride ld, or (MN-major) [K][rows]
  auto mat = [](const lact_bmm_desc& q, const void* ptr, int mn, int64_t rows, int64_t ld, int64_t bs) {
    return mn ? Mat{ptr, q.K, rows, ld, q.batch, bs} : Mat{ptr, rows, q.K, ld, q.batch, bs};
  };
  const int bt = group_bt(d, n);
  const Split split = scratch.part != nullptr ? group_split(d, n) : Split{1, 0};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto fill = [&](auto& g, int btv) -> int {
    for (int p = 0; p < n; ++p) {
      const lact_bmm_desc& q = d[p];
      auto& P = g.prob[p];
      LACT_TRY(make_operand(form_of(P), &P.a[0], &P.ai[0], mat(q, q.a0, q.a0_mn, q.M, q.a0_ld, q.a0_bs), q.a0_mn, kBM, 0, 0));
      LACT_TRY(make_operand(form_of(P), &P.b[0], &P.bi[0], mat(q, q.b0, q.b0_mn, q.N, q.b0_ld, q.b0_bs), q.b0_mn, btv, 0, 0));
      if constexpr (std::remove_reference_t<decltype(g)>::OpType::NA == 2) {
        LACT_TRY(make_operand(form_of(P), &P.a[1], &P.ai[1], mat(q, q.a1, q.a1_mn, q.M, q.a1_ld, q.a1_bs), q.a1_mn, kBM, 0, 0));
        LACT_TRY(make_operand(form_of(P), &P.b[1], &P.bi[1], mat(q, q.b1, q.b1_mn, q.N, q.b1_ld, q.b1_bs), q.b1_mn, btv, 0, 0));
      }
      P.M = static_cast<int>(q.M); P.N = static_cast<int>(q.N); P.K = static_cast<int>(q.K);
      P.batch = static_cast<int>(q.batch);
      P.ep = EpiStore{q.c, q.c_bs, q.c_ld, 0, q.c_dtype == LACT_F32, q.accumulate, alpha};
      set_split(P, split, scratch);
    }
    g.status = status_word;
    return LACT_OK;
  };
  if (n == 1) return two ? launch_op<OpStore2T, 1>(bt, fill, s, kClsOther, 1) : launch_op<OpStoreDirectT, 1>(bt, fill, s, kClsOther, 1);
  return two ? launch_op<OpStore2T, 2>(bt, fill, s, kClsOther, 2) : launch_op<OpStoreDirectT, 2>(bt, fill, s, kClsOther, 2);
}

int lact_bmm_group_split_bytes(const lact_bmm_desc* problems, int32_t n, size_t* bytes, int64_t* counters) {
  if (!problems || !bytes || !counters) return LACT_ERR_NULL;
  if (n < 1 || n > 2) return LACT_ERR_CONFIG;
  *bytes = 0;
  *counters = 0;
  for (int p = 0; p < n; ++p)
    if (problems[p].batch < 1 || problems[p].M < 1 || problems[p].N < 1 || problems[p].K < 1) return LACT_ERR_SHAPE;
  const int splits = group_split(problems, n).splits, bt = group_bt(problems, n);
  if (splits == 1) return LACT_OK;
  for (int p = 0; p < n; ++p) *counters += output_tiles(problems[p].M, problems[p].N, problems[p].batch, bt);
  *bytes = static_cast<size_t>(*counters) * splits * kBM * bt * sizeof(float);
  return LACT_OK;
}

int lact_bmm_group_split_bf16(const lact_bmm_desc* problems, int32_t n, void* counters, void* scratch, size_t scratch_bytes,
                              int32_t* status_word, void* stream) {
  size_t need = 0;
  int64_t words = 0;
  LACT_TRY(lact_bmm_group_split_bytes(problems, n, &need, &words));
  SplitScratch ws;
  if (need > 0) {
    if (!counters || !scratch) return LACT_ERR_NULL;
    if (scratch_bytes < need || (reinterpret_cast<uintptr_t>(scratch) & 15) != 0) return LACT_ERR_WORKSPACE;
    ws = SplitScratch{static_cast<float*>(scratch), static_cast<uint32_t*>(counters)};
  }
  return bmm_group(problems, n, status_word, stream, 1.0f, ws);
}

int lact_bmm_group_bf16(const lact_bmm_desc* problems, int32_t n, int32_t* status_word, void* stream) {
  return bmm_group(problems, n, status_word, stream, 1.0f);
}

static int bmm2_strided(const void* a0, int32_t a0_mn, int64_t a0_ld, int64_t a0_bs, const void* b0, int32_t b0_mn,
                        int64_t b0_ld, int64_t b0_bs, const void* a1, int32_t a1_mn, int64_t a1_ld, int64_t a1_bs,
                        const void* b1, int32_t b1_mn, int64_t b1_ld, int64_t b1_bs, void* c, int32_t c_dtype,
                        int64_t c_ld, int64_t c_bs, int32_t accumulate, int64_t batch, int64_t M, int64_t N, int64_t K,
                        int32_t* status_word, void* stream, float alpha) {
  if (!a0 || !b0 || !c) return LACT_ERR_NULL;
  lact_bmm_desc q;
  std::memset(&q, 0, sizeof(q));
  q.a0 = a0; q.b0 = b0; q.a1 = a1; q.b1 = b1; q.c = c;
  q.a0_ld = a0_ld; q.a0_bs = a0_bs; q.b0_ld = b0_ld; q.b0_bs = b0_bs;
  q.a1_ld = a1_ld; q.a1_bs = a1_bs; q.b1_ld = b1_ld; q.b1_bs = b1_bs;
  q.c_ld = c_ld; q.c_bs = c_bs;
  q.batch = batch; q.M = M; q.N = N; q.K = K;
  q.a0_mn = a0_mn; q.b0_mn = b0_mn; q.a1_mn = a1_mn; q.b1_mn = b1_mn;
  q.c_dtype = c_dtype; q.accumulate = accumulate;
  return bmm_group(&q, 1, status_word, stream, alpha);
}

// Pointwise stage of the fast-weight gradient on its own (see lact_fw_grad): also the backward of apply's
// pre-activations with (k, v) = (q, dO) and unit learning rates.
int lact_fw_grad_pointwise(const void* w0w2, const void* w1, const void* k, int64_t k_ts, int64_t k_bs, const void* v,
                           int64_t v_ts, int64_t v_bs, const void* lr0, const void* lr1, const void* lr2, int32_t lr_dtype,
                           int64_t lr_bs, float w_scale, void* dy02, void* hid, int64_t B, int64_t N, int64_t D, int64_t H,
                           int32_t* status_word, void* stream) {
  if (!w0w2 || !w1 || !k || !v || !dy02 || !hid || !status_word) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  if (B < 1 || B > 65535 || N < 1 || D < 8 || H < 8 || (D % 8) || (H % 8)) return LACT_ERR_SHAPE;
  if (k_ts < D || v_ts < D || (k_ts % 8) || (v_ts % 8) || (k_bs % 8) || (v_bs % 8)) return LACT_ERR_SHAPE;
  if (lr_dtype != LACT_F32 && lr_dtype != LACT_BF16) return LACT_ERR_DTYPE;
  GradArgs a{};
  a.w02b = static_cast<const bf16*>(w0w2);
  a.w1b = static_cast<const bf16*>(w1);
  a.k = k; a.v = v;
  a.k_ts = k_ts; a.k_bs = k_bs; a.v_ts = v_ts; a.v_bs = v_bs;
  a.start = 0; a.end = N;
  a.lr0 = lr0; a.lr1 = lr1; a.lr2 = lr2;
  a.lr_f32 = lr_dtype == LACT_F32;
  a.lr_bs = lr_bs;
  a.w_scale = w_scale;
  a.dy02 = static_cast<bf16*>(dy02);
  a.hid = static_cast<bf16*>(hid);
  a.B = B; a.D = D; a.H = H;
  return run_grad_pointwise(a, status_word, static_cast<cudaStream_t>(stream));
}

int lact_bmm2_strided_bf16(const void* a0, int32_t a0_mn, int64_t a0_ld, int64_t a0_bs, const void* b0, int32_t b0_mn,
                           int64_t b0_ld, int64_t b0_bs, const void* a1, int32_t a1_mn, int64_t a1_ld, int64_t a1_bs,
                           const void* b1, int32_t b1_mn, int64_t b1_ld, int64_t b1_bs, void* c, int32_t c_dtype,
                           int64_t c_ld, int64_t c_bs, int32_t accumulate, int64_t batch, int64_t M, int64_t N, int64_t K,
                           int32_t* status_word, void* stream) {
  return bmm2_strided(a0, a0_mn, a0_ld, a0_bs, b0, b0_mn, b0_ld, b0_bs, a1, a1_mn, a1_ld, a1_bs, b1, b1_mn, b1_ld, b1_bs, c,
                      c_dtype, c_ld, c_bs, accumulate, batch, M, N, K, status_word, stream, 1.0f);
}

// contiguous two-product with the accumulator scaled by alpha before the store (internal)
static int bmm2_scaled(const void* a0, int32_t a0_mn, const void* b0, int32_t b0_mn, const void* a1, int32_t a1_mn,
                       const void* b1, int32_t b1_mn, void* c, int32_t c_dtype, int64_t batch, int64_t M, int64_t N,
                       int64_t K, int32_t* status_word, void* stream, float alpha) {
  auto ld = [&](int mn, int64_t rows) { return mn ? rows : K; };
  return bmm2_strided(a0, a0_mn, ld(a0_mn, M), M * K, b0, b0_mn, ld(b0_mn, N), N * K, a1, a1_mn, ld(a1_mn, M), M * K, b1,
                      b1_mn, ld(b1_mn, N), N * K, c, c_dtype, N, M * N, 0, batch, M, N, K, status_word, stream, alpha);
}

int lact_bmm2_bf16(const void* a0, int32_t a0_mn, const void* b0, int32_t b0_mn, const void* a1, int32_t a1_mn,
                   const void* b1, int32_t b1_mn, void* c, int32_t c_dtype, int32_t accumulate, int64_t batch,
                   int64_t M, int64_t N, int64_t K, int32_t* status_word, void* stream) {
  // contiguous operands: [batch][rows][K] or (MN-major) [batch][K][rows]
  auto ld = [&](int mn, int64_t rows) { return mn ? rows : K; };
  return lact_bmm2_strided_bf16(a0, a0_mn, ld(a0_mn, M), M * K, b0, b0_mn, ld(b0_mn, N), N * K, a1, a1_mn, ld(a1_mn, M),
                                M * K, b1, b1_mn, ld(b1_mn, N), N * K, c, c_dtype, N, M * N, accumulate, batch, M, N, K,
                                status_word, stream);
}

static PlaneArgs make_plane_args(const void* y02, const void* dh, const void* g_dy02, const void* g_hid,
                                 const void* lr0, const void* lr1, const void* lr2, int32_t lr_dtype, float w_scale,
                                 void* dy02, void* hid, void* g_y02, void* g_dh, void* g_lr0, void* g_lr1, void* g_lr2,
                                 int64_t rows, int64_t H) {
  PlaneArgs a;
  std::memset(&a, 0, sizeof(a));
  a.y02 = static_cast<const bf16*>(y02); a.dh = static_cast<const bf16*>(dh);
  a.g_dy02 = static_cast<const bf16*>(g_dy02); a.g_hid = static_cast<const bf16*>(g_hid);
  a.lr0 = lr0; a.lr1 = lr1; a.lr2 = lr2; a.lr_f32 = lr_dtype == LACT_F32; a.w_scale = w_scale;
  a.dy02 = static_cast<bf16*>(dy02); a.hid = static_cast<bf16*>(hid);
  a.g_y02 = static_cast<bf16*>(g_y02); a.g_dh = static_cast<bf16*>(g_dh);
  a.g_lr0 = static_cast<float*>(g_lr0); a.g_lr1 = static_cast<float*>(g_lr1); a.g_lr2 = static_cast<float*>(g_lr2);
  a.rows = rows; a.H = static_cast<int32_t>(H);
  return a;
}

int lact_swiglu_bwd_planes(const void* y02, const void* dh, const void* lr0, const void* lr1, const void* lr2,
                           int32_t lr_dtype, float w_scale, void* dy02, void* hid, int64_t rows, int64_t H,
                           void* stream) {
  if (!y02 || !dh || !dy02 || !hid) return LACT_ERR_NULL;
  if (rows < 1 || H < 8 || (H % 8) != 0) return LACT_ERR_SHAPE;  // planes move as 16-byte vectors
  const PlaneArgs a = make_plane_args(y02, dh, nullptr, nullptr, lr0, lr1, lr2, lr_dtype, w_scale, dy02, hid, nullptr,
                                      nullptr, nullptr, nullptr, nullptr, rows, H);
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  swiglu_bwd_planes_kernel<<<ceil_div(rows, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_fw_grad_bwd_pointwise(const void* y02, const void* dh, const void* g_dy02, const void* g_hid, const void* lr0,
                               const void* lr1, const void* lr2, int32_t lr_dtype, float w_scale, void* g_y02,
                               void* g_dh, void* dy02, void* hid, void* g_lr0, void* g_lr1, void* g_lr2, int64_t B,
                               int64_t n, int64_t H, int64_t lr_bs, int64_t g_lr_bs, int32_t g_lr_add, void* stream) {
  if (!y02 || !dh || !g_dy02 || !g_hid || !lr0 || !lr1 || !lr2 || !g_y02 || !g_dh || !dy02 || !hid || !g_lr0 ||
      !g_lr1 || !g_lr2)
    return LACT_ERR_NULL;
  if (B < 1 || B > 65535 || n < 1 || H < 8 || (H % 8) != 0) return LACT_ERR_SHAPE;  // planes move as 16-byte vectors
  const int64_t rows = B * n;
  PlaneArgs a = make_plane_args(y02, dh, g_dy02, g_hid, lr0, lr1, lr2, lr_dtype, w_scale, dy02, hid, g_y02, g_dh,
                                g_lr0, g_lr1, g_lr2, rows, H);
  a.n = n; a.lr_bs = lr_bs; a.g_lr_bs = g_lr_bs; a.g_lr_add = g_lr_add;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  // lanes per token: the most that divide its units, or a warp where eight do not
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto grid = [&](int lanes) { return dim3(ceil_div(n, 256 / lanes), static_cast<unsigned>(B)); };
  if (H % 256 != 0 && H % 128 == 0) fw_grad_bwd_pointwise_kernel<16><<<grid(16), 256, 0, st>>>(a);
  else if (H % 256 != 0 && H % 64 == 0) fw_grad_bwd_pointwise_kernel<8><<<grid(8), 256, 0, st>>>(a);
  else fw_grad_bwd_pointwise_kernel<32><<<grid(32), 256, 0, st>>>(a);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_renorm_bwd(const void* base, const void* upd, int32_t upd_dtype, const void* n0, const void* dy, void* dw,
                    void* dw_bf16, void* dn0, int64_t rows, int64_t C, int32_t mode, void* stream) {
  if (!base || !upd || !n0 || !dy || !dw) return LACT_ERR_NULL;
  if (rows < 1 || C < 1 || mode < 0 || mode > 2) return LACT_ERR_SHAPE;
  RenormBwdArgs a{static_cast<const float*>(base), upd, upd_dtype == LACT_F32, static_cast<const float*>(n0),
                  static_cast<const float*>(dy), static_cast<float*>(dw), static_cast<bf16*>(dw_bf16),
                  static_cast<float*>(dn0), rows, static_cast<int32_t>(C), mode};
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  renorm_bwd_kernel<<<ceil_div(rows, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_ns_norm_bwd(const void* g, void* dx0, void* partials, int64_t nmat, int64_t elems_per_matrix, void* stream) {
  if (!g || !dx0 || !partials) return LACT_ERR_NULL;
  return ns_norm_bwd_launch(static_cast<const float*>(g), dx0, 0, static_cast<float*>(dx0), static_cast<float*>(partials),
                            nmat, elems_per_matrix, static_cast<cudaStream_t>(stream));
}

int lact_ns_trace_bwd_fused(const lact_ns_bwd_group* groups, int32_t ngroups, int32_t steps, int32_t const_coeffs,
                            int32_t gram_right, int32_t* status_word, void* stream) {
  if (!groups || !status_word) return LACT_ERR_NULL;
  if (ngroups < 1 || ngroups > 2 || steps < 1 || steps > 5) return LACT_ERR_CONFIG;
  LACT_TRY(check_device());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  NsTrace tr[2];
  NsGroup grp[2];
  const bf16* du[2] = {nullptr, nullptr};
  for (int g = 0; g < ngroups; ++g) {
    const lact_ns_bwd_group& G = groups[g];
    if (!G.du || !G.g || !G.dg || !G.trace || !G.partials) return LACT_ERR_NULL;
    LACT_TRY(plan_ns_trace(G.trace, G.nmat, G.rows, G.cols, steps, gram_right, &tr[g]));
    if (tr[g].bytes > G.trace_bytes) return LACT_ERR_WORKSPACE;
    grp[g] = tr[g].grp;
    du[g] = static_cast<const bf16*>(G.du);
  }
  // Tile width (one for all phases).  Among the widths that give the m x m phases enough tiles to occupy most SMs,
  // the one with the least padded work (wider on a tie); with few matrices the kernel is bound by each matrix's
  // chain of phases, so the width with the most tiles (again wider on a tie).
  auto mm_tiles = [&](int bt) {
    int64_t t = 0;
    for (int g = 0; g < ngroups; ++g) t += static_cast<int64_t>(grp[g].nmat) * ceil_div(grp[g].m, kBM) * ceil_div(grp[g].m, bt);
    return t;
  };
  auto padded_work = [&](int bt) {
    int64_t w = 0;
    for (int g = 0; g < ngroups; ++g)
      w += static_cast<int64_t>(grp[g].nmat) * bt *
           (2 * ceil_div(grp[g].m, kBM) * ceil_div(grp[g].m, bt) * static_cast<int64_t>(grp[g].m + grp[g].n) / 2 +
            ceil_div(ns_upd_rows(grp[g]), kBM) * ceil_div(ns_upd_cols(grp[g]), bt) * static_cast<int64_t>(grp[g].m));
    return w;
  };
  const int64_t want = static_cast<int64_t>(sm_count()) * 3 / 4;
  int bt = 0;
  for (int cand : {192, 128, 64})
    if (mm_tiles(cand) >= want && (bt == 0 || padded_work(cand) < padded_work(bt))) bt = cand;
  if (bt == 0) bt = mm_tiles(64) > mm_tiles(128) ? 64 : (mm_tiles(128) > mm_tiles(192) ? 128 : 192);
  // Q and T are symmetric: with Gram sides that are multiples of 128 their phases run on the 128 x 128 tiles on and
  // above the diagonal only
  bool sym_ok = bt == 192;
  for (int g = 0; g < ngroups; ++g) sym_ok = sym_ok && grp[g].m % kBM == 0 && grp[g].m >= 2 * kBM;
  int rc = LACT_ERR_CONFIG;
  if (sym_ok) rc = launch_ns_bwd_fused<128, 192, true>(tr, du, ngroups, steps, const_coeffs, status_word, s);
  else if (bt == 192) rc = launch_ns_bwd_fused<192, 192, false>(tr, du, ngroups, steps, const_coeffs, status_word, s);
  else if (bt == 128) rc = launch_ns_bwd_fused<128, 128, false>(tr, du, ngroups, steps, const_coeffs, status_word, s);
  else rc = launch_ns_bwd_fused<64, 64, false>(tr, du, ngroups, steps, const_coeffs, status_word, s);
  if (rc != LACT_OK) return rc;
  // the gradient w.r.t. the first iterate is the bf16 buffer the last phase wrote; the Frobenius normalisation
  // X0 = bf16(G) / (||G|| + 1e-7) is differentiated into the caller's fp32 dG
  for (int g = 0; g < ngroups; ++g) {
    const lact_ns_bwd_group& G = groups[g];
    LACT_TRY(ns_norm_bwd_launch(static_cast<const float*>(G.g), tr[g].dXb, 1, static_cast<float*>(G.dg),
                                static_cast<float*>(G.partials), G.nmat, G.rows * G.cols, s));
  }
  return LACT_OK;
}

int lact_momentum_bwd_slices(void) { return kNormBwdSlices; }

int lact_momentum_bwd(const void* dg0, const void* dg1, void* carry0, void* carry1, const void* mprev0, const void* mprev1,
                      void* dgb0, void* dgb1, const void* beta, void* dbeta, int64_t B, int64_t n0, int64_t n1,
                      int32_t add_carry, void* stream) {
  if (!dg0 || !dg1 || !dgb0 || !dgb1) return LACT_ERR_NULL;
  if ((carry0 == nullptr) != (carry1 == nullptr) || (mprev0 == nullptr) != (mprev1 == nullptr)) return LACT_ERR_NULL;
  if (B < 1 || B > 65535 * 16 || n0 < 4 || n1 < 4 || (n0 % 4) != 0 || (n1 % 4) != 0) return LACT_ERR_SHAPE;
  MomentumBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  a.dg[0] = static_cast<const float*>(dg0); a.dg[1] = static_cast<const float*>(dg1);
  a.carry[0] = static_cast<float*>(carry0); a.carry[1] = static_cast<float*>(carry1);
  a.mprev[0] = static_cast<const float*>(mprev0); a.mprev[1] = static_cast<const float*>(mprev1);
  a.dgb[0] = static_cast<bf16*>(dgb0); a.dgb[1] = static_cast<bf16*>(dgb1);
  a.beta = static_cast<const float*>(beta);
  a.dbeta = static_cast<float*>(dbeta);
  a.n[0] = n0; a.n[1] = n1;
  a.add_carry = add_carry;
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  momentum_bwd_kernel<<<dim3(static_cast<unsigned>(B), kNormBwdSlices), 512, 0, static_cast<cudaStream_t>(stream)>>>(a);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_momentum_means(const void* momentum, int32_t dtype, int64_t B, int64_t L, int32_t n, const int64_t* start,
                        const int64_t* end, float* beta, void* stream) {
  if (!momentum || !beta || (n > 0 && (!start || !end))) return LACT_ERR_NULL;
  if (B < 1 || B > 65535 || L < 1 || n < 0) return LACT_ERR_SHAPE;
  for (int32_t i = 0; i < n; ++i)
    if (start[i] < 0 || end[i] > L || end[i] <= start[i]) return LACT_ERR_STEPS;
  lact_scan_config c;
  std::memset(&c, 0, sizeof(c));
  c.B = B; c.L = L; c.mom_dtype = dtype;
  lact_scan_io io;
  std::memset(&io, 0, sizeof(io));
  io.momentum = momentum;
  const std::vector<int32_t> kind(static_cast<size_t>(n), LACT_STEP_UPDATE);
  return launch_momentum_means(c, io, n, kind.data(), start, end, beta, static_cast<cudaStream_t>(stream));
}

int lact_momentum_gate_grad(const float* dbeta, int64_t B, int64_t L, int32_t n, const int64_t* start, const int64_t* end,
                            void* out, int32_t out_dtype, void* stream) {
  if (!dbeta || !out || (n > 0 && (!start || !end))) return LACT_ERR_NULL;
  if (B < 1 || B > 65535 || L < 1 || n < 0) return LACT_ERR_SHAPE;
  static_assert(kMeanBatch == LACT_GATE_GRAD_UPDATES, "the header names the launch's size");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int first = 0;
  do {
    MeanArgs ma;
    std::memset(&ma, 0, sizeof(ma));
    ma.n = std::min(kMeanBatch, n - first);
    for (int i = 0; i < ma.n; ++i) {
      ma.s[i] = static_cast<int32_t>(start[first + i]);
      ma.e[i] = static_cast<int32_t>(end[first + i]);
    }
    KernelScope scope(kClsOther, s);
    momentum_gate_grad_kernel<<<dim3(ceil_div(L, 256), static_cast<unsigned>(B)), 256, 0, s>>>(
        ma, dbeta, kNormBwdSlices, static_cast<int>(B), first, first > 0, out, out_dtype == LACT_F32, L);
    LACT_CUDA(cudaGetLastError());
    first += kMeanBatch;
  } while (first < n);
  return LACT_OK;
}

int lact_weight_grad(const float* dW02, const float* dW1, const float* dWm02, const float* dWm1, const float* dn02,
                     const float* dn1, const float* n02, const float* n1, const float* W02, const float* W1, void* dw0,
                     void* dw1, void* dw2, int32_t dtype, int64_t B, int64_t D, int64_t H, void* stream) {
  if (!dW02 || !dW1 || !dw0 || !dw1 || !dw2 || ((dWm02 == nullptr) != (dWm1 == nullptr))) return LACT_ERR_NULL;
  if (dn02 != nullptr && (!dn1 || !n02 || !n1 || !W02 || !W1)) return LACT_ERR_NULL;
  if (B < 1 || D < 1 || H < 1 || B * (2 * H + D) > (1ll << 33)) return LACT_ERR_SHAPE;
  const WeightGradArgs a{dW02, dW1, dWm02, dWm1, dn02, dn1, n02, n1, W02, W1, dw0, dw1, dw2, dtype == LACT_F32,
                         static_cast<int32_t>(B), static_cast<int32_t>(H), static_cast<int32_t>(D)};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  KernelScope scope(kClsOther, s);
  weight_grad_kernel<<<ceil_div(B * (2 * H + D), 8), 256, 0, s>>>(a);
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

// ---------------------------------------------------------------- fp32 mode building blocks
int lact_sgemm_f32(const void* a, int32_t a_t, const void* b, int32_t b_t, void* c, int32_t accumulate,
                   const void* beta, int64_t batch, int64_t M, int64_t N, int64_t K, void* stream) {
  if (!a || !b || !c) return LACT_ERR_NULL;
  if (batch < 1 || batch > 65535 || M < 1 || N < 1 || K < 1 || M > (1ll << 30) || N > (1ll << 30) || K > (1ll << 30))
    return LACT_ERR_SHAPE;
  F32Args g;
  std::memset(&g, 0, sizeof(g));
  g.a = f32_mat(static_cast<const float*>(a), a_t ? M : K, M * K, a_t ? 1 : 0, M, K);
  g.b = f32_mat(static_cast<const float*>(b), b_t ? N : K, N * K, b_t ? 1 : 0, N, K);
  g.M = static_cast<int32_t>(M); g.N = static_cast<int32_t>(N); g.K = static_cast<int32_t>(K);
  g.batch = static_cast<int32_t>(batch);
  g.c = static_cast<float*>(c); g.c_ld = N; g.c_bs = M * N;
  g.accumulate = accumulate;
  g.beta = static_cast<const float*>(beta);
  const dim3 grid(ceil_div(N, kFN), ceil_div(M, kFM), static_cast<unsigned>(batch));
  if (grid.y > 65535) return LACT_ERR_SHAPE;
  g.c_vec = (reinterpret_cast<uintptr_t>(g.c) & 15) == 0 && (g.c_ld % 4) == 0 && (g.c_bs % 4) == 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  KernelScope scope(kClsOther, s);
  LACT_CUDA(launch_pdl(f32_gemm_kernel, grid, dim3(kFThreads), 0, s, g));
  return LACT_OK;
}

int lact_swiglu_planes_f32(const void* y02, const void* dh, const void* lr0, const void* lr1, const void* lr2,
                           int32_t lr_dtype, float w_scale, void* dy02, void* hid, int64_t rows, int64_t H,
                           void* stream) {
  if (!y02 || !hid || (dh != nullptr && !dy02)) return LACT_ERR_NULL;
  if (rows < 1 || H < 8 || (H % 8) != 0) return LACT_ERR_SHAPE;  // planes move as 16-byte vectors
  KernelScope scope(kClsOther, static_cast<cudaStream_t>(stream));
  swiglu_planes_f32_kernel<<<ceil_div(rows, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(y02), static_cast<const float*>(dh), lr0, lr1, lr2, lr_dtype == LACT_F32, w_scale,
      static_cast<float*>(dy02), static_cast<float*>(hid), rows, static_cast<int>(H));
  LACT_CUDA(cudaGetLastError());
  return LACT_OK;
}

int lact_add_renorm(void* master, void* compute, void* shadow, const void* n0, const void* g, const void* x,
                    int64_t B, int64_t R, int64_t C, int32_t mode, int32_t prenorm, int32_t prenorm_bf16,
                    int32_t quirk, void* stream) {
  if (!master || !shadow || !n0 || !g) return LACT_ERR_NULL;
  if (B < 1 || R < 1 || C < 4 || (C % 4) || C > kRenormMaxCols || mode < 0 || mode > 2) return LACT_ERR_SHAPE;
  RenormArgs r;
  std::memset(&r, 0, sizeof(r));
  r.master = static_cast<float*>(master);
  r.compute = static_cast<float*>(compute);
  r.shadow = static_cast<bf16*>(shadow);
  r.n0 = static_cast<const float*>(n0);
  r.g = static_cast<const float*>(g);
  r.x = static_cast<const bf16*>(x);
  r.x_bs = R * C;
  r.B = static_cast<int>(B); r.R = static_cast<int>(R); r.C = static_cast<int>(C);
  r.mode = mode; r.prenorm = prenorm; r.prenorm_bf16 = prenorm_bf16; r.quirk = quirk;
  RenormArgs none = r;
  none.B = 0;
  return launch_add_renorm(r, none, static_cast<cudaStream_t>(stream));
}

int lact_bmm_bf16(const void* a, int32_t a_mn_major, const void* b, int32_t b_mn_major, void* c, int32_t c_dtype,
                  int64_t batch, int64_t M, int64_t N, int64_t K, int32_t* status_word, void* stream) {
  if (!a || !b || !c || !status_word) return LACT_ERR_NULL;
  LACT_TRY(check_device());
  if (batch < 1 || batch > 65535 || M < 1 || N < 8 || K < 1 || (M % 8) || (N % 8) || (K % 8)) return LACT_ERR_SHAPE;
  const Mat A = a_mn_major ? Mat{a, K, M, M, batch, K * M} : Mat{a, M, K, K, batch, M * K};
  const Mat Bm = b_mn_major ? Mat{b, K, N, N, batch, K * N} : Mat{b, N, K, K, batch, N * K};
  auto fill = [&](auto& g, int btv) -> int {
    auto& P = g.prob[0];
    LACT_TRY(make_operand(form_of(P), &P.a[0], &P.ai[0], A, a_mn_major, kBM, 0, 0));
    LACT_TRY(make_operand(form_of(P), &P.b[0], &P.bi[0], Bm, b_mn_major, btv, 0, 0));
    P.M = static_cast<int>(M); P.N = static_cast<int>(N); P.K = static_cast<int>(K);
    P.batch = static_cast<int>(batch);
    P.ep = EpiStore{c, M * N, N, 0, 1, 0};
    g.status = status_word;
    return LACT_OK;
  };
  auto fill_bf16 = [&](auto& g, int btv) -> int {
    auto& P = g.prob[0];
    LACT_TRY(make_operand(form_of(P), &P.a[0], &P.ai[0], A, a_mn_major, kBM, 0, 0));
    LACT_TRY(make_operand(form_of(P), &P.b[0], &P.bi[0], Bm, b_mn_major, btv, 0, 0));
    LACT_TRY(make_output(form_of(P), &P.out[0], &P.oi[0], Mat{c, M, N, N, batch, M * N}, 0, 0));
    P.M = static_cast<int>(M); P.N = static_cast<int>(N); P.K = static_cast<int>(K);
    P.batch = static_cast<int>(batch);
    g.status = status_word;
    return LACT_OK;
  };
  const int bt = choose_bt({{N, 1}});
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (c_dtype == LACT_F32) return launch_op<OpStoreDirectT, 1>(bt, fill, s, kClsOther, 1);
  return launch_op<OpBmmStore, 1>(bt, fill_bf16, s, kClsOther, 1);
}

}  // extern "C"
