// bf16 GEMM for sm_100a on the 5th-generation tensor cores, written by hand:
//   C[M,N] = A[M,K] * B[N,K]^T      (A, B row-major / "K-major", fp32 accumulate)
// One persistent CTA per SM, warp-specialised:
//   warp 0      TMA producer: cp.async.bulk.tensor tiles of A (128 x 64) and
//               B (256 x 64) into a 4-stage shared-memory ring (128B swizzle)
//   warp 1      MMA issuer: one thread issues tcgen05.mma 128x256x16 from the
//               shared-memory descriptors into tensor memory; tcgen05.commit
//               releases ring stages and publishes finished accumulators
//   warps 2-5   epilogue: tcgen05.ld the fp32 accumulators (TMEM lanes = rows),
//               convert, store; two 256-column accumulators alternate so the
//               epilogue of one tile overlaps the MMAs of the next
// The same kernel body serves the tensor-parallel fused paths through two
// optional hooks: rows of A that become valid chunk by chunk (all-gather ->
// GEMM) and an epilogue that pushes partial tiles to the rank that owns the
// rows (GEMM -> reduce-scatter); see gemm_fused.cu.
//
// Every wait is bounded: a wait that runs out sets a flag, all roles wind down,
// tensor memory is freed and the kernel reports an error word to the host.
// The reference has no GEMM and no tensor-core code; this exists because the
// tensor-parallel workload fuses it with the collectives of this library.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <mutex>
#include <vector>

#include "core/graph_capture.h"
#include "kernels/gemm2_kernel.cuh"
#include "kernels/gemm_small.h"
#include "mem/cuda_driver.h"

namespace mnccl {
namespace gemm {

// -------------------------------------------------------------------- host

namespace {

std::mutex g_mu;
// -1: automatic, 0: single-CTA kernel, 1: CTA-pair kernel; MINI_NCCL_GEMM_PAIR sets the initial value
int pair_mode_from_env() {
  const char* e = getenv("MINI_NCCL_GEMM_PAIR");
  if (e == nullptr || *e == 0) return -1;
  const int v = atoi(e);
  return v < 0 ? -1 : (v > 0 ? 1 : 0);
}
int g_use_pair = pair_mode_from_env();
uint32_t* g_err_dev[kMaxDevices] = {};  // one error word per device of the process
// Split-K workspaces (20 MB each, for the life of the process).  Products that may run at once must not add into
// each other's partial tiles:
//   * a product that runs when it is called takes the workspace its stream used last, one of kSplitPools per
//     device; a stream beyond that many takes over the one that has been idle longest, and waits on the GPU for
//     the product that used it.  (Streams are told apart by their ids: a handle can be given out again, and
//     cudaStreamPerThread is another stream in every thread.)
//   * a captured product may be replayed anywhere, beside anything: it gets one of kSplitGraphPools that its graph
//     holds until it is destroyed; products of one capture on one stream follow one another and share it.  Where
//     none is left it is captured without the split.  (Two executable graphs made from one captured graph must not
//     run at once: they share its workspace as they share the product's output.)
struct SplitPool {
  float* ws = nullptr;       // fp32 partial tiles
  uint32_t* cnt = nullptr;   // one counter per 32-row quarter
  // not captured: the end of the last product, its stream, and when that was
  cudaEvent_t last = nullptr;
  unsigned long long stream_id = 0;
  uint64_t used = 0;
  // captured: held by a graph, for products on this stream of this capture
  std::shared_ptr<std::atomic<bool>> in_graph;
  unsigned long long capture_id = 0;
  cudaStream_t capture_stream = nullptr;
};
constexpr size_t kSplitPools = 8, kSplitGraphPools = 8;
struct SplitPools {
  std::mutex mu;
  uint64_t clock = 0;
  std::vector<SplitPool> live[kMaxDevices], graph[kMaxDevices];
};
SplitPools& split_pools() {
  static auto* pools = new SplitPools;   // outlives the destructors of a process that exits with graphs alive
  return *pools;
}
constexpr int kSplitMaxItems = 80;      // K-slices in flight: at most one per CTA pair

}  // namespace

bool make_tensor_map_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t row_stride_elems,
                          uint32_t box_rows, uint32_t box_cols, std::string* why) {
  const CudaDriver* d = CudaDriver::get();
  if (!d || !d->TensorMapEncodeTiled) {
    if (why) *why = "cuTensorMapEncodeTiled unavailable";
    return false;
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0 || (row_stride_elems * 2) % 16 != 0) {
    if (why) *why = "operand base and row stride must be 16-byte aligned";
    return false;
  }
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {row_stride_elems * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  const auto encode = [&] {
    return d->TensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  int dev = 0;
  // a thread's first call: the runtime binds its device's context when it is told the device
  if (r == CUDA_ERROR_INVALID_CONTEXT && cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
  if (r != CUDA_SUCCESS) {
    if (why) *why = "cuTensorMapEncodeTiled: " + d->error_string(r);
    return false;
  }
  return true;
}

uint32_t* error_word() {
  std::lock_guard<std::mutex> lk(g_mu);
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kMaxDevices) dev = 0;
  if (g_err_dev[dev] == nullptr) {
    uint32_t* p = nullptr;
    if (cudaMalloc(&p, 64) != cudaSuccess) return nullptr;
    cudaMemset(p, 0, 64);
    g_err_dev[dev] = p;
  }
  return g_err_dev[dev];
}

namespace {

// kSplitMaxItems partial tiles of 256 x 256 fp32 and one zeroed counter per 32-row quarter.
bool create_split_pool(SplitPool* p, bool captured) {
  AllowAllocationsWhileCapturing allow;
  constexpr size_t kCntBytes = size_t(kSplitMaxItems) * 8 * 4;
  cudaStream_t s = nullptr;   // the zeroes must not be captured, nor wait behind other work
  bool ok = cudaMalloc(&p->ws, size_t(kSplitMaxItems) * 256 * 256 * 4) == cudaSuccess && cudaMalloc(&p->cnt, kCntBytes) == cudaSuccess &&
            cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess && cudaMemsetAsync(p->cnt, 0, kCntBytes, s) == cudaSuccess &&
            cudaStreamSynchronize(s) == cudaSuccess;
  if (ok && !captured) ok = cudaEventCreateWithFlags(&p->last, cudaEventDisableTiming) == cudaSuccess;
  if (s) cudaStreamDestroy(s);
  if (ok) return true;
  (void)cudaGetLastError();
  if (p->ws) cudaFree(p->ws);
  if (p->cnt) cudaFree(p->cnt);
  *p = SplitPool{};
  return false;
}

// A workspace for one product on `stream`, taken before its launch; launched() goes after it.  Other threads wait
// in between, so that none takes the workspace over before the product is in its stream.
class SplitLease {
 public:
  bool take(cudaStream_t stream) {
    try {
      SplitPools& all = split_pools();
      lock_ = std::unique_lock<std::mutex>(all.mu);
      const int dev = current_device_slot();
      const CaptureInfo cap = capture_info(stream);
      return cap.active ? take_captured(all.graph[dev], cap, stream) : take_live(all.live[dev], stream);
    } catch (...) {   // out of host memory, behind a C entry point: no split
      pool_ = nullptr;
      return false;
    }
  }
  float* ws() const { return pool_->ws; }
  uint32_t* cnt() const { return pool_->cnt; }
  void launched(cudaStream_t stream) {
    if (pool_ == nullptr || pool_->last == nullptr) return;
    if (cudaEventRecord(pool_->last, stream) != cudaSuccess) (void)cudaGetLastError();
    pool_->stream_id = id_;
    pool_->used = ++split_pools().clock;
  }

 private:
  bool take_live(std::vector<SplitPool>& pools, cudaStream_t stream) {
    if (cudaStreamGetId(stream, &id_) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    SplitPool* oldest = nullptr;
    for (SplitPool& p : pools) {
      if (p.used != 0 && p.stream_id == id_) return (pool_ = &p) != nullptr;
      if (oldest == nullptr || p.used < oldest->used) oldest = &p;
    }
    SplitPool fresh;
    if (pools.size() < kSplitPools && create_split_pool(&fresh, false)) {
      pools.push_back(fresh);
      pool_ = &pools.back();
      return true;
    }
    if (oldest == nullptr) return false;
    if (cudaStreamWaitEvent(stream, oldest->last, 0) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    pool_ = oldest;
    return true;
  }
  bool take_captured(std::vector<SplitPool>& pools, const CaptureInfo& cap, cudaStream_t stream) {
    SplitPool* idle = nullptr;
    for (SplitPool& p : pools) {
      if (!p.in_graph->load(std::memory_order_acquire)) idle = &p;
      else if (p.capture_id == cap.id && p.capture_stream == stream) return (pool_ = &p) != nullptr;
    }
    if (idle == nullptr) {
      SplitPool fresh;
      if (pools.size() >= kSplitGraphPools || !create_split_pool(&fresh, true)) return false;
      fresh.in_graph = std::make_shared<std::atomic<bool>>(false);
      pools.push_back(fresh);
      idle = &pools.back();
    }
    if (!hold_while_graph_lives(cap.graph, idle->in_graph)) return false;
    idle->capture_id = cap.id;
    idle->capture_stream = stream;
    pool_ = idle;
    return true;
  }

  std::unique_lock<std::mutex> lock_;
  SplitPool* pool_ = nullptr;
  unsigned long long id_ = 0;
};

}  // namespace

// Split-K plan of the CTA-pair kernel: tiles2 tiles on n_pairs pairs, num_kb k-blocks per tile.  When
// the last wave holds at most half as many tiles as there are pairs, each of its tiles is cut into at
// most 8 slices of at least 4 k-blocks so that all slices still form ONE wave (their warps wait for one
// another, which is only safe because they are all resident at the same time).  Returns false for "no split".
bool plan_split(int tiles2, int n_pairs, int num_kb, int* first, int* s, int* kb) {
  const char* e = getenv("MINI_NCCL_GEMM_SPLIT_K");
  if (e != nullptr && *e == '0') return false;
  if (n_pairs < 2 || tiles2 <= n_pairs) return false;        // a single wave: nothing to balance
  const int rem = tiles2 % n_pairs;
  if (rem == 0 || 2 * rem > n_pairs) return false;
  int slices = n_pairs / rem;
  if (slices > kBN / 32) slices = kBN / 32;                     // a slice's warp sums whole 32-column pieces
  if (slices > num_kb / 4) slices = num_kb / 4;
  if (slices * rem > kSplitMaxItems) slices = kSplitMaxItems / rem;
  if (slices < 2) return false;
  const int per = (num_kb + slices - 1) / slices;
  *first = tiles2 - rem;
  *kb = per;
  *s = (num_kb + per - 1) / per;                                // no empty slice
  if (*s < 2) return false;
  // Measured on B200: a 256 x 256 pair tile takes about 3 us + 0.33 us per k-block, and cutting it costs
  // about 7 us (partial sums to the workspace, the meeting of the slices, the sum): 4096 x 3584 x 4096
  // gains 12 us with 8 slices, 4096 x 4096 x 1792 loses 1 us with 2, 4096 x 4096 x 512 loses 4 us.
  const long tile_ns = 3000 + 330L * num_kb;
  return tile_ns * (*s - 1) / *s > 9000;
}

int pick_tile_n(int M, int N, int ctas, bool allow_224) {
  const int cand[4] = {256, 224, 192, 128};  // 128: small products that leave most SMs without a tile
  int best = 256;
  long best_cost = -1;
  const int tiles_m = (M + kBM - 1) / kBM;
  for (int i = 0; i < 4; ++i) {
    const int bn = cand[i];
    if ((bn == 224 || bn == 128) && !allow_224) continue;
    const long tiles = static_cast<long>(tiles_m) * ((N + bn - 1) / bn);
    const long waves = (tiles + ctas - 1) / ctas;
    // Measured on B200 (4096 x 4096 x 1792): a wave of 256-wide tiles takes 13.9 us, of 192-wide
    // tiles 12.2 us: the time per tile is about a + b * bn with a / b ~ 256 columns, so a narrower
    // tile only pays when it removes a whole wave.
    const long cost = waves * (bn + 256);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

bool want_pair(int M, int N, int ctas) {
  if (g_use_pair == 0 || M < 2 * kBM || N < kBN || ctas < 2) return false;
  if (g_use_pair == 1) return true;
  // Measured on B200: pairs win by 5-15 % (a third less operand traffic from L2 per FLOP) once
  // they have enough tiles; with far fewer tiles than pairs, or a worse last wave, single tiles win.
  const long pairs = ctas / 2;
  const long t2 = static_cast<long>((M + 2 * kBM - 1) / (2 * kBM)) * ((N + kBN - 1) / kBN);
  const long t1 = static_cast<long>((M + kBM - 1) / kBM) * ((N + kBN - 1) / kBN);
  if (2 * t2 < pairs) return false;  // small products: narrower single-CTA tiles reach more SMs
  const double fill2 = static_cast<double>(t2) / static_cast<double>(((t2 + pairs - 1) / pairs) * pairs);
  const double fill1 = static_cast<double>(t1) / static_cast<double>(((t1 + ctas - 1) / ctas) * ctas);
  return fill2 >= fill1 - 0.04;
}

int pair_mode() { return g_use_pair; }
void set_pair_mode(int m) { g_use_pair = m; }

int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

namespace {

// Estimated times (ns) on this GPU's 148 SMs, measured for square-ish and for thin products with K from 64 to
// 14336 (graph replay, operands not in L2).  They only have to rank the candidates.
//
// Small kernel (gemm_small.cu), tiles of 128 rows of B x tn rows of A, K over `slices` CTAs: a fixed part
// (launch, first loads, epilogue, meeting of the slices), a time per k-block and SM, which is what L2 can
// hand one SM, and never faster than DRAM delivers the operands.
struct SmallCost {
  int tn, kps;              // rows of A per tile, k-blocks per stage
  long fixed, fixed_split;  // one slice, several slices
  long per_kb;
};
constexpr SmallCost kSmallCost[] = {{16, 2, 3500, 4500, 130}, {32, 2, 4100, 4900, 145}, {64, 2, 4400, 5000, 173}, {128, 1, 5900, 6300, 240}};

long dram_ns(int M, int N, int K, int out_bytes) {
  return static_cast<long>((2.0 * K * (static_cast<double>(M) + N) + static_cast<double>(out_bytes) * M * N) / 6200.0);
}

long plan_small(int M, int N, int K, int out_bytes, int sms, SmallPlan* best) {
  const int num_kb = (K + kBK - 1) / kBK;
  const long tiles_n = (N + 127) / 128, floor_ns = 3000 + dram_ns(M, N, K, out_bytes);
  long best_ns = -1;
  for (const SmallCost& c : kSmallCost) {
    if (c.tn > 16 && c.tn / 2 >= M) break;  // half of the tile would be padding
    const long tiles = tiles_n * ((M + c.tn - 1) / c.tn);
    if (tiles > 4L * sms) continue;
    const int stages = (num_kb + c.kps - 1) / c.kps;
    for (int s = 1; s <= 8; s *= 2) {
      const int per = (stages + s - 1) / s;
      if ((s - 1) * per >= stages) break;  // a slice would be empty
      const long items = tiles * s;
      if (s > 1 && items > 2L * sms) break;
      // One CTA per SM where all of them fit at once (clusters of 4 and 8 do not tile every GPC: 15 clusters of
      // 8 start together, a 16th waits for a whole round); else two share an SM and its L2 port.
      const bool deep = items <= (s == 8 ? 15 * sms / 18 : s == 4 ? 7 * sms / 8 : sms);
      const long rounds = deep ? 1 : 2 * ((items + 2L * sms - 1) / (2L * sms));
      const long fixed = s == 1 ? c.fixed : s == 8 ? c.fixed_split + 1300 : c.fixed_split;
      const long ns = std::max(fixed + rounds * per * c.kps * c.per_kb, floor_ns);
      if (best_ns < 0 || ns < best_ns) {
        best_ns = ns;
        best->tn = c.tn;
        best->slices = s;
        best->kb_per_slice = per;
        best->tiles = static_cast<int>(tiles);
        best->deep = deep;
      }
    }
  }
  return best_ns;
}

// Persistent kernels: waves of tiles, a k-block of a 256 x 256 pair tile in 330 ns, of a 128 x bn tile at what L2
// hands one SM (165 bytes per ns) or, narrow ones, at a quarter of the latency that the four-stage ring covers.
long persistent_ns(int M, int N, int K, int out_bytes, int sms, bool pair, int bn) {
  const long num_kb = (K + kBK - 1) / kBK;
  const long floor_ns = 5000 + dram_ns(M, N, K, out_bytes);
  if (pair) {
    const long tiles = static_cast<long>((M + 2 * kBM - 1) / (2 * kBM)) * ((N + kBN - 1) / kBN);
    const long waves = (tiles + sms / 2 - 1) / (sms / 2);
    return std::max(5600 + waves * num_kb * 330, floor_ns);
  }
  const long tiles = static_cast<long>((M + kBM - 1) / kBM) * ((N + bn - 1) / bn);
  const long waves = (tiles + sms - 1) / sms;
  return std::max(4800 + waves * num_kb * std::max((kBM + bn) * 128 / 165, 285), floor_ns);
}

}  // namespace

int run_gemm(const char* who, const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, GemmOut out,
             cudaStream_t stream) {
  const int sms = sm_count();
  const int out_bytes = out == kOutF32 ? 4 : 2;
  const bool pair = want_pair(M, N, sms);
  const int bn = pair ? kBN : pick_tile_n(M, N, sms, out != kOutSwiGlu);  // (the SwiGLU store collects whole rows of 32-column pieces)
  std::string why;
  if (g_use_pair < 0) {
    // Small products, in automatic mode only: a pinned choice names one of the persistent kernels.
    SmallPlan p;
    const long small_ns = plan_small(M, N, K, out_bytes, sms, &p);
    if (small_ns > 0 && small_ns < persistent_ns(M, N, K, out_bytes, sms, pair, bn)) {
      const cudaError_t e = launch_small(A, B, C, M, N, K, lda, ldb, ldc, static_cast<int>(out), p, error_word(), stream, &why);
      if (!why.empty()) {
        fprintf(stderr, "[Mini-NCCL] %s: %s\n", who, why.c_str());
        return -3;
      }
      return e == cudaSuccess ? 0 : static_cast<int>(e) + 1000;
    }
  }
  CUtensorMap ta, tb;
  // CTA pairs: 256 x 256 tiles, each CTA loads 128 rows of A and 128 rows (half of N) of B
  if (!make_tensor_map_bf16(&ta, A, M, K, lda, kBM, kBK, &why) ||
      !make_tensor_map_bf16(&tb, B, N, K, ldb, pair ? kBN / 2 : bn, kBK, &why)) {
    fprintf(stderr, "[Mini-NCCL] %s: %s\n", who, why.c_str());
    return -3;
  }
  GemmArgs g{};
  g.M = M;
  g.N = N;
  g.K = K;
  g.c = C;
  g.ldc = ldc;
  g.err = error_word();
  g.wait_budget_ns = 2000000000ull;
  g.group_m = 8;
  int grid;
  SplitLease lease;
  if (pair) {
    const int tiles2 = ((M + 2 * kBM - 1) / (2 * kBM)) * ((N + kBN - 1) / kBN);
    grid = std::min(2 * tiles2, sms & ~1);
    const int pairs = std::min(grid / 2, out == kOutSwiGlu ? max_pairs<SwiGluEpilogue>() : max_pairs<StoreEpilogue<false>>());
    int first = 0, slices = 0, per = 0;
    if (plan_split(tiles2, pairs, (K + kBK - 1) / kBK, &first, &slices, &per) && lease.take(stream)) {
      g.split_ws = lease.ws();
      g.split_cnt = lease.cnt();
      g.split_first = first;
      g.split_s = slices;
      g.split_kb = per;
    }
  } else {
    grid = std::min(((M + kBM - 1) / kBM) * ((N + bn - 1) / bn), sms);
  }
  const auto fire = [&](const auto& epi) { return pair ? launch_pair(ta, tb, g, epi, grid, stream) : launch(ta, tb, g, epi, grid, stream, bn); };
  cudaError_t e;
  if (out == kOutF32) e = fire(StoreEpilogue<true>{});
  else if (out == kOutSwiGlu) e = fire(SwiGluEpilogue{bn / 32});
  else e = fire(StoreEpilogue<false>{});
  if (e == cudaSuccess) lease.launched(stream);
  return e == cudaSuccess ? 0 : static_cast<int>(e) + 1000;
}

}  // namespace gemm
}  // namespace mnccl

using namespace mnccl;
using namespace mnccl::gemm;

extern "C" {
#define MNCCL_EXPORT __attribute__((visibility("default")))

// C[M,N] = A[M,K] * B[N,K]^T, bf16 operands, fp32 accumulation.
// out_f32 = 0: C is bf16; 1: C is fp32.  lda / ldb / ldc are row strides in
// elements (0 = dense).  Requirements: A, B 16-byte aligned, lda and ldb
// multiples of 8, K >= 8.  Returns 0, or a negative code for bad arguments, or
// a cudaError_t + 1000.
MNCCL_EXPORT int mncclGemmBf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                               int out_f32, cudaStream_t stream) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return -1;
  if (lda == 0) lda = K;
  if (ldb == 0) ldb = K;
  if (ldc == 0) ldc = N;
  if (lda < K || ldb < K || ldc < N) return -2;
  return run_gemm("GEMM", A, B, C, M, N, K, lda, ldb, ldc, out_f32 ? kOutF32 : kOutBf16, stream);
}

// Pairs of CTAs (clusters of 2) of the GEMM kernel that fit the current device at once.
MNCCL_EXPORT int mncclGemmMaxPairs(void) { return max_pairs<StoreEpilogue<false>>(); }

// Kernel choice for the calls that follow: -1 automatic, 0 single-CTA tiles, 1 CTA pairs (cta_group::2).
MNCCL_EXPORT void mncclGemmSetPairMode(int mode) { set_pair_mode(mode); }

// The host-side choice for an M x N product on `ctas` CTAs, without launching anything (needs no
// GPU): *tile_n = tile width of the single-CTA kernel (`narrow` = 1 admits 224 and 128), *pair = 1
// when the CTA-pair kernel would be taken instead.
MNCCL_EXPORT void mncclGemmPlan(int M, int N, int ctas, int narrow, int* tile_n, int* pair) {
  if (tile_n) *tile_n = pick_tile_n(M, N, ctas, narrow != 0);
  if (pair) *pair = want_pair(M, N, ctas) ? 1 : 0;
}

// Whether an M x N x K product (out: 0 bf16, 1 fp32, 2 SwiGLU) takes the kernel for small products on `sms` SMs in
// automatic mode, and its plan: rows of A per tile, CTAs that share a tile's K, one CTA per SM or two.  Host
// arithmetic only (needs no GPU).
MNCCL_EXPORT int mncclGemmSmallPlan(int M, int N, int K, int out, int sms, int* tn, int* slices, int* deep) {
  if (M <= 0 || N <= 0 || K <= 0 || sms <= 0) return 0;
  SmallPlan p;
  const bool pair = want_pair(M, N, sms);
  const int bn = pair ? kBN : pick_tile_n(M, N, sms, out != kOutSwiGlu), out_bytes = out == kOutF32 ? 4 : 2;
  const long ns = plan_small(M, N, K, out_bytes, sms, &p);
  if (ns < 0 || ns >= persistent_ns(M, N, K, out_bytes, sms, pair, bn)) return 0;
  if (tn) *tn = p.tn;
  if (slices) *slices = p.slices;
  if (deep) *deep = p.deep ? 1 : 0;
  return 1;
}

// The split-K plan of the CTA-pair kernel for an M x N x K product on `pairs` CTA pairs, without launching
// anything (needs no GPU): returns 1 and the first split work item, the slices per tile and the k-blocks
// per slice when the last, partial wave is cut along K, else 0.
MNCCL_EXPORT int mncclGemmSplitPlan(int M, int N, int K, int pairs, int* first, int* slices, int* kb_per_slice) {
  if (M <= 0 || N <= 0 || K <= 0 || pairs <= 0) return 0;
  const int tiles2 = ((M + 2 * kBM - 1) / (2 * kBM)) * ((N + kBN - 1) / kBN);
  int f = 0, s = 0, k = 0;
  if (!plan_split(tiles2, pairs, (K + kBK - 1) / kBK, &f, &s, &k)) return 0;
  if (first) *first = f;
  if (slices) *slices = s;
  if (kb_per_slice) *kb_per_slice = k;
  return 1;
}

// The tiles worker `worker` of `n_workers` visits, in order, exactly as the kernels walk them (host
// arithmetic only, for tests): single-CTA kernel: worker = CTA, tiles of 128 x bn; pair kernel
// (`pair` = 1): worker = CTA pair, 256 x 256 tiles, reported as the two 128-row tiles (tm, tm + 1)
// of its CTAs.  group_m / rotate are the values the entry points put into GemmArgs (in 128-row
// tiles).  Writes up to `max` (tm, tn) pairs; returns the number of 128-row tiles visited.
MNCCL_EXPORT int mncclGemmTileOrder(int M, int N, int bn, int group_m, int rotate, int pair, int n_workers, int worker,
                                    int* out_tm, int* out_tn, int max) {
  if (M <= 0 || N <= 0 || bn <= 0 || n_workers <= 0 || worker < 0 || worker >= n_workers) return -1;
  GemmArgs g{};
  g.M = M;
  g.N = N;
  int n = 0;
  if (pair) {
    g.group_m = group_m > 1 ? group_m / 2 : 1;          // as gemm2_bf16_kernel derives them
    g.m_tile_rotate = rotate / 2;
    const int tiles_m2 = (M + 2 * kBM - 1) / (2 * kBM), tiles_n = (N + kBN - 1) / kBN;
    for (int t = worker; t < tiles_m2 * tiles_n; t += n_workers) {
      int tm2, tn;
      tile_coords(g, t, tiles_m2, tiles_n, &tm2, &tn);
      for (int cta = 0; cta < 2; ++cta, ++n)
        if (n < max) { out_tm[n] = tm2 * 2 + cta; out_tn[n] = tn; }
    }
  } else {
    g.group_m = group_m;
    g.m_tile_rotate = rotate;
    const int tiles_m = (M + kBM - 1) / kBM, tiles_n = (N + bn - 1) / bn;
    for (int t = worker; t < tiles_m * tiles_n; t += n_workers, ++n) {
      int tm, tn;
      tile_coords(g, t, tiles_m, tiles_n, &tm, &tn);
      if (n < max) { out_tm[n] = tm; out_tn[n] = tn; }
    }
  }
  return n;
}

// Reads and clears the GEMM error word of the current device (0 = no bounded
// wait ever ran out).  Synchronises the device.
MNCCL_EXPORT int mncclGemmStatus(uint32_t* status) {
  uint32_t* w = error_word();
  if (!w || !status) return -1;
  if (cudaDeviceSynchronize() != cudaSuccess) return -2;
  if (cudaMemcpy(status, w, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return -2;
  cudaMemset(w, 0, 4);
  return 0;
}

}  // extern "C"
