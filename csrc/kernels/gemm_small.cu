// The sm_100a GEMM for products too small for the persistent kernels: C[M, N] = A[M, K] * B[N, K]^T with few
// rows of A (decode), or with too few 128 x 256 tiles to give every SM one.
//
// What bounds these products is bytes in flight and fixed costs, not the tensor cores: 16 x 14336 x 4096 is
// 117 MB of weights for 1.9 GFLOP.  Hence
//   * the operands are swapped: the 128 rows of the MMA are rows of B (the weight), its TN columns are rows
//     of A (16 .. 128).  A tile of 16 tokens then costs 2 KB of shared memory per k-block instead of 16, the
//     ring holds 6 k-blocks of weights in half an SM's shared memory (two CTAs per SM) or 12 in all of it, and
//     an accumulator column is 128 consecutive elements of one row of C: every store is coalesced whatever
//     N, ldc and the alignment are, without a detour through shared memory;
//   * K is split over the S CTAs of a cluster (S <= 8) where the tiles alone leave SMs idle.  The slices meet
//     in distributed shared memory: slice s receives the S partial copies of its TN / S columns, adds them
//     in slice order and stores them.  No workspace and no counters in global memory, so calls on different
//     streams cannot disturb one another, and a captured call can be replayed anywhere;
//   * the first loads are issued before the CTA's other warps have started: barrier set-up and the allocation
//     of tensor memory overlap the first trip to memory.
// One tile per CTA, nothing is persistent: the hardware's block scheduler balances what little there is.
#include <algorithm>
#include <string>

#include "kernels/gemm_kernel.cuh"
#include "kernels/gemm_small.h"

namespace mnccl {
namespace gemm {

namespace {

constexpr int kWTileBytes = 128 * kBK * 2;  // 128 rows of B per k-block: 16 KB
constexpr int kSmallThreads = 32 * (2 + kEpilogueWarps);

// A stage holds KPS k-blocks: the TN-row tiles of A behind the 128-row tiles of B.
template <int TN, int KPS>
constexpr int kSmallStageBytes = KPS * (kWTileBytes + TN * kBK * 2);

struct __align__(8) SmallCtl {
  uint64_t full[12];
  uint64_t empty[12];
  uint64_t done;
  uint32_t tmem_base;
  volatile uint32_t abort;
};

__device__ __forceinline__ uint32_t cluster_nctaid() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// One column (row m of C) of the tile: this lane's element n.
template <int OUT>
__device__ __forceinline__ void store_column(const SmallArgs& g, int m, int n, float v, int lane) {
  if constexpr (OUT == kOutSwiGlu) {
    // rows [32k, 32k + 16) of B are gate features 16k.., rows [32k + 16, 32k + 32) the up features of the same
    // indices: lanes 0..15 and 16..31 of the warp
    const float up = __shfl_xor_sync(0xffffffffu, v, 16);
    if (lane < 16 && m < g.M && n < g.N)
      static_cast<__nv_bfloat16*>(g.c)[static_cast<size_t>(m) * g.ldc + (n - lane) / 2 + lane] =
          __float2bfloat16_rn(v / (1.0f + __expf(-v)) * up);
  } else {
    if (m >= g.M || n >= g.N) return;
    if constexpr (OUT == kOutF32) static_cast<float*>(g.c)[static_cast<size_t>(m) * g.ldc + n] = v;
    else static_cast<__nv_bfloat16*>(g.c)[static_cast<size_t>(m) * g.ldc + n] = __float2bfloat16_rn(v);
  }
}

template <int TN, int KPS, int NS, int OUT>
__global__ void __launch_bounds__(kSmallThreads)
gemm_small_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                  const __grid_constant__ SmallArgs g) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kStage = kSmallStageBytes<TN, KPS>;
  constexpr uint32_t kCols = TN < 32 ? 32 : TN;
  static_assert(NS <= 12, "ring depth");
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  SmallCtl* ctl = reinterpret_cast<SmallCtl*>(smem + NS * kStage);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slices = static_cast<int>(cluster_nctaid());
  const int slice = static_cast<int>(cluster_ctarank());
  const int tile = static_cast<int>(blockIdx.x) / slices;
  const int n0 = (tile % g.tiles_n) * 128, m0 = (tile / g.tiles_n) * TN;
  // in units of a stage's K (a last stage may reach beyond K: those columns are loaded as zeros)
  const int num_kb = (g.K + KPS * kBK - 1) / (KPS * kBK);
  const int kb0 = slice * g.kb_per_slice;
  const int nkb = min(num_kb, kb0 + g.kb_per_slice) - kb0;  // at least 1: the plan leaves no slice empty

  // The producer and the MMA warp walk their loops as whole warps and one elected lane issues (why: mbar_wait_warp
  // in sm100_ptx.cuh; 0.27 us per k-block of four small MMAs and two loads, now 0.16).
  const bool leader = elect_one();
  auto load = [&](int i, uint32_t s) {  // k-block i of this slice into stage s; the barrier counts both tiles' bytes
    const uint32_t full = smem_u32(&ctl->full[0]) + s * 8u, dst = base + s * kStage;
    mbar_arrive_expect_tx(full, kStage);
#pragma unroll
    for (int p = 0; p < KPS; ++p) {
      const int k = ((kb0 + i) * KPS + p) * kBK;
      tma_load_2d(dst + p * kWTileBytes, &tma_w, full, k, n0);
      tma_load_2d(dst + KPS * kWTileBytes + p * (TN * kBK * 2), &tma_x, full, k, m0);
    }
  };
  if (warp == 0) {
    if (leader) {
      prefetch_tensormap(&tma_w);
      prefetch_tensormap(&tma_x);
      for (int s = 0; s < NS; ++s) {
        mbar_init(smem_u32(&ctl->full[s]), 1);
        mbar_init(smem_u32(&ctl->empty[s]), 1);
      }
      mbar_init(smem_u32(&ctl->done), 1);
      ctl->abort = 0;
      fence_barrier_init();
      fence_proxy_async();
    }
    __syncwarp();
    for (int i = 0; i < NS && i < nkb; ++i)
      if (leader) load(i, i);
  }
  __syncwarp();
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctl->tmem_base), kCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_base;

  if (warp == 0) {
    uint32_t s = 0, ph = 0;
    int i = NS;
    for (; i < nkb; ++i) {
      if (!mbar_wait_warp(smem_u32(&ctl->empty[0]) + s * 8u, ph, &ctl->abort, g.wait_budget_ns)) break;
      if (leader) load(i, s);
      if (++s == NS) { s = 0; ph ^= 1u; }
    }
    loads_land(&ctl->full[0], NS, static_cast<uint32_t>(min(i, nkb)), g.wait_budget_ns);
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(128, TN);
    const uint64_t dw0 = make_smem_desc_sw128(base), dx0 = make_smem_desc_sw128(base + KPS * kWTileBytes);
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int i = 0; i < nkb; ++i) {
      ok = mbar_wait_warp(smem_u32(&ctl->full[0]) + s * 8u, ph, &ctl->abort, g.wait_budget_ns);
      if (!ok) break;
      tc_fence_after_sync();
      const uint64_t dw = dw0 + static_cast<uint64_t>(s * (kStage >> 4)), dx = dx0 + static_cast<uint64_t>(s * (kStage >> 4));
      if (leader) {
#pragma unroll
        for (int k = 0; k < KPS * kBK / kUmmaK; ++k) {
          // 16 elements on inside a 128-byte swizzle row: +2 in the address field; k-blocks are whole tiles apart
          const int p = k / (kBK / kUmmaK), in = k % (kBK / kUmmaK) * 2;
          umma_bf16(tmem, dw + static_cast<uint64_t>(p * (kWTileBytes >> 4) + in),
                    dx + static_cast<uint64_t>(p * ((TN * kBK * 2) >> 4) + in), idesc, (i | k) != 0 ? 1u : 0u);
        }
        umma_commit(smem_u32(&ctl->empty[0]) + s * 8u);
      }
      if (++s == NS) { s = 0; ph ^= 1u; }
    }
    if (ok && leader) umma_commit(smem_u32(&ctl->done));
  }
  __syncwarp();

  // ---- epilogue: warps 2..5, one TMEM lane quarter each
  const int q = warp & 3;
  const int row = q * 32 + lane;  // row of the tile: n0 + row
  const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16);
  bool ok = true;
  if (warp >= 2) {
    ok = mbar_wait_warp(smem_u32(&ctl->done), 0, &ctl->abort, g.wait_budget_ns);
    tc_fence_after_sync();
  }
  constexpr int kPiece = TN < 32 ? TN : 32;  // accumulator columns per TMEM load
  if (slices == 1) {
    if (warp >= 2 && ok) {
#pragma unroll 1
      for (int c = 0; c < TN; c += kPiece) {
        if (m0 + c >= g.M) break;
        uint32_t r[kPiece];
        tmem_ld_cols(taddr + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kPiece; ++j) store_column<OUT>(g, m0 + c + j, n0 + row, __uint_as_float(r[j]), lane);
      }
    }
  } else {
    // Every CTA of the cluster has left its main loop: its ring may be overwritten.
    cluster_sync_all();
    const int own = TN / slices;  // columns this slice finishes (a power of two)
    const int own_log2 = 31 - __clz(own);
    float* recv = reinterpret_cast<float*>(smem);  // [source slice][own columns][128 rows]
    if (warp >= 2 && ok) {
#pragma unroll 1
      for (int c = 0; c < TN; c += kPiece) {
        if (m0 + c >= g.M) break;
        uint32_t r[kPiece];
        tmem_ld_cols(taddr + c, r);
        tmem_ld_wait();
        uint32_t dst = 0;
#pragma unroll
        for (int j = 0; j < kPiece; ++j, dst += 128 * 4) {
          const int col = c + j, at = col & (own - 1);
          if (j == 0 || at == 0)  // the next owner's columns begin
            dst = map_to_cta(smem_u32(recv + (slice * own + at) * 128 + row), static_cast<uint32_t>(col >> own_log2));
          st_cluster_f32(dst, __uint_as_float(r[j]));
        }
      }
    }
    cluster_sync_all();
    if (warp >= 2 && ok) {
      constexpr int kBatch = TN < 64 ? 2 : 8;  // columns in flight; own is a multiple (TN / 8 at least)
#pragma unroll 1
      for (int c = 0; c < own; c += kBatch) {
        const int m = m0 + slice * own + c;
        if (m >= g.M) break;
        float v[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) v[j] = recv[(c + j) * 128 + row];
        for (int s = 1; s < slices; ++s) {
#pragma unroll
          for (int j = 0; j < kBatch; ++j) v[j] += recv[(s * own + c + j) * 128 + row];
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j) store_column<OUT>(g, m + j, n0 + row, v[j], lane);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kCols);
  }
  if (threadIdx.x == 0 && ctl->abort != 0u && g.err != nullptr) atomicCAS(g.err, 0u, ctl->abort);
}

template <int TN, int KPS, int NS, int OUT>
cudaError_t fire(const CUtensorMap& tw, const CUtensorMap& tx, const SmallArgs& g, int tiles, int slices, cudaStream_t stream) {
  auto kernel = gemm_small_kernel<TN, KPS, NS, OUT>;
  constexpr int smem_bytes = NS * kSmallStageBytes<TN, KPS> + 1024 /*alignment slack*/ + static_cast<int>(sizeof(SmallCtl));
  static_assert(smem_bytes <= 227 * 1024, "shared memory of the small GEMM");
  static bool configured[kMaxDevices] = {};
  const int dev = current_device_slot();
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles) * slices);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(slices);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, tw, tx, g);
}

template <int TN, int KPS, int DEEP, int SHALLOW>
cudaError_t fire_out(const CUtensorMap& tw, const CUtensorMap& tx, const SmallArgs& g, const SmallPlan& p, int out, cudaStream_t stream) {
  switch (out) {
    case kOutBf16: return p.deep ? fire<TN, KPS, DEEP, kOutBf16>(tw, tx, g, p.tiles, p.slices, stream) : fire<TN, KPS, SHALLOW, kOutBf16>(tw, tx, g, p.tiles, p.slices, stream);
    case kOutF32: return p.deep ? fire<TN, KPS, DEEP, kOutF32>(tw, tx, g, p.tiles, p.slices, stream) : fire<TN, KPS, SHALLOW, kOutF32>(tw, tx, g, p.tiles, p.slices, stream);
    case kOutSwiGlu: return p.deep ? fire<TN, KPS, DEEP, kOutSwiGlu>(tw, tx, g, p.tiles, p.slices, stream) : fire<TN, KPS, SHALLOW, kOutSwiGlu>(tw, tx, g, p.tiles, p.slices, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_small(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int out,
                         const SmallPlan& p, uint32_t* err, cudaStream_t stream, std::string* why) {
  CUtensorMap tw, tx;
  if (!make_tensor_map_bf16(&tw, B, N, K, ldb, 128, kBK, why) || !make_tensor_map_bf16(&tx, A, M, K, lda, p.tn, kBK, why))
    return cudaErrorInvalidValue;
  SmallArgs g{};
  g.M = M;
  g.N = N;
  g.K = K;
  g.c = C;
  g.ldc = ldc;
  g.tiles_n = (N + 127) / 128;
  g.kb_per_slice = p.kb_per_slice;
  g.err = err;
  g.wait_budget_ns = 2000000000ull;
  // ring depths: all of an SM's shared memory, or half of it
  switch (p.tn) {
    case 16: return fire_out<16, 2, 6, 3>(tw, tx, g, p, out, stream);
    case 32: return fire_out<32, 2, 5, 2>(tw, tx, g, p, out, stream);
    case 64: return fire_out<64, 2, 4, 2>(tw, tx, g, p, out, stream);
    case 128: return fire_out<128, 1, 6, 3>(tw, tx, g, p, out, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gemm
}  // namespace mnccl
