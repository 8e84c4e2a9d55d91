// One rank: out[i] = (OutT)(scale * in[i]), the AllReduce of a communicator of size 1 and the copy-in /
// copy-out step of the chunk pipeline.
//
// Bound by DRAM: every byte is read once and written once, nothing else happens.  What the copy rate
// depends on is how much is in flight and in which order the blocks walk memory (B200, 256 MiB of fp32, per call
// among others): a grid-stride loop of 4 blocks of 512 threads per SM with 16-byte accesses took 91.4 us, one block
// per tile with 32-byte accesses, this kernel, takes 81.9 = 6.55 TB/s.  In a run of the steps one by one, 32-byte accesses
// gave 2 %, a block per tile with 16-byte accesses 3.5 %, both together 6 %.  The hardware's block scheduler keeps the
// tiles that are in flight close together, which the grid-stride loop does not.  A unit is what gives the wider
// of the two types 32 bytes (ld / st .v8.b32), so a cast moves 16 + 32 bytes per unit: 13.1 M elements bf16 -> fp32 in
// 14.5 us, before 22.6 with 8 + 16.  16-byte (or no) alignment takes the narrow form.
#include <type_traits>

#include "kernels/dev_prims.cuh"
#include "kernels/launch.h"

namespace mnccl {
namespace dev {
namespace {

constexpr int kLocalThreads = 256;

__device__ __forceinline__ void load_bytes(const void* p, uint32_t (&w)[8]) {
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void load_bytes(const void* p, uint32_t (&w)[4]) {
  asm volatile("ld.global.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void store_bytes(void* p, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
               "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
__device__ __forceinline__ void store_bytes(void* p, const uint32_t (&w)[4]) {
  asm volatile("st.global.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

// Elements of a unit: the wider type fills 32 bytes.
template <typename InT, typename OutT>
constexpr int kUnitElems = 32 / (sizeof(typename Elem<InT>::Raw) > sizeof(typename Elem<OutT>::Raw)
                                     ? sizeof(typename Elem<InT>::Raw)
                                     : sizeof(typename Elem<OutT>::Raw));

// N raw elements in 32-bit words <-> accumulators.
template <typename T, int N>
union Words {
  static constexpr int kWords = N * sizeof(typename Elem<T>::Raw) / 4;
  uint32_t w[kWords];
  typename Elem<T>::Raw e[N];
};

template <typename OutT, typename A>
__device__ __forceinline__ A scaled(A v, const LocalArgs& a) {
  if constexpr (!Elem<OutT>::kFloat) return v;
  else if constexpr (sizeof(A) == 8) return a.identity ? v : v * a.scale_d;
  else return a.identity ? v : v * a.scale_f;
}

template <typename InT, typename OutT, int N>
__device__ __forceinline__ void convert(const Words<InT, N>& x, Words<OutT, N>& y, const LocalArgs& a) {
  using OAcc = typename Elem<OutT>::Acc;
#pragma unroll
  for (int k = 0; k < N; k += 2) {
    const OAcc v0 = scaled<OutT>(static_cast<OAcc>(Elem<InT>::up(x.e[k])), a);
    const OAcc v1 = scaled<OutT>(static_cast<OAcc>(Elem<InT>::up(x.e[k + 1])), a);
    if constexpr (std::is_same<OutT, __nv_bfloat16>::value) {
      const __nv_bfloat162 p = __floats2bfloat162_rn(v0, v1);   // one instruction for the pair
      y.w[k / 2] = *reinterpret_cast<const uint32_t*>(&p);
    } else if constexpr (std::is_same<OutT, __half>::value) {
      const __half2 p = __floats2half2_rn(v0, v1);
      y.w[k / 2] = *reinterpret_cast<const uint32_t*>(&p);
    } else {
      y.e[k] = Elem<OutT>::down(v0);
      y.e[k + 1] = Elem<OutT>::down(v1);
    }
  }
}

// Tiles of kLocalThreads * U units, dealt to the blocks in order (one each unless the caller capped the grid).
template <typename InT, typename OutT, int U>
__global__ void __launch_bounds__(kLocalThreads) local_wide_kernel(const __grid_constant__ LocalArgs a) {
  constexpr int E = kUnitElems<InT, OutT>;
  using In = Words<InT, E>;
  using Out = Words<OutT, E>;
  constexpr bool kSame = std::is_same<InT, OutT>::value;
  const char* src = static_cast<const char*>(a.send);
  char* dst = static_cast<char*>(a.recv);
  const bool copy = kSame && a.identity != 0;
  const uint64_t units = a.count / E;
  constexpr uint64_t kTile = uint64_t(kLocalThreads) * U;
  for (uint64_t t0 = blockIdx.x * kTile; t0 < units; t0 += gridDim.x * kTile) {
    In x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t i = t0 + u * kLocalThreads + threadIdx.x;
      if (i < units) load_bytes(src + i * sizeof(In), x[u].w);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t i = t0 + u * kLocalThreads + threadIdx.x;
      if (i >= units) continue;
      if constexpr (kSame) {
        if (copy) {
          store_bytes(dst + i * sizeof(In), x[u].w);
          continue;
        }
      }
      Out y;
      convert<InT, OutT, E>(x[u], y, a);
      store_bytes(dst + i * sizeof(Out), y.w);
    }
  }
  // the last count % E elements
  const uint64_t tail = units * E + threadIdx.x;
  if (blockIdx.x == gridDim.x - 1 && tail < a.count) {
    using OAcc = typename Elem<OutT>::Acc;
    const auto v = static_cast<const typename Elem<InT>::Raw*>(a.send)[tail];
    static_cast<typename Elem<OutT>::Raw*>(a.recv)[tail] = Elem<OutT>::down(scaled<OutT>(static_cast<OAcc>(Elem<InT>::up(v)), a));
  }
}

// Any alignment: vectors of at most 16 bytes where a buffer allows it, single elements otherwise.
template <typename InT, typename OutT>
__global__ void __launch_bounds__(kLocalThreads) local_kernel(const __grid_constant__ LocalArgs a) {
  constexpr int VW = kUnitElems<InT, OutT> / 2;
  constexpr int U = 4;
  const bool in_al = vec_aligned<InT, VW>(a.send), out_al = vec_aligned<OutT, VW>(a.recv);
  const uint64_t nvec = (a.count + VW - 1) / VW;
  constexpr uint64_t kTile = uint64_t(kLocalThreads) * U;
  for (uint64_t t0 = blockIdx.x * kTile; t0 < nvec; t0 += gridDim.x * kTile) {
    typename Elem<InT>::Acc x[U][VW];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t v = t0 + u * kLocalThreads + threadIdx.x;
      if (v < nvec) load_vec<InT, VW>(a.send, v * VW, a.count, in_al, x[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t v = t0 + u * kLocalThreads + threadIdx.x;
      if (v >= nvec) continue;
      typename Elem<OutT>::Acc y[VW];
#pragma unroll
      for (int k = 0; k < VW; ++k) y[k] = scaled<OutT>(static_cast<typename Elem<OutT>::Acc>(x[u][k]), a);
      store_vec<OutT, VW>(a.recv, v * VW, a.count, out_al, y);
    }
  }
}

template <typename InT, typename OutT>
cudaError_t fire_local(const LocalArgs& a, int max_blocks, cudaStream_t stream) {
  constexpr int E = kUnitElems<InT, OutT>;
  // two units per thread in flight for a plain copy; a cast has half the bytes on one side and takes four
  // (bf16 -> fp32, 13.1 M elements: two take 2 % longer than four, one 4 %)
  constexpr int U = std::is_same<InT, OutT>::value ? 2 : 4;
  constexpr uintptr_t in_mask = E * sizeof(typename Elem<InT>::Raw) - 1, out_mask = E * sizeof(typename Elem<OutT>::Raw) - 1;
  const bool wide = (reinterpret_cast<uintptr_t>(a.send) & in_mask) == 0 && (reinterpret_cast<uintptr_t>(a.recv) & out_mask) == 0;
  const uint64_t per_block = wide ? uint64_t(kLocalThreads) * U * E : uint64_t(kLocalThreads) * 4 * (E / 2);
  uint64_t blocks = (a.count + per_block - 1) / per_block;
  if (max_blocks > 0 && blocks > static_cast<uint64_t>(max_blocks)) blocks = max_blocks;
  if (blocks > 0x7fffffffull) blocks = 0x7fffffffull;
  if (wide) local_wide_kernel<InT, OutT, U><<<static_cast<unsigned>(blocks), kLocalThreads, 0, stream>>>(a);
  else local_kernel<InT, OutT><<<static_cast<unsigned>(blocks), kLocalThreads, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace
}  // namespace dev

bool local_kernel_exists(DType in, DType out) {
  if (in == out) return true;
  return (in == DType::Float32 && out == DType::Bfloat16) || (in == DType::Bfloat16 && out == DType::Float32);
}

cudaError_t launch_local(DType in, DType out, const LocalArgs& a, int max_blocks, cudaStream_t stream) {
  using namespace dev;
  if (a.count == 0) return cudaSuccess;
  if (in == out) {
    switch (in) {
      case DType::Int8: case DType::Uint8: return fire_local<uint8_t, uint8_t>(a, max_blocks, stream);  // one rank: bytes move as they are
      case DType::Int32: case DType::Uint32: return fire_local<uint32_t, uint32_t>(a, max_blocks, stream);
      case DType::Int64: case DType::Uint64: return fire_local<uint64_t, uint64_t>(a, max_blocks, stream);
      case DType::Float16: return fire_local<__half, __half>(a, max_blocks, stream);
      case DType::Float32: return fire_local<float, float>(a, max_blocks, stream);
      case DType::Float64: return fire_local<double, double>(a, max_blocks, stream);
      case DType::Bfloat16: return fire_local<__nv_bfloat16, __nv_bfloat16>(a, max_blocks, stream);
    }
  }
  if (in == DType::Float32 && out == DType::Bfloat16) return fire_local<float, __nv_bfloat16>(a, max_blocks, stream);
  if (in == DType::Bfloat16 && out == DType::Float32) return fire_local<__nv_bfloat16, float>(a, max_blocks, stream);
  return cudaErrorInvalidDeviceFunction;
}

}  // namespace mnccl
