// See noalloc.h: an AllReduce over several buffers of one GPU that allocates nothing.
//
// All buffers lie in one GPU's memory, so nothing has to be pushed, signalled or waited for: a thread loads
// 16 bytes of every buffer, adds them in buffer order and stores the result to every destination.  At
// these sizes (at most 4 x 64 KiB in and out) the call is launch latency: one ordinary launch with the
// pointers by value, no clearing of state, every load of a thread in flight before the first add.
// 4 x 64 KiB fp32, per call through ctypes: 17.4 us as a cooperative launch of the inbox kernel behind four
// memsets, 8.0 now, of which 1.9 are device time.
#include "kernels/noalloc.h"

#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>

#include "core/dtype.h"
#include "kernels/dev_prims.cuh"

namespace mnccl {
namespace {

constexpr int kThreads = 128;  // 64 KiB: 4096 vectors, 32 blocks

// Outcome of the last call on this GPU: {status, detail}.  Nothing in the kernel can fail, so a call leaves zeros; kept
// because mncclNoAllocLastStatus is part of the interface.
static __device__ unsigned g_outcome[2];

struct LocalSumParams {
  const void* send[kNoAllocMaxRanks];
  void* recv[kNoAllocMaxRanks];
  CollArgs args;   // count, scale_f, int_div
};

template <typename T, int OP>
__global__ void __launch_bounds__(kThreads) local_sum_kernel(const __grid_constant__ LocalSumParams p, int nbuffers) {
  using namespace dev;
  using Acc = typename Elem<T>::Acc;
  constexpr int VW = 16 / sizeof(typename Elem<T>::Raw);
  const uint64_t i0 = (uint64_t(blockIdx.x) * kThreads + threadIdx.x) * VW;
  if (blockIdx.x == 0 && threadIdx.x < 2) g_outcome[threadIdx.x] = 0;
  if (i0 >= p.args.count) return;
  Acc x[kNoAllocMaxRanks][VW];
#pragma unroll
  for (int r = 0; r < kNoAllocMaxRanks; ++r)
    if (r < nbuffers) load_vec<T, VW>(p.send[r], i0, p.args.count, is_aligned16(p.send[r]), x[r]);
#pragma unroll
  for (int r = 1; r < kNoAllocMaxRanks; ++r) {
    if (r >= nbuffers) break;
#pragma unroll
    for (int k = 0; k < VW; ++k) x[0][k] = combine<OP>(x[0][k], x[r][k]);
  }
#pragma unroll
  for (int k = 0; k < VW; ++k) x[0][k] = finalize<T>(x[0][k], p.args);
#pragma unroll
  for (int r = 0; r < kNoAllocMaxRanks; ++r)
    if (r < nbuffers) store_vec<T, VW>(p.recv[r], i0, p.args.count, is_aligned16(p.recv[r]), x[0]);
}

template <typename T>
cudaError_t launch_typed(int op, const LocalSumParams& p, int nbuffers, cudaStream_t stream) {
  constexpr int VW = 16 / sizeof(typename dev::Elem<T>::Raw);
  const unsigned blocks = static_cast<unsigned>((p.args.count + VW * kThreads - 1) / (VW * kThreads));
  switch (op) {
    case 0: local_sum_kernel<T, 0><<<blocks, kThreads, 0, stream>>>(p, nbuffers); break;
    case 1: local_sum_kernel<T, 1><<<blocks, kThreads, 0, stream>>>(p, nbuffers); break;
    case 2: local_sum_kernel<T, 2><<<blocks, kThreads, 0, stream>>>(p, nbuffers); break;
    case 3: local_sum_kernel<T, 3><<<blocks, kThreads, 0, stream>>>(p, nbuffers); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace

// Fills the outcome record with `byte`; the next call must not care.  Not exported: reached through the
// test-suite's own library only (csrc/testing/hooks.cc).
int noalloc_dirty_control(int byte) {
  unsigned words[2];
  memset(words, byte, sizeof(words));
  if (cudaMemcpyToSymbol(g_outcome, words, sizeof(words)) != cudaSuccess) return 1;
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 3;
}

}  // namespace mnccl

using namespace mnccl;

extern "C" {
#define MNCCL_EXPORT __attribute__((visibility("default")))

MNCCL_EXPORT size_t mncclNoAllocScratchBytes(void) { return sizeof(g_outcome); }

MNCCL_EXPORT ncclResult_t mncclNoAllocLastStatus(cudaStream_t stream, unsigned* status, unsigned* detail) {
  if (!status) return ncclInvalidArgument;
  unsigned words[2] = {0, 0};
  cudaError_t e = cudaStreamSynchronize(stream);
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(words, g_outcome, sizeof(words));
  *status = words[0];
  if (detail) *detail = words[1];
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return ncclUnhandledCudaError;
  }
  return ncclSuccess;
}

MNCCL_EXPORT ncclResult_t mncclLocalAllReduceNoAlloc(const void* const* send, void* const* recv, int nbuffers,
                                                     size_t count, ncclDataType_t datatype, ncclRedOp_t op,
                                                     cudaStream_t stream) {
  if (!send || !recv) return ncclInvalidArgument;
  if (nbuffers < 2 || nbuffers > kNoAllocMaxRanks) {
    fprintf(stderr, "[Mini-NCCL] mncclLocalAllReduceNoAlloc: %d buffers requested, supported: 2..%d\n", nbuffers,
            static_cast<int>(kNoAllocMaxRanks));
    return ncclInvalidArgument;
  }
  if (!valid_dtype(datatype) || !valid_op(op)) return ncclInvalidArgument;
  const DType t = static_cast<DType>(datatype);
  if (t != DType::Float32 && t != DType::Float16 && t != DType::Bfloat16 && t != DType::Int32) {
    fprintf(stderr, "[Mini-NCCL] mncclLocalAllReduceNoAlloc: type %s is not supported (fp32, fp16, bf16, int32 are)\n",
            dtype_name(t));
    return ncclInvalidArgument;
  }
  if (count == 0) return ncclSuccess;
  const size_t bytes = count * dtype_size(t);
  if (bytes > kNoAllocMaxBytes) {
    fprintf(stderr, "[Mini-NCCL] mncclLocalAllReduceNoAlloc: %zu bytes per buffer exceed the limit (%d bytes)\n",
            bytes, static_cast<int>(kNoAllocMaxBytes));
    return ncclInvalidArgument;
  }
  LocalSumParams p;
  memset(&p, 0, sizeof(p));
  for (int r = 0; r < nbuffers; ++r) {
    if (!send[r] || !recv[r]) return ncclInvalidArgument;
    p.send[r] = send[r];
    p.recv[r] = recv[r];
  }
  const double factor = (op == ncclAvg) ? 1.0 / nbuffers : 1.0;
  p.args.count = count;
  p.args.scale_f = static_cast<float>(factor);
  p.args.scale_d = factor;
  p.args.int_div = (op == ncclAvg && t == DType::Int32) ? nbuffers : 0;
  const int opi = (op == ncclAvg) ? 0 : static_cast<int>(op);
  cudaError_t e;
  switch (t) {
    case DType::Float32: e = launch_typed<float>(opi, p, nbuffers, stream); break;
    case DType::Float16: e = launch_typed<__half>(opi, p, nbuffers, stream); break;
    case DType::Bfloat16: e = launch_typed<__nv_bfloat16>(opi, p, nbuffers, stream); break;
    default: e = launch_typed<int32_t>(opi, p, nbuffers, stream); break;
  }
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    fprintf(stderr, "[Mini-NCCL] mncclLocalAllReduceNoAlloc: launch failed: %s\n", cudaGetErrorString(e));
    return ncclUnhandledCudaError;
  }
  return ncclSuccess;
}

}  // extern "C"
