// The fused kernels with one rank, for the test-suite only (csrc/testing/hooks.cc).  The entry points of
// mini_nccl_ops.h leave a single rank to the plain GEMM, so on one GPU nothing else launches them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mnccl {
namespace gemm {

// GEMM -> reduce-scatter through staging, tile flags and the reduction pass.  Buffers as for
// mncclGemmReduceScatterBf16, dense operands.
int gemm_rs_fused_one_rank(const void* A, const void* B, void* out, int M, int N, int K, void* stage, void* flags, uint32_t* state,
                           cudaStream_t stream);

// all-gather -> GEMM with its communication CTAs, which have nobody to push to.  Every row block is treated as one that
// a peer delivers: its counter in `ready` has to have reached 4 x the number of the call.
int ag_gemm_fused_one_rank(void* xg, const void* B, void* C, int M, int N, int K, void* ready, void* bar, uint32_t* state, bool swiglu,
                           cudaStream_t stream);

}  // namespace gemm
}  // namespace mnccl
