// Interface of the GEMM for small products (gemm_small.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace mnccl {
namespace gemm {

struct SmallArgs {
  int M, N, K;
  void* c;
  int ldc;
  int tiles_n;        // 128-row tiles of B
  int kb_per_slice;   // ring stages' worth of K per CTA of a cluster
  uint32_t* err;
  uint64_t wait_budget_ns;
};

struct SmallPlan {
  int tn = 0;            // rows of A per tile: 16, 32, 64 or 128
  int slices = 1;        // CTAs of a cluster that share a tile's K: 1, 2, 4 or 8
  int kb_per_slice = 0;  // in units of a ring stage's K: two k-blocks for tiles of up to 64 rows, else one
  int tiles = 0;
  bool deep = false;     // one CTA per SM with the whole shared memory as its ring, or two
};

cudaError_t launch_small(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int out /* GemmOut */,
                         const SmallPlan& p, uint32_t* err, cudaStream_t stream, std::string* why);

}  // namespace gemm
}  // namespace mnccl
