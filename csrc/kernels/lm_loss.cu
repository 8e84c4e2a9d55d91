// Cross-entropy over bf16 logits [T, V] of a language-model head, forward and backward, and the transposes its
// GEMMs need.
//
// What bounds it is memory: 8192 x 50257 logits are 0.82 GB.  As separate operators (a copy to fp32, log-softmax,
// its gradient in fp32, a copy back to bf16) they moved 10.7 GB and took 3.9 ms.  Here the forward pass reads
// the logits once and keeps one fp32 word per row, and the backward pass reads them once more and writes the
// gradient in bf16 twice, as [T, V] and as [V, T]: the layouts in which the two products that follow (gradient of
// the activations, gradient of the weight) have their summation index innermost, which is what the GEMM loads.
// Everything between the bf16 logits and the one rounding of the gradient is fp32.  Rows are padded to a multiple
// of eight elements in memory, so that every access is 16 bytes wide whatever V and T are; what lies in the padding of
// the logits is never used.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace {

constexpr int64_t kIgnore = -100;   // rows with this target count for nothing
constexpr int kRowThreads = 256;
constexpr int kBatch = 4;           // 16-byte loads of a thread in flight

__device__ __forceinline__ void unpack(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ uint32_t pack(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}

// exp(m - of) where m may be -inf (nothing seen yet): 0 instead of exp(-inf + inf).
__device__ __forceinline__ float rescale(float m, float of) { return m == -INFINITY ? 0.0f : expf(m - of); }

__device__ __forceinline__ void merge(float& m, float& s, float m2, float s2) {
  const float top = fmaxf(m, m2);
  s = s * rescale(m, top) + s2 * rescale(m2, top);
  m = top;
}

// One block per row: running maximum and sum of exponentials, then lse = max + log(sum) and the row's loss
// lse - logit[target].  A NaN or +inf logit makes the sum NaN, a row of -inf makes the loss NaN.
__global__ void __launch_bounds__(kRowThreads)
loss_rows_kernel(const __nv_bfloat16* __restrict__ logits, size_t ld, int V, const int64_t* __restrict__ targets,
                 const __nv_bfloat16* __restrict__ picked, float* __restrict__ lse, float* __restrict__ row_loss) {
  const size_t t = blockIdx.x;
  const uint4* row = reinterpret_cast<const uint4*>(logits + t * ld);
  const int nvec = (V + 7) / 8;
  float m = -INFINITY, s = 0.0f;
  for (int v0 = threadIdx.x; v0 < nvec; v0 += kBatch * kRowThreads) {
    uint4 raw[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int v = v0 + b * kRowThreads;
      if (v < nvec) raw[b] = __ldg(row + v);
    }
    float f[kBatch][8], top = m;
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int c = (v0 + b * kRowThreads) * 8;
      if (c < V) unpack(raw[b], f[b]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (c + j >= V) f[b][j] = -INFINITY;
        top = fmaxf(top, f[b][j]);
      }
    }
    s *= rescale(m, top);
    m = top;
    const float base = top == -INFINITY ? 0.0f : top;
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
#pragma unroll
      for (int j = 0; j < 8; ++j) s += expf(f[b][j] - base);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
    merge(m, s, __shfl_xor_sync(0xffffffffu, m, d), __shfl_xor_sync(0xffffffffu, s, d));
  __shared__ float sm[kRowThreads / 32], ss[kRowThreads / 32];
  if ((threadIdx.x & 31) == 0) {
    sm[threadIdx.x >> 5] = m;
    ss[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kRowThreads / 32; ++w) merge(m, s, sm[w], ss[w]);
    const float l = m + logf(s);
    lse[t] = l;
    row_loss[t] = targets[t] == kIgnore ? 0.0f : l - __bfloat162float(picked[t]);
  }
}

// Mean over the rows that count, in one block and a fixed order: out = {mean, number of such rows}.
__global__ void __launch_bounds__(1024)
loss_mean_kernel(const float* __restrict__ row_loss, const int64_t* __restrict__ targets, int T, float* __restrict__ out) {
  float s = 0.0f;
  int n = 0;
  for (int t = threadIdx.x; t < T; t += 1024) {
    if (targets[t] == kIgnore) continue;
    s += row_loss[t];
    ++n;
  }
  __shared__ float ss[32];
  __shared__ int sn[32];
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, d);
      n += __shfl_xor_sync(0xffffffffu, n, d);
    }
    if (pass == 0) {
      if ((threadIdx.x & 31) == 0) {
        ss[threadIdx.x >> 5] = s;
        sn[threadIdx.x >> 5] = n;
      }
      __syncthreads();
      s = ss[threadIdx.x & 31];
      n = sn[threadIdx.x & 31];
    }
  }
  if (threadIdx.x == 0) {
    out[0] = s / static_cast<float>(n);
    out[1] = static_cast<float>(n);
  }
}

// 64 x 64 tiles, 256 threads: a thread takes eight columns of two neighbouring rows, so two elements of a column
// share a word of the tile in shared memory, [column][row pair].  33 words per column: reads of whole columns
// hit 32 banks, writes two lanes per bank.
constexpr int kTile = 64, kTileThreads = 256, kPitch = kTile / 2 + 1;

__device__ __forceinline__ void put_pair(uint32_t* tile, int col, int pair, const float (&a)[8], const float (&b)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) tile[(col + j) * kPitch + pair] = pack(a[j], b[j]);
}

// Columns of the tile out as rows of `dst` [cols, ld], 128 bytes each.
__device__ __forceinline__ void store_transposed(const uint32_t* tile, __nv_bfloat16* dst, size_t ld, int row0, int col0, int rows,
                                                 int cols) {
  const int r = (threadIdx.x & 7) * 8;
  if (row0 + r >= rows) return;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = static_cast<int>(threadIdx.x >> 3) + i * 32;
    if (col0 + c >= cols) continue;
    const uint32_t* w = tile + c * kPitch + r / 2;
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(col0 + c) * ld + row0 + r) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// d = (softmax(logits) - onehot(target)) * grad / count, 0 for rows that count for nothing; written as [T, V] where
// `d` is given and as [V, T] where `dt` is.
__global__ void __launch_bounds__(kTileThreads)
loss_grad_kernel(const __nv_bfloat16* __restrict__ logits, size_t ld, int T, int V, const int64_t* __restrict__ targets,
                 const float* __restrict__ lse, const float* __restrict__ grad, const float* __restrict__ mean,
                 __nv_bfloat16* __restrict__ d, size_t ldd, __nv_bfloat16* __restrict__ dt, size_t ldt) {
  __shared__ uint32_t tile[kTile * kPitch];
  const int col0 = blockIdx.x * kTile, row0 = blockIdx.y * kTile;
  const int c = (threadIdx.x & 7) * 8, pair = threadIdx.x >> 3;
  const float g = grad[0] / mean[1];
  float f[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = row0 + 2 * pair + i, v = col0 + c;
    const bool inside = t < T && v < V;
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (inside) raw = __ldg(reinterpret_cast<const uint4*>(logits + static_cast<size_t>(t) * ld + v));
    const int64_t target = inside ? targets[t] : kIgnore;
    const float l = inside ? lse[t] : 0.0f, factor = target == kIgnore ? 0.0f : g;
    unpack(raw, f[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[i][j] = (expf(f[i][j] - l) - (target == v + j ? 1.0f : 0.0f)) * factor;
    if (d != nullptr && inside)
      *reinterpret_cast<uint4*>(d + static_cast<size_t>(t) * ldd + v) =
          make_uint4(pack(f[i][0], f[i][1]), pack(f[i][2], f[i][3]), pack(f[i][4], f[i][5]), pack(f[i][6], f[i][7]));
  }
  if (dt == nullptr) return;
  put_pair(tile, c, pair, f[0], f[1]);
  __syncthreads();
  store_transposed(tile, dt, ldt, row0, col0, T, V);
}

// dst[cols, ldd] = src[rows, lds]^T; a row of dst is written up to the next multiple of eight elements.
__global__ void __launch_bounds__(kTileThreads)
transpose_kernel(const __nv_bfloat16* __restrict__ src, size_t lds, int rows, int cols, __nv_bfloat16* __restrict__ dst, size_t ldd) {
  __shared__ uint32_t tile[kTile * kPitch];
  const int col0 = blockIdx.x * kTile, row0 = blockIdx.y * kTile;
  const int c = (threadIdx.x & 7) * 8, pair = threadIdx.x >> 3;
  float f[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = row0 + 2 * pair + i;
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (r < rows && col0 + c < cols) raw = __ldg(reinterpret_cast<const uint4*>(src + static_cast<size_t>(r) * lds + col0 + c));
    unpack(raw, f[i]);
  }
  put_pair(tile, c, pair, f[0], f[1]);
  __syncthreads();
  store_transposed(tile, dst, ldd, row0, col0, rows, cols);
}

bool aligned(const void* p, int64_t ld, int64_t width) {
  return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && ld % 8 == 0 && ld >= (width + 7) / 8 * 8;
}

constexpr int kMaxTileRows = 65535 * kTile;  // gridDim.y

int status() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : static_cast<int>(e) + 1000;
}

}  // namespace

extern "C" {
#define MNCCL_EXPORT __attribute__((visibility("default")))

// Mean cross-entropy of bf16 logits [T, V] (row stride ld elements, a multiple of 8 that holds V rounded up to
// one; 16-byte aligned).  targets: T class indices, -100 = the row counts for nothing; picked[t] = the logit of
// row t's target.  Writes lse[T] for the backward pass, row_loss[T] (scratch) and mean[2] = {loss, rows that count}.
// Returns 0, a negative code for bad arguments, or a cudaError_t + 1000.
MNCCL_EXPORT int mncclLmLossForward(const void* logits, int64_t ld, int T, int V, const int64_t* targets, const void* picked,
                                    float* lse, float* row_loss, float* mean, cudaStream_t stream) {
  if (!logits || !targets || !picked || !lse || !row_loss || !mean || T <= 0 || V <= 0) return -1;
  if (!aligned(logits, ld, V)) return -2;
  loss_rows_kernel<<<static_cast<unsigned>(T), kRowThreads, 0, stream>>>(static_cast<const __nv_bfloat16*>(logits), static_cast<size_t>(ld), V,
                                                                         targets, static_cast<const __nv_bfloat16*>(picked), lse, row_loss);
  loss_mean_kernel<<<1, 1024, 0, stream>>>(row_loss, targets, T, mean);
  return status();
}

// Gradient of the above with respect to the logits, times grad[0]: d [T, V] and / or dt [V, T] (either may be
// null), row strides like ld.
MNCCL_EXPORT int mncclLmLossBackward(const void* logits, int64_t ld, int T, int V, const int64_t* targets, const float* lse,
                                     const float* grad, const float* mean, void* d, int64_t ldd, void* dt, int64_t ldt,
                                     cudaStream_t stream) {
  if (!logits || !targets || !lse || !grad || !mean || T <= 0 || V <= 0 || (!d && !dt)) return -1;
  if (!aligned(logits, ld, V) || (d && !aligned(d, ldd, V)) || (dt && !aligned(dt, ldt, T)) || T > kMaxTileRows) return -2;
  const dim3 grid((V + kTile - 1) / kTile, (T + kTile - 1) / kTile);
  loss_grad_kernel<<<grid, kTileThreads, 0, stream>>>(static_cast<const __nv_bfloat16*>(logits), static_cast<size_t>(ld), T, V, targets, lse,
                                                      grad, mean, static_cast<__nv_bfloat16*>(d), static_cast<size_t>(ldd),
                                                      static_cast<__nv_bfloat16*>(dt), static_cast<size_t>(ldt));
  return status();
}

// dst[cols, rows] = src[rows, cols]^T for bf16, both 16-byte aligned with row strides that are multiples of 8 and
// hold a row rounded up to one.
MNCCL_EXPORT int mncclTransposeBf16(const void* src, int64_t lds, int rows, int cols, void* dst, int64_t ldd, cudaStream_t stream) {
  if (!src || !dst || rows <= 0 || cols <= 0) return -1;
  if (!aligned(src, lds, cols) || !aligned(dst, ldd, rows) || rows > kMaxTileRows) return -2;
  const dim3 grid((cols + kTile - 1) / kTile, (rows + kTile - 1) / kTile);
  transpose_kernel<<<grid, kTileThreads, 0, stream>>>(static_cast<const __nv_bfloat16*>(src), static_cast<size_t>(lds), rows, cols,
                                                      static_cast<__nv_bfloat16*>(dst), static_cast<size_t>(ldd));
  return status();
}

}  // extern "C"
