// What a call needs to know about CUDA graph capture, and memory that a captured graph owns.
//
// A captured call keeps the addresses it was captured with, and its graph may be replayed on any stream beside
// later calls.  So device memory that calls share is never captured: a captured call gets memory of its own, held
// until the graph and everything instantiated from it is gone (a CUDA user object of the graph says when).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <memory>

namespace mnccl {

struct CaptureInfo {
  bool active = false;
  unsigned long long id = 0;      // unique per capture
  cudaGraph_t graph = nullptr;    // being captured into; owned by the capture
};

inline CaptureInfo capture_info(cudaStream_t stream) {
  CaptureInfo c;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamGetCaptureInfo_v2(stream, &st, &c.id, &c.graph, nullptr, nullptr) != cudaSuccess) (void)cudaGetLastError();
  c.active = st == cudaStreamCaptureStatusActive;
  return c;
}

// Allocations of this thread are allowed, and stay out of the graph, while any thread captures.
class AllowAllocationsWhileCapturing {
 public:
  AllowAllocationsWhileCapturing() { exchange(); }
  ~AllowAllocationsWhileCapturing() { exchange(); }
  AllowAllocationsWhileCapturing(const AllowAllocationsWhileCapturing&) = delete;
  AllowAllocationsWhileCapturing& operator=(const AllowAllocationsWhileCapturing&) = delete;

 private:
  void exchange() {
    if (cudaThreadExchangeStreamCaptureMode(&mode_) != cudaSuccess) (void)cudaGetLastError();
  }
  cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// Clears *held when `graph` and every executable graph made from it has been destroyed and has finished.  On
// failure *held is clear on return.
inline bool hold_while_graph_lives(cudaGraph_t graph, const std::shared_ptr<std::atomic<bool>>& held) {
  // (no CUDA call is allowed inside the destructor of a user object: it only clears the flag)
  auto* ref = new std::shared_ptr<std::atomic<bool>>(held);
  cudaUserObject_t object = nullptr;
  const cudaHostFn_t let_go = [](void* p) {
    auto* r = static_cast<std::shared_ptr<std::atomic<bool>>*>(p);
    (*r)->store(false, std::memory_order_release);
    delete r;
  };
  held->store(true, std::memory_order_relaxed);
  if (cudaUserObjectCreate(&object, ref, let_go, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
    (void)cudaGetLastError();
    let_go(ref);
    return false;
  }
  if (cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove) != cudaSuccess) {
    (void)cudaGetLastError();
    (void)cudaUserObjectRelease(object, 1);
    held->store(false, std::memory_order_release);
    return false;
  }
  return true;
}

}  // namespace mnccl
