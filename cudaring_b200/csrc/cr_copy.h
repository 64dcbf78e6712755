// Host copies of the setters and getters.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace cr {

// Pinned chunks of one context, made for its first large copy and freed with
// it: two per worker thread.
struct Staging {
  static constexpr int kWorkers = 4;
  static constexpr size_t kChunk = (size_t)1 << 20;
  unsigned char* buf = nullptr;  // [kWorkers][2][kChunk]
  bool failed = false;           // pinned memory or events could not be had: plain copies
  cudaEvent_t ready[kWorkers][2] = {};
  ~Staging();
};

// Synchronous copies between host memory and the device on stream st.  Copies
// of 8 MB and more from or to pageable memory go through pinned chunks, four
// threads at a time: one thread's copy to fresh pages runs at 4.5 GB/s (40 MB:
// 9 ms), most of it page faults.
cudaError_t copy_in(Staging& s, int device, cudaStream_t st, void* dst, const void* src, size_t bytes);
cudaError_t copy_out(Staging& s, int device, cudaStream_t st, void* dst, const void* src, size_t bytes);

}  // namespace cr
