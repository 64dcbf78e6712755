#include "cr_copy.h"

#include <algorithm>
#include <cstring>
#include <exception>
#include <thread>

namespace cr {
namespace {

constexpr size_t kLarge = (size_t)8 << 20;

bool prepare(Staging& s) {
  if (s.buf) return true;
  if (s.failed) return false;
  const size_t n = (size_t)Staging::kWorkers * 2 * Staging::kChunk;
  bool ok = cudaHostAlloc((void**)&s.buf, n, cudaHostAllocDefault) == cudaSuccess;
  for (int w = 0; ok && w < Staging::kWorkers; w++)
    for (int k = 0; ok && k < 2; k++)
      ok = cudaEventCreateWithFlags(&s.ready[w][k], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    if (s.buf) cudaFreeHost(s.buf);
    s.buf = nullptr;
    s.failed = true;
  }
  return ok;
}

// Worker w: chunks w, w + kWorkers, ... through its two buffers in turn.
cudaError_t worker(Staging& s, int device, cudaStream_t st, int w, unsigned char* dst, const unsigned char* src,
                   size_t bytes, bool in) {
  cudaError_t e = cudaSetDevice(device);
  unsigned char* buf = s.buf + (size_t)w * 2 * Staging::kChunk;
  const size_t step = (size_t)Staging::kWorkers * Staging::kChunk;
  size_t held[2] = {0, 0};  // offset of the chunk each buffer holds
  bool busy[2] = {false, false};
  const auto finish = [&](int k) {
    if (!busy[k]) return cudaSuccess;
    busy[k] = false;
    const cudaError_t f = cudaEventSynchronize(s.ready[w][k]);
    if (f == cudaSuccess && !in)
      std::memcpy(dst + held[k], buf + k * Staging::kChunk, std::min(Staging::kChunk, bytes - held[k]));
    return f;
  };
  int k = 0;
  for (size_t at = (size_t)w * Staging::kChunk; e == cudaSuccess && at < bytes; at += step, k ^= 1) {
    if ((e = finish(k)) != cudaSuccess) break;
    const size_t n = std::min(Staging::kChunk, bytes - at);
    unsigned char* b = buf + k * Staging::kChunk;
    if (in) std::memcpy(b, src + at, n);
    e = in ? cudaMemcpyAsync(dst + at, b, n, cudaMemcpyHostToDevice, st)
           : cudaMemcpyAsync(b, src + at, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaEventRecord(s.ready[w][k], st);
    held[k] = at;
    busy[k] = e == cudaSuccess;
  }
  for (int q = 0; q < 2; q++, k ^= 1) {
    const cudaError_t f = finish(k);
    if (e == cudaSuccess) e = f;
  }
  return e;
}

cudaError_t plain(cudaStream_t st, void* dst, const void* src, size_t bytes, bool in) {
  const cudaError_t e =
      cudaMemcpyAsync(dst, src, bytes, in ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st);
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

// The context's device for one copy, the caller's again after it: a plain copy
// runs on a stream of any device, but events belong to the device that was
// current when they were made.
struct OnDevice {
  int before = -1;
  explicit OnDevice(int device) {
    int now;
    if (cudaGetDevice(&now) != cudaSuccess || now == device) return;
    if (cudaSetDevice(device) == cudaSuccess) before = now;
  }
  ~OnDevice() {
    if (before >= 0) cudaSetDevice(before);
  }
};

cudaError_t copy(Staging& s, int device, cudaStream_t st, void* dst, const void* src, size_t bytes, bool in) {
  if (bytes < kLarge) return plain(st, dst, src, bytes, in);
  const OnDevice on(device);
  cudaPointerAttributes at{};
  const cudaError_t e = cudaPointerGetAttributes(&at, in ? src : dst);
  if (e != cudaSuccess) cudaGetLastError();
  if (e != cudaSuccess || at.type != cudaMemoryTypeUnregistered || !prepare(s)) return plain(st, dst, src, bytes, in);
  cudaError_t err[Staging::kWorkers];
  std::thread t[Staging::kWorkers];
  int started = 0;
  for (int w = 1; w < Staging::kWorkers; w++) {
    try {
      t[w] = std::thread([&, w] {
        err[w] = worker(s, device, st, w, (unsigned char*)dst, (const unsigned char*)src, bytes, in);
      });
    } catch (const std::exception&) {
      break;  // no more threads: this one takes the rest
    }
    started = w;
  }
  err[0] = worker(s, device, st, 0, (unsigned char*)dst, (const unsigned char*)src, bytes, in);
  for (int w = started + 1; w < Staging::kWorkers; w++)
    err[w] = worker(s, device, st, w, (unsigned char*)dst, (const unsigned char*)src, bytes, in);
  for (int w = 1; w <= started; w++) t[w].join();
  for (int w = 0; w < Staging::kWorkers; w++)
    if (err[w] != cudaSuccess) return err[w];
  return cudaStreamSynchronize(st);
}

}  // namespace

Staging::~Staging() {
  if (buf) cudaFreeHost(buf);
  for (auto& w : ready)
    for (cudaEvent_t e : w)
      if (e) cudaEventDestroy(e);
}

cudaError_t copy_in(Staging& s, int device, cudaStream_t st, void* dst, const void* src, size_t bytes) {
  return copy(s, device, st, dst, src, bytes, true);
}
cudaError_t copy_out(Staging& s, int device, cudaStream_t st, void* dst, const void* src, size_t bytes) {
  return copy(s, device, st, dst, src, bytes, false);
}

}  // namespace cr
