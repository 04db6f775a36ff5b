// Staged copies between pageable host memory and the device (topx_hostcopy.hpp).
#include "topx_hostcopy.hpp"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "topx_kernels.cuh"

namespace topx {

namespace {

constexpr int kCopyThreads = 4;
constexpr size_t kChunk = size_t(1) << 20;
constexpr size_t kStagedFrom = size_t(3) << 20;  // below, starting the threads costs what they save
// Making and giving back the slots takes 4 to 9 ms, and a staged copy saves about 0.07 ms a MB (100 MB to the device 9.5 ms
// through the runtime, 2.5 staged; back 6.3, 3.1): they pay from about 100 MB on.  Made after 64 MB of long copies, they
// cost a program that makes one context after another, each with a few copies, nothing.
constexpr size_t kSlotsFrom = size_t(64) << 20;

struct Slots {
  std::mutex busy;  // held by the copy that uses the slots
  std::mutex mu;    // guards the rest
  int holders = 0;
  size_t moved = 0;  // bytes of long copies through the runtime since the first holder came
  char* mem = nullptr;
} g_slots;

bool page_locked(const void* h) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, h) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type != cudaMemoryTypeUnregistered;
}

// the slots, or null while a copy of `bytes` goes through the runtime
char* slots_memory(size_t bytes) {
  std::lock_guard<std::mutex> lock(g_slots.mu);
  if (g_slots.mem || g_slots.holders == 0) return g_slots.mem;
  if (g_slots.moved < kSlotsFrom) {
    g_slots.moved += bytes;
    return nullptr;
  }
  if (cudaHostAlloc(reinterpret_cast<void**>(&g_slots.mem), kCopyThreads * 2 * kChunk, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    g_slots.mem = nullptr;
  }
  return g_slots.mem;
}

// One thread's share of a staged copy: chunks w, w + kCopyThreads, ... through its two slots.
cudaError_t share(int w, int device, char* slots, char* d, char* h, size_t bytes, bool to_device, cudaStream_t st) {
  cudaError_t e = cudaSetDevice(device);
  cudaEvent_t ev[2] = {nullptr, nullptr};
  for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
  size_t at[2] = {0, 0}, len[2] = {0, 0};  // the chunk in flight in each slot
  auto settle = [&](int s) {  // waits for slot s; a chunk from the device then goes to its place
    if (len[s] == 0 || e != cudaSuccess) return;
    e = cudaEventSynchronize(ev[s]);
    if (e == cudaSuccess && !to_device) std::memcpy(h + at[s], slots + s * kChunk, len[s]);
    len[s] = 0;
  };
  int s = 0;
  for (size_t o = size_t(w) * kChunk; o < bytes && e == cudaSuccess; o += kCopyThreads * kChunk, s ^= 1) {
    settle(s);
    if (e != cudaSuccess) break;
    const size_t n = std::min(kChunk, bytes - o);
    char* slot = slots + s * kChunk;
    if (to_device) std::memcpy(slot, h + o, n);
    e = to_device ? cudaMemcpyAsync(d + o, slot, n, cudaMemcpyHostToDevice, st)
                  : cudaMemcpyAsync(slot, d + o, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaEventRecord(ev[s], st);
    at[s] = o;
    len[s] = n;
  }
  settle(s);
  settle(s ^ 1);
  for (cudaEvent_t x : ev)
    if (x) cudaEventDestroy(x);
  return e;
}

void copy(char* d, char* h, size_t bytes, bool to_device, cudaStream_t st) {
  if (bytes >= kStagedFrom && !page_locked(h)) {
    std::unique_lock<std::mutex> lock(g_slots.busy, std::try_to_lock);
    char* mem = lock.owns_lock() ? slots_memory(bytes) : nullptr;
    if (mem) {
      int device = 0;
      TOPX_CUDA_OK(cudaGetDevice(&device));
      cudaError_t err[kCopyThreads];
      std::thread helper[kCopyThreads];
      auto part = [&](int w) { err[w] = share(w, device, mem + size_t(w) * 2 * kChunk, d, h, bytes, to_device, st); };
      int started = 1;
      try {
        for (; started < kCopyThreads; ++started) helper[started] = std::thread(part, started);
      } catch (...) {  // no more threads: their shares are done here
      }
      for (int w = started; w < kCopyThreads; ++w) part(w);
      part(0);
      for (int w = 1; w < started; ++w) helper[w].join();
      for (cudaError_t e : err) TOPX_CUDA_OK(e);
      return;
    }
  }
  TOPX_CUDA_OK(to_device ? cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st)
                         : cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, st));
  TOPX_CUDA_OK(cudaStreamSynchronize(st));
}

}  // namespace

void host_to_device(void* d, const void* h, size_t bytes, cudaStream_t st) {
  copy(static_cast<char*>(d), const_cast<char*>(static_cast<const char*>(h)), bytes, true, st);
}
void device_to_host(void* h, const void* d, size_t bytes, cudaStream_t st) {
  copy(const_cast<char*>(static_cast<const char*>(d)), static_cast<char*>(h), bytes, false, st);
}

HostCopyHold::HostCopyHold() {
  std::lock_guard<std::mutex> lock(g_slots.mu);
  ++g_slots.holders;
}
HostCopyHold::~HostCopyHold() {
  std::lock_guard<std::mutex> lock(g_slots.mu);
  if (--g_slots.holders > 0) return;
  if (g_slots.mem) cudaFreeHost(g_slots.mem);
  g_slots.mem = nullptr;
  g_slots.moved = 0;
}

}  // namespace topx
