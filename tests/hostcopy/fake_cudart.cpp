// A CUDA runtime of a few calls for copy_to_host on the CPU: two devices, one
// stream whose copies happen only when they are waited for, and counts of what
// was called and from which threads.
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>
#include <deque>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "host_copy.hpp"

namespace {

struct op {
  void* dst = nullptr;
  const void* src = nullptr;
  size_t bytes = 0;
  cudaEvent_t event = nullptr;
};

std::recursive_mutex mu;
std::deque<op> stream;
std::set<cudaEvent_t> reached;
std::thread::id caller;
int device = 0, allocs = 0, frees = 0, events = 0, foreign = 0, staged = 0, fail_event = -1, waits = 0;
void* pinned = nullptr;

void seen() {
  if (std::this_thread::get_id() != caller) ++foreign;
}
void run_until(cudaEvent_t e) {
  while (!stream.empty()) {
    const op o = stream.front();
    stream.pop_front();
    if (o.bytes) std::memcpy(o.dst, o.src, o.bytes);
    if (o.event) reached.insert(o.event);
    if (e && o.event == e) return;
  }
}

}  // namespace

#define FAKE(name) \
  std::lock_guard<std::recursive_mutex> lock(mu); \
  seen()

extern "C" {

cudaError_t cudaGetDevice(int* d) {
  FAKE();
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  FAKE();
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
  FAKE();
  if (pinned && dst >= pinned && dst < static_cast<char*>(pinned) + (8u << 20)) ++staged;
  std::memset(dst, 0xA5, n);  // what an early reader would find
  stream.push_back(op{dst, src, n, nullptr});
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  FAKE();
  run_until(nullptr);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  FAKE();
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  FAKE();
  ++allocs;
  *p = pinned = ::operator new(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  FAKE();
  ++frees;
  ::operator delete(p);
  pinned = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  FAKE();
  ++events;
  *e = reinterpret_cast<cudaEvent_t>(new int(device));
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  FAKE();
  --events;
  delete reinterpret_cast<int*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  FAKE();
  if (*reinterpret_cast<int*>(e) != device) return cudaErrorInvalidResourceHandle;  // another device's event
  reached.erase(e);
  stream.push_back(op{nullptr, nullptr, 0, e});
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  FAKE();
  if (waits++ == fail_event) return cudaErrorUnknown;
  if (!reached.count(e)) run_until(e);
  return reached.count(e) ? cudaSuccess : cudaErrorUnknown;
}
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}

// ---- the test's side
int test_copy(void* dst, const void* src, size_t bytes, int dev, int fail) {
  {
    std::lock_guard<std::recursive_mutex> lock(mu);
    caller = std::this_thread::get_id();
    device = dev;
    waits = 0;
    fail_event = fail;
  }
  return plato_b200::copy_to_host(dst, src, bytes, nullptr);
}
void* test_user() {
  caller = std::this_thread::get_id();
  return new plato_b200::host_copy_user();
}
void test_user_gone(void* u) {
  caller = std::this_thread::get_id();
  delete static_cast<plato_b200::host_copy_user*>(u);
}
// pinned blocks taken, given back, events alive, CUDA calls of other threads, chunks staged
void test_counts(int* out) {
  const int c[5] = {allocs, frees, events, foreign, staged};
  std::memcpy(out, c, sizeof(c));
}

}  // extern "C"
