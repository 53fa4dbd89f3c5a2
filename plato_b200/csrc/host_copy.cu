// Device to host copies of result vectors.
//
// A caller's result buffer is usually pageable (a numpy array, a vector); the
// driver stages such a copy through its own pinned memory with one thread,
// about 9 GB/s, and a V-sized result then costs more than many of the
// algorithms.  copy_to_host stages it itself: the device writes pinned chunks
// at the link's rate, and several host threads move finished chunks to the
// caller while later ones arrive.  The staging memory is one block per process
// (kHalves * kHalfBytes, portable: every device's copies use it), used by one
// call at a time; a call that finds it busy, a small result and a caller's
// pinned buffer take the plain copy.  Pinning the block costs 2-8 ms, as much as
// staging saves on some 50 MB, so the first kBefore bytes go the plain way: a
// program that takes one result from each graph does not pay for the block (first
// call at RMAT s22, 9.6 MB: 11.4 ms with the block, 8.0 without).  It is freed
// with the last graph.
//
// The other host threads only move bytes.  Whatever they call of the CUDA
// runtime would use their own current device, and set it up if it is not the
// caller's.
#include <omp.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>

#include "common.cuh"
#include "host_copy.hpp"

namespace plato_b200 {
namespace {

constexpr size_t kChunk = 256u << 10, kHalfBytes = 4u << 20, kHalves = 2;
constexpr size_t kChunks = kHalfBytes / kChunk;
constexpr size_t kSmall = 1u << 20;  // below, waking the threads costs more than they save
constexpr size_t kBefore = 4u << 20;
constexpr int kThreads = 8;
constexpr int kDevices = 64;

struct staging {
  std::mutex mu;  // held by the copy that uses the block
  unsigned char* p = nullptr;
  size_t before = 0;  // bytes that went the plain way
  cudaEvent_t* done[kDevices] = {};  // [kHalves * kChunks] of a device
  void release() {
    for (cudaEvent_t*& d : done) {
      for (size_t i = 0; d && i < kHalves * kChunks; ++i)
        if (d[i]) cudaEventDestroy(d[i]);
      delete[] d;
      d = nullptr;
    }
    if (p) cudaFreeHost(p);
    p = nullptr;
    before = 0;
  }
  // The events of device `dev`, or null: no block (yet), take the plain copy.
  cudaEvent_t* ready(int dev, size_t bytes) {
    if (dev < 0 || dev >= kDevices) return nullptr;
    if (!p) {
      if (before < kBefore) {
        before += bytes;
        return nullptr;
      }
      if (cudaHostAlloc(reinterpret_cast<void**>(&p), kHalves * kHalfBytes, cudaHostAllocPortable) != cudaSuccess) {
        p = nullptr;
        cudaGetLastError();
        return nullptr;
      }
    }
    if (!done[dev]) {
      cudaEvent_t* d = new (std::nothrow) cudaEvent_t[kHalves * kChunks]();
      bool ok = d != nullptr;
      for (size_t i = 0; ok && i < kHalves * kChunks; ++i)
        ok = cudaEventCreateWithFlags(&d[i], cudaEventDisableTiming) == cudaSuccess;
      if (!ok) {
        cudaGetLastError();
        for (size_t i = 0; d && i < kHalves * kChunks; ++i)
          if (d[i]) cudaEventDestroy(d[i]);
        delete[] d;
        return nullptr;
      }
      done[dev] = d;
    }
    return done[dev];
  }
};

staging g_stage;
std::mutex g_users_mu;
int g_users = 0;

int plain_copy(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  PLATO_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
  PLATO_CUDA_TRY(cudaStreamSynchronize(st));
  return PLATO_OK;
}

bool pageable(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace

host_copy_user::host_copy_user() {
  std::lock_guard<std::mutex> lock(g_users_mu);
  ++g_users;
}

host_copy_user::~host_copy_user() {
  std::lock_guard<std::mutex> lock(g_users_mu);
  if (--g_users == 0) {
    std::lock_guard<std::mutex> stage(g_stage.mu);
    g_stage.release();
  }
}

int copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (bytes == 0) {
    PLATO_CUDA_TRY(cudaStreamSynchronize(st));
    return PLATO_OK;
  }
  if (bytes < kSmall || !pageable(dst)) return plain_copy(dst, src, bytes, st);
  std::unique_lock<std::mutex> lock(g_stage.mu, std::try_to_lock);
  int dev = 0;
  PLATO_CUDA_TRY(cudaGetDevice(&dev));
  cudaEvent_t* const done = lock.owns_lock() ? g_stage.ready(dev, bytes) : nullptr;
  if (!done) {
    if (lock.owns_lock()) lock.unlock();
    return plain_copy(dst, src, bytes, st);
  }
  unsigned char* out = static_cast<unsigned char*>(dst);
  const unsigned char* in = static_cast<const unsigned char*>(src);
  // part `k` of the result goes through half k % 2, a chunk at a time
  const size_t parts = (bytes + kHalfBytes - 1) / kHalfBytes;
  auto enqueue = [&](size_t k) -> cudaError_t {
    const size_t lo = k * kHalfBytes, hi = std::min(bytes, lo + kHalfBytes);
    for (size_t c = lo, i = (k % kHalves) * kChunks; c < hi; c += kChunk, ++i) {
      cudaError_t e = cudaMemcpyAsync(g_stage.p + (k % kHalves) * kHalfBytes + (c - lo), in + c,
                                      std::min(kChunk, hi - c), cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaEventRecord(done[i], st);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  };
  cudaError_t err = cudaSuccess;
  for (size_t k = 0; k < std::min(kHalves, parts) && err == cudaSuccess; ++k) err = enqueue(k);
  const int threads = std::max(1, std::min(kThreads, omp_get_max_threads()));
  for (size_t k = 0; k < parts && err == cudaSuccess; ++k) {
    const size_t lo = k * kHalfBytes, hi = std::min(bytes, lo + kHalfBytes);
    const int n = static_cast<int>((hi - lo + kChunk - 1) / kChunk);
    const cudaEvent_t* arrived = done + (k % kHalves) * kChunks;
    const unsigned char* half = g_stage.p + (k % kHalves) * kHalfBytes;
    auto move = [&](int i) {
      const size_t at = static_cast<size_t>(i) * kChunk;
      std::memcpy(out + lo + at, half + at, std::min(kChunk, hi - lo - at));
    };
    // This thread waits for the chunks one after another, the others take what has
    // arrived; the wait for the work before the first chunk is this thread's alone.
    err = cudaEventSynchronize(arrived[0]);
    if (err != cudaSuccess) break;
    std::atomic<int> next{0}, in_memory{1};  // chunks taken, chunks there (n + 1: give up)
#pragma omp parallel num_threads(threads)
    {
      if (omp_get_thread_num() == 0)
        for (int i = 1; i < n; ++i) {
          if (omp_get_num_threads() == 1) move(next.fetch_add(1));
          err = cudaEventSynchronize(arrived[i]);
          in_memory.store(err == cudaSuccess ? i + 1 : n + 1, std::memory_order_release);
          if (err != cudaSuccess) break;
        }
      for (int i = next.fetch_add(1); i < n; i = next.fetch_add(1)) {
        int there;
        while ((there = in_memory.load(std::memory_order_acquire)) <= i) std::this_thread::yield();
        if (there > n) break;
        move(i);
      }
    }
    if (err == cudaSuccess && k + kHalves < parts) err = enqueue(k + kHalves);
  }
  const cudaError_t sync = cudaStreamSynchronize(st);  // also before the block is given back after an error
  if (err == cudaSuccess) err = sync;
  if (err != cudaSuccess)
    return set_error(PLATO_ECUDA, std::string("copy of a result to the host failed: ") + cudaGetErrorString(err));
  return PLATO_OK;
}

}  // namespace plato_b200
