// Results to the caller's host memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace plato_b200 {

// Copies `bytes` of device memory at `src` to host memory at `dst` behind the
// work of `st`, and waits for it.
int copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t st);

// The staging memory of copy_to_host exists while a graph does.
struct host_copy_user {
  host_copy_user();
  ~host_copy_user();
  host_copy_user(const host_copy_user&) = delete;
  host_copy_user& operator=(const host_copy_user&) = delete;
};

}  // namespace plato_b200
