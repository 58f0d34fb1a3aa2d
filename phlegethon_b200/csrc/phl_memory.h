// Device memory of one context.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <functional>
#include <string>
#include <unordered_map>

namespace phl {

// Every block a context holds, with its size.  A buffer's capacity is looked up by its pointer, so a
// buffer that could not be replaced has none: after a failed call its pointer is null, and nothing
// remembers the size it had.
struct DeviceMemory {
  std::unordered_map<void *, size_t> blocks;
  std::string error;  // of the last allocation that failed
  // gives up a block that the context can do without; false: there is none (any more)
  std::function<bool()> give_up;

  // a block of its own, or nullptr; the failed allocation is no error of the calls that follow
  void *get(size_t bytes) {
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e != cudaSuccess && give_up && give_up()) {
      cudaGetLastError();
      e = cudaMalloc(&p, bytes);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      error = std::string("cudaMalloc: ") + cudaGetErrorString(e);
      return nullptr;
    }
    blocks[p] = bytes;
    return p;
  }
  size_t size(const void *p) const {
    const auto b = blocks.find(const_cast<void *>(p));
    return b == blocks.end() ? 0 : b->second;
  }
  // room for `count` elements at *p, whose contents are lost when it has to grow
  template <class T>
  bool grow(T **p, size_t count) {
    const size_t bytes = sizeof(T) * (count ? count : 1);
    if (size(*p) >= bytes) return true;
    put(p);
    *p = static_cast<T *>(get(bytes));
    return *p != nullptr;
  }
  template <class T>
  void put(T **p) {
    if (*p) {
      blocks.erase(*p);
      cudaFree(*p);
    }
    *p = nullptr;
  }
  void release() {
    for (auto &b : blocks) cudaFree(b.first);
    blocks.clear();
  }
};

}  // namespace phl
