// spiffe_b200/csrc/slab.hpp -- device memory of the instances (devmem.cu), and
// several arrays in one allocation.
#pragma once

#include <cstddef>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

cudaError_t spiffe_dev_malloc(void **p, size_t bytes);
cudaError_t spiffe_dev_free(void *p);
cudaError_t spiffe_pinned_malloc(void **p, size_t bytes);
cudaError_t spiffe_pinned_free(void *p);

// in place of cudaMalloc and cudaFree, with their meaning
template <typename T> inline cudaError_t dev_malloc(T **p, size_t bytes) { return spiffe_dev_malloc((void **)p, bytes); }
inline cudaError_t dev_free(void *p) { return spiffe_dev_free(p); }

// Arrays that live and go together in one allocation: add() names them, each
// on a 256-byte boundary; make() allocates them.  The first array's pointer is
// the allocation's: it alone is freed.
class DeviceSlab {
  std::vector<std::pair<void **, size_t>> parts_; // pointer, offset
  size_t bytes_ = 0;

public:
  template <typename T> void add(T **p, size_t n)
  {
    parts_.emplace_back((void **)p, bytes_);
    bytes_ += (n * sizeof(T) + 255) / 256 * 256;
  }
  size_t bytes() const { return bytes_; }
  cudaError_t make()
  {
    char *base = nullptr;
    const cudaError_t e = dev_malloc(&base, bytes_);
    for (auto &part : parts_)
      *part.first = e == cudaSuccess ? base + part.second : nullptr;
    return e;
  }
};
