// spiffe_b200/csrc/devmem.cu -- device and pinned memory of the instances.
//
// An instance is made of a dozen blocks.  cudaMalloc takes 20 us below 1 MB,
// but 160 to 320 us from there on and cudaFree nearly as much, and four bytes
// of pinned memory 1.5 ms (B200 under a hypervisor): 7.5 of the 14 ms of a
// short served request.  So a freed block of at most KEEP_BLOCK bytes is kept
// for the next instance, up to KEEP_TOTAL bytes a device; what is larger or
// beyond goes back to the driver at once, and all of it does when an
// allocation fails.  A request's instance made again: created in
// 1.2 ms instead of 5, freed in 0.13 instead of 2.5.
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "slab.hpp"

namespace {

constexpr size_t KEEP_BLOCK = (size_t)32 << 20, KEEP_TOTAL = (size_t)256 << 20;
constexpr size_t PINNED_BLOCK = 8192, KEEP_PINNED = 64; // bytes; blocks

struct Block {
  int dev;
  size_t bytes;
};
struct Memory {
  std::mutex lock;
  std::unordered_map<void *, Block> used;               // blocks that may be kept
  std::map<int, std::multimap<size_t, void *>> idle;    // by device and size
  std::map<int, size_t> kept;                           // bytes idle on a device
  std::vector<void *> pinned;
};
Memory &memory()
{
  static Memory *m = new Memory; // outlives every instance, also one freed while the process ends
  return *m;
}

// everything idle on the device back to the driver
void trim(Memory &m, int dev)
{
  std::vector<void *> all;
  {
    std::lock_guard<std::mutex> g(m.lock);
    for (const auto &b : m.idle[dev])
      all.push_back(b.second);
    m.idle[dev].clear();
    m.kept[dev] = 0;
  }
  for (void *p : all)
    cudaFree(p);
}

} // namespace

cudaError_t spiffe_dev_malloc(void **p, size_t bytes)
{
  *p = nullptr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || bytes == 0)
    return e;
  Memory &m = memory();
  if (bytes <= KEEP_BLOCK) {
    std::lock_guard<std::mutex> g(m.lock);
    auto &idle = m.idle[dev];
    const auto it = idle.lower_bound(bytes);
    if (it != idle.end() && it->first <= bytes + bytes / 4) { // no block lies idle in a much smaller one's place
      *p = it->second;
      m.kept[dev] -= it->first;
      m.used[*p] = Block{dev, it->first};
      idle.erase(it);
      return cudaSuccess;
    }
  }
  e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    trim(m, dev);
    e = cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess)
    cudaGetLastError(); // it is returned here, and is not the next call's
  if (e == cudaSuccess && bytes <= KEEP_BLOCK) {
    std::lock_guard<std::mutex> g(m.lock);
    m.used[*p] = Block{dev, bytes};
  }
  return e;
}

cudaError_t spiffe_dev_free(void *p)
{
  if (!p)
    return cudaSuccess;
  Memory &m = memory();
  Block b{};
  {
    std::lock_guard<std::mutex> g(m.lock);
    const auto it = m.used.find(p);
    if (it != m.used.end()) {
      b = it->second;
      m.used.erase(it);
    }
  }
  if (!b.bytes)
    return cudaFree(p);
  // as cudaFree: work in flight may still use the block (also another stream's)
  int cur = 0;
  cudaError_t e = cudaGetDevice(&cur);
  if (e == cudaSuccess && cur != b.dev)
    e = cudaSetDevice(b.dev);
  if (e == cudaSuccess)
    e = cudaDeviceSynchronize();
  if (cur != b.dev)
    cudaSetDevice(cur);
  if (e == cudaSuccess) {
    std::lock_guard<std::mutex> g(m.lock);
    if (m.kept[b.dev] + b.bytes <= KEEP_TOTAL) {
      m.kept[b.dev] += b.bytes;
      m.idle[b.dev].emplace(b.bytes, p);
      return cudaSuccess;
    }
  }
  return cudaFree(p);
}

cudaError_t spiffe_pinned_malloc(void **p, size_t bytes)
{
  *p = nullptr;
  if (bytes > PINNED_BLOCK)
    return cudaMallocHost(p, bytes);
  Memory &m = memory();
  {
    std::lock_guard<std::mutex> g(m.lock);
    if (!m.pinned.empty()) {
      *p = m.pinned.back();
      m.pinned.pop_back();
      return cudaSuccess;
    }
  }
  return cudaHostAlloc(p, PINNED_BLOCK, cudaHostAllocPortable); // for any device
}

// bytes as allocated; no copy to or from the block may be in flight
cudaError_t spiffe_pinned_free(void *p, size_t bytes)
{
  if (!p)
    return cudaSuccess;
  if (bytes <= PINNED_BLOCK) {
    Memory &m = memory();
    std::lock_guard<std::mutex> g(m.lock);
    if (m.pinned.size() < KEEP_PINNED) {
      m.pinned.push_back(p);
      return cudaSuccess;
    }
  }
  return cudaFreeHost(p);
}
