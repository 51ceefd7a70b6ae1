// spiffe_b200/csrc/devmem.cu -- device and pinned memory of the instances.
//
// An instance is made of a dozen blocks.  cudaMalloc takes 20 us below 1 MB,
// but 160 to 320 us from there on and cudaFree nearly as much, and four bytes
// of pinned memory 1.5 ms (B200 under a hypervisor): 7.5 of the 14 ms of a
// short served request.  So a freed block of at most KEEP_BLOCK bytes is kept
// for the next instance, up to KEEP_TOTAL bytes a context; what is larger or
// beyond goes back to the driver at once, and all of it does when an
// allocation fails or spiffe_gpu_idle_memory asks for it.  A request's
// instance made again: created in 1.2 ms instead of 5, freed in 0.13 instead
// of 2.5.
//
// Blocks belong to a context and are handed out in that one only: a program
// may reset the device between two instances, which ends the context and its
// memory.  The driver numbers contexts; the same handle with another number
// is a new context.
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

#include <cuda.h>

#include "../../include/spiffe_b200.h"
#include "slab.hpp"

extern "C" int spiffe_set_error(int code, const char *msg);

namespace {

constexpr size_t KEEP_BLOCK = (size_t)32 << 20, KEEP_TOTAL = (size_t)256 << 20;
constexpr size_t PINNED_BLOCK = 8192, KEEP_PINNED = 64; // bytes; blocks

struct Context {
  CUcontext handle = nullptr;
  unsigned long long id = 0; // 0: not known, nothing is kept
};
struct Block {
  int dev = 0;
  Context ctx;
  size_t bytes = 0;
};
struct Idle {
  std::multimap<size_t, void *> blocks; // by size
  size_t bytes = 0;
  std::vector<void *> pinned;
};
struct Memory {
  std::mutex lock;
  std::unordered_map<void *, Block> used;     // blocks that may be kept, device and pinned
  std::map<unsigned long long, Idle> idle;    // by context
  std::map<CUcontext, unsigned long long> id; // a handle's context when last seen
};
Memory &memory()
{
  static Memory *m = new Memory; // outlives every instance, also one freed while the process ends
  return *m;
}

// The calling thread's context, made if there is none (or no longer one, after
// a reset).  What lay idle in one that its handle no longer names went with it.
Context context(Memory &m)
{
  typedef CUresult (*Current)(CUcontext *);
  typedef CUresult (*Id)(CUcontext, unsigned long long *);
  struct Driver {
    Current current = nullptr;
    Id id = nullptr;
    Driver()
    {
      cudaDriverEntryPointQueryResult st;
      if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", (void **)&current, 12000, cudaEnableDefault, &st) != cudaSuccess)
        current = nullptr;
      if (cudaGetDriverEntryPointByVersion("cuCtxGetId", (void **)&id, 12000, cudaEnableDefault, &st) != cudaSuccess)
        id = nullptr;
      cudaGetLastError();
    }
  };
  static const Driver d;
  Context c;
  if (!d.current || !d.id)
    return c;
  auto ask = [&]() { return d.current(&c.handle) == CUDA_SUCCESS && c.handle && d.id(c.handle, &c.id) == CUDA_SUCCESS; };
  if (!ask()) {
    c = Context();
    if (cudaFree(nullptr) != cudaSuccess || !ask()) {
      cudaGetLastError();
      return Context();
    }
  }
  std::lock_guard<std::mutex> g(m.lock);
  unsigned long long &seen = m.id[c.handle];
  if (seen != c.id) {
    m.idle.erase(seen);
    seen = c.id;
  }
  return c;
}

// everything idle in the context back to the driver
void trim(Memory &m, const Context &c)
{
  Idle all;
  {
    std::lock_guard<std::mutex> g(m.lock);
    const auto it = m.idle.find(c.id);
    if (it == m.idle.end())
      return;
    all = std::move(it->second);
    m.idle.erase(it);
  }
  for (const auto &b : all.blocks)
    cudaFree(b.second);
  for (void *p : all.pinned)
    cudaFreeHost(p);
}

// p leaves the blocks in use; bytes 0: it is none of them
Block taken(Memory &m, void *p)
{
  std::lock_guard<std::mutex> g(m.lock);
  Block b;
  const auto it = m.used.find(p);
  if (it != m.used.end()) {
    b = it->second;
    m.used.erase(it);
  }
  return b;
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
  const Context c = context(m);
  const bool may_keep = bytes <= KEEP_BLOCK && c.id;
  if (may_keep) {
    std::lock_guard<std::mutex> g(m.lock);
    Idle &idle = m.idle[c.id];
    const auto it = idle.blocks.lower_bound(bytes);
    if (it != idle.blocks.end() && it->first <= bytes + bytes / 4) { // no block lies idle in a much smaller one's place
      *p = it->second;
      idle.bytes -= it->first;
      m.used[*p] = Block{dev, c, it->first};
      idle.blocks.erase(it);
      return cudaSuccess;
    }
  }
  e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    trim(m, c);
    e = cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess)
    cudaGetLastError(); // it is returned here, and is not the next call's
  if (e == cudaSuccess && may_keep) {
    std::lock_guard<std::mutex> g(m.lock);
    m.used[*p] = Block{dev, c, bytes};
  }
  return e;
}

cudaError_t spiffe_dev_free(void *p)
{
  if (!p)
    return cudaSuccess;
  Memory &m = memory();
  const Block b = taken(m, p);
  if (!b.bytes)
    return cudaFree(p);
  // as cudaFree: work in flight may still use the block (also another stream's)
  int cur = 0;
  cudaError_t e = cudaGetDevice(&cur);
  if (e == cudaSuccess && cur != b.dev)
    e = cudaSetDevice(b.dev);
  const Context c = context(m);
  const bool gone = c.handle == b.ctx.handle && c.id != b.ctx.id; // with its context
  if (e == cudaSuccess && c.id == b.ctx.id)
    e = cudaDeviceSynchronize();
  if (cur != b.dev)
    cudaSetDevice(cur);
  if (gone)
    return cudaSuccess;
  if (e == cudaSuccess && c.id == b.ctx.id) {
    std::lock_guard<std::mutex> g(m.lock);
    Idle &idle = m.idle[c.id];
    if (idle.bytes + b.bytes <= KEEP_TOTAL) {
      idle.bytes += b.bytes;
      idle.blocks.emplace(b.bytes, p);
      return cudaSuccess;
    }
  }
  return cudaFree(p);
}

cudaError_t spiffe_pinned_malloc(void **p, size_t bytes)
{
  *p = nullptr;
  Memory &m = memory();
  const Context c = context(m);
  if (bytes > PINNED_BLOCK || !c.id)
    return cudaMallocHost(p, bytes);
  {
    std::lock_guard<std::mutex> g(m.lock);
    std::vector<void *> &idle = m.idle[c.id].pinned;
    if (!idle.empty()) {
      *p = idle.back();
      idle.pop_back();
      m.used[*p] = Block{0, c, PINNED_BLOCK};
      return cudaSuccess;
    }
  }
  const cudaError_t e = cudaHostAlloc(p, PINNED_BLOCK, cudaHostAllocPortable); // for any device
  if (e == cudaSuccess) {
    std::lock_guard<std::mutex> g(m.lock);
    m.used[*p] = Block{0, c, PINNED_BLOCK};
  }
  return e;
}

// no copy to or from the block may be in flight
cudaError_t spiffe_pinned_free(void *p)
{
  if (!p)
    return cudaSuccess;
  Memory &m = memory();
  const Block b = taken(m, p);
  if (b.bytes) {
    context(m); // notes a context that is new under its handle
    std::lock_guard<std::mutex> g(m.lock);
    if (m.id[b.ctx.handle] != b.ctx.id)
      return cudaSuccess; // gone with its context
    std::vector<void *> &idle = m.idle[b.ctx.id].pinned;
    if (idle.size() < KEEP_PINNED) {
      idle.push_back(p);
      return cudaSuccess;
    }
  }
  return cudaFreeHost(p);
}

extern "C" int spiffe_gpu_idle_memory(int32_t release, int64_t *bytes)
{
  Memory &m = memory();
  const Context c = context(m);
  if (!c.id)
    return spiffe_set_error(SPIFFE_ERR_CUDA, "no CUDA context");
  if (bytes) {
    std::lock_guard<std::mutex> g(m.lock);
    *bytes = (int64_t)m.idle[c.id].bytes;
  }
  if (release)
    trim(m, c);
  return 0;
}
