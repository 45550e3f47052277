// Device and pinned-host blocks kept for reuse.
//
// Every prepare, solve and far-field call needs buffers whose sizes repeat from
// call to call (the same target at the next wavelength, the next orientation).
// cudaMalloc and cudaFree cost 0.1-0.3 ms each and stop the device: a prepare
// with one MATVEC at 96x80x96 spent 12 of its 21 ms in 30 allocations and 51
// releases, the FP64 far field of 8 polarisations at 64^3 12 of 20.  Released
// blocks go to a list and serve later requests of about their size.
//
// Rules: a block is handed back only when no work that uses it is in flight
// (the callers wait for their stream first; Engine::release and release_state
// for the device, as cudaFree did), so any thread or stream may take it next.
// The lists hold at most mem_keep's limit and HOST_KEEP bytes; what does not fit
// goes straight back to the driver, mem_trim (ddscat_cuda_release) returns
// everything, and an allocation that fails trims first and tries again.  A block
// serves requests down to half its size, and at most SLACK bytes smaller.
// Contents of a block are undefined.
#include <algorithm>
#include <map>
#include <mutex>
#include <unordered_map>
#include "engine.h"

namespace ddb {

namespace {

// Limit of the idle device bytes (mem_keep).  The default holds what a prepare at
// 128^3 gives back and takes again, 1.5 GB: Green tensor 0.1, its temporaries 0.4,
// vectors 0.7, MATVEC workspace 0.3.
size_t g_dev_keep = (size_t)2 << 30;
constexpr size_t HOST_KEEP = (size_t)64 << 20;
constexpr size_t SLACK = (size_t)256 << 20;

struct Block {
  size_t bytes;
  int dev;  // device ordinal, -1 for pinned host memory
};

struct Cache {
  std::mutex mu;
  std::unordered_map<void*, Block> live;                  // handed out
  std::multimap<std::pair<int, size_t>, void*> idle;      // (device, bytes)
  size_t held[2] = {0, 0};                                // idle bytes: device, host
};
// never destroyed: blocks are released up to process exit
Cache& cache() {
  static Cache* c = new Cache;
  return *c;
}

// request sizes rounded so that near-equal requests share blocks
size_t rounded(size_t b) {
  const size_t g = b < ((size_t)1 << 20) ? 512 : (size_t)1 << 20;
  return (b + g - 1) / g * g;
}

cudaError_t raw_alloc(void** p, size_t bytes, bool host) {
  return host ? cudaMallocHost(p, bytes) : cudaMalloc(p, bytes);
}
void raw_free(void* p, bool host) {
  if (host) cudaFreeHost(p);
  else cudaFree(p);
}

cudaError_t get(void** p, size_t bytes, bool host) {
  *p = nullptr;
  int dev = -1;
  if (!host) {
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
  }
  const size_t want = rounded(bytes ? bytes : 1);
  Cache& c = cache();
  {
    std::lock_guard<std::mutex> lock(c.mu);
    // the smallest idle block that holds the request
    auto it = c.idle.lower_bound({dev, want});
    if (it != c.idle.end() && it->first.first == dev && it->first.second <= want + std::min(want, SLACK)) {
      *p = it->second;
      c.live[*p] = Block{it->first.second, dev};
      c.held[host] -= it->first.second;
      c.idle.erase(it);
      return cudaSuccess;
    }
  }
  cudaError_t e = raw_alloc(p, want, host);
  if (e != cudaSuccess) {
    cudaGetLastError();
    mem_trim();
    e = raw_alloc(p, want, host);
  }
  if (e != cudaSuccess) { *p = nullptr; return e; }
  std::lock_guard<std::mutex> lock(c.mu);
  c.live[*p] = Block{want, dev};
  return cudaSuccess;
}

void put(void* p, bool host) {
  if (!p) return;
  Cache& c = cache();
  {
    std::lock_guard<std::mutex> lock(c.mu);
    auto it = c.live.find(p);
    if (it != c.live.end()) {
      const Block b = it->second;
      c.live.erase(it);
      if (c.held[host] + b.bytes <= (host ? HOST_KEEP : g_dev_keep)) {
        c.held[host] += b.bytes;
        c.idle.emplace(std::make_pair(b.dev, b.bytes), p);
        return;
      }
    }
  }
  raw_free(p, host);
}

}  // namespace

cudaError_t dev_alloc(void** p, size_t bytes) { return get(p, bytes, false); }
void dev_free(void* p) { put(p, false); }
cudaError_t host_alloc(void** p, size_t bytes) { return get(p, bytes, true); }
void host_free(void* p) { put(p, true); }

void mem_keep(size_t device_bytes) {
  std::lock_guard<std::mutex> lock(cache().mu);
  g_dev_keep = device_bytes;
}

void mem_trim() {
  Cache& c = cache();
  std::multimap<std::pair<int, size_t>, void*> idle;
  {
    std::lock_guard<std::mutex> lock(c.mu);
    idle.swap(c.idle);
    c.held[0] = c.held[1] = 0;
  }
  for (auto& k : idle) raw_free(k.second, k.first.first < 0);
}

}  // namespace ddb
