// pool.cu -- caching device allocator of the engine.
//
// The engine, the list store and the split operands allocate and release
// tens of buffers per CC solve (up to tens of GB).  cudaMalloc/cudaFree of
// that much memory costs milliseconds to seconds per solve (the driver maps
// and unmaps pages, cudaFree synchronises the device), which dominates short
// solves such as the 64-system batch.  Released blocks are therefore kept per
// device and size class and handed out again; they return to the driver only
// when an allocation would otherwise fail, or at aces_fin.
#include <atomic>
#include <map>
#include <mutex>
#include <unordered_map>

#include "common.cuh"

namespace acesb200 {

namespace {
using Blocks = std::multimap<std::pair<int, size_t>, void *>;

struct Pool {
  std::mutex mu;
  Blocks free_blocks;                                          // (device, bytes) -> block
  std::unordered_map<void *, std::pair<int, size_t>> live;     // block -> (device, bytes)
  std::map<int, size_t> cached;                                // device -> cached bytes
  std::map<int, size_t> cap;                                   // device -> cache limit
};
// cached bytes per device are held below 35 % of its memory, so other users of
// the device in the same process (e.g. a host program's own allocator) keep room
size_t cache_cap(Pool &P, int dev) {
  auto it = P.cap.find(dev);
  if (it != P.cap.end()) return it->second;
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    tot = 0;
  }
  const size_t c = tot / 100 * 35;
  P.cap[dev] = c;
  return c;
}
// every dev_alloc call, and the ones the cache could not serve (cudaMalloc)
std::atomic<long long> g_alloc_calls{0}, g_driver_allocs{0};
Pool &pool() {
  static Pool *p = new Pool();  // never destroyed: blocks may be released at exit
  return *p;
}
size_t size_class(size_t bytes) {
  if (bytes == 0) bytes = 1;
  if (bytes >= (2u << 20)) return (bytes + (2u << 20) - 1) & ~(size_t)((2u << 20) - 1);
  size_t c = 512;
  while (c < bytes) c <<= 1;
  return c;
}
// the running call of this thread (CallScope): its depth, the blocks it has
// given back, and its workspace
struct Call {
  int depth = 0;
  bool launched = false;
  Blocks held;
  std::map<int, size_t> bytes;  // device -> held bytes
  void *ws = nullptr;
  size_t ws_bytes = 0;
  int ws_dev = -1;
};
Call &call() {
  static thread_local Call c;
  return c;
}

void trim_device(Blocks &blocks, std::map<int, size_t> &bytes, int dev) {
  for (auto it = blocks.begin(); it != blocks.end();) {
    if (it->first.first == dev) {
      cudaFree(it->second);
      it = blocks.erase(it);
    } else {
      ++it;
    }
  }
  bytes[dev] = 0;
}
// smallest block of the device that fits without wasting more than a quarter of
// the size asked for
Blocks::iterator best_fit(Blocks &blocks, int dev, size_t cls) {
  auto it = blocks.lower_bound({dev, cls});
  return it != blocks.end() && it->first.first == dev && it->first.second <= cls + cls / 4
             ? it
             : blocks.end();
}
// largest block of the device
Blocks::iterator largest(Blocks &blocks, int dev) {
  auto it = blocks.lower_bound({dev + 1, 0});
  if (it == blocks.begin()) return blocks.end();
  --it;
  return it->first.first == dev ? it : blocks.end();
}

// keeps a block: with the running call (its kernels may still use it), else in
// the pool; over the limit, cached blocks go to the driver, largest first
// (cudaFree waits for the device), then the block itself if it still does not
// fit
void keep(Pool &P, Call &C, int dev, size_t bytes, void *ptr) {
  int cur = -1;
  cudaGetDevice(&cur);
  const size_t cap = cur == dev ? cache_cap(P, dev) : 0;
  while (P.cached[dev] + C.bytes[dev] + bytes > cap) {
    auto p = largest(P.free_blocks, dev), h = largest(C.held, dev);
    if (p == P.free_blocks.end() && h == C.held.end()) break;
    const bool mine = p == P.free_blocks.end() ||
                      (h != C.held.end() && h->first.second > p->first.second);
    Blocks &from = mine ? C.held : P.free_blocks;
    auto it = mine ? h : p;
    cudaFree(it->second);
    (mine ? C.bytes : P.cached)[dev] -= it->first.second;
    from.erase(it);
  }
  if (P.cached[dev] + C.bytes[dev] + bytes > cap) {
    cudaFree(ptr);
    return;
  }
  (C.depth ? C.held : P.free_blocks).emplace(std::make_pair(dev, bytes), ptr);
  (C.depth ? C.bytes : P.cached)[dev] += bytes;
}
}  // namespace

cudaError_t dev_alloc(void **ptr, size_t bytes) {
  *ptr = nullptr;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const size_t cls = size_class(bytes);
  g_alloc_calls.fetch_add(1, std::memory_order_relaxed);
  Pool &P = pool();
  Call &C = call();
  std::lock_guard<std::mutex> lk(P.mu);
  auto p = best_fit(P.free_blocks, dev, cls), h = best_fit(C.held, dev, cls);
  if (p != P.free_blocks.end() || h != C.held.end()) {
    const bool mine = p == P.free_blocks.end() ||
                      (h != C.held.end() && h->first.second <= p->first.second);
    Blocks &from = mine ? C.held : P.free_blocks;
    auto it = mine ? h : p;
    *ptr = it->second;
    P.live[*ptr] = it->first;
    (mine ? C.bytes : P.cached)[dev] -= it->first.second;
    from.erase(it);
    return cudaSuccess;
  }
  g_driver_allocs.fetch_add(1, std::memory_order_relaxed);
  e = cudaMalloc(ptr, cls);
  if (e != cudaSuccess) {
    cudaGetLastError();
    trim_device(P.free_blocks, P.cached, dev);
    trim_device(C.held, C.bytes, dev);
    e = cudaMalloc(ptr, cls);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *ptr = nullptr;
      return e;
    }
  }
  P.live[*ptr] = {dev, cls};
  return cudaSuccess;
}

bool dev_cached(size_t bytes) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const size_t cls = size_class(bytes);
  Pool &P = pool();
  std::lock_guard<std::mutex> lk(P.mu);
  Call &C = call();
  return best_fit(P.free_blocks, dev, cls) != P.free_blocks.end() ||
         best_fit(C.held, dev, cls) != C.held.end();
}

void dev_free(void *ptr) {
  if (!ptr) return;
  Pool &P = pool();
  std::lock_guard<std::mutex> lk(P.mu);
  auto it = P.live.find(ptr);
  if (it == P.live.end()) return;  // not ours
  const int dev = it->second.first;
  const size_t bytes = it->second.second;
  P.live.erase(it);
  keep(P, call(), dev, bytes, ptr);
}

CallScope::CallScope() {
  Call &C = call();
  if (C.depth++ == 0) C.launched = false;
}

bool call_first_launch() {
  Call &C = call();
  const bool first = !C.launched;
  C.launched = true;
  return first;
}

cudaError_t CallScope::wait() {
  waited = true;
  cudaError_t e = cudaStreamSynchronize(0);
  if (extra && *extra) {
    const cudaError_t x = cudaStreamSynchronize(*extra);
    if (e == cudaSuccess) e = x;
  }
  return e;
}

CallScope::~CallScope() {
  if (!waited) wait();
  Call &C = call();
  if (--C.depth) return;
  if (C.ws) dev_free(C.ws);
  C.ws = nullptr;
  Pool &P = pool();
  std::lock_guard<std::mutex> lk(P.mu);
  Blocks held;
  held.swap(C.held);
  C.bytes.clear();
  for (auto &b : held) keep(P, C, b.first.first, b.first.second, b.second);
}

void *call_workspace(size_t bytes) {
  Call &C = call();
  int dev = 0;
  if (!C.depth || cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (C.ws && C.ws_dev == dev && C.ws_bytes >= bytes) return C.ws;
  if (C.ws) dev_free(C.ws);
  C.ws = nullptr;
  if (dev_alloc(&C.ws, bytes) != cudaSuccess) {
    cudaGetLastError();
    C.ws = nullptr;
    return nullptr;
  }
  C.ws_dev = dev;
  C.ws_bytes = bytes;
  return C.ws;
}

void pool_trim() {
  Pool &P = pool();
  std::lock_guard<std::mutex> lk(P.mu);
  for (auto &kv : P.free_blocks) cudaFree(kv.second);
  P.free_blocks.clear();
  P.cached.clear();
}

}  // namespace acesb200

extern "C" int aces_pool_stats(long long *alloc_calls, long long *driver_allocs,
                               long long *cached_bytes) {
  using namespace acesb200;
  if (alloc_calls) *alloc_calls = g_alloc_calls.load();
  if (driver_allocs) *driver_allocs = g_driver_allocs.load();
  if (cached_bytes) {
    Pool &P = pool();
    std::lock_guard<std::mutex> lk(P.mu);
    long long c = 0;
    for (auto &kv : P.cached) c += (long long)kv.second;
    *cached_bytes = c;
  }
  return ACES_OK;
}
