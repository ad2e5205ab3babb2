// common.cuh -- shared state and helpers of the B200 CC engine.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <atomic>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/aces_b200.h"

namespace acesb200 {

void set_error(const char *fmt, ...);
// destroys the CC engine (amplitudes, intermediates, split caches) of this process
void engine_reset();

// caching device allocator (pool.cu): dev_free keeps the block for reuse by a
// later dev_alloc of the same size class on the same device; pool_trim
// returns every cached block to the driver
cudaError_t dev_alloc(void **ptr, size_t bytes);
void dev_free(void *ptr);
// whether dev_alloc would serve this size from a cached block
bool dev_cached(size_t bytes);
void pool_trim();

// One call of an entry point on its host thread.  A block that dev_free takes
// back during the call may still be read or written by kernels the call has
// launched, so it stays with the thread: the thread's own dev_alloc hands it out
// again (the later use is ordered by the stream), other threads get it only
// after the call has waited for its streams.
class CallScope {
 public:
  CallScope();
  ~CallScope();  // waits, unless wait() has been called
  CallScope(const CallScope &) = delete;
  CallScope &operator=(const CallScope &) = delete;
  // a stream of the call besides stream 0 (read when the scope waits)
  void also(const cudaStream_t *st) { extra = st; }
  // waits for the call's streams; no launch may follow
  cudaError_t wait();

 private:
  const cudaStream_t *extra = nullptr;
  bool waited = false;
};
// scratch of the running call, at least `bytes` long: one buffer that the
// call's products use in turn, given back when the call ends; nullptr outside a
// call or when there is no memory
void *call_workspace(size_t bytes);
// whether the running call has launched nothing yet; true once per call
bool call_first_launch();

// number of kernels the library has launched (reported by the benchmarks)
extern std::atomic<long long> g_launches;
// Launches that follow one another on a stream.  A kernel launched with
// launch_after may be set up while the kernel before it drains (programmatic
// stream serialization); it must therefore begin with after_previous(), which
// returns when that kernel is complete and its writes are visible.  No kernel
// here releases its successor before its blocks have ended: the early release
// measured slower (its blocks take slots from a last wave: EOM o = 6, v = 50
// 14.2 ms), and this way no load of the old kernel can refill an L1 line after
// the new one has started.  Back-to-back dependent launches, direct or from a
// captured graph, lose 1-1.5 us each without it: EOM o = 6, v = 50 (2600
// launches) 15.2 -> 13.4 ms, CCSD o = 5, v = 21 3.10 -> 2.72 ms.
// The first kernel of a call follows a kernel of the caller, which may release
// its successors early: it is launched in plain stream order.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                         A &&...args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = call_first_launch() ? 0 : 1;
  // an error stays for the caller's cudaGetLastError, as after <<< >>>
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

inline void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

#define ACES_CUDA(call)                                                        \
  do {                                                                         \
    cudaError_t _e = (call);                                                   \
    if (_e != cudaSuccess) {                                                   \
      ::acesb200::set_error("%s:%d %s: %s", __FILE__, __LINE__, #call,         \
                            cudaGetErrorString(_e));                           \
      return ACES_ERR_CUDA;                                                    \
    }                                                                          \
  } while (0)

#define ACES_TRY(call)                                                         \
  do {                                                                         \
    int _s = (call);                                                           \
    if (_s != ACES_OK) return _s;                                              \
  } while (0)

// Division of 32-bit indices below 2^31 by a run-time invariant divisor with
// a multiply-high, add and shift (Granlund and Montgomery, "Division by
// invariant integers using multiplication", PLDI 1994): with
// s = ceil(log2 d) and m = floor(2^32 (2^s - d) / d) + 1,
// n / d = (umulhi(n, m) + n) >> s for 0 <= n < 2^31.
struct FastDiv {
  unsigned d = 1, m = 1, s = 0;
  FastDiv() = default;
  explicit FastDiv(unsigned divisor) : d(divisor ? divisor : 1) {
    s = 0;
    while ((1ull << s) < d) ++s;
    m = (unsigned)(((1ull << 32) * ((1ull << s) - d)) / d + 1);
  }
  __host__ __device__ __forceinline__ unsigned div(unsigned n) const {
#ifdef __CUDA_ARCH__
    return (__umulhi(n, m) + n) >> s;
#else
    return (unsigned)((((unsigned long long)n * m) >> 32) + n) >> s;
#endif
  }
};

// One irrep block of a list: nrows x ncols doubles, column-major, on device.
struct ListBlock {
  int nrows = 0;
  int ncols = 0;
  double *dev = nullptr;
};

// Bump allocator over large device chunks: lists live until aces_fin, like
// the reference's single ICORE heap (acescore/aces_malloc.c).
struct DeviceArena {
  struct Chunk { char *base; size_t size; size_t used; };
  std::vector<Chunk> chunks;
  size_t chunk_bytes = size_t(256) << 20;
  void *alloc(size_t bytes);
  void release();
  size_t total() const;
};

struct SymInfo {
  int nirrep = 0;
  int pop[8] = {0};
  int vrt[8] = {0};
  int irpdpd[8][22] = {{0}};     // [irrep][type]
  int isymoff[8][8][25] = {{{0}}};  // [irp_q][irp_pq][type], 1-based
  bool ready = false;
};

struct State {
  std::recursive_mutex mu;
  int device = -1;
  SymInfo sym;
  std::map<int, std::vector<ListBlock>> lists;  // list id -> 8 irreps
  std::map<int, std::pair<int, int>> isytyp;    // list -> (left, right) type
  std::map<std::string, std::vector<char>> records;
  DeviceArena arena;
};

State &state();

// pair-type description: spins and occupied/virtual character of each index
struct PairType {
  char p, q;       // 'O' or 'V'
  int packing;     // 0 FULL, 1 PACK (p<q), 2 PCK2 (p<=q)
};
PairType pair_type(int type);   // type 1..25

// New list blocks whose memory a producer writes whole: created without the
// zero fill, and zeroed after all when the producer ends without calling
// written() (an error must not leave old device memory in a list).
class UnfilledLists {
 public:
  ~UnfilledLists();
  void add(double *p, size_t bytes) { blocks.push_back({p, bytes}); }
  void written() { blocks.clear(); }

 private:
  std::vector<std::pair<double *, size_t>> blocks;
};
// aces_inipck; with `unfilled`, the memory of new blocks is left to the producer
int list_inipck(int irrepx, int sytypl, int sytypr, int list, int iset, UnfilledLists *unfilled);

// Orbital count of irrep h (0-based) for 'O'/'V' (RHF: alpha == beta).
inline int norb(const SymInfo &s, char c, int h) { return c == 'O' ? s.pop[h] : s.vrt[h]; }

// 0-based pair index (within the pairs of total irrep hpq) of local orbitals
// p (irrep hp) and q (irrep hq), or -1 when the pair is not stored
// (p >= q in a PACK block, p > q in a PCK2 block).
long long pair_index(const SymInfo &s, int type, int hp, int p, int hq, int q);

}  // namespace acesb200
