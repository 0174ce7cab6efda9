// Library context: device properties, a growable scratch arena, the device
// status word, a pinned read-back buffer and optional per-kernel timing.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <map>
#include <string>
#include <vector>

#include "common.cuh"
#include "tuned_classes.h"

namespace ks {
// A call's list elements: level-0 records, which keep their successors, and
// where the elements are in the caller's arrays.
struct Listed {
  const void* rec = nullptr;  // nullptr: none
  bool wide = false;          // 16 B records
  uint32_t n = 0;
  SegMap seg;
};
}  // namespace ks

struct kascade_ctx {
  int device = 0;
  int sm_count = 148;
  size_t l2_bytes = 0;
  size_t smem_optin = 0;
  ks::DevStatus* d_status = nullptr;
  unsigned long long* h_pinned = nullptr;  // KS_PINNED_WORDS words
  // the device status: whether a call since its last clearing may have left it
  // non-zero, and whether the call's last kernel copies it to h_pinned
  bool status_dirty = false, published = false;
  ks::Listed listed;  // the last call's, if it ranked lists by their records
  // scratch arena: blocks are never freed inside a call, so pointers handed
  // out by alloc() stay valid until the next begin_call()
  struct Block {
    char* ptr;
    size_t cap;
    size_t used;
    bool owned = true;  // false: memory lent by the caller (arena_adopt)
  };
  std::vector<Block> blocks;
  size_t reserve_bytes = 0;
  bool arena_fixed = false;  // the arena may not grow (a stream capture)
  bool arena_exact = false;  // it grows by no more than it is asked for
  // profiling
  bool profile = false;
  struct Pending {
    const char* name;
    cudaEvent_t a, b;
  };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> event_pool;
  std::map<std::string, std::pair<double, unsigned long long>> times;
  std::vector<std::string> time_names;  // stable storage for returned names
  std::vector<unsigned long long> last_levels;
  unsigned long long error_info = 0;
  kascade_status last_status = KASCADE_OK;
  // ordering between calls issued on different streams: the next call's
  // stream waits for the previous call's completion event before it reuses
  // the arena
  cudaEvent_t done_event = nullptr;
  cudaStream_t last_stream = nullptr;
  bool async_pending = false;
  // a second stream for device work that is independent within a call
  cudaStream_t side = nullptr;
  int side_priority = 0;
  cudaEvent_t fork = nullptr, join = nullptr;
  // size classes: a batch of at most class_max[i] records uses a ruler spacing
  // of class_spacing[i], a call that ranks one list of that size
  // class_spacing_single[i]; both chase in blocks of class_block[i] threads.
  // (class_chains: kept for its callers, no effect.)  Defaults: the tuned table.
  std::vector<unsigned long long> class_max = KS_TUNED_MAX;
  std::vector<uint32_t> class_spacing = KS_TUNED_SPACING;
  std::vector<uint32_t> class_chains = KS_TUNED_CHAINS;
  std::vector<uint32_t> class_block = KS_TUNED_BLOCK;
  std::vector<uint32_t> class_spacing_single = KS_TUNED_SPACING_SINGLE;
  int class_of(unsigned long long n) const {
    for (size_t i = 0; i < class_max.size(); ++i)
      if (n <= class_max[i]) return (int)i;
    return (int)class_max.size() - 1;
  }
  // SMs' worth of block slots this context's kernels may occupy (0 = all):
  // grids are sized for this many SMs, so that work on other streams (a
  // server's latency lane) always finds free slots.  Read at every launch;
  // another thread may change it between launches.
  std::atomic<int> sm_budget{0};
  int usable_sms() const {
    const int b = sm_budget.load(std::memory_order_relaxed);
    return (b > 0 && b < sm_count) ? b : sm_count;
  }
};

namespace ks {

constexpr int KS_PINNED_WORDS = 64;

// Arena -------------------------------------------------------------------
kascade_status arena_begin_call(kascade_ctx& ctx, cudaStream_t s);
// Use `bytes` of caller-owned device memory as the arena (the caller frees
// it after the context); contexts that never run concurrently may share one.
void arena_adopt(kascade_ctx& ctx, char* p, size_t bytes);
// Make `device` current unless the current context already belongs to it
// (which keeps a context the caller made current, e.g. an SM partition).
cudaError_t ensure_device(int device);
void* arena_alloc(kascade_ctx& ctx, size_t bytes);  // nullptr on OOM
// A point to go back to: what was allocated since, and not yet used by any
// enqueued work, is given back.
struct ArenaMark {
  size_t blocks, used;
};
ArenaMark arena_mark(const kascade_ctx& ctx);
void arena_rewind(kascade_ctx& ctx, const ArenaMark& m);
// Run `f`, which allocates and enqueues nothing.  Blocks are at least as large
// as the last one; where that does not fit, it runs again with blocks of the
// size asked for.  Out of memory all the same: nothing stays allocated.
template <class F>
kascade_status arena_try(kascade_ctx& ctx, F f) {
  const ArenaMark m = arena_mark(ctx);
  kascade_status st = f();
  if (st != KASCADE_ERR_OOM) return st;
  arena_rewind(ctx, m);
  ctx.arena_exact = true;
  st = f();
  ctx.arena_exact = false;
  if (st == KASCADE_ERR_OOM) arena_rewind(ctx, m);
  return st;
}
template <class T>
T* alloc(kascade_ctx& ctx, size_t count) {
  return reinterpret_cast<T*>(arena_alloc(ctx, count * sizeof(T) + 16));
}

// Status --------------------------------------------------------------------
kascade_status cuda_status(cudaError_t e);
// Start a call: the device status is zero (stream-ordered).
kascade_status status_reset(kascade_ctx& ctx, cudaStream_t s);
// For the launch that ends a call's device work (last): where its
// publish_status puts the status.
unsigned long long* status_host(kascade_ctx& ctx, bool last = true);
// Copy the status to the host by a launch of its own unless a kernel does.
kascade_status status_publish(kascade_ctx& ctx, cudaStream_t s);
// Synchronise `s`, read the status, collect kernel timings.
kascade_status status_finish(kascade_ctx& ctx, cudaStream_t s);
// The smallest place in the caller's arrays of an element with two
// predecessors, a list's end aside (ctx.listed; waits for it); ~0: none.
kascade_status find_two_predecessors(kascade_ctx& ctx, uint32_t* place, cudaStream_t s);
// Read one device word into the pinned buffer and wait for it.
kascade_status read_u32(kascade_ctx& ctx, const uint32_t* dptr, uint32_t* out, cudaStream_t s);

// A driver function by name; false where the driver has none.
template <class F>
bool driver_fn(const char* name, F*& fn) {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q{};
  if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess ||
      !p) {
    cudaGetLastError();
    return false;
  }
  fn = reinterpret_cast<F*>(p);
  return true;
}

// Whether `s` belongs to an SM partition (a green context), which another
// stream would leave.
bool in_partition(cudaStream_t s);
// Work on ctx.side, of the priority of `s`, that may run beside what is
// enqueued on `s` from here on, and its end: `s` waits for it.  Every fork is
// joined, in error paths too.
kascade_status side_fork(kascade_ctx& ctx, cudaStream_t s);
kascade_status side_join(kascade_ctx& ctx, cudaStream_t s);

// Profiling ----------------------------------------------------------------
struct ProfScope {
  kascade_ctx& ctx;
  cudaStream_t s;
  const char* name;
  cudaEvent_t b = nullptr;
  ProfScope(kascade_ctx& c, const char* nm, cudaStream_t st);
  ~ProfScope();
};

// Launch of a kernel that begins with kernel_begin: its blocks are put in place
// before the kernel ahead has ended, ~1 us less per launch of a call that is a
// chain of small ones (50K forest 96 -> 84 us, pointer doubling of 1M 190 ->
// 174, a list of 100K 88 -> 82, 32 instances of 3e4 94 -> 80).  Such a kernel
// reads global memory by ld_ca, ld_cg and ld_cs.  Not while a context has a
// budget of SMs: waiting blocks take slots.
template <class... P, class... A>
kascade_status launch(const kascade_ctx& ctx, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                      cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = ctx.usable_sms() == ctx.sm_count ? 1 : 0;
  return cuda_status(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

inline unsigned grid_for(const kascade_ctx& ctx, uint64_t work, unsigned block, unsigned per_sm_cap) {
  uint64_t g = (work + block - 1) / block;
  uint64_t cap = (uint64_t)ctx.usable_sms() * per_sm_cap;
  if (g > cap) g = cap;
  if (g == 0) g = 1;
  return (unsigned)g;
}

}  // namespace ks

#define KS_CHECK_LAUNCH()                                   \
  do {                                                      \
    cudaError_t _e = cudaGetLastError();                    \
    if (_e != cudaSuccess) return ks::cuda_status(_e);      \
  } while (0)

#define KS_TRY(expr)                                        \
  do {                                                      \
    kascade_status _s = (expr);                             \
    if (_s != KASCADE_OK) return _s;                        \
  } while (0)

#define KS_CUDA(expr)                                       \
  do {                                                      \
    cudaError_t _e = (expr);                                \
    if (_e != cudaSuccess) return ks::cuda_status(_e);      \
  } while (0)
