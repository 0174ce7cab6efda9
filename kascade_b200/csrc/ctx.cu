// Context plumbing: arena, status word, read-backs, kernel timing.
#include "ctx.cuh"

#include <cstddef>

namespace ks {

kascade_status cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return KASCADE_OK;
  if (e == cudaErrorMemoryAllocation) return KASCADE_ERR_OOM;
  return KASCADE_ERR_CUDA;
}

kascade_status arena_begin_call(kascade_ctx& ctx, cudaStream_t s) {
  (void)s;
  ctx.listed = Listed{};  // (in the arena)
  if (ctx.blocks.size() > 1) {
    // The previous call grew the arena: fold the blocks into one so that the
    // next call of the same size needs no allocation.  Growth is rare, so a
    // device-wide wait here is acceptable.
    KS_CUDA(cudaDeviceSynchronize());
    size_t total = 0;
    for (auto& b : ctx.blocks) {
      total += b.cap;
      if (b.owned) cudaFree(b.ptr);
    }
    ctx.blocks.clear();
    char* p = nullptr;
    if (cudaMalloc(&p, total) != cudaSuccess) {
      cudaGetLastError();
      return KASCADE_ERR_OOM;
    }
    ctx.blocks.push_back({p, total, 0});
  }
  for (auto& b : ctx.blocks) b.used = 0;
  return KASCADE_OK;
}

void* arena_alloc(kascade_ctx& ctx, size_t bytes) {
  bytes = (bytes + 255) & ~size_t(255);
  if (!ctx.blocks.empty()) {
    auto& b = ctx.blocks.back();
    if (b.used + bytes <= b.cap) {
      void* p = b.ptr + b.used;
      b.used += bytes;
      return p;
    }
  }
  if (ctx.arena_fixed) return nullptr;
  size_t prev = ctx.blocks.empty() ? 0 : ctx.blocks.back().cap;
  size_t cap = bytes;
  if (!ctx.arena_exact) {
    if (cap < prev) cap = prev;
    if (cap < ctx.reserve_bytes) cap = ctx.reserve_bytes;
    if (cap < (size_t(64) << 20)) cap = size_t(64) << 20;
  }
  char* p = nullptr;
  if (cudaMalloc(&p, cap) != cudaSuccess) {
    cudaGetLastError();
    // retry with exactly what is needed
    if (cap == bytes || cudaMalloc(&p, bytes) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    cap = bytes;
  }
  ctx.blocks.push_back({p, cap, bytes, true});
  return p;
}

ArenaMark arena_mark(const kascade_ctx& ctx) {
  return ArenaMark{ctx.blocks.size(), ctx.blocks.empty() ? 0 : ctx.blocks.back().used};
}

void arena_rewind(kascade_ctx& ctx, const ArenaMark& m) {
  for (; ctx.blocks.size() > m.blocks; ctx.blocks.pop_back())
    if (ctx.blocks.back().owned) cudaFree(ctx.blocks.back().ptr);
  if (m.blocks) ctx.blocks.back().used = m.used;
}

void arena_adopt(kascade_ctx& ctx, char* p, size_t bytes) {
  ctx.listed = Listed{};
  for (auto& b : ctx.blocks)
    if (b.owned) cudaFree(b.ptr);
  ctx.blocks.clear();
  ctx.blocks.push_back({p, bytes, 0, false});
  ctx.reserve_bytes = bytes;
}

cudaError_t ensure_device(int device) {
  int cur = -1;
  if (cudaGetDevice(&cur) == cudaSuccess && cur == device) return cudaSuccess;
  return cudaSetDevice(device);
}

kascade_status status_reset(kascade_ctx& ctx, cudaStream_t s) {
  if (ctx.status_dirty) KS_CUDA(cudaMemsetAsync(ctx.d_status, 0, sizeof(DevStatus), s));
  ctx.status_dirty = true;
  ctx.published = false;
  return KASCADE_OK;
}

unsigned long long* status_host(kascade_ctx& ctx, bool last) {
  if (!last) return nullptr;
  ctx.published = true;
  ctx.status_dirty = false;
  return ctx.h_pinned;
}

static __global__ void k_publish_status(DevStatus* st, unsigned long long* host) { publish_status(st, host); }

kascade_status status_publish(kascade_ctx& ctx, cudaStream_t s) {
  if (ctx.published) return KASCADE_OK;
  k_publish_status<<<1, 32, 0, s>>>(ctx.d_status, status_host(ctx));
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

// Which element has two predecessors, once a call has found that one has.
static __global__ void __launch_bounds__(256) k_two_predecessors(Listed l, uint32_t* bits, uint32_t* place) {
  auto succ = [&](uint32_t x) {
    return l.wide ? static_cast<const Rec*>(l.rec)[x].b : static_cast<const Rec8*>(l.rec)[x].b & ~REC8_RULER;
  };
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < l.n; x += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t y = succ((uint32_t)x), bit = 1u << (y & 31);
    if (y == x || !(atomicOr(bits + (y >> 5), bit) & bit) || succ(y) == y) continue;
    atomicMin(place, l.seg.n ? y + l.seg.delta[l.seg.find(y)] : y);
  }
}

kascade_status find_two_predecessors(kascade_ctx& ctx, uint32_t* place, cudaStream_t s) {
  const uint64_t words = ((uint64_t)ctx.listed.n + 31) / 32;
  const ArenaMark m = arena_mark(ctx);
  uint32_t* bits = alloc<uint32_t>(ctx, words + 1);
  if (!bits) return KASCADE_ERR_OOM;
  kascade_status st = cuda_status(cudaMemsetAsync(bits, 0, words * 4, s));
  if (st == KASCADE_OK) st = cuda_status(cudaMemsetAsync(bits + words, 0xFF, 4, s));
  if (st == KASCADE_OK) {
    k_two_predecessors<<<grid_for(ctx, ctx.listed.n, 256, 8), 256, 0, s>>>(ctx.listed, bits, bits + words);
    st = cuda_status(cudaGetLastError());
  }
  if (st == KASCADE_OK) st = read_u32(ctx, bits + words, place, s);
  arena_rewind(ctx, m);
  return st;
}

static void collect_times(kascade_ctx& ctx) {
  for (auto& p : ctx.pending) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
      auto& t = ctx.times[p.name];
      t.first += ms;
      t.second += 1;
    } else {
      cudaGetLastError();
    }
    ctx.event_pool.push_back(p.a);
    ctx.event_pool.push_back(p.b);
  }
  ctx.pending.clear();
}

kascade_status status_finish(kascade_ctx& ctx, cudaStream_t s) {
  kascade_status ps = status_publish(ctx, s);
  if (ps == KASCADE_OK) ps = cuda_status(cudaStreamSynchronize(s));
  ctx.published = false;  // (a call's later kernels are read by another status_finish)
  if (ps != KASCADE_OK) {
    ctx.status_dirty = true;
    ctx.last_status = ps;
    return ps;
  }
  collect_times(ctx);
  const DevStatus* st = reinterpret_cast<const DevStatus*>(ctx.h_pinned);
  // level 0's size when only the device knew it (a forest's)
  if (st->counter[1] && !ctx.last_levels.empty()) ctx.last_levels[0] = st->counter[1];
  ctx.error_info = st->info;
  ctx.last_status = (kascade_status)st->code;
  // two chains stamped one element: it has two predecessors
  if (ctx.last_status == KASCADE_OK && st->counter[2] != st->counter[3]) ctx.last_status = KASCADE_ERR_NOT_A_LIST;
  if (ctx.last_status == KASCADE_ERR_NOT_A_LIST && ctx.listed.rec) {
    uint32_t place = ~0u;
    if (find_two_predecessors(ctx, &place, s) == KASCADE_OK && place != ~0u) ctx.error_info = place;
  }
  return ctx.last_status;
}

kascade_status read_u32(kascade_ctx& ctx, const uint32_t* dptr, uint32_t* out, cudaStream_t s) {
  uint32_t* hp = reinterpret_cast<uint32_t*>(ctx.h_pinned + 32);
  KS_CUDA(cudaMemcpyAsync(hp, dptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  KS_CUDA(cudaStreamSynchronize(s));
  *out = *hp;
  return KASCADE_OK;
}

bool in_partition(cudaStream_t s) {
  using Fn = CUresult(CUstream, CUgreenCtx*);
  static Fn* const green = [] {
    Fn* fn = nullptr;
    return driver_fn("cuStreamGetGreenCtx", fn) ? fn : nullptr;
  }();
  CUgreenCtx g = nullptr;
  return green && green(s, &g) == CUDA_SUCCESS && g;
}

kascade_status side_fork(kascade_ctx& ctx, cudaStream_t s) {
  int priority = 0;
  KS_CUDA(cudaStreamGetPriority(s, &priority));
  if (ctx.side && priority != ctx.side_priority) {
    cudaStreamDestroy(ctx.side);  // (every fork was joined)
    ctx.side = nullptr;
  }
  if (!ctx.side) {
    KS_CUDA(cudaStreamCreateWithPriority(&ctx.side, cudaStreamNonBlocking, priority));
    ctx.side_priority = priority;
  }
  if (!ctx.fork) KS_CUDA(cudaEventCreateWithFlags(&ctx.fork, cudaEventDisableTiming));
  if (!ctx.join) KS_CUDA(cudaEventCreateWithFlags(&ctx.join, cudaEventDisableTiming));
  KS_CUDA(cudaEventRecord(ctx.fork, s));
  KS_CUDA(cudaStreamWaitEvent(ctx.side, ctx.fork, 0));
  return KASCADE_OK;
}

kascade_status side_join(kascade_ctx& ctx, cudaStream_t s) {
  KS_CUDA(cudaEventRecord(ctx.join, ctx.side));
  KS_CUDA(cudaStreamWaitEvent(s, ctx.join, 0));
  return KASCADE_OK;
}

static cudaEvent_t take_event(kascade_ctx& ctx) {
  if (!ctx.event_pool.empty()) {
    cudaEvent_t e = ctx.event_pool.back();
    ctx.event_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  if (cudaEventCreate(&e) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return e;
}

ProfScope::ProfScope(kascade_ctx& c, const char* nm, cudaStream_t st) : ctx(c), s(st), name(nm) {
  if (!ctx.profile) return;
  b = take_event(ctx);
  if (b) cudaEventRecord(b, s);
}

ProfScope::~ProfScope() {
  if (!ctx.profile || !b) return;
  cudaEvent_t e = take_event(ctx);
  if (!e) return;
  cudaEventRecord(e, s);
  ctx.pending.push_back({name, b, e});
}

}  // namespace ks
