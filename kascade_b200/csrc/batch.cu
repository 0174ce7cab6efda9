// Batched ranking: thousands of independent lists and forests of uneven size
// ranked together.
//
// The instances arrive concatenated (instance-local indices) with a segment
// table.  They are laid out in one record space so that a single ruler chase
// -- one persistent launch with one device work queue -- serves every
// instance:
//   list element g (concatenated position)  -> record g
//   forest vertex g                         -> record g (its up edge / tour end;
//                                              a leaf's down and up edge in one)
//   down edges of all forests (F of them)   -> records total_n .. total_n+F-1
//                                              (a leaf's or a root's: a dead self loop)
// The ruler spacing is one per batch, from the size class of its record count
// (the context's size-class table, filled by the autotuner).
// Roots are reported relative to their own instance.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "ranker.cuh"

namespace ks {

kascade_status batch_tours(kascade_ctx& ctx, const uint64_t* fpar, uint32_t F, const uint32_t* fd, const uint32_t* foff,
                           const uint32_t* fhint, uint32_t nf, uint32_t down_base, const Level0& l0,
                           const Rulers& rl, uint32_t* leaf_out, Heads* heads, cudaStream_t s);

namespace {

constexpr uint32_t ITEM = 4096;  // elements per work item
constexpr int BP_THREADS = 256;
constexpr int BP_PER = ITEM / BP_THREADS;

struct __align__(16) DSeg {
  unsigned long long off;
  uint32_t size;
  uint32_t kind;
  uint32_t fd;  // forests: base in the compact forest vertex space
  uint32_t pad;
};

struct __align__(16) Item {
  uint32_t seg;
  uint32_t start;
  uint32_t count;
  uint32_t pad;
};

struct BWUnit {
  __device__ __forceinline__ uint32_t operator()(uint64_t) const { return 1u; }
};
struct BWU32 {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator()(uint64_t g) const { return __ldcs(p + g); }
};

template <class F, class W>
__global__ void __launch_bounds__(BP_THREADS) k_batch_prepare(const Item* __restrict__ items, uint32_t nitems,
                                                              const DSeg* __restrict__ segs,
                                                              const uint64_t* __restrict__ in, W w, Rulers rl,
                                                              typename F::R* __restrict__ rec,
                                                              typename F::S* __restrict__ stamp,
                                                              uint64_t* __restrict__ fpar, DevStatus* st) {
  for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item item = items[it];
    const DSeg sg = segs[item.seg];
    if (sg.kind == KASCADE_SEG_LIST) {
      uint32_t wv[BP_PER];
      unsigned long long lv[BP_PER];
      // every load of the item first (independent, all in flight together),
      // then the checks
#pragma unroll
      for (int i = 0; i < BP_PER; ++i) {
        const uint32_t k = item.start + i * BP_THREADS + threadIdx.x;
        lv[i] = 0;
        wv[i] = 0;
        if (k < item.start + item.count) {
          const uint64_t g = sg.off + k;
          lv[i] = __ldcs(reinterpret_cast<const unsigned long long*>(in) + g);
          wv[i] = w(g);
        }
      }
      uint64_t bad = ~0ull;  // the first element whose successor is out of its instance
#pragma unroll
      for (int i = 0; i < BP_PER; ++i) {
        const uint32_t k = item.start + i * BP_THREADS + threadIdx.x;
        if (k >= item.start + item.count) continue;
        const uint64_t g = sg.off + k;
        unsigned long long loc = lv[i];
        if (loc >= sg.size) {
          if (bad == ~0ull) bad = g;
          loc = k;
        }
        const uint32_t b = (uint32_t)(sg.off + loc);
        uint32_t j;
        F::put(rec + g, loc == k ? 0u : wv[i], b, rl.is(b, &j));  // a root's weight is no part of any rank
        if (stamp) F::clear(stamp + g);
      }
      if (bad != ~0ull) set_error(st, KASCADE_ERR_OUT_OF_RANGE, bad);
    } else {
      unsigned long long pv[BP_PER];
#pragma unroll
      for (int i = 0; i < BP_PER; ++i) {
        const uint32_t k = item.start + i * BP_THREADS + threadIdx.x;
        pv[i] = k < item.start + item.count ? __ldcs(reinterpret_cast<const unsigned long long*>(in) + sg.off + k) : 0;
      }
      uint64_t bad = ~0ull;
#pragma unroll
      for (int i = 0; i < BP_PER; ++i) {
        const uint32_t k = item.start + i * BP_THREADS + threadIdx.x;
        if (k >= item.start + item.count) continue;
        unsigned long long par = pv[i];
        if (par >= sg.size) {
          if (bad == ~0ull) bad = sg.off + k;
          par = k;
        }
        __stcs(reinterpret_cast<unsigned long long*>(fpar) + sg.fd + k, (unsigned long long)(sg.fd + par));
      }
      if (bad != ~0ull) set_error(st, KASCADE_ERR_OUT_OF_RANGE, bad);
    }
  }
}

// The list ends among the inputs (counted when a plan is made).
__global__ void __launch_bounds__(BP_THREADS) k_count_ends(const Item* __restrict__ items, uint32_t nitems,
                                                           const DSeg* __restrict__ segs,
                                                           const uint64_t* __restrict__ in,
                                                           uint32_t* __restrict__ count) {
  uint32_t c = 0;
  for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item item = items[it];
    const uint64_t off = segs[item.seg].off;
    for (uint32_t k = item.start + threadIdx.x; k < item.start + item.count; k += BP_THREADS)
      c += in[off + k] == k ? 1u : 0u;
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

}  // namespace

// Host tables of one batch: built from the segment list, uploaded into the
// context's arena.  Kept apart from the launches so that a plan can upload
// them once and capture only the device work.
struct BatchTables {
  std::vector<DSeg> dsegs;
  std::vector<Item> items;
  std::vector<uint32_t> fd, foff, hint, fhint, tour;  // tour: bit j set when instance j is a forest
  std::vector<unsigned long long> seg_off;
  uint64_t total = 0, F = 0;
  uint32_t nseg = 0, nf = 0, M = 0;
  // device copies
  DSeg* d_segs = nullptr;
  Item* d_items = nullptr;
  uint32_t *d_fd = nullptr, *d_foff = nullptr, *d_hint = nullptr, *d_fhint = nullptr, *d_tour = nullptr;
  unsigned long long* d_off = nullptr;
};

kascade_status batch_build_tables(const kascade_segment* segs, uint32_t nseg, uint64_t total, BatchTables& t) {
  t = BatchTables{};
  t.nseg = nseg;
  t.total = total;
  t.dsegs.resize(nseg);
  t.seg_off.resize(nseg);
  t.tour.assign((nseg + 31) / 32, 0u);
  t.items.reserve(total / ITEM + nseg);
  uint64_t expect = 0;
  for (uint32_t i = 0; i < nseg; ++i) {
    const kascade_segment& g = segs[i];
    if (g.offset != expect || g.size > 0x7FFFFFFFull || (g.kind != KASCADE_SEG_LIST && g.kind != KASCADE_SEG_FOREST))
      return KASCADE_ERR_INVALID_ARG;
    expect += g.size;
    const bool forest = g.kind == KASCADE_SEG_FOREST;
    t.dsegs[i] = DSeg{g.offset, (uint32_t)g.size, g.kind, (uint32_t)t.F, 0};
    t.seg_off[i] = g.offset;
    if (forest) {
      t.fd.push_back((uint32_t)t.F);
      t.foff.push_back((uint32_t)g.offset);
      t.tour[i >> 5] |= 1u << (i & 31);
      t.F += g.size;
    }
    for (uint64_t st = 0; st < g.size; st += ITEM)
      t.items.push_back(Item{i, (uint32_t)st, (uint32_t)std::min<uint64_t>(ITEM, g.size - st), 0});
  }
  if (expect != total) return KASCADE_ERR_INVALID_ARG;
  if (total + t.F > MAX_ELEMS) return KASCADE_ERR_TOO_LARGE;
  t.nf = (uint32_t)t.fd.size();
  t.fd.push_back((uint32_t)t.F);
  t.hint.resize((size_t)((total + 4095) / 4096) + 1);
  {
    uint32_t j = 0;
    for (size_t k = 0; k < t.hint.size(); ++k) {
      const uint64_t x = (uint64_t)k * 4096;
      while (j + 1 < nseg && t.seg_off[j + 1] <= x) ++j;
      t.hint[k] = j;
    }
  }
  // per 4096 compact forest vertices: the forest holding the first (and one
  // entry past the last block, so a block's search range is [fhint[k], fhint[k+1]])
  t.fhint.resize((size_t)((t.F + 4095) / 4096) + 1);
  {
    uint32_t j = 0;
    for (size_t k = 0; k < t.fhint.size(); ++k) {
      const uint64_t c = (uint64_t)k * 4096;
      while (j + 1 < t.nf && t.fd[j + 1] <= c) ++j;
      t.fhint[k] = j;
    }
  }
  t.M = (uint32_t)(total + t.F);
  return KASCADE_OK;
}

kascade_status batch_upload_tables(kascade_ctx& ctx, BatchTables& t, cudaStream_t s) {
  t.d_segs = alloc<DSeg>(ctx, t.nseg);
  t.d_items = alloc<Item>(ctx, t.items.size() + 1);
  t.d_fd = alloc<uint32_t>(ctx, t.fd.size());
  t.d_foff = alloc<uint32_t>(ctx, t.foff.size() + 1);
  t.d_off = alloc<unsigned long long>(ctx, t.nseg);
  t.d_hint = alloc<uint32_t>(ctx, t.hint.size());
  t.d_fhint = alloc<uint32_t>(ctx, t.fhint.size());
  t.d_tour = alloc<uint32_t>(ctx, t.tour.size());
  if (!t.d_segs || !t.d_items || !t.d_fd || !t.d_foff || !t.d_off || !t.d_hint || !t.d_fhint || !t.d_tour)
    return KASCADE_ERR_OOM;
  KS_CUDA(cudaMemcpyAsync(t.d_segs, t.dsegs.data(), sizeof(DSeg) * t.nseg, cudaMemcpyHostToDevice, s));
  KS_CUDA(cudaMemcpyAsync(t.d_items, t.items.data(), sizeof(Item) * t.items.size(), cudaMemcpyHostToDevice, s));
  KS_CUDA(cudaMemcpyAsync(t.d_fd, t.fd.data(), sizeof(uint32_t) * t.fd.size(), cudaMemcpyHostToDevice, s));
  if (t.nf) {
    KS_CUDA(cudaMemcpyAsync(t.d_foff, t.foff.data(), sizeof(uint32_t) * t.nf, cudaMemcpyHostToDevice, s));
    KS_CUDA(cudaMemcpyAsync(t.d_tour, t.tour.data(), sizeof(uint32_t) * t.tour.size(), cudaMemcpyHostToDevice, s));
  }
  KS_CUDA(cudaMemcpyAsync(t.d_off, t.seg_off.data(), sizeof(unsigned long long) * t.nseg, cudaMemcpyHostToDevice, s));
  KS_CUDA(cudaMemcpyAsync(t.d_hint, t.hint.data(), sizeof(uint32_t) * t.hint.size(), cudaMemcpyHostToDevice, s));
  KS_CUDA(cudaMemcpyAsync(t.d_fhint, t.fhint.data(), sizeof(uint32_t) * t.fhint.size(), cudaMemcpyHostToDevice, s));
  return KASCADE_OK;
}

// The batch's parameters: ruler spacing and block size from the class of its
// record count (one chase launch serves every instance).
Params batch_params(const kascade_ctx& ctx, const BatchTables& t, const kascade_opts* opts) {
  Params p = make_params(ctx, opts, t.M);
  if (!(opts && opts->ruler_spacing)) p.spacing0 = std::max(2u, ctx.class_spacing[ctx.class_of(t.M)]);
  p.algorithm = KASCADE_ALGO_SPARSE_RULING_SET;
  return p;
}

// The device work of one batch over uploaded tables: no host tables are read
// and there are no host waits -- a stream capture of this call is a replayable
// CUDA graph.
kascade_status batch_enqueue(kascade_ctx& ctx, const BatchTables& t, const uint64_t* in, const uint32_t* weights,
                             uint64_t* root_out, uint64_t* rank_out, const kascade_opts* opts, cudaStream_t s) {
  const uint32_t M = t.M;
  const Params p = batch_params(ctx, t, opts);
  Level0 l0;
  KS_TRY(alloc_level0(ctx, plan_level0(p, M, weights ? WKind::U32 : WKind::Unit), M, &l0));
  const Rulers rl = level0_rulers(p);
  uint64_t* fpar = alloc<uint64_t>(ctx, t.F + 1);
  // forest leaves by output position: their rank is one less than their depth
  const uint64_t leaf_words = t.F ? (t.total + 31) / 32 : 0;
  uint32_t* leaf_out = leaf_words ? alloc<uint32_t>(ctx, leaf_words) : nullptr;
  if (!fpar || (leaf_words && !leaf_out)) return KASCADE_ERR_OOM;
  if (leaf_out) KS_CUDA(cudaMemsetAsync(leaf_out, 0, sizeof(uint32_t) * leaf_words, s));
  {
    ProfScope ps(ctx, "batch_prepare", s);
    const uint32_t items = (uint32_t)t.items.size();
    const unsigned grid = (unsigned)std::min<uint64_t>(items, (uint64_t)ctx.usable_sms() * 8);
    auto prepare = [&](auto f, auto w) {
      using F = decltype(f);
      k_batch_prepare<F><<<grid, BP_THREADS, 0, s>>>(t.d_items, items, t.d_segs, in, w, rl, l0.records<F>(),
                                                     l0.stamps<F>(), fpar, ctx.d_status);
    };
    if (l0.fmt == Format::F8x16)
      prepare(F8x16{}, BWU32{weights});
    else if (l0.fmt == Format::F8x8)
      prepare(F8x8{}, BWUnit{});
    else if (l0.fmt == Format::F16i && weights)
      prepare(F16i{}, BWU32{weights});
    else if (l0.fmt == Format::F16i)
      prepare(F16i{}, BWUnit{});
    else if (weights)
      prepare(F16x16{}, BWU32{weights});
    else
      prepare(F16x16{}, BWUnit{});
    KS_CHECK_LAUNCH();
  }
  Heads heads;
  KS_TRY(batch_tours(ctx, fpar, (uint32_t)t.F, t.d_fd, t.d_foff, t.d_fhint, t.nf, (uint32_t)t.total, l0, rl,
                     leaf_out, &heads, s));
  SinkBatch sink{root_out, rank_out, (uint32_t)t.total, reinterpret_cast<const uint64_t*>(t.d_off), t.d_hint, t.nseg,
                 leaf_out, t.F ? t.d_tour : nullptr};
  Extent ext;
  ext.cap = M;
  return rank_records(ctx, l0, M, ext, heads, sink, p, s);
}

kascade_status rank_batch_impl(kascade_ctx& ctx, const kascade_segment* segs, uint32_t nseg, const uint64_t* in,
                               const uint32_t* weights, uint64_t total, uint64_t* root_out, uint64_t* rank_out,
                               const kascade_opts* opts, cudaStream_t s) {
  if (total == 0) return KASCADE_OK;
  BatchTables t;
  KS_TRY(batch_build_tables(segs, nseg, total, t));
  KS_TRY(batch_upload_tables(ctx, t, s));
  return batch_enqueue(ctx, t, in, weights, root_out, rank_out, opts, s);
}

// Whether a batch may be planned: one made mostly of list ends may not (as
// documented).  Waits for the count.
static kascade_status plan_admits(kascade_ctx& ctx, const BatchTables& t, const uint64_t* in,
                                  const kascade_opts* opts, cudaStream_t s) {
  uint32_t* count = alloc<uint32_t>(ctx, 1);
  if (!count) return KASCADE_ERR_OOM;
  KS_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), s));
  const unsigned grid = (unsigned)std::min<uint64_t>(t.items.size(), (uint64_t)ctx.usable_sms() * 8);
  k_count_ends<<<grid, BP_THREADS, 0, s>>>(t.d_items, (uint32_t)t.items.size(), t.d_segs, in, count);
  KS_CHECK_LAUNCH();
  uint32_t ends = 0;
  KS_TRY(read_u32(ctx, count, &ends, s));
  const uint64_t rulers = t.M / batch_params(ctx, t, opts).spacing0;
  const uint64_t most = rulers * 3 / 2 + 65536;
  return ends + rulers > std::min<uint64_t>(most, t.M) ? KASCADE_ERR_UNSUPPORTED : KASCADE_OK;
}

// ---------------------------------------------------------------------------
// Plans: one batch captured as a CUDA graph and replayed.
// ---------------------------------------------------------------------------
// A complete call (status read back), in capi.cu.
kascade_status rank_batch_device_call(kascade_ctx* c, const kascade_segment* segs, uint32_t nseg, const uint64_t* in,
                                      const uint32_t* weights, uint64_t total, uint64_t* root_out,
                                      uint64_t* rank_out, const kascade_opts* opts, cudaStream_t s);
}  // namespace ks

struct kascade_batch_plan {
  kascade_ctx* ctx = nullptr;
  cudaStream_t stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

namespace ks {

kascade_status batch_plan_create(int device, const kascade_segment* segs, uint32_t nseg, const uint64_t* in,
                                 const uint32_t* weights, uint64_t total, uint64_t* root_out, uint64_t* rank_out,
                                 const kascade_opts* opts_in, kascade_batch_plan** out) {
  *out = nullptr;
  if (total == 0 || !segs || !nseg || !in || !root_out || !rank_out) return KASCADE_ERR_INVALID_ARG;
  kascade_opts opts;
  kascade_opts_init(&opts);
  if (opts_in) std::memcpy(&opts, opts_in, std::min<size_t>(sizeof(opts), opts_in->struct_size ? opts_in->struct_size
                                                                                                : sizeof(opts)));
  opts.struct_size = sizeof(opts);
  opts.profile = 0;
  opts.async = 0;
  auto* plan = new (std::nothrow) kascade_batch_plan();
  if (!plan) return KASCADE_ERR_OOM;
  auto fail = [&](kascade_status st) {
    kascade_batch_plan_destroy(plan);
    return st;
  };
  KS_TRY(kascade_ctx_create(device, &plan->ctx));
  kascade_ctx& ctx = *plan->ctx;
  if (cudaStreamCreateWithFlags(&plan->stream, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    return fail(KASCADE_ERR_CUDA);
  }
  cudaStream_t s = plan->stream;
  // 1. one eager run, which grows the plan's arena to what the batch needs
  kascade_status st = rank_batch_device_call(plan->ctx, segs, nseg, in, weights, total, root_out, rank_out, &opts, s);
  if (st != KASCADE_OK) return fail(st);
  // 2. tables uploaded outside the capture, the device work captured
  st = arena_begin_call(ctx, s);
  BatchTables t;
  if (st == KASCADE_OK) st = batch_build_tables(segs, nseg, total, t);
  if (st == KASCADE_OK) st = batch_upload_tables(ctx, t, s);
  if (st == KASCADE_OK) st = plan_admits(ctx, t, in, &opts, s);
  if (st == KASCADE_OK && cudaStreamSynchronize(s) != cudaSuccess) st = KASCADE_ERR_CUDA;
  if (st != KASCADE_OK) return fail(st);
  const size_t blocks_before = ctx.blocks.size();
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return fail(KASCADE_ERR_CUDA);
  }
  st = status_reset(ctx, s);
  if (st == KASCADE_OK) st = batch_enqueue(ctx, t, in, weights, root_out, rank_out, &opts, s);
  if (st == KASCADE_OK) st = status_publish(ctx, s);
  cudaGraph_t g = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(s, &g);
  plan->graph = g;
  if (st == KASCADE_OK && (ce != cudaSuccess || !g)) st = KASCADE_ERR_CUDA;
  // the capture must not have grown the arena (the eager run sized it)
  if (st == KASCADE_OK && ctx.blocks.size() != blocks_before) st = KASCADE_ERR_UNSUPPORTED;
  if (st == KASCADE_OK && cudaGraphInstantiate(&plan->exec, g, 0) != cudaSuccess) st = KASCADE_ERR_CUDA;
  cudaGetLastError();
  if (st != KASCADE_OK) return fail(st);
  *out = plan;
  return KASCADE_OK;
}

kascade_status batch_plan_launch(kascade_batch_plan* plan, cudaStream_t s) {
  if (!plan || !plan->exec) return KASCADE_ERR_INVALID_ARG;
  kascade_ctx& ctx = *plan->ctx;
  // the plan's scratch is reused by every launch: order after the previous one
  if (ctx.done_event && ctx.last_stream != s) KS_CUDA(cudaStreamWaitEvent(s, ctx.done_event, 0));
  KS_CUDA(cudaGraphLaunch(plan->exec, s));
  ctx.published = true;  // by a captured kernel
  cudaEventRecord(ctx.done_event, s);
  ctx.last_stream = s;
  return status_finish(ctx, s);
}

}  // namespace ks

extern "C" KASCADE_API kascade_status kascade_batch_plan_destroy(kascade_batch_plan* plan) {
  if (!plan) return KASCADE_OK;
  if (plan->stream) cudaStreamSynchronize(plan->stream);
  if (plan->exec) cudaGraphExecDestroy(plan->exec);
  if (plan->graph) cudaGraphDestroy(plan->graph);
  if (plan->stream) cudaStreamDestroy(plan->stream);
  if (plan->ctx) kascade_ctx_destroy(plan->ctx);
  cudaGetLastError();
  delete plan;
  return KASCADE_OK;
}
