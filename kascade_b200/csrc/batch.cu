// Batched ranking: thousands of independent lists and forests of uneven size
// ranked together.
//
// The instances arrive concatenated (instance-local indices) with a segment
// table.  One pass over them numbers the lists' elements densely in one space
// and the forests' vertices in another; all lists are then ranked as one
// (rank_records) and all forests as one (tree.cu): a single ruler chase, one
// launch with one work queue, serves every list.  Ruler spacing and block size
// are one per batch, from the size class of its list elements (the context's
// size-class table, filled by the autotuner).  Outputs go straight to the
// instances' places, roots relative to their own instance.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "ranker.cuh"

namespace ks {

namespace {

constexpr uint32_t TILE = 4096;  // positions per tile, and per entry of a segment hint
constexpr int BP_THREADS = 256;
constexpr int BP_PER = 8;  // positions a thread has in flight

// (first element in its kind's dense numbering, kind) of every instance.
struct BatchIn {
  const uint64_t* in;
  SegMap pos;  // the instances in the caller's arrays (no delta)
  const uint2* kinds;
};

// The segment hints of an element range: hint[k] is the segment of element
// 4096 k, the last entry that of the last element.  One launch for a batch's
// three ranges.
struct HintJob {
  const uint32_t* base;
  uint32_t* hint;
  uint32_t n, elems, entries;
};
struct HintJobs {
  HintJob job[3];
};
__global__ void __launch_bounds__(BP_THREADS) k_batch_hints(HintJobs jobs) {
  kernel_begin();
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const HintJob& j = jobs.job[q];
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < j.entries; k += gridDim.x * blockDim.x) {
      const uint32_t x = (uint32_t)min((uint64_t)k * TILE, (uint64_t)j.elems - 1);
      uint32_t lo = 0, hi = j.n;  // the last segment with base <= x
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (ld_ca(j.base + mid) <= x)
          lo = mid;
        else
          hi = mid;
      }
      j.hint[k] = lo;
    }
  }
}

struct BWUnit {
  __device__ __forceinline__ uint32_t operator()(uint64_t) const { return 1u; }
};
struct BWU32 {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator()(uint64_t g) const { return ld_cs(p + g); }
};

// List elements' records, and forest vertices' parents, from the caller's
// arrays.  Streaming; a tile inside one instance (hints alike) looks its
// segment up once.
template <class F, class W>
__global__ void __launch_bounds__(BP_THREADS) k_batch_prepare(BatchIn b, uint32_t total, W w, Rulers rl,
                                                              typename F::R* __restrict__ rec,
                                                              typename F::S* __restrict__ stamp,
                                                              uint32_t* __restrict__ fpar, DevStatus* st) {
  kernel_begin();
  constexpr uint32_t STEP = BP_THREADS * BP_PER;
  const uint32_t steps = (uint32_t)(((uint64_t)total + STEP - 1) / STEP);
  for (uint32_t t = blockIdx.x; t < steps; t += gridDim.x) {
    const uint64_t g0 = (uint64_t)t * STEP;
    uint64_t v[BP_PER];
    uint32_t wv[BP_PER];
#pragma unroll
    for (int i = 0; i < BP_PER; ++i) {
      const uint64_t g = g0 + i * BP_THREADS + threadIdx.x;
      v[i] = g < total ? ld_cs(b.in + g) : 0;
      wv[i] = g < total ? w(g) : 0u;
    }
    // (a step lies within one tile of the hints)
    const uint32_t j0 = ld_ca(b.pos.hint + (uint32_t)(g0 / TILE)), j1 = ld_ca(b.pos.hint + (uint32_t)(g0 / TILE) + 1);
    uint32_t j = j0, off = 0, size = 0;
    uint2 kind = make_uint2(0, 0);
    auto segment = [&]() {
      off = ld_ca(b.pos.base + j);
      size = ld_ca(b.pos.base + j + 1) - off;
      kind = ld_ca(b.kinds + j);
    };
    if (j0 == j1) segment();
#pragma unroll
    for (int i = 0; i < BP_PER; ++i) {
      const uint64_t g = g0 + i * BP_THREADS + threadIdx.x;
      if (g >= total) continue;
      if (j0 != j1) {
        j = b.pos.find((uint32_t)g);
        segment();
      }
      const uint32_t k = (uint32_t)g - off;
      if (v[i] >= size) {
        set_error(st, KASCADE_ERR_OUT_OF_RANGE, g);
        v[i] = k;
      }
      const uint32_t x = kind.x + k, y = kind.x + (uint32_t)v[i];
      if (kind.y == KASCADE_SEG_LIST) {
        uint32_t q;
        F::put(rec + x, x == y ? 0u : wv[i], y, rl.is(y, &q));  // a root's weight is no part of any rank
        if (stamp) F::clear(stamp + x);
      } else {
        __stcs(fpar + x, y);
      }
    }
  }
}
static_assert(TILE % (BP_THREADS * BP_PER) == 0, "a step lies within a tile");

// The list ends and roots among the inputs (counted when a plan is made).
__global__ void __launch_bounds__(BP_THREADS) k_count_ends(BatchIn b, uint32_t total, uint32_t* __restrict__ count) {
  uint32_t c = 0;
  for (uint64_t g = (uint64_t)blockIdx.x * BP_THREADS + threadIdx.x; g < total; g += (uint64_t)gridDim.x * BP_THREADS)
    c += b.in[g] == g - __ldg(b.pos.base + b.pos.find((uint32_t)g)) ? 1u : 0u;
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

}  // namespace

// Tables of one batch: what the host knows of the segments in one upload, the
// hints filled in on the device.  Kept apart from the launches so that a plan
// can upload them once and capture only the device work.
struct BatchTables {
  std::vector<uint32_t> host;
  uint64_t total = 0;
  uint32_t nseg = 0, L = 0, F = 0;  // list elements, forest vertices
  uint32_t nl = 0, nf = 0;
  // device copies
  SegMap pos, lists, forests;
  const uint2* kinds = nullptr;
};

kascade_status batch_build_tables(const kascade_segment* segs, uint32_t nseg, uint64_t total, BatchTables& t) {
  t = BatchTables{};
  t.nseg = nseg;
  t.total = total;
  uint64_t expect = 0, F = 0;
  for (uint32_t i = 0; i < nseg; ++i) {
    const kascade_segment& g = segs[i];
    if (g.offset != expect || g.size > 0x7FFFFFFFull || (g.kind != KASCADE_SEG_LIST && g.kind != KASCADE_SEG_FOREST))
      return KASCADE_ERR_INVALID_ARG;
    expect += g.size;
    if (g.kind == KASCADE_SEG_FOREST) {
      F += g.size;
      ++t.nf;
    } else {
      ++t.nl;
    }
  }
  if (expect != total) return KASCADE_ERR_INVALID_ARG;
  if (total + F > MAX_ELEMS) return KASCADE_ERR_TOO_LARGE;
  t.F = (uint32_t)F;
  t.L = (uint32_t)(total - F);
  // kinds (pairs), positions, lists (base, delta), forests (base, delta)
  t.host.resize(2ull * nseg + (nseg + 1) + (2ull * t.nl + 1) + (2ull * t.nf + 1));
  uint32_t* kinds = t.host.data();
  uint32_t* pos = kinds + 2ull * nseg;
  uint32_t* base[2] = {pos + nseg + 1, pos + nseg + 1 + 2ull * t.nl + 1};  // lists, forests
  uint32_t* delta[2] = {base[0] + t.nl + 1, base[1] + t.nf + 1};
  uint32_t at[2] = {0, 0}, q[2] = {0, 0};
  for (uint32_t i = 0; i < nseg; ++i) {
    const int f = segs[i].kind == KASCADE_SEG_FOREST;
    kinds[2ull * i] = at[f];
    kinds[2ull * i + 1] = segs[i].kind;
    pos[i] = (uint32_t)segs[i].offset;
    base[f][q[f]] = at[f];
    delta[f][q[f]] = (uint32_t)segs[i].offset - at[f];
    ++q[f];
    at[f] += (uint32_t)segs[i].size;
  }
  pos[nseg] = (uint32_t)total;
  base[0][t.nl] = t.L;
  base[1][t.nf] = t.F;
  return KASCADE_OK;
}

kascade_status batch_upload_tables(kascade_ctx& ctx, BatchTables& t, cudaStream_t s) {
  uint32_t* d = alloc<uint32_t>(ctx, t.host.size());
  if (!d) return KASCADE_ERR_OOM;
  KS_CUDA(cudaMemcpyAsync(d, t.host.data(), sizeof(uint32_t) * t.host.size(), cudaMemcpyHostToDevice, s));
  t.kinds = reinterpret_cast<const uint2*>(d);
  const uint32_t* pos = d + 2ull * t.nseg;
  const uint32_t* lists = pos + t.nseg + 1;
  const uint32_t* forests = lists + 2ull * t.nl + 1;
  HintJobs jobs{};
  uint32_t most = 1;
  auto map = [&](SegMap* m, HintJob* j, const uint32_t* base, uint32_t n, uint64_t elems) {
    m->base = base;
    m->delta = base + n + 1;
    m->n = n;
    if (elems == 0) return KASCADE_OK;
    *j = HintJob{base, nullptr, n, (uint32_t)elems, (uint32_t)((elems + TILE - 1) / TILE) + 1};
    j->hint = alloc<uint32_t>(ctx, j->entries);
    if (!j->hint) return KASCADE_ERR_OOM;
    m->hint = j->hint;
    most = std::max(most, j->entries);
    return KASCADE_OK;
  };
  KS_TRY(map(&t.pos, &jobs.job[0], pos, t.nseg, t.total));
  KS_TRY(map(&t.lists, &jobs.job[1], lists, t.nl, t.L));
  KS_TRY(map(&t.forests, &jobs.job[2], forests, t.nf, t.F));
  return launch(ctx, k_batch_hints, grid_for(ctx, most, BP_THREADS, 8), BP_THREADS, 0, s, jobs);
}

// A batch's parameters: ruler spacing and block size from the class of its
// record count.
Params batch_params(const kascade_ctx& ctx, uint64_t records, const kascade_opts* opts) {
  Params p = make_params(ctx, opts, records);
  if (!(opts && opts->ruler_spacing)) p.spacing0 = std::max(2u, ctx.class_spacing[ctx.class_of(records)]);
  p.algorithm = KASCADE_ALGO_SPARSE_RULING_SET;
  return p;
}

// The device work of one batch over uploaded tables: no host tables are read
// and there are no host waits -- a stream capture of this call is a replayable
// CUDA graph.
kascade_status batch_enqueue(kascade_ctx& ctx, const BatchTables& t, const uint64_t* in, const uint32_t* weights,
                             uint64_t* root_out, uint64_t* rank_out, const kascade_opts* opts, cudaStream_t s) {
  const Params p = batch_params(ctx, t.L, opts);
  ctx.last_levels.assign(1, 0);
  uint32_t* fpar = alloc<uint32_t>(ctx, t.F);
  if (!fpar) return KASCADE_ERR_OOM;
  Forest f;
  KS_TRY(alloc_forests(ctx, t.F, p, &f));
  Lists l;  // last: they can do with less
  KS_TRY(alloc_lists(ctx, p, t.L, weights ? WKind::U32 : WKind::Unit, &l));
  const Level0& l0 = l.l0;
  const Rulers rl = level0_rulers(p);
  {
    ProfScope ps(ctx, "batch_prepare", s);
    const unsigned grid = grid_for(ctx, (t.total + BP_PER - 1) / BP_PER, BP_THREADS, 8);
    auto prepare = [&](auto f, auto w) {
      using F = decltype(f);
      return launch(ctx, k_batch_prepare<F, decltype(w)>, grid, BP_THREADS, 0, s, BatchIn{in, t.pos, t.kinds},
                    (uint32_t)t.total, w, rl, l0.records<F>(), l0.stamps<F>(), fpar, ctx.d_status);
    };
    if (l0.fmt == Format::F8x16)
      KS_TRY(prepare(F8x16{}, BWU32{weights}));
    else if (l0.fmt == Format::F8x8)
      KS_TRY(prepare(F8x8{}, BWUnit{}));
    else if (l0.fmt == Format::F16i && weights)
      KS_TRY(prepare(F16i{}, BWU32{weights}));
    else if (l0.fmt == Format::F16i)
      KS_TRY(prepare(F16i{}, BWUnit{}));
    else if (weights)
      KS_TRY(prepare(F16x16{}, BWU32{weights}));
    else
      KS_TRY(prepare(F16x16{}, BWUnit{}));
  }
  // The forests' levels run beside the lists': neither fills the chip for long
  // (128 instances of 3e6 elements 380 -> 270 us, 4096 of 2^28 11.2 -> 10.5 ms).  A
  // context with a budget of SMs, a stream in a partition of them, and profiled
  // calls keep one stream.
  const SinkBatch lists{root_out, rank_out, t.lists}, forests{root_out, rank_out, t.forests};
  // (trees among the lists of a small batch are ranked, as in a small call)
  const CtaMode mode = t.total + t.F > ONE_CTA_TREES ? CTA_LISTS : CTA_SMALL_TREES;
  const bool beside = t.L && t.F && !ctx.profile && ctx.usable_sms() == ctx.sm_count && !in_partition(s);
  if (beside) {
    Params q = p;
    q.last = false;
    KS_TRY(side_fork(ctx, s));
    kascade_status st = rank_records(ctx, l, lists, mode, q, s);
    const kascade_status sf = root_forests(ctx, fpar, f, forests, false, ctx.side);
    const kascade_status sj = side_join(ctx, s);
    if (st == KASCADE_OK) st = sf == KASCADE_OK ? sj : sf;
    KS_TRY(st);
  } else {
    KS_TRY(root_forests(ctx, fpar, f, forests, t.L == 0, s));
    KS_TRY(rank_records(ctx, l, lists, mode, p, s));
  }
  ctx.last_levels[0] = t.total + t.F;  // as a batch's size is reported: a forest's vertex counts twice
  return KASCADE_OK;
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

// Whether a batch may be planned.  One made mostly of list ends may not: the
// bound is that of a recursion whose levels could overflow.  Nothing here can;
// the refusal is part of the call's documented contract.  Waits for the count.
static kascade_status plan_admits(kascade_ctx& ctx, const BatchTables& t, const uint64_t* in,
                                  const kascade_opts* opts, cudaStream_t s) {
  uint32_t* count = alloc<uint32_t>(ctx, 1);
  if (!count) return KASCADE_ERR_OOM;
  KS_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), s));
  k_count_ends<<<grid_for(ctx, t.total, BP_THREADS, 8), BP_THREADS, 0, s>>>(BatchIn{in, t.pos, t.kinds},
                                                                            (uint32_t)t.total, count);
  KS_CHECK_LAUNCH();
  uint32_t ends = 0;
  KS_TRY(read_u32(ctx, count, &ends, s));
  const uint64_t records = t.total + t.F;
  const uint64_t rulers = records / batch_params(ctx, records, opts).spacing0;
  const uint64_t most = rulers * 3 / 2 + 65536;
  return ends + rulers > std::min<uint64_t>(most, records) ? KASCADE_ERR_UNSUPPORTED : KASCADE_OK;
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
  ctx.arena_fixed = true;  // (the eager run sized it)
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return fail(KASCADE_ERR_CUDA);
  }
  st = status_reset(ctx, s);
  if (st == KASCADE_OK) st = batch_enqueue(ctx, t, in, weights, root_out, rank_out, &opts, s);
  if (st == KASCADE_OK) st = status_publish(ctx, s);
  cudaGraph_t g = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(s, &g);
  ctx.arena_fixed = false;
  plan->graph = g;
  if (st == KASCADE_OK && (ce != cudaSuccess || !g)) st = KASCADE_ERR_CUDA;
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
