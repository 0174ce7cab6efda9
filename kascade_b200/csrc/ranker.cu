// Ruling-set list ranker for one B200.
//
// Reference counterparts (niklas-uhl/kascade):
//   ruler sampling      lib/kascade/sparse_ruling_set_detail/ruler_selection.hpp:18-115,
//                       sparse_ruling_set.cpp:106-136 (shuffled candidates) -> here one
//                       element of every block of s indices, at a hashed offset
//   ruler chasing       sparse_ruling_set.cpp:147-273 (init / work_on_item) and
//                       ruler_chasing_engine.hpp:57-101 (sync rounds) -> one
//                       persistent kernel, every hop a dependent 16 B load
//   unreached fix-up    post_invert.hpp:195-264 -> elements ahead of their list's
//                       first ruler walk forward during propagation
//   pack / recursion    pack.hpp:23-79, sparse_ruling_set.cpp:291-310, 376-392
//                       -> the chase writes the ruler sub-list directly in
//                       dense ruler-id space
//   propagation (pull)  ruler_propagation.hpp:148-256 -> one coalesced pass
//   pointer doubling    pointer_doubling_generic.hpp:43-60, 171-212, 418-438,
//                       609-700 -> the jump kernel of a last level that the caller's
//                       depth limit leaves larger than one CTA; the calls: tree.cu
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>

#include "ranker.cuh"
#include "tma.cuh"

namespace ks {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int PREP_ITEMS = 8;

// Weight sources; T is the narrowest type that holds one weight (fewer live
// registers in the prepare kernel).
struct WUnit {
  using T = uint32_t;
  __device__ __forceinline__ T operator()(uint64_t) const { return 1u; }
};
struct WU32 {
  using T = uint32_t;
  const uint32_t* p;
  __device__ __forceinline__ T operator()(uint64_t x) const { return ld_cs(p + x); }
};
struct WI64 {
  using T = uint64_t;
  const int64_t* p;
  __device__ __forceinline__ T operator()(uint64_t x) const {
    return ld_cs(reinterpret_cast<const uint64_t*>(p) + x);
  }
};

// ---------------------------------------------------------------------------
// prepare: build records, clear the stamps (stamp == nullptr: the write-free
// path has none).  A root's weight is no part of any rank: its record carries
// 0, so that a chain ending at it adds the record's word like any.
// ---------------------------------------------------------------------------
template <class F, class W>
__global__ void __launch_bounds__(256, 4) k_prepare_arrays(const uint64_t* succ, W w, uint32_t n,
                                                        uint64_t start, Rulers rl, typename F::R* __restrict__ rec,
                                                        typename F::S* __restrict__ stamp, DevStatus* st) {
  kernel_begin();
  const uint64_t tile_sz = (uint64_t)blockDim.x * PREP_ITEMS;
  for (uint64_t tile = start + (uint64_t)blockIdx.x * tile_sz; tile < n; tile += (uint64_t)gridDim.x * tile_sz) {
    unsigned long long sv[PREP_ITEMS];
    typename W::T wv[PREP_ITEMS];
#pragma unroll
    for (int i = 0; i < PREP_ITEMS; ++i) {
      const uint64_t x = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      sv[i] = 0;
      wv[i] = 0;
      if (x < n) {
        sv[i] = ld_cs(reinterpret_cast<const unsigned long long*>(succ) + x);
        wv[i] = w(x);
      }
    }
#pragma unroll
    for (int i = 0; i < PREP_ITEMS; ++i) {
      const uint64_t x = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      if (x >= n) continue;
      if (sv[i] >= n) {
        set_error(st, KASCADE_ERR_OUT_OF_RANGE, x);
        sv[i] = x;
      }
      uint32_t j;
      F::put(rec + x, sv[i] == x ? 0 : wv[i], (uint32_t)sv[i], rl.is((uint32_t)sv[i], &j));
      if (stamp) F::clear(stamp + x);
    }
  }
}

// The same work for 16 B-aligned inputs with 32-bit weights, with the input
// tiles moved by bulk (TMA) copies: a persistent block keeps PT_STAGES tiles
// of succ (and weights) in flight into shared memory while it writes the
// records of an earlier tile.  Full tiles only; the caller hands the tail to
// k_prepare_arrays.
constexpr int PT_TILE = 2048;
constexpr int PT_STAGES = 4;
constexpr int PT_ITEMS = PT_TILE / 256;

template <class F, bool W32>
__global__ void __launch_bounds__(256) k_prepare_tma(const uint64_t* succ, const uint32_t* w,
                                                     uint32_t n, uint32_t ntiles, Rulers rl,
                                                     typename F::R* __restrict__ rec,
                                                     typename F::S* __restrict__ stamp, DevStatus* st) {
  kernel_begin();
  constexpr uint32_t SB = PT_TILE * 8, WB = W32 ? PT_TILE * 4 : 0, STAGE = SB + WB;
  extern __shared__ __align__(128) unsigned char dyn[];
  __shared__ __align__(8) uint64_t bar[PT_STAGES];
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    for (int i = 0; i < PT_STAGES; ++i) mbar_init(&bar[i], 1);
    fence_mbar_init();
  }
  __syncthreads();
  // the k-th tile of this block goes to stage k % PT_STAGES
  auto issue = [&](uint32_t k) {
    const uint32_t t = blockIdx.x + k * gridDim.x;
    if (t >= ntiles) return;
    unsigned char* dst = dyn + (k % PT_STAGES) * STAGE;
    uint64_t* b = &bar[k % PT_STAGES];
    mbar_expect_tx(b, STAGE);
    bulk_g2s(dst, succ + (uint64_t)t * PT_TILE, SB, b);
    if (W32) bulk_g2s(dst + SB, w + (uint64_t)t * PT_TILE, WB, b);
  };
  if (tid == 0)
    for (uint32_t k = 0; k < PT_STAGES; ++k) issue(k);
  for (uint32_t k = 0;; ++k) {
    const uint32_t t = blockIdx.x + k * gridDim.x;
    if (t >= ntiles) break;
    const uint32_t sg = k % PT_STAGES;
    const bool ok = mbar_wait_bounded(&bar[sg], (k / PT_STAGES) & 1u);
    if (__syncthreads_or(!ok)) {
      // a copy never completed: report it and let the copies in flight land
      // before the block's shared memory goes away
      if (tid == 0) {
        set_error(st, KASCADE_ERR_TIMEOUT, t);
        for (uint32_t j = k; j < k + PT_STAGES; ++j)
          if (blockIdx.x + j * gridDim.x < ntiles) mbar_wait_bounded(&bar[j % PT_STAGES], (j / PT_STAGES) & 1u);
      }
      __syncthreads();
      return;
    }
    const uint64_t* ss = reinterpret_cast<const uint64_t*>(dyn + sg * STAGE);
    const uint32_t* ws = reinterpret_cast<const uint32_t*>(dyn + sg * STAGE + SB);
    const uint64_t base = (uint64_t)t * PT_TILE;
    uint32_t sv[PT_ITEMS], wv[PT_ITEMS];
#pragma unroll
    for (int i = 0; i < PT_ITEMS; ++i) {
      const uint32_t j = i * 256 + tid;
      const uint32_t x = (uint32_t)(base + j);
      unsigned long long sx = ss[j];
      if (sx >= n) {
        set_error(st, KASCADE_ERR_OUT_OF_RANGE, x);
        sx = x;
      }
      sv[i] = (uint32_t)sx;
      wv[i] = W32 ? ws[j] : 1u;
    }
    __syncthreads();  // the stage is read: refill it with this block's tile k + PT_STAGES
    if (tid == 0) {
      fence_proxy_async();
      issue(k + PT_STAGES);
    }
#pragma unroll
    for (int i = 0; i < PT_ITEMS; ++i) {
      const uint32_t x = (uint32_t)(base + i * 256 + tid);
      uint32_t j;
      F::put(rec + x, sv[i] == x ? 0u : wv[i], sv[i], rl.is(sv[i], &j));
      if (stamp) F::clear(stamp + x);
    }
  }
}

// ---------------------------------------------------------------------------
// chase: one chain per thread, one per ruler.  A hop reads the record of the
// next element and stamps (distance from ruler, ruler id) for it.  A chain
// ends in front of the next ruler or at the list's end.  A warp's first rulers
// are its own share, later ones come from one counter, for several idle lanes
// at a time; only the first `lanes` lanes of a warp work, so that few rulers
// spread over all SMs and a warp's hop waits for few loads.
//
// Bound by the longest chains' dependent hops, and by instructions while most
// chains run (a warp issues them for its last running lane too).  The next
// record is asked for as soon as its index is known, before the element at
// hand is stamped.
//
// Stamps are counted; propagation counts the elements it finds stamped, and
// fewer than stamps made mean that two chains met.  hop_cap: a chain this long
// looks for a cycle ahead.
// ---------------------------------------------------------------------------
constexpr int CHASE_REFILL = 8;  // idle lanes worth a refill

template <class F>
__global__ void __launch_bounds__(512) k_chase(const typename F::R* rec, typename F::S* stamp, uint32_t n, Rulers rl,
                                               uint32_t r, const uint32_t* rootel, NextLevel nx,
                                               uint32_t* __restrict__ work, uint32_t lanes, uint32_t hop_cap,
                                               DevStatus* st) {
  kernel_begin();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint32_t first = warps * lanes;  // ids from here on are handed out by the counter
  uint32_t id = 0, x = 0, hops = 0, stamps = 0;
  uint64_t acc = 0;
  Hop h{0, 0, false};             // the record of x, asked for
  bool act = false, own = false;  // own: x is the chain's ruler (not stamped)
  auto begin = [&](uint32_t i) {
    id = i;
    const uint64_t x0 = rl.elem(i);
    if (x0 >= n) {
      nx.put(i, 0, i);  // the last block's ruler, beyond the elements
    } else {
      x = (uint32_t)x0;
      h = F::hop(rec + x);
      acc = 0;
      hops = 0;
      act = own = true;
    }
  };
  if (lane < lanes && warp * lanes + lane < r) begin(warp * lanes + lane);
  bool more = first < r;  // warp-uniform
  while (true) {
    const uint32_t running = __ballot_sync(FULL, act);
    if (more && (running == 0u || __popc(running) + CHASE_REFILL <= (int)lanes)) {
      const uint32_t idle = ~running & (lanes == 32 ? FULL : (1u << lanes) - 1u);
      uint32_t b = 0;
      if (lane == 0) b = first + atomicAdd(work, (uint32_t)__popc(idle));
      b = __shfl_sync(FULL, b, 0);
      if (b >= r) more = false;
      const uint32_t i = b + __popc(idle & lanemask_lt());
      if (((idle >> lane) & 1u) && i < r) begin(i);
      continue;
    }
    if (running == 0u) {
      if (!more) break;
      continue;
    }
    if (!act) continue;
    const uint32_t y = h.b;
    const uint64_t d = acc + h.w;
    const bool end = y == x, stop = end || h.ruler;
    // the next record's request goes out ahead of a stamp of its own array (a
    // stamp in the record goes first: the next record may share its sector)
    const Hop at = h;
    if (!F::kInPlace && !stop) h = F::hop(rec + y);
    if (!end && !own) {
      F::stamp(stamp + x, id, acc, at);
      ++stamps;
    }
    if (F::kInPlace && !stop) h = F::hop(rec + y);
    if (stop) {  // (a list's end is not stamped: any number of chains may end there)
      uint32_t next = id;
      if (end) {
        nx.rootel[id] = rootel ? ld_ca(rootel + x) : x;
      } else {
        next = rl.block_of(y);
        // back at its own ruler: a cycle without a root that holds one ruler
        if (next == id) set_error(st, KASCADE_ERR_CYCLE, id);
      }
      nx.put(id, d, next);
      act = false;
      continue;
    }
    own = false;
    acc = d;
    x = y;
    if (++hops == hop_cap) {
      hops = 0;
      if (endless<F>(rec, y)) {
        set_error(st, KASCADE_ERR_CYCLE, id);
        nx.put(id, 0, id);
        act = false;
      }
    }
  }
  stamps = __reduce_add_sync(FULL, stamps);
  if (lane == 0 && stamps) atomicAdd(&st->counter[2], (unsigned long long)stamps);
}

// ---------------------------------------------------------------------------
// propagate: rank(x) = rank(ruler) - distance(ruler, x); elements no chase
// reached (ahead of their list's first ruler) walk forward to the first
// ruler, stamped element or list end and add the weights they pass.  A block
// collects those and walks them together after its streaming work, one per
// thread: walked where they are met, each stalled its warp for its whole walk
// (512 lists in 2.6e7 elements: 2.0 -> 1.7 ms for the whole call).
// ---------------------------------------------------------------------------
constexpr uint32_t PROP_WALKS = 512;  // elements a block collects

template <class F, class Sink>
__device__ __forceinline__ void walk_to_result(const typename F::R* rec, const typename F::S* stamp, uint32_t x,
                                               const Rulers& rl, const uint32_t* rootel, const Out* out_next,
                                               const Sink& sink, DevStatus* st) {
  Hop h = F::hop(rec + x);
  uint64_t acc = h.w;
  uint32_t y = h.b, hops = 0, mark = x;
  while (true) {
    if (h.ruler) {
      const Out o = ld_out(out_next + rl.block_of(y));
      sink.put(x, acc + o.rank, o.root, false);
      return;
    }
    h = F::hop(rec + y);
    const Stamp t = F::get(stamp + y);
    if (t.id != TAG_UNREACHED) {
      const Out o = ld_out(out_next + t.id);
      sink.put(x, acc + o.rank - t.dist, o.root, false);
      return;
    }
    acc += h.w;
    if (h.b == y) {
      sink.put(x, acc, rootel ? ld_ca(rootel + y) : y, false);
      return;
    }
    // an invalid (rootless, ruler-free) cycle comes back to a marked element
    // in a number of steps proportional to its length
    if (y == mark) {
      set_error(st, KASCADE_ERR_CYCLE, x);
      return;
    }
    ++hops;
    if ((hops & (hops - 1)) == 0) mark = y;
    y = h.b;
  }
}

template <class F, class Sink, int ITEMS>
__global__ void __launch_bounds__(256) k_propagate(const typename F::R* rec, const typename F::S* stamp,
                                                   uint32_t n, Rulers rl, const uint32_t* rootel, const Out* out_next,
                                                   Sink sink, DevStatus* st, unsigned long long* status) {
  kernel_begin();
  __shared__ uint32_t walks[PROP_WALKS];
  __shared__ uint32_t nwalks, nfound;
  if (threadIdx.x == 0) nwalks = nfound = 0;
  __syncthreads();
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint64_t pol = l2_keep_policy();
  uint32_t stamped = 0;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x * ITEMS + threadIdx.x; base < n;
       base += (uint64_t)stride * ITEMS) {
    Stamp sv[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint64_t x = base + (uint64_t)i * blockDim.x;
      if (x < n) sv[i] = F::get_stream(stamp + x);
    }
    // every ruler's or stamped element's result, all loads in flight together
    // (they would otherwise wait behind the previous element's stores)
    Out ov[ITEMS];
    uint32_t found = 0;  // bit i: ov[i] holds the result of item i's ruler
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint64_t x = base + (uint64_t)i * blockDim.x;
      ov[i] = Out{0, 0, 0};
      if (x >= n) continue;
      uint32_t id;
      if (rl.is((uint32_t)x, &id)) {
        sv[i].dist = 0;
        found |= 1u << i;
      } else if (sv[i].id != TAG_UNREACHED) {
        id = sv[i].id;
        found |= 1u << i;
        ++stamped;
      }
      if ((found >> i) & 1u) ov[i] = ld_out_keep(out_next + id, pol);
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint64_t x = base + (uint64_t)i * blockDim.x;
      if (x >= n) continue;
      if ((found >> i) & 1u) {
        // a result whose root is the element itself: it is a ruler and a root
        sink.put((uint32_t)x, ov[i].rank - sv[i].dist, ov[i].root, !rootel && ov[i].root == (uint32_t)x);
        continue;
      }
      const Hop h = F::hop(rec + x);
      if (h.b == (uint32_t)x) {
        sink.put((uint32_t)x, h.w, rootel ? ld_ca(rootel + x) : (uint32_t)x, true);
      } else {
        const uint32_t w = atomicAdd(&nwalks, 1u);
        if (w < PROP_WALKS)
          walks[w] = (uint32_t)x;
        else
          walk_to_result<F>(rec, stamp, (uint32_t)x, rl, rootel, out_next, sink, st);
      }
    }
  }
  stamped = __reduce_add_sync(FULL, stamped);
  if ((threadIdx.x & 31u) == 0 && stamped) atomicAdd(&nfound, stamped);
  __syncthreads();
  if (threadIdx.x == 0 && nfound) atomicAdd(&st->counter[3], (unsigned long long)nfound);
  for (uint32_t w = threadIdx.x; w < min(nwalks, PROP_WALKS); w += blockDim.x)
    walk_to_result<F>(rec, stamp, walks[w], rl, rootel, out_next, sink, st);
  publish_status(st, status);
}

// ---------------------------------------------------------------------------
// One CTA ranks up to ONE_CTA_MAX elements in shared memory: the last level
// of the recursion, or a whole small input straight from the caller's arrays.
// The elements are loaded once; at most CTA_RULERS rulers (placed as on every
// level) walk and stamp as in k_chase, pointer jumping ranks the rulers
// (three steps per round), and every element reads its ruler's result.
// Against pointer jumping over all elements (13 rounds of 16 elements per
// thread at 8192: 51 us) each element is touched once.  Each element's word
// also says whether its successor is a ruler, so a hop is one read and one
// write of the word and of the distance.  Bound by one SM's shared-memory
// pipe and instructions: 1000 elements 9.9 us, 4000 14.7, 8000 18.2, 14.3
// thousand 27 (46 with a pass of its own for the ruler bits, three barriers a
// jumping round and a predecessor byte per element in every case).
// With several lists, their heads (no predecessor) start chains as well, so
// that no run of elements ahead of a first ruler is walked element by element.
// Two chains that meet (a tree, not a list) leave fewer stamped elements than
// stamps; CTA_SMALL_TREES does an input of at most ONE_CTA_TREES elements again
// without stamps, every element walking to its first ruler, which ranks any
// forest; CTA_TREES and CTA_ROOTING do so from the start.
// ---------------------------------------------------------------------------
constexpr uint32_t CTA_THREADS = 1024;
constexpr uint32_t CTA_HEADS = 1024;
constexpr uint32_t CTA_LOADS = 8;           // elements a thread has in flight while loading
constexpr uint32_t CTA_ILP = 4;             // elements a thread has in flight in shared memory
constexpr uint32_t CTA_FLAG = 0x80000000u;  // next: stamped, low bits the chain; rnext: the list's end
constexpr uint32_t CTA_RUL = 0x20000000u;   // next: the successor is a ruler
constexpr uint32_t CTA_IDX = 0x1FFFFFFFu;
constexpr size_t cta_smem(uint64_t n) {
  return (size_t)((n + CTA_RULERS + CTA_HEADS) * 12 + CTA_RULERS * 12 + CTA_HEADS * 2 + (n + 3) / 4 * 4);
}

// Element sources: the records of a level (a list end's carries its rank), or
// the caller's arrays (a root's weight is no part of any rank).
// FLAGGED: the records' ruler bits are for this ranker's rulers.
template <class F, bool FLAGGED>
struct CtaRecords {
  static constexpr bool kEndWeight = true, kFlagged = FLAGGED;
  const typename F::R* rec;
  const uint32_t* rootel;
  __device__ __forceinline__ void load(uint32_t x, uint64_t* a, uint32_t* b, bool* ruler) const {
    const Hop h = F::hop(rec + x);
    *a = h.w;
    *b = h.b;
    *ruler = h.ruler;
  }
  __device__ __forceinline__ uint32_t root_of(uint32_t x) const { return rootel ? ld_ca(rootel + x) : x; }
};
template <class W, class I = uint64_t>
struct CtaArrays {
  static constexpr bool kEndWeight = false, kFlagged = false;
  const I* succ;
  W w;
  __device__ __forceinline__ void load(uint32_t x, uint64_t* a, uint32_t* b, bool* ruler) const {
    *ruler = false;
    const uint64_t s = ld_cg(succ + x);
    *a = w(x);
    *b = s > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)s;  // beyond any element: found out of range
  }
  __device__ __forceinline__ uint32_t root_of(uint32_t x) const { return x; }
};

// The first element that has two predecessors, a list's end aside (~0: none).
// predw: a byte for each element, found: one word, both in shared memory.
template <class Src>
__device__ __noinline__ uint32_t two_predecessors(const Src& src, uint32_t n, uint32_t* predw, uint32_t* found) {
  uint64_t a;
  uint32_t y, z;
  bool f;
  if (threadIdx.x == 0) *found = ~0u;
  for (uint32_t w = threadIdx.x; w < (n + 3) / 4; w += blockDim.x) predw[w] = 0;
  __syncthreads();
  for (uint32_t x = threadIdx.x; x < n; x += blockDim.x) {
    src.load(x, &a, &y, &f);
    const uint32_t bit = 1u << (8 * (y & 3));
    if (y >= n || y == x || !(atomicOr(predw + (y >> 2), bit) & bit)) continue;
    src.load(y, &a, &z, &f);
    if (z != y) atomicMin(found, y);
  }
  __syncthreads();
  return *found;
}

template <class Src, class Sink>
__device__ __forceinline__ void rank_cta(const Src& src, const Extent& ext, const Sink& sink, CtaMode mode,
                                         DevStatus* st) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t nends, nheads, nstamps;
  const uint32_t n = ext.get();
  unsigned long long* dist = reinterpret_cast<unsigned long long*>(smem);  // weight, once stamped the distance
  unsigned long long* rdist = dist + ext.cap;                              // per chain: distance, then rank
  unsigned long long* jdist = rdist + CTA_RULERS + CTA_HEADS;              // (the jumping rounds' other copy)
  uint32_t* next = reinterpret_cast<uint32_t*>(jdist + CTA_RULERS);
  uint32_t* rnext = next + ext.cap;  // per chain: next ruler or CTA_FLAG | list end, then the root
  uint32_t* jnext = rnext + CTA_RULERS + CTA_HEADS;
  uint32_t* predw = jnext + CTA_RULERS;
  unsigned char* pred = reinterpret_cast<unsigned char*>(predw);  // 1: has a predecessor
  uint16_t* hlist = reinterpret_cast<uint16_t*>(predw + (ext.cap + 3) / 4);
  const uint32_t tid = threadIdx.x, nthreads = blockDim.x;
  const Rulers rl = cta_rulers(n);
  const bool all = rl.s == 1;  // every element is a ruler
  const uint32_t rulers = all ? n : (n + rl.s - 1) / rl.s;
  auto ruler = [&](uint32_t x) {
    uint32_t j;
    return all || rl.is(x, &j);
  };
  auto elem = [&](uint32_t j) { return all ? j : (uint32_t)rl.elem(j); };
  bool stamp = mode <= CTA_SMALL_TREES && !all;  // (chains of one element pass none)
  uint32_t heads = 0;
  while (true) {
    if (tid == 0) nends = nheads = nstamps = 0;
    __syncthreads();
    uint32_t ends = 0;
    for (uint32_t x0 = tid; x0 < n; x0 += nthreads * CTA_LOADS) {
      uint64_t a[CTA_LOADS];
      uint32_t b[CTA_LOADS], rul = 0;
#pragma unroll
      for (uint32_t i = 0; i < CTA_LOADS; ++i) {
        const uint32_t x = x0 + i * nthreads;
        bool f = false;
        if (x < n) src.load(x, &a[i], &b[i], &f);
        rul |= f ? 1u << i : 0u;
      }
#pragma unroll
      for (uint32_t i = 0; i < CTA_LOADS; ++i) {
        const uint32_t x = x0 + i * nthreads;
        if (x >= n) continue;
        if (b[i] >= n) {
          set_error(st, KASCADE_ERR_OUT_OF_RANGE, x);
          b[i] = x;
        }
        const bool end = b[i] == x;
        dist[x] = (Src::kEndWeight || !end) ? a[i] : 0ull;
        // (a list's end is its own word, whether it is a ruler or not)
        next[x] = b[i] | (!end && (Src::kFlagged ? (rul >> i) & 1u : ruler(b[i])) ? CTA_RUL : 0u);
        ends += end ? 1u : 0u;
      }
    }
    ends = __reduce_add_sync(FULL, ends);
    if ((tid & 31u) == 0 && ends) atomicAdd(&nends, ends);
    __syncthreads();
    if (mode == CTA_ROOTING) {  // the call's size: the vertices, and again those between a root and a leaf
      for (uint32_t w = tid; w < (n + 3) / 4; w += nthreads) predw[w] = 0;
      __syncthreads();
      for (uint32_t x = tid; x < n; x += nthreads) {
        const uint32_t y = next[x] & CTA_IDX;
        if (y != x) pred[y] = 1;
      }
      __syncthreads();
      uint32_t downs = 0;
      for (uint32_t x = tid; x < n; x += nthreads) downs += pred[x] && next[x] != x ? 1u : 0u;
      downs = __reduce_add_sync(FULL, downs);
      if ((tid & 31u) == 0) atomicAdd(&st->counter[1], (unsigned long long)(downs + (tid == 0 ? n : 0u)));
    }
    // with several lists, their heads start chains too
    if (stamp && !all && nends > 2) {
      for (uint32_t w = tid; w < (n + 3) / 4; w += nthreads) predw[w] = 0;
      __syncthreads();
      for (uint32_t x = tid; x < n; x += nthreads) {
        const uint32_t y = next[x] & CTA_IDX;
        if (y != x) pred[y] = 1;
      }
      __syncthreads();
      for (uint32_t w = tid; w < (n + 3) / 4; w += nthreads) {
        const uint32_t pw = predw[w];
        if (pw == 0x01010101u) continue;
        for (uint32_t i = 0; i < 4; ++i) {
          const uint32_t x = w * 4 + i;
          if (((pw >> (8 * i)) & 1u) || x >= n || next[x] == x || ruler(x)) continue;
          const uint32_t e = atomicAdd(&nheads, 1u);
          if (e < CTA_HEADS) hlist[e] = (uint16_t)x;
        }
      }
      __syncthreads();
      heads = min(nheads, CTA_HEADS);
    }
    // chains of the rulers, then (ids from CTA_RULERS on) of the heads
    uint32_t stamps = 0, loops = 0;
    for (uint32_t k = tid; k < rulers + heads; k += nthreads) {
      const uint32_t id = k < rulers ? k : CTA_RULERS + (k - rulers);
      const uint32_t x0 = k < rulers ? elem(k) : hlist[k - rulers];
      if (x0 >= n) {  // the last block's ruler, beyond the elements
        rnext[id] = CTA_FLAG;
        continue;
      }
      uint32_t f = next[x0], x = x0;
      unsigned long long acc = dist[x0];
      if (f == x0) {  // a list's end
        rdist[id] = acc;
        rnext[id] = CTA_FLAG | x0;
        continue;
      }
      if (stamp) {  // no other chain passes a ruler or a head
        next[x0] = CTA_FLAG | id;
        dist[x0] = 0;
      }
      uint32_t hops = 0;
      while (!(f & (CTA_FLAG | CTA_RUL))) {
        x = f;
        f = next[x];
        const unsigned long long w = dist[x];
        if (f == x) {  // the list's end
          acc += w;
          break;
        }
        if (stamp) {
          next[x] = CTA_FLAG | id;
          dist[x] = acc;
          ++stamps;
        } else if (++hops > n) {  // a cycle without a ruler
          f = CTA_FLAG;
        }
        acc += w;
      }
      rdist[id] = acc;
      if (f & CTA_FLAG) {  // another chain's element (counted below), or a cycle: never ends
        loops = 1;
        rnext[id] = id < CTA_RULERS ? id : 0u;
      } else if (f & CTA_RUL) {
        rnext[id] = all ? f & CTA_IDX : rl.block_of(f & CTA_IDX);
      } else {
        rnext[id] = CTA_FLAG | x;
      }
    }
    if (!stamp) break;
    stamps = __reduce_add_sync(FULL, stamps);
    if ((tid & 31u) == 0 && stamps) atomicAdd(&nstamps, stamps);
    const int clash = __syncthreads_or((int)loops);
    uint32_t marks = 0;  // stamped elements that are no chain's first
    for (uint32_t x = tid; x < n; x += nthreads) marks += next[x] >> 31;
    for (uint32_t k = tid; k < rulers + heads; k += nthreads) {
      const uint32_t x0 = k < rulers ? elem(k) : hlist[k - rulers];
      if (x0 < n && (next[x0] & CTA_FLAG)) --marks;
    }
    marks = __reduce_add_sync(FULL, marks);
    if ((tid & 31u) == 0 && marks) atomicSub(&nstamps, marks);
    __syncthreads();
    if (!clash && nstamps == 0) break;
    if (mode == CTA_LISTS || n > ONE_CTA_TREES) {
      const uint32_t x = two_predecessors(src, n, predw, &nheads);
      if (tid == 0) set_error(st, KASCADE_ERR_NOT_A_LIST, x);
      return;
    }
    __syncthreads();
    stamp = false;  // again from the source, without stamps
    heads = 0;
  }
  __syncthreads();
  // pointer jumping over the rulers through the previous round's copy: one
  // barrier per round (three steps per round were slower: the rounds are bound
  // by the shared-memory pipe, not by their barriers)
  {
    unsigned long long *da = rdist, *db = jdist;
    uint32_t *na = rnext, *nb = jnext;
    for (int round = 0;; ++round) {
      int busy = 0;
#pragma unroll 4
      for (uint32_t j = tid; j < rulers; j += nthreads) {
        uint32_t nx = na[j];
        unsigned long long d = da[j];
        if (!(nx & CTA_FLAG)) {
          d += da[nx];
          nx = na[nx];
          busy = 1;
        }
        nb[j] = nx;
        db[j] = d;
      }
      unsigned long long* td = da;
      da = db;
      db = td;
      uint32_t* tn = na;
      na = nb;
      nb = tn;
      if (!__syncthreads_or(busy)) break;
      if (round > 11) {  // 2^11 > CTA_RULERS: what has not ended by now never does
        if (tid == 0) set_error(st, KASCADE_ERR_CYCLE, n);
        return;
      }
    }
    if (da != rdist) {  // (the heads' entries are in rdist and rnext)
      for (uint32_t j = tid; j < rulers; j += nthreads) {
        rdist[j] = da[j];
        rnext[j] = na[j];
      }
      __syncthreads();
    }
  }
  // the heads' chains end at a ruler or a list end; then every chain's root
  for (uint32_t h = tid; h < heads; h += nthreads) {
    const uint32_t j = CTA_RULERS + h, nx = rnext[j];
    if (!(nx & CTA_FLAG)) {
      rdist[j] += rdist[nx];
      rnext[j] = rnext[nx];
    }
  }
  __syncthreads();
  for (uint32_t k = tid; k < rulers + heads; k += nthreads) {
    const uint32_t j = k < rulers ? k : CTA_RULERS + (k - rulers);
    rnext[j] = src.root_of(rnext[j] & ~CTA_FLAG);
  }
  __syncthreads();
  for (uint32_t x0 = tid; x0 < n; x0 += nthreads * CTA_ILP) {
    uint32_t f[CTA_ILP];
    unsigned long long d[CTA_ILP];
#pragma unroll
    for (uint32_t i = 0; i < CTA_ILP; ++i) {
      const uint32_t x = x0 + i * nthreads;
      f[i] = x < n ? next[x] : 0u;
      d[i] = x < n ? dist[x] : 0ull;
    }
#pragma unroll
    for (uint32_t i = 0; i < CTA_ILP; ++i) {
      const uint32_t x = x0 + i * nthreads;
      if (x >= n) continue;
      uint32_t root = 0, j;
      if (f[i] & CTA_FLAG) {
        d[i] = rdist[f[i] & CTA_IDX] - d[i];
        root = rnext[f[i] & CTA_IDX];
      } else if (f[i] == x) {
        root = src.root_of(x);
      } else if (!stamp && (all || rl.is(x, &j))) {
        j = all ? x : rl.block_of(x);
        d[i] = rdist[j];
        root = rnext[j];
      } else {  // ahead of its list's first ruler (or nothing is stamped): walk
        uint32_t hops = 0, w = f[i];
        bool ok = true;
        while (true) {
          const uint32_t y = w & CTA_IDX;
          if (w & CTA_RUL) {
            const uint32_t k = all ? y : rl.block_of(y);
            d[i] += rdist[k];
            root = rnext[k];
            break;
          }
          w = next[y];
          if (w & CTA_FLAG) {
            d[i] += rdist[w & CTA_IDX] - dist[y];
            root = rnext[w & CTA_IDX];
            break;
          }
          d[i] += dist[y];
          if (w == y) {
            root = src.root_of(y);
            break;
          }
          if (++hops > n) {
            set_error(st, KASCADE_ERR_CYCLE, x);
            ok = false;
            break;
          }
        }
        if (!ok) continue;
      }
      sink.put(x, d[i], root, f[i] == x);
    }
  }
}

// status: see publish_status.
template <class Src, class Sink>
__global__ void __launch_bounds__(CTA_THREADS, 1) k_rank_cta(Src src, Extent ext, Sink sink, CtaMode mode,
                                                             DevStatus* st, unsigned long long* status) {
  kernel_begin();
  rank_cta(src, ext, sink, mode, st);
  publish_status(st, status);
}

// ---------------------------------------------------------------------------
// pointer doubling: double-buffered jump rounds over 16 B records.
// done bit 0: successor is a root; bit 1: the element is a root.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_pd_init(const Rec* __restrict__ rec, Extent ext,
                                                 PdRec* __restrict__ a, DevStatus* st) {
  const uint32_t n = ext.get();
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (uint64_t)gridDim.x * blockDim.x) {
    Rec r = rec[x];
    if (r.b >= n) {  // guard: treat as a root and report
      set_error(st, KASCADE_ERR_OUT_OF_RANGE, x);
      r.b = (uint32_t)x;
    }
    bool root = (r.b == (uint32_t)x);
    PdRec p;
    p.rank = r.a;  // a list end's record holds its own rank: 0 on level 0
    p.succ = r.b;
    p.done = root ? 3u : 0u;
    a[x] = p;
  }
}

// One round of pointer jumping over the previous round's records `a`: an
// element not yet at its root follows its pointer three times there (a chain
// of dependent reads of `a` only, never of `b`), so a round multiplies every
// pointer's reach by four: half the launches of single jumps.
__global__ void __launch_bounds__(256) k_pd_round(const PdRec* __restrict__ a, PdRec* __restrict__ b, Extent ext) {
  const uint32_t n = ext.get();
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (uint64_t)gridDim.x * blockDim.x) {
    PdRec e = a[x];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (e.done & 1u) break;
      const PdRec t = a[e.succ];
      e.rank += t.rank;
      e.succ = t.succ;
      e.done = t.done & 1u;
    }
    b[x] = e;
  }
}

template <class Sink>
__global__ void __launch_bounds__(256) k_pd_final(const PdRec* __restrict__ a, Extent ext,
                                                  const uint32_t* __restrict__ elem0, Sink sink) {
  const uint32_t n = ext.get();
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (uint64_t)gridDim.x * blockDim.x) {
    PdRec e = a[x];
    uint32_t rt = e.succ;
    if (elem0) rt = elem0[rt];
    sink.put((uint32_t)x, e.rank, rt, (e.done & 2u) != 0u);
  }
}

// After a fixed number of rounds every element must point at a root; one that
// does not sits on a rootless cycle.
__global__ void __launch_bounds__(256) k_pd_check(const PdRec* __restrict__ a, Extent ext, DevStatus* st) {
  const uint32_t n = ext.get();
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (uint64_t)gridDim.x * blockDim.x)
    if (!(a[x].done & 1u)) set_error(st, KASCADE_ERR_CYCLE, x);
}

// ---------------------------------------------------------------------------
// is_list: count predecessors.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_count_preds(const uint64_t* __restrict__ succ, uint64_t n,
                                                     uint32_t* __restrict__ cnt, uint32_t* __restrict__ bad) {
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t s = succ[x];
    if (s >= n) {
      atomicOr(bad, 2u);
      continue;
    }
    if (s == x) continue;
    if (atomicAdd(cnt + s, 1u) >= 1u) atomicOr(bad, 1u);
  }
}

// ---------------------------------------------------------------------------
// Host-side launch helpers
// ---------------------------------------------------------------------------
template <class K>
int occupancy(K kernel, int block, size_t smem) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, block, smem) != cudaSuccess) {
    cudaGetLastError();
    nb = 1;
  }
  return nb < 1 ? 1 : nb;
}

// Resident blocks per SM of the chase.
template <class F>
int chase_occupancy(uint32_t block) {
  static std::atomic<int> occ[3] = {{-1}, {-1}, {-1}};  // blocks of 128, 256, 512 threads
  const int bi = block == 128 ? 0 : block == 512 ? 2 : 1;
  int v = occ[bi].load();
  if (v < 0) occ[bi].store(v = occupancy(k_chase<F>, (int)block, 0));
  return v;
}

// Warps that share a level's rulers before a warp works with more lanes: the
// L2 serves dependent hops of this many resident warps at full speed.
constexpr uint64_t CHASE_SPREAD_WARPS_PER_SM = 32;

// Level k's chase.
template <class F>
kascade_status launch_chase(kascade_ctx& ctx, const Levels& lv, int k, const typename F::R* rec, typename F::S* stamp,
                            uint32_t block, cudaStream_t s) {
  const uint32_t r = lv.n[k + 1];
  const uint64_t wpb = block / 32;
  const uint64_t max_grid = (uint64_t)ctx.usable_sms() * chase_occupancy<F>(block);
  const uint64_t spread = std::min<uint64_t>(max_grid * wpb, (uint64_t)ctx.usable_sms() * CHASE_SPREAD_WARPS_PER_SM);
  const uint32_t lanes = (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, (r + spread - 1) / spread));
  const uint64_t need = ((uint64_t)r + lanes - 1) / lanes;  // warps worth of work
  const unsigned grid = (unsigned)std::min<uint64_t>(max_grid, (need + wpb - 1) / wpb);
  ProfScope ps(ctx, "chase", s);
  KS_TRY(launch(ctx, k_chase<F>, grid, block, 0, s, rec, stamp, lv.n[k], lv.rulers[k], r, lv.rootel[k], next_level(lv,
                k + 1), &ctx.d_status->work[k], lanes, hop_cap(lv.rulers[k]), ctx.d_status));
  return KASCADE_OK;
}

// Level k's results from level k + 1's.  Four elements a thread (eight took 86
// registers, a quarter of the SM's warps: 6e6 elements in place 403 -> 394 us,
// a list of 2e6 176 -> 170; two: 401 and 171), two on small levels, so that
// they fill the chip.
template <class F, class Sink>
kascade_status launch_propagate(kascade_ctx& ctx, const Levels& lv, int k, const typename F::R* rec,
                                const typename F::S* stamp, const Sink& sink, bool last, cudaStream_t s) {
  const uint32_t n = lv.n[k];
  ProfScope ps(ctx, "propagate", s);
  unsigned long long* status = status_host(ctx, last);
  if (n <= (uint64_t)ctx.usable_sms() * 256 * 8 * 4) {
    const unsigned grid = grid_for(ctx, ((uint64_t)n + 1) / 2, 256, 8);
    KS_TRY(launch(ctx, k_propagate<F, Sink, 2>, grid, 256, 0, s, rec, stamp, n, lv.rulers[k], lv.rootel[k],
                  lv.out[k + 1], sink, ctx.d_status, status));
  } else {
    const unsigned grid = grid_for(ctx, ((uint64_t)n + 3) / 4, 256, 8);
    KS_TRY(launch(ctx, k_propagate<F, Sink, 4>, grid, 256, 0, s, rec, stamp, n, lv.rulers[k], lv.rootel[k],
                  lv.out[k + 1], sink, ctx.d_status, status));
  }
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

template <class Src, class Sink>
kascade_status launch_rank_cta(kascade_ctx& ctx, const Src& src, const Extent& ext, const Sink& sink,
                               CtaMode mode, bool last, cudaStream_t s) {
  static std::atomic<uint64_t> raised{0};  // kernel attributes are per device
  const uint64_t bit = 1ull << (ctx.device & 63);
  if (!(raised.load() & bit)) {
    KS_CUDA(cudaFuncSetAttribute(k_rank_cta<Src, Sink>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)cta_smem(ONE_CTA_MAX)));
    raised.fetch_or(bit);
  }
  ProfScope ps(ctx, "base_case", s);
  // one ruler per thread; a small input's few barriers are cheaper with fewer
  // warps (a list of 1000: 128 / 256 / 512 / 1024 threads 14.9 / 11.0 / 9.9 / 10.2
  // us, of 64: 6.2 / 6.2 / 6.3 / 6.9)
  const unsigned threads = ext.cap <= 256 ? 256 : ext.cap <= 1024 ? 512 : CTA_THREADS;
  KS_TRY(launch(ctx, k_rank_cta<Src, Sink>, 1, threads, cta_smem(ext.cap), s, src, ext, sink, mode, ctx.d_status,
                status_host(ctx, last)));
  return KASCADE_OK;
}

// Ruler spacing of a deeper level of n elements: levels of equal spacing down
// to `target`, as many as cost least.  The target is three quarters of what
// one CTA ranks: its time grows with its elements (2^20: 87382 elements to
// 12484 153 us, to 9710 138; 2e6: 200 and 193, 4e6: 278 and 285).  A level costs its longest
// chain, spacing x ln(rulers) dependent hops, and launches worth ~36 hops
// (measured on L2-resident levels: 0.25 us a hop, ~9 us for a level's chase
// and propagation launches).
uint32_t deep_spacing(uint32_t n, uint32_t target) {
  uint32_t best = 4;
  double best_cost = 1e300;
  for (int levels = 1; levels <= 8; ++levels) {
    const double sp = std::max(4.0, std::ceil(std::pow((double)n / target, 1.0 / levels)));
    double cost = 36.0 * levels, m = n;
    for (int i = 0; i < levels; ++i) {
      m = std::max(2.0, m / sp);
      cost += sp * std::log(m);
    }
    if (cost < best_cost) {
      best_cost = cost;
      best = (uint32_t)sp;
    }
  }
  return best;
}

}  // namespace

// ---------------------------------------------------------------------------
// Public (library-internal) entry points
// ---------------------------------------------------------------------------
Params make_params(const kascade_ctx& ctx, const kascade_opts* o, uint64_t n) {
  Params p;
  // Spacing trades chase critical path (~ spacing * ln(n/spacing) hops)
  // against ruler-table size; the defaults are the context's size classes
  // (tuned_classes.h).
  {
    const int k = ctx.class_of(n);
    p.spacing0 = ctx.class_spacing_single[k];
    p.block = ctx.class_block[k];
  }
  if (o) {
    if (o->ruler_spacing) p.spacing0 = p.spacing_given = o->ruler_spacing;
    if (o->ruler_spacing_deep) p.spacing_deep = o->ruler_spacing_deep;
    if (o->max_levels) p.max_levels = o->max_levels;
    if (o->base_case_size) p.base_max = o->base_case_size;
    if (o->block_size) p.block = o->block_size;
    if (o->seed) p.seed = o->seed;
    p.algorithm = o->algorithm;
    if (o->struct_size >= offsetof(kascade_opts, max_chain) + sizeof(uint32_t)) p.level0_mode = o->level0_mode;
  }
  if (p.base_max > ONE_CTA_MAX) p.base_max = ONE_CTA_MAX;
  if (p.block != 128 && p.block != 512) p.block = 256;
  if (p.spacing0 < 2) p.spacing0 = 2;
  if (p.spacing_deep == 1) p.spacing_deep = 2;
  return p;
}

Rulers level0_rulers(const Params& p) { return make_rulers(p.spacing0, salt_for(p.seed, 0)); }

namespace {

// How level 0 of n elements of that weight kind runs: the records' format, and
// whether it takes the write-free path.
struct Level0Plan {
  Format fmt;
  bool write_free;
};

// The three ways to run level 0, by what stays in L2 (lists of random order,
// unit / 32-bit / 64-bit weights, us):
//   split records and stamps while both fit: 4e6 elements 247 / 310 / 417
//     against 279 / 287 / 331 with the stamp in the record, 3e6 213 / 224
//     against 242 / 249, 6e6 396 / 500 / 617 against 384 / 389 / 444
//   stamps in 16 B records while those fit, 8e6: 531 / 536 / 605
//   write-free above: 8e6 522 / 528 / 653, 1.2e7 711 / 719 against 815 / 823
// F16i has 31 bits for ruler ids, Record8 for successors.
Level0Plan plan_level0(const Params& p, uint64_t n, WKind wk) {
  constexpr uint64_t SPLIT_BYTES = 88ull << 20;
  const uint64_t split = n * (wk == WKind::Unit ? 16 : wk == WKind::U32 ? 24 : 32);
  const uint64_t log_min = wk == WKind::I64 ? 12000000 : 8000000;
  Level0Plan plan;
  plan.write_free = p.level0_mode == 2 || (p.level0_mode != 1 && n >= log_min);
  if (!plan.write_free && split > SPLIT_BYTES && n / p.spacing0 + 1 < F16i::NONE)
    plan.fmt = Format::F16i;
  else if (n > REC8_MAX || wk == WKind::I64)
    plan.fmt = Format::F16x16;
  else
    plan.fmt = wk == WKind::Unit ? Format::F8x8 : Format::F8x16;
  return plan;
}

kascade_status alloc_level0(kascade_ctx& ctx, const Level0Plan& plan, uint64_t cap, Level0* l0) {
  const bool wide = plan.fmt == Format::F16x16 || plan.fmt == Format::F16i;
  l0->fmt = plan.fmt;
  l0->stamp = nullptr;
  l0->rec = alloc<char>(ctx, cap * (wide ? 16 : 8));
  if (!l0->rec) return KASCADE_ERR_OOM;
  if (plan.write_free) return KASCADE_OK;
  l0->stamp = plan.fmt == Format::F16i ? l0->rec : alloc<char>(ctx, cap * (plan.fmt == Format::F8x8 ? 8 : 16));
  return l0->stamp ? KASCADE_OK : KASCADE_ERR_OOM;
}

// The levels of n elements, and their arrays.
kascade_status alloc_levels(kascade_ctx& ctx, uint32_t n, const Params& p, Levels* lv) {
  *lv = Levels{};
  const int max_levels = (int)std::min<uint32_t>(p.max_levels, MAX_LEVELS);
  const uint32_t base = std::max(1u, p.base_max);
  int k = 0;
  lv->n[0] = n;
  while (lv->n[k] > base && k < max_levels) {
    const uint32_t sp = p.spacing_deep ? p.spacing_deep : deep_spacing(lv->n[k], ONE_CTA_MAX * 3 / 4);
    lv->rulers[k] = k == 0 ? level0_rulers(p) : make_rulers(sp, salt_for(p.seed, k));
    lv->n[k + 1] = ruler_count(lv->n[k], lv->rulers[k]);
    ++k;
  }
  lv->last = k;
  lv->rulers[k] = cta_rulers(lv->n[k]);
  ctx.last_levels.assign(lv->n, lv->n + k + 1);
  for (int i = 1; i <= k; ++i) {
    lv->rec[i] = alloc<Rec>(ctx, lv->n[i]);
    lv->stamp[i] = i < k ? alloc<uint4>(ctx, lv->n[i]) : nullptr;
    lv->rootel[i] = alloc<uint32_t>(ctx, lv->n[i]);
    lv->out[i] = alloc<Out>(ctx, lv->n[i]);
    if (!lv->rec[i] || (i < k && !lv->stamp[i]) || !lv->rootel[i] || !lv->out[i]) return KASCADE_ERR_OOM;
  }
  if (lv->n[k] > ONE_CTA_MAX) {
    for (PdRec*& j : lv->jump) {
      j = alloc<PdRec>(ctx, lv->n[k]);
      if (!j) return KASCADE_ERR_OOM;
    }
  }
  return KASCADE_OK;
}

kascade_status alloc_lists_as(kascade_ctx& ctx, const Params& p, const Level0Plan& plan, uint64_t n, Lists* l) {
  *l = Lists{};
  l->n = (uint32_t)n;
  l->write_free = plan.write_free;
  KS_TRY(alloc_level0(ctx, plan, n, &l->l0));
  if (n <= p.base_max) return KASCADE_OK;
  KS_TRY(alloc_levels(ctx, l->n, p, &l->lv));
  return plan.write_free ? alloc_log(ctx, l->n, l->lv.n[1], p, &l->log) : KASCADE_OK;
}

}  // namespace

kascade_status alloc_lists(kascade_ctx& ctx, const Params& p, uint64_t n, WKind wk, Lists* l) {
  const Level0Plan plan = plan_level0(p, n, wk);
  const kascade_status st = arena_try(ctx, [&] { return alloc_lists_as(ctx, p, plan, n, l); });
  if (st != KASCADE_ERR_OOM || !plan.write_free) return st;
  Params q = p;
  q.level0_mode = 1;
  return arena_try(ctx, [&] { return alloc_lists_as(ctx, q, plan_level0(q, n, wk), n, l); });
}

namespace {

template <class F, class W>
kascade_status prepare_plain(kascade_ctx& ctx, const uint64_t* succ, const W& w, uint32_t n, uint64_t start,
                             const Level0& l0, const Rulers& rl, cudaStream_t s) {
  if (start >= n) return KASCADE_OK;
  const uint64_t rest = n - start;
  const unsigned grid = grid_for(ctx, (rest + 256 * PREP_ITEMS - 1) / (256 * PREP_ITEMS) * 256, 256, 8);
  KS_TRY(launch(ctx, k_prepare_arrays<F, W>, grid, 256, 0, s, succ, w, n, start, rl, l0.records<F>(), l0.stamps<F>(),
                ctx.d_status));
  return KASCADE_OK;
}

// Full tiles of 16 B-aligned inputs go through the bulk-copy kernel, the rest
// through the plain one.
template <class F, bool W32, class W>
kascade_status prepare_tiles(kascade_ctx& ctx, const uint64_t* succ, const uint32_t* w32, const W& w, uint32_t n,
                             const Level0& l0, const Rulers& rl, cudaStream_t s) {
  uint64_t start = 0;
  const bool aligned = reinterpret_cast<uintptr_t>(succ) % 16 == 0 &&
                       (!W32 || reinterpret_cast<uintptr_t>(w32) % 16 == 0);
  const uint32_t ntiles = n / PT_TILE;
  if (aligned && ntiles >= (uint32_t)ctx.usable_sms()) {
    const unsigned g = (unsigned)std::min<uint64_t>(ntiles, (uint64_t)ctx.usable_sms() * 2);
    constexpr int smem = PT_STAGES * PT_TILE * (W32 ? 12 : 8);
    static std::atomic<uint64_t> raised{0};
    const uint64_t bit = 1ull << (ctx.device & 63);
    if (!(raised.load() & bit)) {
      KS_CUDA(cudaFuncSetAttribute(k_prepare_tma<F, W32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      raised.fetch_or(bit);
    }
    KS_TRY(launch(ctx, k_prepare_tma<F, W32>, g, 256, smem, s, succ, w32, n, ntiles, rl, l0.records<F>(),
                  l0.stamps<F>(), ctx.d_status));
    start = (uint64_t)ntiles * PT_TILE;
  }
  return prepare_plain<F>(ctx, succ, w, n, start, l0, rl, s);
}

}  // namespace

kascade_status prepare_arrays(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                              const Level0& l0, const Rulers& rl, cudaStream_t s) {
  ProfScope ps(ctx, "prepare", s);
  const uint32_t* w32 = static_cast<const uint32_t*>(w);
  if (wk == WKind::Unit && l0.fmt == Format::F8x8)
    return prepare_tiles<F8x8, false>(ctx, succ, nullptr, WUnit{}, n, l0, rl, s);
  if (wk == WKind::U32 && l0.fmt == Format::F8x16)
    return prepare_tiles<F8x16, true>(ctx, succ, w32, WU32{w32}, n, l0, rl, s);
  if (l0.fmt == Format::F16i) {
    if (wk == WKind::Unit) return prepare_tiles<F16i, false>(ctx, succ, nullptr, WUnit{}, n, l0, rl, s);
    if (wk == WKind::U32) return prepare_tiles<F16i, true>(ctx, succ, w32, WU32{w32}, n, l0, rl, s);
    return prepare_plain<F16i>(ctx, succ, WI64{static_cast<const int64_t*>(w)}, n, 0, l0, rl, s);
  }
  // 64-bit records (pointer doubling takes these for every weight kind)
  switch (wk) {
    case WKind::Unit:
      return prepare_plain<F16x16>(ctx, succ, WUnit{}, n, 0, l0, rl, s);
    case WKind::U32:
      return prepare_plain<F16x16>(ctx, succ, WU32{w32}, n, 0, l0, rl, s);
    default:
      return prepare_plain<F16x16>(ctx, succ, WI64{static_cast<const int64_t*>(w)}, n, 0, l0, rl, s);
  }
}

kascade_status rank_arrays_one_cta(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                                   const SinkPlain& sink, CtaMode mode, cudaStream_t s) {
  ctx.last_levels.assign(1, n);
  Extent ext;
  ext.cap = n;
  switch (wk) {
    case WKind::Unit:
      return launch_rank_cta(ctx, CtaArrays<WUnit>{succ, WUnit{}}, ext, sink, mode, true, s);
    case WKind::U32:
      return launch_rank_cta(ctx, CtaArrays<WU32>{succ, WU32{(const uint32_t*)w}}, ext, sink, mode, true, s);
    default:
      return launch_rank_cta(ctx, CtaArrays<WI64>{succ, WI64{(const int64_t*)w}}, ext, sink, mode, true, s);
  }
}

kascade_status rank_parents_one_cta(kascade_ctx& ctx, const uint32_t* parent, uint32_t n, const SinkBatch& sink,
                                    bool last, cudaStream_t s) {
  Extent ext;
  ext.cap = n;
  return launch_rank_cta(ctx, CtaArrays<WUnit, uint32_t>{parent, WUnit{}}, ext, sink, CTA_TREES, last, s);
}
kascade_status rank_trees_one_cta(kascade_ctx& ctx, const Rec8* rec, const uint32_t* rootel, const Extent& ext,
                                  uint2* out, cudaStream_t s) {
  return launch_rank_cta(ctx, CtaRecords<F8x8, true>{rec, rootel}, ext, SinkOut8{out}, CTA_TREES, false, s);
}
kascade_status rank_trees_one_cta(kascade_ctx& ctx, const Rec* rec, const uint32_t* rootel, const Extent& ext,
                                  Out* out, cudaStream_t s) {
  return launch_rank_cta(ctx, CtaRecords<F16x16, true>{rec, rootel}, ext, SinkOut{out}, CTA_TREES, false, s);
}

// Doubling for a fixed number of rounds, enough for any list the level can
// hold: no host wait.  Only a recursion depth limited by the caller ends on a
// level larger than one CTA ranks.
static kascade_status pointer_double_level(kascade_ctx& ctx, const Levels& lv, const Extent& ext, cudaStream_t s) {
  const uint32_t m = ext.cap;
  const Rec* rec = lv.rec[lv.last];
  PdRec *a = lv.jump[0], *b = lv.jump[1];
  const unsigned grid = grid_for(ctx, m, 256, 8);
  ProfScope ps(ctx, "pd_final_level", s);
  k_pd_init<<<grid, 256, 0, s>>>(rec, ext, a, ctx.d_status);
  KS_CHECK_LAUNCH();
  // rounds of reach x4 until 4^rounds >= 4m: any list of at most m elements
  int lg = 0;
  while ((1ull << lg) < m) ++lg;
  const int rounds = (lg + 1) / 2 + 1;
  for (int i = 0; i < rounds; ++i) {
    k_pd_round<<<grid, 256, 0, s>>>(a, b, ext);
    KS_CHECK_LAUNCH();
    std::swap(a, b);
  }
  k_pd_check<<<grid, 256, 0, s>>>(a, ext, ctx.d_status);
  KS_CHECK_LAUNCH();
  k_pd_final<SinkOut><<<grid, 256, 0, s>>>(a, ext, lv.rootel[lv.last], SinkOut{lv.out[lv.last]});
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

// Ruler gaps are geometric: longer than this has probability ~e^-64.
uint32_t hop_cap(const Rulers& rl) { return (uint32_t)std::min<uint64_t>(64ull * rl.s + 1024, 0xFFFFFFFFull); }

kascade_status rank_deep(kascade_ctx& ctx, const Levels& lv, cudaStream_t s) {
  for (int k = 1; k < lv.last; ++k)
    KS_TRY(launch_chase<F16x16>(ctx, lv, k, lv.rec[k], lv.stamp[k], 256, s));
  const int L = lv.last;
  Extent ext;
  ext.cap = lv.n[L];
  if (lv.n[L] <= ONE_CTA_MAX) {
    KS_TRY(launch_rank_cta(ctx, CtaRecords<F16x16, true>{lv.rec[L], lv.rootel[L]}, ext, SinkOut{lv.out[L]}, CTA_LISTS,
                           false, s));
  } else {
    KS_TRY(pointer_double_level(ctx, lv, ext, s));
  }
  for (int k = L - 1; k >= 1; --k)
    KS_TRY(launch_propagate<F16x16>(ctx, lv, k, lv.rec[k], lv.stamp[k], SinkOut{lv.out[k]}, false, s));
  return KASCADE_OK;
}

namespace {

template <class F, class Sink>
kascade_status rank_records_as(kascade_ctx& ctx, const Lists& l, const Sink& sink, CtaMode mode, const Params& p,
                               cudaStream_t s) {
  const typename F::R* rec = l.l0.records<F>();
  if (l.n <= p.base_max) {
    ctx.last_levels.assign(1, l.n);
    Extent ext;
    ext.cap = l.n;
    return launch_rank_cta(ctx, CtaRecords<F, false>{rec, nullptr}, ext, sink, mode, p.last, s);
  }
  KS_TRY(launch_chase<F>(ctx, l.lv, 0, rec, l.l0.stamps<F>(), p.block, s));
  KS_TRY(rank_deep(ctx, l.lv, s));
  return launch_propagate<F>(ctx, l.lv, 0, rec, l.l0.stamps<F>(), sink, p.last, s);
}

}  // namespace

template <class Sink>
kascade_status rank_records(kascade_ctx& ctx, const Lists& l, const Sink& sink, CtaMode mode, const Params& p,
                            cudaStream_t s) {
  if (l.n == 0) return KASCADE_OK;
  const bool wide = l.l0.fmt == Format::F16x16 || l.l0.fmt == Format::F16i;
  ctx.listed = Listed{l.l0.rec, wide, l.n, sink.log_target().seg};
  if (l.n > p.base_max && l.write_free) return rank_level0_log(ctx, l, sink.log_target(), p, s);
  switch (l.l0.fmt) {
    case Format::F8x8:
      return rank_records_as<F8x8>(ctx, l, sink, mode, p, s);
    case Format::F8x16:
      return rank_records_as<F8x16>(ctx, l, sink, mode, p, s);
    case Format::F16i:
      return rank_records_as<F16i>(ctx, l, sink, mode, p, s);
    default:
      return rank_records_as<F16x16>(ctx, l, sink, mode, p, s);
  }
}

kascade_status check_is_list(kascade_ctx& ctx, const uint64_t* succ, uint64_t n, int* ok, cudaStream_t s) {
  uint32_t* cnt = alloc<uint32_t>(ctx, n);
  uint32_t* bad = alloc<uint32_t>(ctx, 1);
  if (!cnt || !bad) return KASCADE_ERR_OOM;
  KS_CUDA(cudaMemsetAsync(cnt, 0, n * sizeof(uint32_t), s));
  KS_CUDA(cudaMemsetAsync(bad, 0, sizeof(uint32_t), s));
  unsigned grid = grid_for(ctx, n, 256, 8);
  {
    ProfScope ps(ctx, "is_list", s);
    k_count_preds<<<grid, 256, 0, s>>>(succ, n, cnt, bad);
    KS_CHECK_LAUNCH();
  }
  uint32_t b = 0;
  KS_TRY(read_u32(ctx, bad, &b, s));
  if (b & 2u) return KASCADE_ERR_OUT_OF_RANGE;
  *ok = (b & 1u) ? 0 : 1;
  return KASCADE_OK;
}

// explicit instantiations for the level-0 sinks
template kascade_status rank_records<SinkPlain>(kascade_ctx&, const Lists&, const SinkPlain&, CtaMode, const Params&,
                                                cudaStream_t);
template kascade_status rank_records<SinkBatch>(kascade_ctx&, const Lists&, const SinkBatch&, CtaMode, const Params&,
                                                cudaStream_t);

}  // namespace ks
