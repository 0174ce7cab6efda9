// Ruling-set list ranker and pointer doubling for one B200.
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
//                       609-700 -> double-buffered jump kernel
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
  __device__ __forceinline__ T operator()(uint64_t x) const { return __ldcs(p + x); }
};
struct WI64 {
  using T = uint64_t;
  const int64_t* p;
  __device__ __forceinline__ T operator()(uint64_t x) const {
    return (uint64_t)__ldcs(reinterpret_cast<const long long*>(p) + x);
  }
};

inline uint32_t salt_for(uint32_t seed, int level) { return mix32(seed + 0x9E3779B9u * (uint32_t)(level + 1)); }

// ---------------------------------------------------------------------------
// prepare: build records.  A root's weight is no part of any rank: its record
// carries 0, so that a chain ending at it adds the record's word like any.
// ---------------------------------------------------------------------------
__device__ __forceinline__ Rec make_rec(uint64_t w, uint64_t succ, uint64_t x) {
  Rec r;
  r.a = succ == x ? 0ull : w;
  r.b = (uint32_t)succ;
  r.c = TAG_UNREACHED;
  return r;
}

template <class W>
__global__ void __launch_bounds__(256, 4) k_prepare_arrays(const uint64_t* __restrict__ succ, W w, uint32_t n,
                                                        uint64_t start, Rec* __restrict__ rec, DevStatus* st) {
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
        sv[i] = __ldcs(reinterpret_cast<const unsigned long long*>(succ) + x);
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
      rec[x] = make_rec(wv[i], sv[i], x);
    }
  }
}

// The same work for 16 B-aligned inputs, with the input tiles moved by bulk
// (TMA) copies: a persistent block keeps PT_STAGES tiles of succ (and
// weights) in flight into shared memory while it writes the records of an
// earlier tile.  Full tiles only; the caller hands the tail to
// k_prepare_arrays.
constexpr int PT_TILE = 2048;
constexpr int PT_STAGES = 4;
constexpr int PT_ITEMS = PT_TILE / 256;

template <bool W32>
__global__ void __launch_bounds__(256) k_prepare_tma(const uint64_t* __restrict__ succ, const uint32_t* __restrict__ w,
                                                     uint32_t n, uint32_t ntiles, Rec* __restrict__ rec,
                                                     DevStatus* st) {
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
      st_rec_cs(rec + x, make_rec(wv[i], sv[i], x));
    }
  }
}

// The record of ruler `id` at the next level: its chain ended at ruler `next`,
// or (next == id) at the list's end, whose level-0 root goes to *rootel.
__device__ __forceinline__ void end_chain(Rec* rec_next, uint32_t id, uint64_t dist, uint32_t next) {
  Rec o;
  o.a = dist;
  o.b = next;
  o.c = TAG_UNREACHED;
  st_rec_cg(rec_next + id, o);
}

// ---------------------------------------------------------------------------
// chase: C chains in flight per thread, one per ruler.  A hop reads the 16 B
// record of the next element and stamps (distance from ruler, ruler id) into
// it.  A chain ends in front of the next ruler, known from the index alone,
// or at the list's end.  A warp's first rulers are its own share, later ones
// come from one counter; only the first `lanes` lanes of a warp work, so that
// few rulers spread over all SMs and a warp's hop waits for few loads (a
// dependent L2 hop costs 0.23 us alone and 0.43 us for 32 lanes together).
// A new chain's first load shares an iteration with the other lanes' hops.
// ---------------------------------------------------------------------------
// head_base: where level k >= 1 keeps its heads (level 0: heads.elem lists
// them).  A head's own record is stamped at distance 0.
template <int C>
__global__ void __launch_bounds__(512) k_chase(Rec* __restrict__ rec, Extent ext, Rulers rl, uint32_t rulers,
                                               Heads heads, uint32_t head_base,
                                               const uint32_t* __restrict__ rootel, Rec* __restrict__ rec_next,
                                               uint32_t* __restrict__ rootel_next, uint32_t* __restrict__ work,
                                               uint32_t lanes, DevStatus* st) {
  const uint32_t n = ext.get();
  const uint32_t r = rulers + heads.get();
  // level 0's size, reported by the call
  if (!rootel && ext.add && blockIdx.x == 0 && threadIdx.x == 0) st->counter[1] = n;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = lanemask_lt();
  const uint32_t batch = lanes * C;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  uint32_t cid[C], cx[C], hops[C];
  uint64_t acc[C];
  uint32_t act = 0, fresh = 0;  // bit c: chain c runs / has not read its ruler's record yet
  // warp-uniform: this warp's ruler ids at hand, and whether more may follow
  uint32_t q_base = warp * batch;
  uint32_t q_left = q_base < r ? r - q_base : 0u;
  if (q_left > batch) q_left = batch;
  const uint32_t first = warps * batch;  // ids from here on are handed out by the counter
  bool drained = false;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    cid[c] = cx[c] = hops[c] = 0;
    acc[c] = 0;
  }
  while (true) {
    if (!drained) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        bool need = lane < lanes && !((act >> c) & 1u);
        uint32_t m = __ballot_sync(FULL, need);
        while (m != 0u && !drained) {
          if (q_left == 0u) {
            uint32_t b = r;
            if (first < r) {
              uint32_t t = 0;
              if (lane == 0) t = atomicAdd(work, batch);
              b = first + __shfl_sync(FULL, t, 0);
            }
            if (b >= r) {
              drained = true;
              break;
            }
            q_base = b;
            q_left = r - b;
            if (q_left > batch) q_left = batch;
          }
          const uint32_t take = min((uint32_t)__popc(m), q_left);
          const uint32_t my_rank = __popc(m & lt);
          const bool mine = need && my_rank < take;
          if (mine) {
            const uint32_t id = q_base + my_rank;
            uint64_t x0;
            if (id < rulers)
              x0 = rl.elem(id);
            else
              x0 = rootel ? head_base + (id - rulers) : __ldg(heads.elem + (id - rulers));
            uint32_t j;
            if (x0 >= n) {
              end_chain(rec_next, id, 0, id);  // the last block's ruler, beyond the elements
            } else if (id >= rulers && rl.is((uint32_t)x0, &j) && j < rulers) {
              end_chain(rec_next, id, 0, j);  // a head that is a ruler itself
              rootel_next[id] = 0;
            } else {
              cid[c] = id;
              cx[c] = (uint32_t)x0;
              acc[c] = 0;
              hops[c] = 0;
              act |= 1u << c;
              fresh |= 1u << c;
            }
          }
          m &= ~__ballot_sync(FULL, mine);
          need = need && !mine;
          q_base += take;
          q_left -= take;
        }
      }
    }
    if (!__any_sync(FULL, act != 0u)) {
      if (drained) break;
      continue;
    }
    Rec rr[C];
#pragma unroll
    for (int c = 0; c < C; ++c)
      if ((act >> c) & 1u) rr[c] = ld_rec_cg(rec + cx[c]);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (!((act >> c) & 1u)) continue;
      const uint32_t x = cx[c], y = rr[c].b;
      const uint64_t d = acc[c];
      if (y == x) {  // the list's end (never stamped: any number of chains may end here)
        end_chain(rec_next, cid[c], d + rr[c].a, cid[c]);
        rootel_next[cid[c]] = rootel ? __ldg(rootel + x) : x;
        act &= ~(1u << c);
        fresh &= ~(1u << c);
        continue;
      }
      const bool start = (fresh >> c) & 1u;
      fresh &= ~(1u << c);
      if (!start || cid[c] >= rulers) {
        if (!tag_unreached(rr[c].c)) {  // stamped by another chain: two predecessors
          set_error(st, KASCADE_ERR_NOT_A_LIST, x);
          end_chain(rec_next, cid[c], 0, cid[c]);
          rootel_next[cid[c]] = 0;
          act &= ~(1u << c);
          continue;
        }
        Rec wv;
        wv.a = d;
        wv.b = y;
        wv.c = cid[c];
        st_rec_cg(rec + x, wv);
      }
      acc[c] = d + rr[c].a;
      cx[c] = y;
      uint32_t j;
      if (rl.is(y, &j)) {
        // back at its own ruler: a cycle without a root that holds one ruler
        if (j == cid[c]) set_error(st, KASCADE_ERR_CYCLE, j);
        end_chain(rec_next, cid[c], acc[c], j);
        rootel_next[cid[c]] = 0;
        act &= ~(1u << c);
      } else if (++hops[c] > n) {
        set_error(st, KASCADE_ERR_CYCLE, cid[c]);
        end_chain(rec_next, cid[c], 0, cid[c]);
        rootel_next[cid[c]] = 0;
        act &= ~(1u << c);
      }
    }
  }
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

template <class Sink>
__device__ __forceinline__ void walk_to_result(const Rec* __restrict__ rec, uint32_t x, uint32_t n_all,
                                               const Rulers& rl, const uint32_t* __restrict__ rootel,
                                               const Out* __restrict__ out_next, const Sink& sink, DevStatus* st) {
  Rec r = ld_rec_cg(rec + x);
  // Brent's cycle detection keeps an invalid (rootless, ruler-free) cycle to
  // O(cycle length) steps instead of n per element
  uint64_t acc = r.a;
  uint32_t y = r.b, hops = 0, lam = 0, power = 1, mark = x;
  while (true) {
    uint32_t id;
    if (rl.is(y, &id)) {
      const Out o = ld_out(out_next + id);
      sink.put(x, acc + o.rank, o.root, false);
      return;
    }
    r = ld_rec_cg(rec + y);
    if (!tag_unreached(r.c)) {
      const Out o = ld_out(out_next + r.c);
      sink.put(x, acc + o.rank - r.a, o.root, false);
      return;
    }
    acc += r.a;
    if (r.b == y) {
      sink.put(x, acc, rootel ? __ldg(rootel + y) : y, false);
      return;
    }
    if (y == mark || ++hops > n_all) {
      set_error(st, KASCADE_ERR_CYCLE, x);
      return;
    }
    if (++lam == power) {
      mark = y;
      power <<= 1;
      lam = 0;
    }
    y = r.b;
  }
}

template <class Sink, int ITEMS>
__global__ void __launch_bounds__(256) k_propagate(const Rec* __restrict__ rec, uint32_t n_out, Extent ext,
                                                   Rulers rl, uint32_t rulers, const uint32_t* __restrict__ rootel,
                                                   const Out* __restrict__ out_next, Sink sink, DevStatus* st) {
  __shared__ uint32_t walks[PROP_WALKS];
  __shared__ uint32_t nwalks;
  if (threadIdx.x == 0) nwalks = 0;
  __syncthreads();
  const uint32_t n_all = ext.get();  // records exist up to here
  n_out = min(n_out, n_all);
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint64_t pol = l2_keep_policy();
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x * ITEMS + threadIdx.x; base < n_out;
       base += (uint64_t)stride * ITEMS) {
    Rec rv[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint64_t x = base + (uint64_t)i * blockDim.x;
      if (x < n_out) rv[i] = ld_rec_cs(rec + x);
    }
    // every ruler's or stamped element's result, all loads in flight together
    // (they would otherwise wait behind the previous element's stores)
    Out ov[ITEMS];
    uint32_t found = 0;  // bit i: ov[i] holds the result of item i's ruler
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint64_t x = base + (uint64_t)i * blockDim.x;
      ov[i] = Out{0, 0, 0};
      if (x >= n_out) continue;
      uint32_t id;
      if (rl.is((uint32_t)x, &id) && id < rulers) {  // (a head's index may lie past the last block)
        rv[i].c = TAG_RULER;
        found |= 1u << i;
      } else if (!tag_unreached(rv[i].c)) {
        id = rv[i].c;
        found |= 1u << i;
      }
      if ((found >> i) & 1u) ov[i] = ld_out_keep(out_next + id, pol);
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint64_t x = base + (uint64_t)i * blockDim.x;
      if (x >= n_out) continue;
      const Rec r = rv[i];
      const bool is_root = r.b == (uint32_t)x && (r.c == TAG_RULER || tag_unreached(r.c));
      if ((found >> i) & 1u) {
        sink.put((uint32_t)x, ov[i].rank - (r.c == TAG_RULER ? 0ull : r.a), ov[i].root, is_root);
      } else if (is_root) {
        sink.put((uint32_t)x, r.a, rootel ? __ldg(rootel + x) : (uint32_t)x, true);
      } else {
        const uint32_t w = atomicAdd(&nwalks, 1u);
        if (w < PROP_WALKS)
          walks[w] = (uint32_t)x;
        else
          walk_to_result(rec, (uint32_t)x, n_all, rl, rootel, out_next, sink, st);
      }
    }
  }
  __syncthreads();
  for (uint32_t w = threadIdx.x; w < min(nwalks, PROP_WALKS); w += blockDim.x)
    walk_to_result(rec, walks[w], n_all, rl, rootel, out_next, sink, st);
}

// ---------------------------------------------------------------------------
// One CTA ranks up to ONE_CTA_MAX elements in shared memory: the last level
// of the recursion, or a whole small input straight from the caller's arrays.
// The elements are loaded once; at most CTA_RULERS rulers (placed as on every
// level) walk and stamp as in k_chase, pointer jumping ranks the rulers
// (<= 10 rounds), and every element reads its ruler's result.  Against
// pointer jumping over all elements (13 rounds of 16 elements per thread at
// 8192: 51 us) each element is touched once.  Each element's word also says
// whether its successor is a ruler or a list's end, so a hop is one exchange.
// With several lists, their heads (no predecessor) start chains as well, so
// that no run of elements ahead of a first ruler is walked element by element.
// Two chains that meet (a tree, not a list) are found by the exchange; an
// input of at most `tree_max` elements is then done again without stamps,
// every element walking to its first ruler, which ranks any forest.
// ---------------------------------------------------------------------------
constexpr uint32_t CTA_THREADS = 1024;
constexpr uint32_t CTA_RULERS = 1024;
constexpr uint32_t CTA_HEADS = 1024;
constexpr uint32_t CTA_CHAINS = CTA_RULERS / CTA_THREADS;
constexpr uint32_t CTA_LOADS = 8;           // elements a thread has in flight while loading
constexpr uint32_t CTA_ILP = 4;             // elements a thread has in flight in shared memory
constexpr uint32_t CTA_FLAG = 0x80000000u;  // next: stamped, low bits the chain; rnext: the list's end
constexpr uint32_t CTA_END = 0x40000000u;   // next: the successor ends the list
constexpr uint32_t CTA_RUL = 0x20000000u;   // next: the successor is a ruler
constexpr uint32_t CTA_IDX = 0x1FFFFFFFu;
constexpr size_t cta_smem(uint64_t n) {
  return (size_t)((n + CTA_RULERS + CTA_HEADS) * 12 + CTA_HEADS * 2 + (n + 31) / 32 * 4);
}

// Element sources: the records of a level (a list end's carries its rank), or
// the caller's arrays (a root's weight is no part of any rank).
struct CtaRecords {
  static constexpr bool kEndWeight = true;
  const Rec* rec;
  const uint32_t* rootel;
  __device__ __forceinline__ void load(uint32_t x, uint64_t* a, uint32_t* b) const {
    const Rec r = ld_rec_cg(rec + x);
    *a = r.a;
    *b = r.b;
  }
  __device__ __forceinline__ uint32_t root_of(uint32_t x) const { return rootel ? __ldg(rootel + x) : x; }
};
template <class W>
struct CtaArrays {
  static constexpr bool kEndWeight = false;
  const uint64_t* succ;
  W w;
  __device__ __forceinline__ void load(uint32_t x, uint64_t* a, uint32_t* b) const {
    const unsigned long long s = __ldcg(reinterpret_cast<const unsigned long long*>(succ) + x);
    *a = w(x);
    *b = s > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)s;  // beyond any element: found out of range
  }
  __device__ __forceinline__ uint32_t root_of(uint32_t x) const { return x; }
};

template <class Src, class Sink>
__global__ void __launch_bounds__(CTA_THREADS, 1) k_rank_cta(Src src, Extent ext, Sink sink, uint32_t tree_max,
                                                             int level0, DevStatus* st) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t nends, nheads;
  const uint32_t n = ext.get();
  unsigned long long* dist = reinterpret_cast<unsigned long long*>(smem);  // weight, once stamped the distance
  unsigned long long* rdist = dist + ext.cap;                              // per chain: distance, then rank
  uint32_t* next = reinterpret_cast<uint32_t*>(rdist + CTA_RULERS + CTA_HEADS);
  uint32_t* rnext = next + ext.cap;  // per chain: next ruler or CTA_FLAG | list end, then the root
  uint32_t* pred = rnext + CTA_RULERS + CTA_HEADS;
  uint16_t* hlist = reinterpret_cast<uint16_t*>(pred + (ext.cap + 31) / 32);
  const uint32_t tid = threadIdx.x;
  const uint32_t words = (n + 31) / 32;
  if (level0 && ext.add && tid == 0) st->counter[1] = n;
  const bool all = n <= CTA_RULERS;  // every element is a ruler
  const Rulers rl = make_rulers((n + CTA_RULERS - 1) / CTA_RULERS, 0x63746121u);
  const uint32_t rulers = all ? n : (n + rl.s - 1) / rl.s;
  auto ruler = [&](uint32_t x, uint32_t* j) {
    if (all) {
      *j = x;
      return true;
    }
    return rl.is(x, j);
  };
  bool stamp = true;
  uint32_t heads = 0;
  while (true) {
    if (tid == 0) nends = nheads = 0;
    for (uint32_t w = tid; w < words; w += CTA_THREADS) pred[w] = 0;
    __syncthreads();
    uint32_t ends = 0;
    for (uint32_t x0 = tid; x0 < n; x0 += CTA_THREADS * CTA_LOADS) {
      uint64_t a[CTA_LOADS];
      uint32_t b[CTA_LOADS];
#pragma unroll
      for (uint32_t i = 0; i < CTA_LOADS; ++i) {
        const uint32_t x = x0 + i * CTA_THREADS;
        if (x < n) src.load(x, &a[i], &b[i]);
      }
#pragma unroll
      for (uint32_t i = 0; i < CTA_LOADS; ++i) {
        const uint32_t x = x0 + i * CTA_THREADS;
        if (x >= n) continue;
        if (b[i] >= n) {
          set_error(st, KASCADE_ERR_OUT_OF_RANGE, x);
          b[i] = x;
        }
        dist[x] = (Src::kEndWeight || b[i] != x) ? a[i] : 0ull;
        next[x] = b[i];
        ends += b[i] == x ? 1u : 0u;
      }
    }
    ends = __reduce_add_sync(FULL, ends);
    if ((tid & 31u) == 0 && ends) atomicAdd(&nends, ends);
    __syncthreads();
    // what each successor is; with several lists, who has a predecessor
    const bool many = stamp && !all && nends > 2;
    for (uint32_t x0 = tid; x0 < n; x0 += CTA_THREADS * CTA_ILP) {
      uint32_t y[CTA_ILP], z[CTA_ILP];
#pragma unroll
      for (uint32_t i = 0; i < CTA_ILP; ++i) {
        const uint32_t x = x0 + i * CTA_THREADS;
        y[i] = x < n ? next[x] : x;
      }
#pragma unroll
      for (uint32_t i = 0; i < CTA_ILP; ++i) z[i] = x0 + i * CTA_THREADS < n ? next[y[i]] & CTA_IDX : 0u;
#pragma unroll
      for (uint32_t i = 0; i < CTA_ILP; ++i) {
        const uint32_t x = x0 + i * CTA_THREADS;
        uint32_t j;
        if (x >= n || y[i] == x) continue;
        next[x] = y[i] | (z[i] == y[i] ? CTA_END : 0u) | (ruler(y[i], &j) ? CTA_RUL : 0u);
        if (many) atomicOr(&pred[y[i] >> 5], 1u << (y[i] & 31));
      }
    }
    __syncthreads();
    if (many) {
      for (uint32_t w = tid; w < words; w += CTA_THREADS) {
        uint32_t m = ~pred[w];
        while (m) {
          const uint32_t x = w * 32 + (uint32_t)__ffs(m) - 1;
          m &= m - 1;
          uint32_t j;
          if (x >= n || next[x] == x || rl.is(x, &j)) continue;
          const uint32_t e = atomicAdd(&nheads, 1u);
          if (e < CTA_HEADS) hlist[e] = (uint16_t)x;
        }
      }
      __syncthreads();
      heads = min(nheads, CTA_HEADS);
    }
    // chains: ids of rulers, then (from CTA_RULERS on) of heads; a thread's
    // chains go hop by hop together
    uint32_t id[CTA_CHAINS], cur[CTA_CHAINS], hops = 0, act = 0;
    unsigned long long acc[CTA_CHAINS];
    int clash = 0;
    // the chain has passed acc and its next word is f: at its end, or at cur
    auto arrive = [&](uint32_t c, uint32_t f) {
      const uint32_t y = f & CTA_IDX;
      if (f & CTA_RUL) {
        rdist[id[c]] = acc[c];
        rnext[id[c]] = all ? y : rl.block_of(y);
        return false;
      }
      if (f & CTA_END) {
        rdist[id[c]] = acc[c] + dist[y];
        rnext[id[c]] = CTA_FLAG | y;
        return false;
      }
      cur[c] = y;
      return true;
    };
    auto begin = [&](uint32_t c) {
      uint32_t x0 = n;
      if (id[c] < rulers)
        x0 = all ? id[c] : (uint32_t)rl.elem(id[c]);
      else if (id[c] >= CTA_RULERS && id[c] - CTA_RULERS < heads)
        x0 = hlist[id[c] - CTA_RULERS];
      if (x0 >= n) return false;
      const uint32_t f = next[x0];
      acc[c] = dist[x0];
      if (f == x0) {
        rdist[id[c]] = acc[c];
        rnext[id[c]] = CTA_FLAG | x0;
        return false;
      }
      if (id[c] >= CTA_RULERS) {  // a head is stamped by its own chain
        next[x0] = CTA_FLAG | id[c];
        dist[x0] = 0;
      }
      return arrive(c, f);
    };
#pragma unroll
    for (uint32_t c = 0; c < CTA_CHAINS; ++c) {
      id[c] = tid + c * CTA_THREADS;
      cur[c] = 0;
      acc[c] = 0;
      bool on = begin(c);
      if (!on && heads) {
        id[c] += CTA_RULERS;
        on = begin(c);
      }
      if (on) act |= 1u << c;
    }
    while (act) {
      ++hops;
#pragma unroll
      for (uint32_t c = 0; c < CTA_CHAINS; ++c) {
        if (!((act >> c) & 1u)) continue;
        const uint32_t x = cur[c];
        const uint32_t f = stamp ? atomicExch(&next[x], CTA_FLAG | id[c]) : next[x];
        bool on = false;
        if ((f & CTA_FLAG) || hops > 2 * n) {
          // two chains met, or a cycle without a ruler
          if (f & CTA_FLAG) clash = 1;
          rdist[id[c]] = 0;
          rnext[id[c]] = id[c];  // never ends: the rounds below report the cycle
        } else {
          const unsigned long long w = dist[x];
          if (stamp) dist[x] = acc[c];
          acc[c] += w;
          on = arrive(c, f);
        }
        if (!on && id[c] < CTA_RULERS && heads) {
          id[c] += CTA_RULERS;
          on = begin(c);
        }
        if (!on) act &= ~(1u << c);
      }
    }
    clash = __syncthreads_or(clash);
    if (!clash) break;
    if (n > tree_max) {
      if (tid == 0) set_error(st, KASCADE_ERR_NOT_A_LIST, n);
      return;
    }
    stamp = false;  // again from the source, without stamps
    heads = 0;
  }
  // pointer jumping over the rulers
  for (int round = 0;; ++round) {
    unsigned long long d[CTA_CHAINS];
    uint32_t nx[CTA_CHAINS];
    int busy = 0;
#pragma unroll
    for (uint32_t c = 0; c < CTA_CHAINS; ++c) {
      const uint32_t j = tid + c * CTA_THREADS;
      nx[c] = CTA_FLAG;
      d[c] = 0;
      if (j >= rulers || (!all && rl.elem(j) >= n)) continue;
      nx[c] = rnext[j];
      d[c] = rdist[j];
      if (!(nx[c] & CTA_FLAG)) {
        d[c] += rdist[nx[c]];
        nx[c] = rnext[nx[c]];
        busy = 1;
      }
    }
    if (!__syncthreads_or(busy)) break;
    if (round > 11) {  // 2^11 > CTA_RULERS: what has not ended by now never does
      if (tid == 0) set_error(st, KASCADE_ERR_CYCLE, n);
      return;
    }
#pragma unroll
    for (uint32_t c = 0; c < CTA_CHAINS; ++c) {
      const uint32_t j = tid + c * CTA_THREADS;
      if (j >= rulers || (!all && rl.elem(j) >= n)) continue;
      rdist[j] = d[c];
      rnext[j] = nx[c];
    }
    __syncthreads();
  }
  // the heads' chains end at a ruler or a list end; then every chain's root
  for (uint32_t h = tid; h < heads; h += CTA_THREADS) {
    const uint32_t j = CTA_RULERS + h, nx = rnext[j];
    if (!(nx & CTA_FLAG)) {
      rdist[j] += rdist[nx];
      rnext[j] = rnext[nx];
    }
  }
  __syncthreads();
  for (uint32_t j = tid; j < CTA_RULERS + heads; j += CTA_THREADS)
    if (j < rulers ? (all || rl.elem(j) < n) : j >= CTA_RULERS) rnext[j] = src.root_of(rnext[j] & ~CTA_FLAG);
  __syncthreads();
  for (uint32_t x0 = tid; x0 < n; x0 += CTA_THREADS * CTA_ILP) {
    uint32_t f[CTA_ILP], j[CTA_ILP];
    unsigned long long d[CTA_ILP];
#pragma unroll
    for (uint32_t i = 0; i < CTA_ILP; ++i) {
      const uint32_t x = x0 + i * CTA_THREADS;
      f[i] = x < n ? next[x] : 0u;
      d[i] = x < n ? dist[x] : 0ull;
    }
#pragma unroll
    for (uint32_t i = 0; i < CTA_ILP; ++i) {
      const uint32_t x = x0 + i * CTA_THREADS;
      if (x >= n) continue;
      const bool end = f[i] == x;
      uint32_t root = 0;
      if (ruler(x, &j[i])) {
        d[i] = rdist[j[i]];
        root = rnext[j[i]];
      } else if (f[i] & CTA_FLAG) {
        d[i] = rdist[f[i] & CTA_IDX] - d[i];
        root = rnext[f[i] & CTA_IDX];
      } else if (end) {
        root = src.root_of(x);
      } else {  // ahead of its list's first ruler: walk
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
          if (w & CTA_END) {
            d[i] += dist[y];
            root = src.root_of(y);
            break;
          }
          w = next[y];
          if (w & CTA_FLAG) {
            d[i] += rdist[w & CTA_IDX] - dist[y];
            root = rnext[w & CTA_IDX];
            break;
          }
          d[i] += dist[y];
          if (++hops > n) {
            set_error(st, KASCADE_ERR_CYCLE, x);
            ok = false;
            break;
          }
        }
        if (!ok) continue;
      }
      sink.put(x, d[i], root, end);
    }
  }
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
// element not yet at its root follows its pointer JUMPS times there (a chain
// of dependent reads of `a` only, never of `b`), so a round multiplies every
// pointer's reach by JUMPS + 1.  JUMPS = 1 is classic doubling; the last level
// of the device-driven recursion (at most 2^17 elements, L2-resident, a fixed
// number of launches) takes JUMPS = 3: half the launches for three reads each.
template <int JUMPS>
__global__ void __launch_bounds__(256) k_pd_round(const PdRec* __restrict__ a, PdRec* __restrict__ b, Extent ext,
                                                  uint32_t* __restrict__ active) {
  const uint32_t n = ext.get();
  uint32_t cnt = 0;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (uint64_t)gridDim.x * blockDim.x) {
    PdRec e = a[x];
#pragma unroll
    for (int j = 0; j < JUMPS; ++j) {
      if (e.done & 1u) break;
      const PdRec t = a[e.succ];
      e.rank += t.rank;
      e.succ = t.succ;
      e.done = t.done & 1u;
    }
    cnt += (e.done & 1u) ? 0u : 1u;
    b[x] = e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(FULL, cnt, o);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(active, cnt);
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

// Resident blocks per SM of the chase, by chains per thread and block size.
template <int C>
int chase_occupancy(uint32_t block) {
  static std::atomic<int> occ[3] = {{-1}, {-1}, {-1}};  // blocks of 128, 256, 512 threads
  const int bi = block == 128 ? 0 : block == 512 ? 2 : 1;
  int v = occ[bi].load();
  if (v < 0) occ[bi].store(v = occupancy(k_chase<C>, (int)block, 0));
  return v;
}

// Warps that share a level's rulers before a warp works with more lanes: the
// L2 serves dependent hops of this many resident warps at full speed.
constexpr uint64_t CHASE_SPREAD_WARPS_PER_SM = 32;

template <int C>
kascade_status launch_chase_c(kascade_ctx& ctx, const Levels& lv, int k, const Extent& ext, uint32_t block,
                              cudaStream_t s) {
  const uint32_t r = lv.n[k + 1];
  const uint64_t wpb = block / 32;
  const uint64_t max_grid = (uint64_t)ctx.usable_sms() * chase_occupancy<C>(block);
  const uint64_t spread = std::min<uint64_t>(max_grid * wpb, (uint64_t)ctx.usable_sms() * CHASE_SPREAD_WARPS_PER_SM);
  const uint32_t lanes = (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, (r + spread * C - 1) / (spread * C)));
  const uint64_t need = ((uint64_t)r + lanes * C - 1) / (lanes * C);  // warps worth of work
  const unsigned grid = (unsigned)std::min<uint64_t>(max_grid, (need + wpb - 1) / wpb);
  ProfScope ps(ctx, "chase", s);
  k_chase<C><<<grid, block, 0, s>>>(lv.rec[k], ext, lv.rulers[k], lv.r[k], lv.heads, k ? lv.r[k - 1] : 0u,
                                    lv.rootel[k], lv.rec[k + 1], lv.rootel[k + 1], &ctx.d_status->work[k], lanes,
                                    ctx.d_status);
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

// Level k's chase (k = 0: the caller's records).
kascade_status launch_chase(kascade_ctx& ctx, const Levels& lv, int k, const Extent& ext, uint32_t chains,
                            uint32_t block, cudaStream_t s) {
  switch (chains) {
    case 1:
      return launch_chase_c<1>(ctx, lv, k, ext, block, s);
    case 4:
      return launch_chase_c<4>(ctx, lv, k, ext, block, s);
    default:
      return launch_chase_c<2>(ctx, lv, k, ext, block, s);
  }
}

// Level k's results from level k + 1's.  Small levels take two elements per
// thread instead of eight, so that they fill the chip.
template <class Sink>
kascade_status launch_propagate(kascade_ctx& ctx, const Levels& lv, int k, uint32_t n_out, const Extent& ext,
                                const Sink& sink, cudaStream_t s) {
  ProfScope ps(ctx, "propagate", s);
  if (n_out <= (uint64_t)ctx.usable_sms() * 256 * 8 * 4) {
    const unsigned grid = grid_for(ctx, ((uint64_t)n_out + 1) / 2, 256, 8);
    k_propagate<Sink, 2><<<grid, 256, 0, s>>>(lv.rec[k], n_out, ext, lv.rulers[k], lv.r[k], lv.rootel[k],
                                              lv.out[k + 1], sink, ctx.d_status);
  } else {
    const unsigned grid = grid_for(ctx, ((uint64_t)n_out + 7) / 8, 256, 8);
    k_propagate<Sink, 8><<<grid, 256, 0, s>>>(lv.rec[k], n_out, ext, lv.rulers[k], lv.r[k], lv.rootel[k],
                                              lv.out[k + 1], sink, ctx.d_status);
  }
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

template <class Src, class Sink>
kascade_status launch_rank_cta(kascade_ctx& ctx, const Src& src, const Extent& ext, const Sink& sink,
                               uint32_t tree_max, int level0, cudaStream_t s) {
  static std::atomic<uint64_t> raised{0};  // kernel attributes are per device
  const uint64_t bit = 1ull << (ctx.device & 63);
  if (!(raised.load() & bit)) {
    KS_CUDA(cudaFuncSetAttribute(k_rank_cta<Src, Sink>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)cta_smem(ONE_CTA_MAX)));
    raised.fetch_or(bit);
  }
  ProfScope ps(ctx, "base_case", s);
  k_rank_cta<Src, Sink><<<1, CTA_THREADS, cta_smem(ext.cap), s>>>(src, ext, sink, tree_max, level0, ctx.d_status);
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

// Ruler spacing of a deeper level of n elements: levels of equal spacing down
// to the one-CTA size, as many as cost least.  A level costs its longest
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
  // against ruler-table size; these defaults are the tuned values for
  // random lists on B200 (see the autotune table in the batch path).
  {
    const int k = ctx.class_of(n);
    p.spacing0 = ctx.class_spacing_single[k];
    p.chains = ctx.class_chains[k];
    p.block = ctx.class_block[k];
  }
  if (o) {
    if (o->ruler_spacing) p.spacing0 = o->ruler_spacing;
    if (o->ruler_spacing_deep) p.spacing_deep = o->ruler_spacing_deep;
    if (o->max_levels) p.max_levels = o->max_levels;
    if (o->base_case_size) p.base_max = o->base_case_size;
    if (o->chains_per_thread) p.chains = o->chains_per_thread;
    if (o->block_size) p.block = o->block_size;
    if (o->seed) p.seed = o->seed;
    p.algorithm = o->algorithm;
    if (o->struct_size >= offsetof(kascade_opts, max_chain) + sizeof(uint32_t)) {
      if (o->level0_mode == 1) p.level0_log_min = 0xFFFFFFFFu;
      if (o->level0_mode == 2) p.level0_log_min = 0;
      p.max_chain = o->max_chain;
    }
  }
  if (p.base_max > ONE_CTA_MAX) p.base_max = ONE_CTA_MAX;
  if (p.block != 128 && p.block != 512) p.block = 256;
  if (p.spacing0 < 2) p.spacing0 = 2;
  if (p.spacing_deep == 1) p.spacing_deep = 2;
  return p;
}

kascade_status prepare_arrays(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n, Rec* rec,
                              const Params& p, cudaStream_t s) {
  (void)p;
  ProfScope ps(ctx, "prepare", s);
  // full tiles of 16 B-aligned inputs go through the bulk-copy kernel
  uint64_t start = 0;
  const bool aligned = (reinterpret_cast<uintptr_t>(succ) % 16 == 0) &&
                       (wk == WKind::Unit || (wk == WKind::U32 && reinterpret_cast<uintptr_t>(w) % 16 == 0));
  const uint32_t ntiles = n / PT_TILE;
  if (aligned && ntiles >= (uint32_t)ctx.usable_sms()) {
    const unsigned g = (unsigned)std::min<uint64_t>(ntiles, (uint64_t)ctx.usable_sms() * 2);
    if (wk == WKind::U32) {
      constexpr int smem = PT_STAGES * PT_TILE * 12;
      static bool raised = false;
      if (!raised) {
        KS_CUDA(cudaFuncSetAttribute(k_prepare_tma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        raised = true;
      }
      k_prepare_tma<true><<<g, 256, smem, s>>>(succ, (const uint32_t*)w, n, ntiles, rec, ctx.d_status);
    } else {
      constexpr int smem = PT_STAGES * PT_TILE * 8;
      static bool raised = false;
      if (!raised) {
        KS_CUDA(cudaFuncSetAttribute(k_prepare_tma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        raised = true;
      }
      k_prepare_tma<false><<<g, 256, smem, s>>>(succ, nullptr, n, ntiles, rec, ctx.d_status);
    }
    KS_CHECK_LAUNCH();
    start = (uint64_t)ntiles * PT_TILE;
  }
  if (start < n) {
    const uint64_t rest = n - start;
    const unsigned grid = grid_for(ctx, (rest + 256 * PREP_ITEMS - 1) / (256 * PREP_ITEMS) * 256, 256, 8);
    switch (wk) {
      case WKind::Unit:
        k_prepare_arrays<WUnit><<<grid, 256, 0, s>>>(succ, WUnit{}, n, start, rec, ctx.d_status);
        break;
      case WKind::U32:
        k_prepare_arrays<WU32><<<grid, 256, 0, s>>>(succ, WU32{(const uint32_t*)w}, n, start, rec, ctx.d_status);
        break;
      case WKind::I64:
        k_prepare_arrays<WI64><<<grid, 256, 0, s>>>(succ, WI64{(const int64_t*)w}, n, start, rec, ctx.d_status);
        break;
    }
    KS_CHECK_LAUNCH();
  }
  return KASCADE_OK;
}

kascade_status rank_arrays_one_cta(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                                   const SinkPlain& sink, cudaStream_t s) {
  ctx.last_levels.assign(1, n);
  Extent ext;
  ext.cap = n;
  switch (wk) {
    case WKind::Unit:
      return launch_rank_cta(ctx, CtaArrays<WUnit>{succ, WUnit{}}, ext, sink, ONE_CTA_TREES, 1, s);
    case WKind::U32:
      return launch_rank_cta(ctx, CtaArrays<WU32>{succ, WU32{(const uint32_t*)w}}, ext, sink, ONE_CTA_TREES, 1, s);
    default:
      return launch_rank_cta(ctx, CtaArrays<WI64>{succ, WI64{(const int64_t*)w}}, ext, sink, ONE_CTA_TREES, 1, s);
  }
}

template <class Sink>
kascade_status pointer_double_records(kascade_ctx& ctx, const Rec* rec, uint32_t n, const uint32_t* elem0,
                                      const Sink& sink, cudaStream_t s) {
  if (n == 0) return KASCADE_OK;
  PdRec* a = alloc<PdRec>(ctx, n);
  PdRec* b = alloc<PdRec>(ctx, n);
  uint32_t* active = alloc<uint32_t>(ctx, 1);
  if (!a || !b || !active) return KASCADE_ERR_OOM;
  unsigned grid = grid_for(ctx, n, 256, 8);
  Extent ext;
  ext.cap = n;
  {
    ProfScope ps(ctx, "pd_init", s);
    k_pd_init<<<grid, 256, 0, s>>>(rec, ext, a, ctx.d_status);
    KS_CHECK_LAUNCH();
  }
  int rounds = 0;
  while (true) {
    KS_CUDA(cudaMemsetAsync(active, 0, sizeof(uint32_t), s));
    {
      ProfScope ps(ctx, "pd_round", s);
      k_pd_round<1><<<grid, 256, 0, s>>>(a, b, ext, active);
      KS_CHECK_LAUNCH();
    }
    PdRec* t = a;
    a = b;
    b = t;
    uint32_t left = 0;
    KS_TRY(read_u32(ctx, active, &left, s));
    if (left == 0) break;
    if (++rounds > 64) {
      ctx.error_info = left;
      return KASCADE_ERR_CYCLE;
    }
  }
  {
    ProfScope ps(ctx, "pd_final", s);
    k_pd_final<Sink><<<grid, 256, 0, s>>>(a, ext, elem0, sink);
    KS_CHECK_LAUNCH();
  }
  return KASCADE_OK;
}

// Doubling for a fixed number of rounds, enough for any list the level can
// hold: no host wait.  Only a recursion depth limited by the caller ends on a
// level larger than one CTA ranks.
static kascade_status pointer_double_level(kascade_ctx& ctx, const Rec* rec, const Extent& ext,
                                           const uint32_t* rootel, Out* out, cudaStream_t s) {
  const uint32_t m = ext.cap;
  PdRec* a = alloc<PdRec>(ctx, m);
  PdRec* b = alloc<PdRec>(ctx, m);
  uint32_t* active = alloc<uint32_t>(ctx, 1);
  if (!a || !b || !active) return KASCADE_ERR_OOM;
  const unsigned grid = grid_for(ctx, m, 256, 8);
  ProfScope ps(ctx, "pd_final_level", s);
  k_pd_init<<<grid, 256, 0, s>>>(rec, ext, a, ctx.d_status);
  KS_CHECK_LAUNCH();
  // rounds of reach x4 until 4^rounds >= 4m: any list of at most m elements
  int lg = 0;
  while ((1ull << lg) < m) ++lg;
  const int rounds = (lg + 1) / 2 + 1;
  for (int i = 0; i < rounds; ++i) {
    k_pd_round<3><<<grid, 256, 0, s>>>(a, b, ext, active);
    KS_CHECK_LAUNCH();
    std::swap(a, b);
  }
  k_pd_check<<<grid, 256, 0, s>>>(a, ext, ctx.d_status);
  KS_CHECK_LAUNCH();
  k_pd_final<SinkOut><<<grid, 256, 0, s>>>(a, ext, rootel, SinkOut{out});
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

kascade_status plan_levels(kascade_ctx& ctx, uint32_t n, const Heads& heads, const Params& p, Levels* lv) {
  *lv = Levels{};
  const int max_levels = (int)std::min<uint32_t>(p.max_levels, MAX_LEVELS);
  lv->heads = heads;
  // the last level holds the heads too: a caller's base case below them takes none
  if (p.base_max < 2 * heads.cap) lv->heads = Heads{};
  const uint32_t extra = lv->heads.cap;
  const uint32_t base = std::max(1u, p.base_max - extra);
  int k = 0;
  uint32_t m = n;  // the elements of level k that rulers are placed among
  lv->n[0] = n;
  while (m > base && k < max_levels) {
    const uint32_t sp = k == 0           ? p.spacing0
                        : p.spacing_deep ? p.spacing_deep
                                         : deep_spacing(m, ONE_CTA_MAX - extra);
    lv->rulers[k] = make_rulers(sp, salt_for(p.seed, k));
    lv->r[k] = m = ruler_count(m, lv->rulers[k]);
    lv->n[k + 1] = m + extra;
    ++k;
  }
  lv->last = k;
  ctx.last_levels.assign(1, n);
  for (int i = 1; i <= k; ++i) {
    ctx.last_levels.push_back(lv->r[i - 1]);
    lv->rec[i] = alloc<Rec>(ctx, lv->n[i]);
    lv->rootel[i] = alloc<uint32_t>(ctx, lv->n[i]);
    lv->out[i] = alloc<Out>(ctx, lv->n[i]);
    if (!lv->rec[i] || !lv->rootel[i] || !lv->out[i]) return KASCADE_ERR_OOM;
  }
  return KASCADE_OK;
}

kascade_status rank_deep(kascade_ctx& ctx, const Levels& lv, const Params& p, cudaStream_t s) {
  // deeper levels are L2-resident: one chain per thread saturates the L2
  (void)p;
  for (int k = 1; k < lv.last; ++k) KS_TRY(launch_chase(ctx, lv, k, lv.extent(k), 1, 256, s));
  const int L = lv.last;
  if (lv.n[L] <= ONE_CTA_MAX) {
    KS_TRY(launch_rank_cta(ctx, CtaRecords{lv.rec[L], lv.rootel[L]}, lv.extent(L), SinkOut{lv.out[L]}, 0, 0, s));
  } else {
    KS_TRY(pointer_double_level(ctx, lv.rec[L], lv.extent(L), lv.rootel[L], lv.out[L], s));
  }
  for (int k = L - 1; k >= 1; --k) KS_TRY(launch_propagate(ctx, lv, k, lv.n[k], lv.extent(k), SinkOut{lv.out[k]}, s));
  return KASCADE_OK;
}

template <class Sink>
kascade_status rank_records(kascade_ctx& ctx, Rec* rec, uint32_t n, const Extent& ext, const Heads& heads,
                            const Sink& sink, const Params& p, cudaStream_t s, bool host_check) {
  if (n == 0) return KASCADE_OK;
  if (n <= p.base_max) {
    ctx.last_levels.assign(1, n);
    return launch_rank_cta(ctx, CtaRecords{rec, nullptr}, ext, sink, ONE_CTA_TREES, 1, s);
  }
  if (Sink::kWriteFree && n >= p.level0_log_min && !sink.log_target(n).keep_roots) {
    const kascade_status st = rank_level0_log(ctx, rec, n, ext, heads, sink.log_target(n), p, s, host_check);
    if (!host_check || st != KASCADE_ERR_TIMEOUT) return st;
    // a chain exceeded the write-free path's hop cap (invalid input, or an
    // astronomically unlikely ruler gap): redo level 0 on the stamping path
    KS_TRY(status_reset(ctx, s));
  }
  Levels lv;
  KS_TRY(plan_levels(ctx, n, heads, p, &lv));
  lv.rec[0] = rec;
  KS_TRY(launch_chase(ctx, lv, 0, ext, p.chains, p.block, s));
  KS_TRY(rank_deep(ctx, lv, p, s));
  return launch_propagate(ctx, lv, 0, sink.limit(n), ext, sink, s);
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
template kascade_status rank_records<SinkPlain>(kascade_ctx&, Rec*, uint32_t, const Extent&, const Heads&,
                                                const SinkPlain&, const Params&, cudaStream_t, bool);
template kascade_status rank_records<SinkTour>(kascade_ctx&, Rec*, uint32_t, const Extent&, const Heads&,
                                               const SinkTour&, const Params&, cudaStream_t, bool);
template kascade_status rank_records<SinkBatch>(kascade_ctx&, Rec*, uint32_t, const Extent&, const Heads&,
                                                const SinkBatch&, const Params&, cudaStream_t, bool);
template kascade_status pointer_double_records<SinkPlain>(kascade_ctx&, const Rec*, uint32_t, const uint32_t*,
                                                          const SinkPlain&, cudaStream_t);

}  // namespace ks
