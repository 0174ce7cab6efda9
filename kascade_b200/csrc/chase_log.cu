// Write-free level 0 of the ruling-set ranker.
//
// On B200 a random read costs a DRAM fetch of about 100 B whatever its width (98
// for the 8 B records here), and writing a record back after reading it roughly
// halves the random-access rate (16 B records: random read ~45 G/s, read + write
// back ~17-22 G/s; see `bench.py --calibrate`).  This path therefore never writes
// at a random address:
//
//   chase     read-only walk of every chain; each visited element appends
//             (element, ruler id, distance from ruler) to a log made of
//             1024-entry chunks that each warp takes from a global counter,
//             so the log is written with coalesced 16 B stores
//   recurse   the ruler sub-list (written by the chase in dense id space) is
//             ranked by the deeper levels
//   resolve   first radix pass over the log by element window (2^20
//             elements), resolving each entry on the way: rank = rank(ruler)
//             - distance, root = root(ruler).  Tiles of 2 K entries are
//             sorted by window in shared memory and written as one run per
//             window; the ruler lookups mostly hit L1 (a log chunk holds the
//             entries of a few hundred chains)
//   partition second radix pass: each window into 128 sub-windows of 2^13
//   place     one sub-window at a time: outputs assembled in shared memory
//             and written densely, so no output store is random
//   heads     elements ahead of their list's first ruler were never visited:
//             the place step finds them (no entry in their slot), presets
//             their root output to a NOT_REACHED sentinel and lists them;
//             each walks forward to the first element with outputs; a list
//             end that is no ruler itself is one of them
//
// Reference counterparts: the chase of sparse_ruling_set.cpp:147-273 (whose
// per-element writes are the reference's messages), ruler_propagation.hpp:
// 148-256 (pull) and post_invert.hpp:195-264 (unreached fix-up).
#include <algorithm>
#include <atomic>

#include "ranker.cuh"

namespace ks {

struct __align__(16) LogEnt {
  uint32_t x;
  uint32_t id;
  uint64_t off;
};

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr uint32_t LOG_CHUNK = 1024;  // entries per warp-owned log chunk
constexpr int LOG_REFILL = 6;         // idle lanes worth a refill
constexpr uint32_t LOG_CHAINS_PER_SM = 1024;
constexpr uint32_t WIN_SHIFT = 20;    // 2^20 elements per window (first partition pass)
constexpr uint32_t WIN = 1u << WIN_SHIFT;
constexpr uint32_t SUB_SHIFT = 13;  // 2^13 elements per sub-window (second pass; resolved in shared memory)
constexpr uint32_t SUB = 1u << SUB_SHIFT;
constexpr uint32_t SUBS = WIN / SUB;    // sub-windows per window
constexpr uint32_t MAX_BUCKETS = 4096;  // windows for 2^32 elements
constexpr uint32_t PT_THREADS = 256;    // partition: threads per block
// entries per thread (a tile is PT_THREADS x ITEMS entries) and resident
// blocks per SM of the two partition passes: 2048-entry tiles, 4 blocks per
// SM (more tiles in flight per SM than 4096-entry tiles at 2 blocks)
constexpr uint32_t P1_ITEMS = 8, P1_BLOCKS = 4;
constexpr uint32_t P2_ITEMS = 8, P2_BLOCKS = 4;
// One partition pass, straight to the sub-windows, up to as many of these as
// leave room for four blocks' counters on an SM (24.6 million elements); with
// three the pass loses to two of them whatever the order.  One / two passes, us:
//   runs of 64    1.6e7 645 / 706, 2e7 760 / 850, 2.4e7 911 / 993,
//                 2.8e7 1219 / 1148, 2^25 1922 / 1353
//   random order  1.4e7 777 / 787, 2e7 1130 / 1088, 2.4e7 1399 / 1297,
//                 2.8e7 1842 / 1503, 2^25 2806 / 1792
// (a tile of a random order has as many sub-windows as entries, and neither way
// of writing them coalesces).  A call that asks for this path takes two passes
// from 2^22 elements on.
constexpr uint32_t DIRECT_SUBS = 3000;
constexpr uint32_t DIRECT_MAX = DIRECT_SUBS * SUB, DIRECT_MAX_FORCED = 1u << 22;
static_assert(DIRECT_SUBS <= MAX_BUCKETS &&
                  P1_BLOCKS * (PT_THREADS * P1_ITEMS * 16 + DIRECT_SUBS * 8 + 1088) <= 228 * 1024,
              "four blocks on an SM");
constexpr uint32_t CURSOR_STRIDE = 8;   // one 32 B sector per cursor (spreads the atomics)
constexpr uint32_t FIN_THREADS = 512;  // place: threads per block (one sub-window per iteration; 2 blocks per SM)
constexpr uint32_t FIN_GROUP = 8;      // place: entries a thread has in flight
constexpr uint32_t NO_ROOT = 0xFFFFFFFFu;          // shared-memory root slot not written
constexpr unsigned long long NOT_REACHED = ~0ull;  // root output of an element no chain reached

__device__ __forceinline__ void st_log(LogEnt* p, uint32_t x, uint32_t id, uint64_t off) {
  __stcs(reinterpret_cast<uint4*>(p), make_uint4(x, id, (uint32_t)off, (uint32_t)(off >> 32)));
}

// A warp's place in the log: the chunk it owns (all values warp-uniform).
struct LogCursor {
  uint32_t pos = 0, end = 0;
};

// Warp-cooperative append of one entry per emitting lane.
__device__ __forceinline__ void log_append(bool emit, uint32_t x, uint32_t id, uint64_t off, LogCursor& cur,
                                           LogEnt* __restrict__ log, uint32_t* __restrict__ chunk_fill,
                                           uint32_t* __restrict__ chunk_cursor, uint32_t nchunks, uint32_t lane,
                                           uint32_t lt, DevStatus* st) {
  uint32_t m = __ballot_sync(FULL, emit);
  const uint32_t cnt = (uint32_t)__popc(m);
  if (cur.pos + cnt < cur.end) {  // all of them fit, and the chunk is not full after
    if (emit) st_log(log + cur.pos + __popc(m & lt), x, id, off);
    cur.pos += cnt;
    return;
  }
  while (m != 0u) {
    if (cur.pos == cur.end) {
      uint32_t ch = 0;
      if (lane == 0) ch = atomicAdd(chunk_cursor, 1u);
      ch = __shfl_sync(FULL, ch, 0);
      if (ch >= nchunks) {
        // more entries than elements: the input is not a forest of lists
        if (lane == 0) set_error(st, KASCADE_ERR_NOT_A_LIST, ch);
        return;
      }
      cur.pos = ch * LOG_CHUNK;
      cur.end = cur.pos + LOG_CHUNK;
    }
    const uint32_t take = min((uint32_t)__popc(m), cur.end - cur.pos);
    const uint32_t my = __popc(m & lt);
    const bool mine = emit && my < take;
    if (mine) st_log(log + cur.pos + my, x, id, off);
    m &= ~__ballot_sync(FULL, mine);
    emit = emit && !mine;
    cur.pos += take;
    if (cur.pos == cur.end && lane == 0) chunk_fill[(cur.pos - 1) / LOG_CHUNK] = LOG_CHUNK;
  }
}

// The read-only chase: one chain per thread, rulers and chain ends as in
// k_chase.  Every ruler and every element a chain passes is logged; a list's
// end is not (any number of chains may end there).  Bound by the random reads'
// DRAM fetches at large sizes and by instructions at L2-resident ones; 1024
// chains per SM are enough for either (2^28 elements: 768 / 1024 / 1536 / 2048
// chains 7.27 / 7.30 / 7.41 / 7.48 ms; two or four chains per thread are
// slower).
template <class F>
__global__ void __launch_bounds__(512) k_chase_log(const typename F::R* __restrict__ rec, uint32_t n, Rulers rl,
                                                   uint32_t r, NextLevel nx,
                                                   uint32_t* __restrict__ work, LogEnt* __restrict__ log, uint32_t* __restrict__ chunk_fill,
                                                   uint32_t* __restrict__ chunk_cursor, uint32_t nchunks,
                                                   uint32_t hop_cap, DevStatus* st) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = lanemask_lt();
  const uint32_t first = gridDim.x * blockDim.x;  // ids from here on are handed out by the counter
  uint32_t id = 0, x = 0, hops = 0;
  uint64_t acc = 0;
  Hop h{0, 0, false};  // the record of x, asked for
  bool act = false, own = false;  // own: x is the chain's first element
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
  const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i0 < r) begin(i0);
  bool more = first < r;  // warp-uniform
  LogCursor cur;
  while (true) {
    const uint32_t running = __ballot_sync(FULL, act);
    if (more && (running == 0u || __popc(running) <= 32 - LOG_REFILL)) {
      const uint32_t idle = ~running;
      uint32_t b = 0;
      if (lane == 0) b = first + atomicAdd(work, (uint32_t)__popc(idle));
      b = __shfl_sync(FULL, b, 0);
      if (b >= r) more = false;
      const uint32_t i = b + __popc(idle & lt);
      if (!act && i < r) begin(i);
      continue;
    }
    if (running == 0u) {
      if (!more) break;
      continue;
    }
    bool emit = false;
    const uint32_t lx = x, lid = id;
    const uint64_t ld = acc;
    if (act) {
      const uint32_t y = h.b;
      const uint64_t d = acc + h.w;
      const bool end = y == x, stop = end || h.ruler;
      emit = own || !end;
      own = false;
      if (!stop) {
        h = F::hop(rec + y);
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
      } else {
        uint32_t next = id;
        if (end) {
          nx.rootel[id] = x;
        } else {
          next = rl.block_of(y);
          // back at its own ruler: a rootless cycle holding one ruler
          if (next == id) set_error(st, KASCADE_ERR_CYCLE, id);
        }
        nx.put(id, d, next);
        act = false;
      }
    }
    log_append(emit, lx, lid, ld, cur, log, chunk_fill, chunk_cursor, nchunks, lane, lt, st);
  }
  if (lane == 0 && cur.end != 0 && cur.pos != cur.end)
    chunk_fill[(cur.end - 1) / LOG_CHUNK] = LOG_CHUNK - (cur.end - cur.pos);
}

// Exclusive prefix sum of v[0, m) in place (shared memory, m <= MAX_BUCKETS);
// returns the total to every thread.  Called by all threads of the block.
__device__ uint32_t block_exclusive_scan(uint32_t* v, uint32_t m) {
  __shared__ uint32_t warp_sum[PT_THREADS / 32];
  const uint32_t per = (m + PT_THREADS - 1) / PT_THREADS;
  const uint32_t lo = min(threadIdx.x * per, m), hi = min(lo + per, m);
  uint32_t sum = 0;
  for (uint32_t i = lo; i < hi; ++i) sum += v[i];
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  uint32_t inc = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, inc, d);
    if (lane >= (uint32_t)d) inc += t;
  }
  if (lane == 31) warp_sum[wid] = inc;
  __syncthreads();
  uint32_t before = 0, total = 0;
  for (uint32_t k = 0; k < PT_THREADS / 32; ++k) {
    if (k < wid) before += warp_sum[k];
    total += warp_sum[k];
  }
  uint32_t run = before + inc - sum;
  for (uint32_t i = lo; i < hi; ++i) {
    const uint32_t c = v[i];
    v[i] = run;
    run += c;
  }
  __syncthreads();
  return total;
}

// Radix partition of 16 B entries by element index.  A block loads a
// tile of PT_TILE entries into registers, counts them per bucket in shared
// memory, takes one global cursor step per bucket the tile touches, sorts
// the tile by bucket in shared memory and writes each bucket's run with
// consecutive threads: every global store is part of a contiguous run, so
// L2 sees whole lines instead of one 16 B piece per store.
//   FROM_LOG (first pass): tiles of PT_TILE_CHUNKS log chunks, buckets are
//     windows of 2^shift elements -- the sub-windows themselves where there
//     are few enough, and there is no second pass then.  Each log entry
//     (element, ruler id, distance)
//     is resolved on the way: rank = rank(ruler) - distance, root =
//     root(ruler), from the rulers' results of the recursion.  A log chunk
//     holds the entries of a few hundred chains, so most of these lookups
//     hit L1
//   otherwise (second pass): tiles inside one window's region, buckets are
//     its SUBS sub-windows
// More entries than a bucket holds means some element was logged twice.
//   used (first pass, optional): the chunks the chase took (its chunk
//     cursor); the chunks after them are empty and are skipped
template <bool FROM_LOG, uint32_t ITEMS, uint32_t BLOCKS>
__global__ void __launch_bounds__(PT_THREADS, BLOCKS) k_partition(const LogEnt* __restrict__ src,
                                                             const uint32_t* __restrict__ src_info, uint32_t nchunks,
                                                             const Out* __restrict__ out1, uint32_t limit,
                                                             uint32_t shift, uint32_t nb, LogEnt* __restrict__ dst,
                                                             uint32_t* __restrict__ dcursor,
                                                             const uint32_t* __restrict__ used, DevStatus* st) {
  constexpr uint32_t PT_TILE = PT_THREADS * ITEMS;
  constexpr uint32_t PT_TILE_CHUNKS = PT_TILE / LOG_CHUNK;
  static_assert(PT_TILE % LOG_CHUNK == 0 && WIN % PT_TILE == 0, "tiles hold whole log chunks");
  extern __shared__ __align__(16) unsigned char smraw[];
  uint4* stage = reinterpret_cast<uint4*>(smraw);
  const uint32_t nbk = FROM_LOG ? nb : SUBS;
  uint32_t* cnt = reinterpret_cast<uint32_t*>(stage + PT_TILE);  // counts, then the tile's offsets
  uint32_t* gbase = cnt + nbk;                                   // the tile's start in each bucket
  __shared__ uint32_t fills[PT_TILE_CHUNKS];
  if (FROM_LOG && used) nchunks = min(nchunks, __ldcg(used));
  const uint32_t ntiles =
      FROM_LOG ? (nchunks + PT_TILE_CHUNKS - 1) / PT_TILE_CHUNKS : nb * (WIN / PT_TILE);
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    uint32_t w = 0, valid_end = 0;  // second pass: window and its entry count
    uint64_t src0;                  // index of the tile's first entry
    if (FROM_LOG) {
      src0 = (uint64_t)t * PT_TILE;
    } else {
      w = t / (WIN / PT_TILE);
      const uint32_t k0 = (t % (WIN / PT_TILE)) * PT_TILE;
      const uint32_t c = min(__ldcg(src_info + (uint64_t)w * CURSOR_STRIDE), WIN);
      if (k0 >= c) continue;  // block-uniform
      valid_end = c - k0;
      src0 = (uint64_t)w * WIN + k0;
    }
    for (uint32_t b = threadIdx.x; b < nbk; b += PT_THREADS) cnt[b] = 0;
    if (FROM_LOG && threadIdx.x < PT_TILE_CHUNKS) {
      // a flat source (no fill table) holds `limit` entries in full chunks
      const uint32_t c = t * PT_TILE_CHUNKS + threadIdx.x;
      fills[threadIdx.x] = c >= nchunks ? 0u : src_info ? __ldcg(src_info + c) : min(LOG_CHUNK, limit - c * LOG_CHUNK);
    }
    __syncthreads();
    uint4 v[ITEMS];
    uint32_t pos[ITEMS];
#pragma unroll
    for (uint32_t k = 0; k < ITEMS; ++k) {
      const uint32_t e = k * PT_THREADS + threadIdx.x;
      const bool valid = FROM_LOG ? (e % LOG_CHUNK) < fills[e / LOG_CHUNK] : e < valid_end;
      v[k] = valid ? __ldcs(reinterpret_cast<const uint4*>(src + src0 + e)) : make_uint4(NO_ROOT, 0, 0, 0);
    }
    if (FROM_LOG && out1) {
      const uint64_t pol = l2_keep_policy();
#pragma unroll
      for (uint32_t k = 0; k < ITEMS; ++k) {
        if (v[k].x >= limit) continue;
        const Out o = ld_out_nc_keep(out1 + v[k].y, pol);
        const uint64_t rank = o.rank - ((uint64_t)v[k].z | ((uint64_t)v[k].w << 32));
        v[k] = make_uint4(v[k].x, o.root, (uint32_t)rank, (uint32_t)(rank >> 32));
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < ITEMS; ++k) {
      pos[k] = NO_ROOT;
      const uint32_t x = v[k].x;
      if (x < limit) {
        const uint32_t b = FROM_LOG ? x >> shift : (x >> SUB_SHIFT) & (SUBS - 1);
        pos[k] = atomicAdd(&cnt[b], 1u);
      }
    }
    __syncthreads();
    // one cursor step per bucket the tile touches.  In the second pass (one
    // bucket per thread) the step's result stays in a register until the
    // sorted tile is in place, so its round trip overlaps the scan and the
    // sort (1.60 -> 1.58 ms at 2^28; the first pass measured slower so)
    const bool one_per_thread = !FROM_LOG && nbk <= PT_THREADS;
    uint32_t g_mine = 0;
    for (uint32_t b = threadIdx.x; b < nbk; b += PT_THREADS) {
      const uint32_t c = cnt[b];
      const uint64_t ci = FROM_LOG ? (uint64_t)b * CURSOR_STRIDE : ((uint64_t)w * SUBS + b) * CURSOR_STRIDE;
      const uint32_t g = c ? atomicAdd(dcursor + ci, c) : 0u;
      if (one_per_thread)
        g_mine = g;
      else
        gbase[b] = g;
    }
    const uint32_t total = block_exclusive_scan(cnt, nbk);  // cnt now holds the tile's offsets
#pragma unroll
    for (uint32_t k = 0; k < ITEMS; ++k) {
      if (pos[k] == NO_ROOT) continue;
      const uint32_t x = v[k].x;
      const uint32_t b = FROM_LOG ? x >> shift : (x >> SUB_SHIFT) & (SUBS - 1);
      stage[cnt[b] + pos[k]] = v[k];
    }
    if (one_per_thread && threadIdx.x < nbk) gbase[threadIdx.x] = g_mine;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < total; i += PT_THREADS) {
      const uint4 e = stage[i];
      const uint32_t b = FROM_LOG ? e.x >> shift : (e.x >> SUB_SHIFT) & (SUBS - 1);
      const uint32_t p = gbase[b] + (i - cnt[b]);
      const uint32_t cap = FROM_LOG ? 1u << shift : SUB;
      if (p >= cap) {
        set_error(st, KASCADE_ERR_NOT_A_LIST, e.x);  // an element logged twice
        continue;
      }
      const uint64_t d = FROM_LOG ? ((uint64_t)b << shift) + p : (uint64_t)w * WIN + (uint64_t)b * SUB + p;
      __stcg(reinterpret_cast<uint4*>(dst + d), e);
    }
    __syncthreads();
  }
}

// Place: one sub-window (SUB elements) per block iteration.  Its entries
// (element, root, rank) are read in order and placed in shared memory by
// element, then the sub-window's outputs are written densely.  Elements
// without an entry were reached by no chain: their root output becomes
// NOT_REACHED and they join the unreached list.  seg: a batch's outputs.
// keep_roots: a root's rank output stays as it is (its root output already
// names it).
__global__ void __launch_bounds__(FIN_THREADS, 2) k_place(const LogEnt* __restrict__ part2,
                                                            const uint32_t* __restrict__ cursor2, uint32_t nb,
                                                            uint32_t limit, uint64_t* __restrict__ root_out,
                                                            uint64_t* __restrict__ rank_out,
                                                            uint32_t* __restrict__ ulist,
                                                            uint32_t* __restrict__ ucount, uint32_t ucap,
                                                            SegMap seg, int keep_roots, DevStatus* st) {
  extern __shared__ __align__(16) unsigned char smraw[];
  unsigned long long* rank_s = reinterpret_cast<unsigned long long*>(smraw);  // SUB entries
  uint32_t* root_s = reinterpret_cast<uint32_t*>(rank_s + SUB);               // SUB entries
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t items = nb * SUBS;
  for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
    const uint32_t lo = it * SUB;  // == window * WIN + sub-window * SUB
    if (lo >= limit) continue;     // block-uniform
    const uint32_t len = min(SUB, limit - lo);
    const uint32_t cnt = min(__ldcg(cursor2 + (uint64_t)it * CURSOR_STRIDE), SUB);
    for (uint32_t i = threadIdx.x; i < SUB; i += FIN_THREADS) root_s[i] = NO_ROOT;
    __syncthreads();
    const LogEnt* src = part2 + (uint64_t)it * SUB;
    for (uint32_t g = 0; g < SUB / FIN_THREADS; g += FIN_GROUP) {
      uint4 e[FIN_GROUP];
#pragma unroll
      for (uint32_t j = 0; j < FIN_GROUP; ++j) {
        const uint32_t i = (g + j) * FIN_THREADS + threadIdx.x;
        e[j] = i < cnt ? __ldcs(reinterpret_cast<const uint4*>(src + i)) : make_uint4(NO_ROOT, 0, 0, 0);
      }
#pragma unroll
      for (uint32_t j = 0; j < FIN_GROUP; ++j) {
        if (e[j].x == NO_ROOT) continue;
        const uint32_t xl = e[j].x - lo;
        if (xl >= len) {  // not this sub-window's: the partition passes wrote nothing like it
          set_error(st, KASCADE_ERR_NOT_A_LIST, e[j].x);
          continue;
        }
        if (atomicExch(&root_s[xl], e[j].y) != NO_ROOT) set_error(st, KASCADE_ERR_NOT_A_LIST, e[j].x);
        rank_s[xl] = (uint64_t)e[j].z | ((uint64_t)e[j].w << 32);
      }
    }
    __syncthreads();
    // a batch: the segment holding this thread's first element, its base and
    // the next one's; a thread's elements only move forward
    uint32_t jseg = 0, cur_base = 0, delta = 0, next_base = 0xFFFFFFFFu;
    if (seg.n && threadIdx.x < len) {
      jseg = seg.find(lo + threadIdx.x);
      cur_base = __ldg(seg.base + jseg);
      delta = __ldg(seg.delta + jseg);
      next_base = __ldg(seg.base + jseg + 1);
    }
    for (uint32_t i0 = 0; i0 < len; i0 += FIN_THREADS) {
      const uint32_t i = i0 + threadIdx.x;
      bool un = false;
      if (i < len) {
        const uint32_t r = root_s[i];
        un = r == NO_ROOT;
        while (seg.n && lo + i >= next_base) {  // (the last segment ends where the elements do)
          ++jseg;
          cur_base = next_base;
          delta = __ldg(seg.delta + jseg);
          next_base = __ldg(seg.base + jseg + 1);
        }
        const uint32_t g = lo + i + delta;
        __stcs(reinterpret_cast<unsigned long long*>(root_out) + g, un ? NOT_REACHED : (unsigned long long)(r - cur_base));
        const unsigned long long k = un ? 0ull : rank_s[i];
        if (!(keep_roots && (un || r == lo + i))) __stcs(reinterpret_cast<unsigned long long*>(rank_out) + g, k);
      }
      const uint32_t m = __ballot_sync(FULL, un);
      if (m == 0u) continue;
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(ucount, (uint32_t)__popc(m));
      base = __shfl_sync(FULL, base, 0);
      if (un) {
        const uint32_t p = base + __popc(m & lanemask_lt());
        if (p < ucap)
          ulist[p] = lo + i;
        else
          set_error(st, KASCADE_ERR_TOO_LARGE, p);
      }
    }
    __syncthreads();
  }
}

// Each unreached element walks forward to its list's end or to the first
// element with outputs: one the place step wrote (root output not
// NOT_REACHED) or one another walker finished.  Walkers write the rank,
// fence, then the root, and readers load the root, fence, then the rank, so a
// root seen set comes with its rank.  Roots already relative to their instance
// stay so (a walker and the element it stops at share an instance); a list
// end's root is made relative here.  keep_roots: a root's rank output is the
// caller's, its rank 0.
template <class F>
__global__ void __launch_bounds__(256) k_walk_unreached(const typename F::R* __restrict__ rec,
                                                        const uint32_t* __restrict__ ulist,
                                                        const uint32_t* __restrict__ ucount, uint32_t n,
                                                        uint64_t* root_out, uint64_t* rank_out, SegMap seg,
                                                        int keep_roots, DevStatus* st, unsigned long long* status) {
  const uint32_t cnt = min(*ucount, n);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
    const uint32_t u = ulist[i];
    uint32_t base = 0, delta = 0;
    if (seg.n) {
      const uint32_t j = seg.find(u);
      base = __ldg(seg.base + j);
      delta = __ldg(seg.delta + j);
    }
    uint64_t acc = 0;
    uint32_t y = u, mark = u, hops = 0;
    unsigned long long base_root = NOT_REACHED;
    bool ok = true;
    while (true) {
      const Hop h = F::hop(rec + y);
      acc += h.w;
      if (h.b == y) {  // the list's end
        base_root = y - base;
        break;
      }
      y = h.b;
      if (y >= n) {  // not reachable for a validated input; keeps every load in range
        set_error(st, KASCADE_ERR_OUT_OF_RANGE, u);
        ok = false;
        break;
      }
      const uint32_t g = y + delta;
      base_root = __ldcg(reinterpret_cast<const unsigned long long*>(root_out) + g);
      if (base_root != NOT_REACHED) {
        __threadfence();
        if (base_root + base != y || !keep_roots) acc += __ldcg(reinterpret_cast<const unsigned long long*>(rank_out) + g);
        break;
      }
      if (y == mark) {
        set_error(st, KASCADE_ERR_CYCLE, u);
        ok = false;
        break;
      }
      ++hops;
      if ((hops & (hops - 1)) == 0) mark = y;
    }
    if (!ok) continue;
    const uint32_t g = u + delta;
    if (!(keep_roots && base_root + base == u)) rank_out[g] = acc;
    __threadfence();
    root_out[g] = base_root;
  }
  publish_status(st, status);
}

constexpr uint32_t TILE1 = PT_THREADS * P1_ITEMS, TILE2 = PT_THREADS * P2_ITEMS;
auto k_part1 = k_partition<true, P1_ITEMS, P1_BLOCKS>;
auto k_part2 = k_partition<false, P2_ITEMS, P2_BLOCKS>;

// Kernel attributes are per device: the shared-memory limits are raised once
// on each.
kascade_status raise_smem_limits() {
  static std::atomic<uint64_t> raised{0};
  int dev = 0;
  KS_CUDA(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (raised.load() & bit) return KASCADE_OK;
  KS_CUDA(cudaFuncSetAttribute(k_part1, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(TILE1 * sizeof(LogEnt) + 2 * sizeof(uint32_t) * MAX_BUCKETS)));
  KS_CUDA(cudaFuncSetAttribute(k_part2, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(TILE2 * sizeof(LogEnt) + 2 * sizeof(uint32_t) * SUBS)));
  KS_CUDA(cudaFuncSetAttribute(k_place, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(SUB * (sizeof(unsigned long long) + sizeof(uint32_t)))));
  raised.fetch_or(bit);
  return KASCADE_OK;
}

template <class F>
kascade_status rank_level0_log_as(kascade_ctx& ctx, const Lists& l, const LogTarget& t, const Params& p,
                                  cudaStream_t s) {
  const Levels& lv = l.lv;
  const Log& log = l.log;
  const uint32_t n = l.n, r = lv.n[1];
  const uint32_t nb = (uint32_t)(((uint64_t)n + WIN - 1) / WIN);
  KS_CUDA(cudaMemsetAsync(log.zero, 0, sizeof(uint32_t) * log.zero_words, s));
  {
    ProfScope ps(ctx, "chase", s);
    k_chase_log<F><<<log.grid, p.block, 0, s>>>(l.l0.records<F>(), n, lv.rulers[0], r, next_level(lv, 1),
                                          &ctx.d_status->work[0], log.ent,
                                          log.fill, log.cursor, log.nchunks, hop_cap(lv.rulers[0]), ctx.d_status);
    KS_CHECK_LAUNCH();
  }
  KS_TRY(rank_deep(ctx, lv, s));

  // Up to DIRECT_MAX elements the log goes straight to the sub-windows;
  // larger ones in two passes, windows (part), then sub-windows (part2).
  const bool direct = log.direct;
  const uint32_t nsub = (uint32_t)(((uint64_t)n + SUB - 1) / SUB);
  KS_TRY(raise_smem_limits());
  if (direct) {
    ProfScope ps(ctx, "resolve", s);
    const uint32_t tiles = (log.nchunks + TILE1 / LOG_CHUNK - 1) / (TILE1 / LOG_CHUNK);
    const size_t smem = TILE1 * sizeof(LogEnt) + 2 * sizeof(uint32_t) * std::max(nsub, 1u);
    k_part1<<<(unsigned)std::min<uint64_t>(tiles, (uint64_t)ctx.usable_sms() * P1_BLOCKS), PT_THREADS, smem, s>>>(
        log.ent, log.fill, log.nchunks, lv.out[1], n, SUB_SHIFT, nsub, log.part, log.cursor2, log.cursor, ctx.d_status);
    KS_CHECK_LAUNCH();
  } else {
    const size_t smem1 = TILE1 * sizeof(LogEnt) + 2 * sizeof(uint32_t) * nb;
    const size_t smem2 = TILE2 * sizeof(LogEnt) + 2 * sizeof(uint32_t) * SUBS;
    {
      ProfScope ps(ctx, "resolve", s);
      const uint32_t tiles1 = (log.nchunks + TILE1 / LOG_CHUNK - 1) / (TILE1 / LOG_CHUNK);
      k_part1<<<(unsigned)std::min<uint64_t>(tiles1, (uint64_t)ctx.usable_sms() * P1_BLOCKS), PT_THREADS, smem1, s>>>(
          log.ent, log.fill, log.nchunks, lv.out[1], n, WIN_SHIFT, nb, log.part, log.cursor1, log.cursor, ctx.d_status);
      KS_CHECK_LAUNCH();
    }
    const uint32_t tiles2 = nb * (WIN / TILE2);
    if (tiles2) {
      ProfScope ps(ctx, "partition", s);
      k_part2<<<(unsigned)std::min<uint64_t>(tiles2, (uint64_t)ctx.usable_sms() * P2_BLOCKS), PT_THREADS, smem2, s>>>(
          log.part, log.cursor1, 0, nullptr, n, 0, nb, log.part2, log.cursor2, nullptr, ctx.d_status);
      KS_CHECK_LAUNCH();
    }
  }
  // the first pass's source or output is dead by now: it holds the unreached list
  uint32_t* ulist = reinterpret_cast<uint32_t*>(direct ? log.ent : log.part);
  {
    ProfScope ps(ctx, "place", s);
    const uint32_t items = nb * SUBS;
    const size_t smem = SUB * (sizeof(unsigned long long) + sizeof(uint32_t));
    k_place<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>(items, (uint64_t)ctx.usable_sms() * 2)),
                FIN_THREADS, smem, s>>>(log.part2, log.cursor2, nb, n, t.root, t.rank, ulist, log.ucount, n, t.seg, t.keep_roots,
                                        ctx.d_status);
    KS_CHECK_LAUNCH();
  }
  {
    ProfScope ps(ctx, "heads", s);
    k_walk_unreached<F><<<ctx.usable_sms() * 4, 256, 0, s>>>(l.l0.records<F>(), ulist, log.ucount, n, t.root, t.rank, t.seg,
                                                             t.keep_roots, ctx.d_status, status_host(ctx, p.last));
    KS_CHECK_LAUNCH();
  }
  return KASCADE_OK;
}

}  // namespace

kascade_status alloc_log(kascade_ctx& ctx, uint32_t n, uint32_t rulers, const Params& p, Log* log) {
  const uint64_t blocks = (uint64_t)ctx.usable_sms() * std::max(1u, LOG_CHAINS_PER_SM / p.block);
  log->grid = (unsigned)std::max<uint64_t>(1, std::min(blocks, ((uint64_t)rulers + p.block - 1) / p.block));
  const uint64_t warps = (uint64_t)log->grid * (p.block / 32);
  log->nchunks = (uint32_t)(((uint64_t)n + LOG_CHUNK - 1) / LOG_CHUNK + warps + 1);
  log->direct = n <= (p.level0_mode == 2 ? DIRECT_MAX_FORCED : DIRECT_MAX);
  const uint64_t nb = ((uint64_t)n + WIN - 1) / WIN, nsub = ((uint64_t)n + SUB - 1) / SUB;
  const uint64_t cursors = nb * (SUBS + 1) * CURSOR_STRIDE;
  log->ent = alloc<LogEnt>(ctx, (uint64_t)log->nchunks * LOG_CHUNK);
  log->zero_words = 8 + cursors + log->nchunks;
  log->zero = alloc<uint32_t>(ctx, log->zero_words);
  log->part = alloc<LogEnt>(ctx, log->direct ? nsub * SUB : nb * WIN);
  // the second pass's output takes the log's memory where that is large enough
  // (the log is dead by then)
  log->part2 = log->direct                                          ? log->part
               : (uint64_t)log->nchunks * LOG_CHUNK >= nsub * SUB ? log->ent
                                                                    : alloc<LogEnt>(ctx, nsub * SUB);
  if (!log->ent || !log->zero || !log->part || !log->part2) return KASCADE_ERR_OOM;
  log->cursor = log->zero;
  log->ucount = log->zero + 1;
  log->cursor1 = log->zero + 8;
  log->cursor2 = log->cursor1 + nb * CURSOR_STRIDE;
  log->fill = log->cursor1 + cursors;
  return KASCADE_OK;
}

kascade_status rank_level0_log(kascade_ctx& ctx, const Lists& l, const LogTarget& t, const Params& p, cudaStream_t s) {
  // records of 32-bit weights are alike with and without 64-bit stamps
  if (l.l0.fmt == Format::F16x16) return rank_level0_log_as<F16x16>(ctx, l, t, p, s);
  return rank_level0_log_as<F8x16>(ctx, l, t, p, s);
}

}  // namespace ks
