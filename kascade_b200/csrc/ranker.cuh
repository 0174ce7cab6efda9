// Internal interface of the ruling-set list ranker.
//
// Pipeline for a list of n elements:
//   prepare   : records {weight, successor} from the caller's arrays
//   chase     : every ruler walks its successors until the next ruler or the
//               list's end, stamping (ruler id, distance) for each element it
//               passes and writing the ruler's record of the next level
//   recurse   : the list of rulers is ranked the same way, down to a one-CTA
//               shared-memory ranker
//   propagate : one coalesced pass: rank = rank(ruler) - distance, root =
//               root(ruler); elements ahead of their list's first ruler walk
//               forward to the first element with a result
//
// Rulers are placed by position (struct Rulers): one in every block of s
// consecutive indices, at an offset hashed from the block's number.  A
// ruler's id is its block's number, so ids need no numbering pass, no list of
// ruler elements and no tag in the records: a chain knows from the index
// alone that the next element is a ruler and ends without reading it, and
// every level's size is ceil(n / s), known on the host before the first
// launch.  A gap between rulers along a list is at most as long as with
// independent samples of rate 1 / s (blocks that a gap meets more than once
// only help).
#pragma once

#include "common.cuh"
#include "ctx.cuh"

namespace ks {

struct Params {
  uint32_t spacing0 = 48;     // mean elements per ruler, level 0
  uint32_t spacing_given = 0;  // the caller's, if any
  uint32_t spacing_deep = 0;  // mean elements per ruler, deeper levels (0: by level size)
  uint32_t max_levels = 6;
  uint32_t base_max = 0x7FFFFFFFu;  // one-CTA ranker bound, at most ONE_CTA_MAX
  uint32_t block = 256;
  uint32_t seed = 0x6b617363u;
  uint32_t algorithm = KASCADE_ALGO_SPARSE_RULING_SET;
  uint32_t level0_mode = 0;  // 0: by size, 1: stamps, 2: write-free
  bool last = true;          // the ranking is the call's last device work
};

Params make_params(const kascade_ctx& ctx, const kascade_opts* opts, uint64_t n);

// Ruler placement of one level: element x lies in block x / s, whose ruler is
// at offset hash(block) in [0, s).  The last block's ruler may fall beyond
// the level's elements; its id is then dead (a record no element points to).
// Division by s: the round-up multiply-and-shift for any 32-bit x (Granlund and
// Montgomery, Division by Invariant Integers using Multiplication, 1994).
struct Rulers {
  uint32_t s = 2, mul = 0, sh = 0, salt = 0;
  __device__ __forceinline__ uint32_t offset(uint32_t j) const { return __umulhi(mix32(j ^ salt), s); }
  __device__ __forceinline__ uint64_t elem(uint32_t j) const { return (uint64_t)j * s + offset(j); }
  __device__ __forceinline__ uint32_t block_of(uint32_t x) const {
    const uint32_t t = __umulhi(x, mul);
    return (t + ((x - t) >> 1)) >> sh;
  }
  // whether x is a ruler; *j: its block (its id when it is one)
  __device__ __forceinline__ bool is(uint32_t x, uint32_t* j) const {
    const uint32_t b = block_of(x);
    *j = b;
    return x - b * s == offset(b);
  }
};
__host__ __device__ inline Rulers make_rulers(uint32_t s, uint32_t salt) {
  Rulers r;
  if (s < 2) {  // every element a ruler: the one-CTA ranker's placement on few elements
    r.s = 1;
    r.salt = salt;
    return r;
  }
  if (s > 0x80000000u) s = 0x80000000u;
  uint32_t l = 1;
  while (l < 31 && (1ull << l) < s) ++l;
  r.s = s;
  r.mul = (uint32_t)(((1ull << 32) * ((1ull << l) - s)) / s + 1);
  r.sh = l - 1;
  r.salt = salt;
  return r;
}
// The one-CTA ranker's rulers: at most CTA_RULERS.
constexpr uint32_t CTA_RULERS = 1024;
__host__ __device__ inline Rulers cta_rulers(uint32_t n) {
  return make_rulers((n + CTA_RULERS - 1) / CTA_RULERS, 0x63746121u);
}
inline uint32_t salt_for(uint32_t seed, int level) { return mix32(seed + 0x9E3779B9u * (uint32_t)(level + 1)); }
inline uint32_t ruler_count(uint32_t n, const Rulers& r) { return (uint32_t)(((uint64_t)n + r.s - 1) / r.s); }

// A level's element count when only the device knows it: *count / div, rounded
// up, at most the capacity the launch was sized for (count == nullptr: the
// capacity).
struct Extent {
  uint32_t cap = 0;
  const uint32_t* count = nullptr;
  uint32_t div = 1;
  __device__ __forceinline__ uint32_t get() const {
    if (!count) return cap;
    uint32_t v = ld_ca(count);
    if (div != 1) v = v / div + (v % div != 0u ? 1u : 0u);
    return min(cap, v);
  }
};

// Where results of level 0 go ------------------------------------------------
// A sink receives, for element x, its rank, its root (level-0 index) and
// whether x itself is a root.

// Level-0 output description for the write-free (log) pipeline.
struct LogTarget {
  uint64_t* root;
  uint64_t* rank;
  int keep_roots;  // leave roots' entries untouched
  SegMap seg;
};

// Plain arrays. keep_roots: leave root entries untouched (the reference's
// in-place contract); otherwise roots get (x, 0).
struct SinkPlain {
  uint64_t* root;
  uint64_t* rank;
  int keep_roots;
  LogTarget log_target() const { return LogTarget{root, rank, keep_roots, SegMap{}}; }
  __device__ __forceinline__ void put(uint32_t x, uint64_t rk, uint32_t rt, bool is_root) const {
    if (is_root) {
      if (!keep_roots) {
        __stcs(root + x, (unsigned long long)x);
        __stcs(rank + x, 0ull);
      }
      return;
    }
    __stcs(root + x, (unsigned long long)rt);
    __stcs(rank + x, (unsigned long long)rk);
  }
};

// A batch's lists or forests.
struct SinkBatch {
  uint64_t* root;
  uint64_t* rank;
  SegMap seg;
  LogTarget log_target() const { return LogTarget{root, rank, 0, seg}; }
  __device__ __forceinline__ void put(uint32_t x, uint64_t rk, uint32_t rt, bool is_root) const {
    const uint32_t j = seg.find(x);
    const uint32_t b = ld_ca(seg.base + j), g = x + ld_ca(seg.delta + j);
    __stcs(root + g, (unsigned long long)((is_root ? x : rt) - b));
    __stcs(rank + g, is_root ? 0ull : (unsigned long long)rk);
  }
};

// Deeper levels write Out records.
struct SinkOut {
  Out* out;
  __device__ __forceinline__ void put(uint32_t x, uint64_t rk, uint32_t rt, bool is_root) const {
    (void)is_root;  // a deeper level's list end carries its rank like every element
    st_out(out + x, rk, rt);
  }
};

// Results of a tree rooting's deeper levels: depths fit 32 bits.
struct SinkOut8 {
  uint2* out;  // (depth, root)
  __device__ __forceinline__ void put(uint32_t x, uint64_t rk, uint32_t rt, bool is_root) const {
    (void)is_root;
    __stcg(out + x, make_uint2((uint32_t)rk, rt));
  }
};

// Weight readers for building level-0 records.
enum class WKind { Unit, U32, I64 };

// Level 0 of a call: its records, and their stamps on the stamping path (null
// on the write-free one).
struct Level0 {
  Format fmt = Format::F16x16;
  void* rec = nullptr;
  void* stamp = nullptr;
  template <class F>
  typename F::R* records() const { return static_cast<typename F::R*>(rec); }
  template <class F>
  typename F::S* stamps() const { return static_cast<typename F::S*>(stamp); }
};

// The levels of one call.  Level k >= 1 holds level k - 1's rulers: records
// {distance, next ruler}, the root of a list end and results.
constexpr int MAX_LEVELS = 24;
struct Levels {
  int last = 0;                  // the level ranked by one CTA (or by doubling)
  uint32_t n[MAX_LEVELS + 1];    // elements per level
  Rulers rulers[MAX_LEVELS + 1];  // each level's rulers; the last one's: the one-CTA ranker's
  Rec* rec[MAX_LEVELS + 1];      // from level 1 on
  uint4* stamp[MAX_LEVELS + 1];  // from level 1 on, but not of the last level
  uint32_t* rootel[MAX_LEVELS + 1];  // level k >= 1: a list end's root as a level-0 element
  Out* out[MAX_LEVELS + 1];
  PdRec* jump[2];                // a last level that doubling ranks
};

// The write-free chase's log and what its entries are partitioned with
// (chase_log.cu).
struct LogEnt;
struct Log {
  LogEnt* ent = nullptr;
  uint32_t nchunks = 0;
  unsigned grid = 1;                 // blocks of the chase
  bool direct = false;               // one partition pass
  uint32_t* zero = nullptr;          // zeroed by one memset:
  uint64_t zero_words = 0;
  uint32_t *cursor = nullptr, *ucount = nullptr;   // the log's next chunk, unreached elements
  uint32_t *cursor1 = nullptr, *cursor2 = nullptr;  // windows, sub-windows
  uint32_t* fill = nullptr;                        // per chunk
  LogEnt *part = nullptr, *part2 = nullptr;
};

// What ranking a call's n list elements takes, allocated before anything that
// uses it is enqueued.
struct Lists {
  uint32_t n = 0;
  bool write_free = false;
  Level0 l0;
  Levels lv;  // above base_max elements
  Log log;    // write-free
};
// Write-free takes up to 2.8 times the stamping path's memory (2^26 elements in
// place 51 B an element against 18.1): a call whose memory does not suffice for
// it stamps.
kascade_status alloc_lists(kascade_ctx& ctx, const Params& p, uint64_t n, WKind wk, Lists* l);

// Level-0 records of a list from (succ, weights), stamps cleared; a root's
// record carries weight 0.
kascade_status prepare_arrays(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                              const Level0& l0, const Rulers& rl, cudaStream_t s);
Rulers level0_rulers(const Params& p);
uint32_t hop_cap(const Rulers& rl);

// Rank n <= ONE_CTA_MAX elements straight from the caller's arrays in one
// launch.  Any forest is accepted up to ONE_CTA_TREES elements; above, lists.
constexpr uint32_t ONE_CTA_MAX = 14336;
constexpr uint32_t ONE_CTA_TREES = 8192;
// What the one-CTA ranker takes: lists only; lists, and trees up to
// ONE_CTA_TREES elements; trees; trees, reporting their size as an Euler tour.
enum CtaMode : uint32_t { CTA_LISTS, CTA_SMALL_TREES, CTA_TREES, CTA_ROOTING };
kascade_status rank_arrays_one_cta(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                                   const SinkPlain& sink, CtaMode mode, cudaStream_t s);
// A forest's last level (its records' ruler bits are for cta_rulers(n)).
kascade_status rank_trees_one_cta(kascade_ctx& ctx, const Rec8* rec, const uint32_t* rootel, const Extent& ext,
                                  uint2* out, cudaStream_t s);
kascade_status rank_trees_one_cta(kascade_ctx& ctx, const Rec* rec, const uint32_t* rootel, const Extent& ext,
                                  Out* out, cudaStream_t s);
kascade_status rank_parents_one_cta(kascade_ctx& ctx, const uint32_t* parent, uint32_t n, const SinkBatch& sink,
                                    bool last, cudaStream_t s);
// A forest's levels: level k + 1 holds level k's rulers.
struct TreeLevels {
  int last = 0;
  Extent ext[MAX_LEVELS + 1];
  Rulers rulers[MAX_LEVELS + 1];
};
// Records, roots and results of the levels from 1 on.
template <class R, class O>
struct TreeRulers {
  R* rec[MAX_LEVELS + 1] = {};
  uint32_t* root[MAX_LEVELS + 1] = {};
  O* out[MAX_LEVELS + 1] = {};
};
// What rooting a forest takes, allocated before anything is enqueued (tree.cu).
struct Forest {
  uint32_t n = 0;
  TreeLevels lv;
  bool bits = false;  // child flags in bits
  char* inner = nullptr;
  uint32_t *sums = nullptr, *count = nullptr, *rec = nullptr, *vert = nullptr;
  uint2 *iw = nullptr, *out = nullptr;
  TreeRulers<Rec8, uint2> up;
};
// A batch's forests, parents in one compact vertex space.  last: the call's
// last device work.
kascade_status alloc_forests(kascade_ctx& ctx, uint32_t n, const Params& p, Forest* f);
kascade_status root_forests(kascade_ctx& ctx, const uint32_t* parent, const Forest& f, const SinkBatch& sink, bool last,
                            cudaStream_t s);
// Any forest: results of every element (tree.cu).
kascade_status rank_forest_weighted(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                                    const SinkPlain& sink, const Params& p, cudaStream_t s);

// Rank level-0 records and deliver the results to the sink.  Every level's
// size is known on the host: no host wait between the launches.
template <class Sink>
kascade_status rank_records(kascade_ctx& ctx, const Lists& l, const Sink& sink, CtaMode mode, const Params& p,
                            cudaStream_t s);

// Levels 1..last once the level-0 chase has written level 1: fills lv.out[1].
kascade_status rank_deep(kascade_ctx& ctx, const Levels& lv, cudaStream_t s);

// Where a level's chains put their rulers' records.  The last level has no
// stamps.
struct NextLevel {
  Rec* rec = nullptr;
  uint4* stamp = nullptr;
  uint32_t* rootel = nullptr;
  Rulers rl;
  // its chain ended at ruler `next`, or (next == id) at a list's end
  __device__ __forceinline__ void put(uint32_t id, uint64_t dist, uint32_t next) const {
    uint32_t j;
    Record16::put(rec + id, dist, next, rl.s == 1 || rl.is(next, &j));
    if (stamp) Stamp16::clear(stamp + id);
  }
};
inline NextLevel next_level(const Levels& lv, int k) {
  NextLevel nx;
  nx.rec = lv.rec[k];
  nx.stamp = lv.stamp[k];
  nx.rootel = lv.rootel[k];
  nx.rl = lv.rulers[k];
  return nx;
}

// Whether a walk from y never meets a ruler or a list's end (an invalid input's
// ruler-free cycle).  Only chains far beyond any plausible ruler gap ask.
template <class F>
__device__ __noinline__ bool endless(const typename F::R* rec, uint32_t y) {
  uint32_t mark = y;
  for (uint32_t hops = 1;; ++hops) {
    const Hop h = F::hop(rec + y);
    if (h.ruler || h.b == y) return false;
    y = h.b;
    if (y == mark) return true;
    if ((hops & (hops - 1)) == 0) mark = y;
  }
}

kascade_status compute_stats(kascade_ctx& ctx, const uint64_t* root, const int64_t* rank, uint64_t n, int level,
                             kascade_stats* out, kascade_tree_stats* per_tree, uint64_t per_tree_cap,
                             uint64_t* per_tree_count, cudaStream_t s);

// Write-free level 0: read-only chase that logs (element, ruler, distance),
// recursion on the ruler list, then two radix passes over the log by element
// and a dense placement into the outputs.
kascade_status alloc_log(kascade_ctx& ctx, uint32_t n, uint32_t rulers, const Params& p, Log* log);
kascade_status rank_level0_log(kascade_ctx& ctx, const Lists& l, const LogTarget& t, const Params& p, cudaStream_t s);

// Validation: *ok = 1 if no element has two predecessors.
kascade_status check_is_list(kascade_ctx& ctx, const uint64_t* succ, uint64_t n, int* ok,
                             cudaStream_t s);

}  // namespace ks
