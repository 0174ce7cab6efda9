// Ranking in-trees: every element's distance to its root and that root, for
// any forest -- tree rooting (unit weights: depths) and the pointer-doubling
// entry points (any weights).
//
// Reference: rank_via_euler_tour (lib/kascade/eulertour.cpp:337-377) and
// pointer_doubling (lib/kascade/pointer_doubling.hpp:18-43).  The reference
// roots a forest by ranking its Euler tour, a list of up to 2n elements; the
// results, a vertex's root and depth, are those of the path from the vertex to
// its root, so paths are contracted instead and no tour is built.
//
// Rulers are placed by position as for lists.  Every ruler walks to the next
// ruler or root above it; those distances are a forest on the rulers, which is
// ranked the same way, down to the size one CTA ranks; then every element
// walks to its first ruler and adds that ruler's result.  Paths merge, so
// nothing is stamped: elements above several rulers are read by each of them,
// which costs no more, as a walk's expected length is the spacing s whatever
// the forest's shape (rulers are placed independently of it), and the longest
// of n walks is s ln n.  Walks only read: elements near the roots, which many
// walks pass, stay in L1.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "ranker.cuh"

namespace ks {

namespace {

constexpr int TREE_THREADS = 256;
constexpr int TREE_PREP_ITEMS = 8;
// Child flags in bytes up to here, see k_tree_inner; beside a batch's lists to
// twice that (8e7 vertices of a 2^28-element batch: 10.0 ms, 10.7 in bits, whose
// atomics wait behind the chase's traffic).
constexpr uint32_t TREE_BYTES_MAX = 1u << 26, TREE_BYTES_MAX_BATCH = 1u << 27;
constexpr int TREE_REC_ITEMS = 4;  // (8: 95 registers; 2^26 vertices 3.89 -> 3.83 ms, 4.2e6 228 -> 221 us)
constexpr int TREE_OUT_ITEMS = 4;  // (2: 1.07 ms, 4 and 8: 0.95 for 2^26 vertices)
// Mean elements per ruler.  Large levels are bound by what they read at
// random, (s + 1) s / (s - 1) reads an element over all levels; small ones by
// their longest walks and by launches.  2^26 caterpillars, s = 2 / 3 / 4:
// 4.0 / 4.2 / 4.4 ms; 4.2M random recursive trees 314 / 275 / 250 us.  A
// caller's spacing counts up to TREE_SPACING: without stamps a walk reads all of
// its gap, so that the spacings lists are fast with are slow here (a path of
// 2^25 vertices, s = 2 / 8 / 24 / 48: 2.9 / 5.3 / 10.1 / 17.3 ms).
constexpr uint32_t TREE_SPACING = 4, TREE_SPACING_LARGE = 2, TREE_LARGE = 1u << 23;
// Largest last level: without stamps the one-CTA ranker's walks grow with its
// spacing (3100 elements 15 us, 6200 24, 8300 44, 12500 75; a level above it
// costs ~13 us).
constexpr uint32_t TREE_BASE = 4096;

// Level formats.  kEndWeight: a root's record carries its rank.
// Level 0 of a tree rooting: the parent and whether it is a ruler, 4 B.
struct TreeUnit {
  using R = uint32_t;
  static constexpr bool kEndWeight = false;
  static __device__ __forceinline__ Hop hop(const R* p) {
    const uint32_t v = ld_ca(p);
    return Hop{1, v & ~REC8_RULER, (v & REC8_RULER) != 0u};
  }
};
// Deeper levels of one: depths in 32 bits.
struct Tree8 {
  using R = Rec8;
  using O = uint2;  // rank, root
  static constexpr bool kEndWeight = true;
  static __device__ __forceinline__ Hop hop(const R* p) {
    return Record8::unpack(ld_ca(reinterpret_cast<const uint2*>(p)));
  }
  static __device__ __forceinline__ Out out(const O* p) {
    const uint2 v = ld_ca(p);
    return Out{v.x, v.y, 0};
  }
  static __device__ __forceinline__ void put(R* p, uint64_t w, uint32_t b, bool ruler) { Record8::put(p, w, b, ruler); }
};
// 64-bit weights.
struct Tree16 {
  using R = Rec;
  using O = Out;
  static constexpr bool kEndWeight = true;  // (level 0: prepared as 0)
  static __device__ __forceinline__ Hop hop(const R* p) {
    const uint4 v = ld_ca(reinterpret_cast<const uint4*>(p));
    return Hop{(uint64_t)v.x | ((uint64_t)v.y << 32), v.z, v.w != 0u};
  }
  static __device__ __forceinline__ Out out(const O* p) { return ld_out(p); }
  static __device__ __forceinline__ void put(R* p, uint64_t w, uint32_t b, bool ruler) {
    Record16::put(p, w, b, ruler);
  }
};

// ---------------------------------------------------------------------------
// Tree rooting works on the vertices that have children, renumbered densely:
// a leaf is on nobody's path, and its result is its parent's with one more
// step.  Half the vertices of random recursive trees and of caterpillars are
// leaves; what the walks read at random is then half as large (2^26
// caterpillars: 134 MB instead of 268, about the L2).
// ---------------------------------------------------------------------------
constexpr int WORDS_PER = 8;  // words of 32 vertices a thread counts
constexpr uint32_t WORDS_TILE = TREE_THREADS * WORDS_PER;

// Parents are the caller's 64-bit indices, or a batch's in one vertex space.
template <class P>
__device__ __forceinline__ uint64_t parent_of(const P* parent, uint64_t v, uint32_t n) {
  return v < n ? ld_cs(parent + v) : v;
}

// A flag set for every vertex with a child (zeroed by the caller).  A parent
// out of range is reported; its vertex counts as a root everywhere.
// Bytes, stored plainly, while they stay in L2; above 2^26 vertices bits, asked
// for before the atomic (an atomic for every vertex comes one at a time where
// a few hubs have all the leaves: 15 ms instead of 1 at 2^26).  Flags and
// numbering of random recursive trees, bytes / bits: 2^25 vertices 0.45 / 0.45
// ms, 2^26 0.87 / 0.92, 2^27 3.61 / 2.01, 2^28 10.7 / 4.3; ten thousand hubs at
// 2^26 6.0 / 4.5.
template <class P, class I>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_inner(const P* parent, uint32_t n,
                                                             I* __restrict__ inner, DevStatus* st) {
  kernel_begin();
  const uint64_t tile_sz = (uint64_t)blockDim.x * TREE_PREP_ITEMS;
  for (uint64_t tile = (uint64_t)blockIdx.x * tile_sz; tile < n; tile += (uint64_t)gridDim.x * tile_sz) {
    uint64_t p[TREE_PREP_ITEMS];
#pragma unroll
    for (int i = 0; i < TREE_PREP_ITEMS; ++i) p[i] = parent_of(parent, tile + (uint64_t)i * blockDim.x + threadIdx.x, n);
#pragma unroll
    for (int i = 0; i < TREE_PREP_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      if (p[i] >= n) {
        if (v < n) set_error(st, KASCADE_ERR_OUT_OF_RANGE, v);
        p[i] = v;
      }
      if (p[i] == v) continue;
      if constexpr (sizeof(I) == 1) {
        __stcg(inner + p[i], (unsigned char)1);
      } else {
        const uint32_t b = (uint32_t)p[i], bit = 1u << (b & 31);
        if (!(ld_cg(inner + (b >> 5)) & bit)) atomicOr(inner + (b >> 5), bit);
      }
    }
  }
}

__device__ __forceinline__ uint32_t inner_word(const uint32_t* inner, uint32_t w) { return ld_cg(inner + w); }
// The bits of 32 vertices' bytes (each 0 or 1).
__device__ __forceinline__ uint32_t inner_word(const unsigned char* inner, uint32_t w) {
  const uint4 a = ld_cg(reinterpret_cast<const uint4*>(inner) + 2ull * w);
  const uint4 b = ld_cg(reinterpret_cast<const uint4*>(inner) + 2ull * w + 1);
  auto four = [](uint32_t v) { return (v * 0x01020408u) >> 24; };  // byte i's bit to bit i
  return four(a.x) | four(a.y) << 4 | four(a.z) << 8 | four(a.w) << 12 | four(b.x) << 16 | four(b.y) << 20 |
         four(b.z) << 24 | four(b.w) << 28;
}

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* sm) {  // all threads get it
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31u) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
#pragma unroll
  for (int i = 0; i < TREE_THREADS / 32; ++i) t += sm[i];
  __syncthreads();
  return t;
}

// Vertices with children per tile of words.
template <class I>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_count(const I* inner, uint32_t words,
                                                             uint32_t* __restrict__ sums) {
  kernel_begin();
  __shared__ uint32_t sm[TREE_THREADS / 32];
  const uint32_t base = blockIdx.x * WORDS_TILE;
  uint32_t c = 0;
#pragma unroll
  for (int i = 0; i < WORDS_PER; ++i) {
    const uint32_t w = base + i * TREE_THREADS + threadIdx.x;
    if (w < words) c += __popc(inner_word(inner, w));
  }
  c = block_sum(c, sm);
  if (threadIdx.x == 0) sums[blockIdx.x] = c;
}

// iw[w] = (bits, bits set before word w), and their number.  A block adds up
// the tiles before its own.
template <class I>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_number(const I* inner, uint32_t words,
                                                              const uint32_t* sums,
                                                              uint2* __restrict__ iw, uint32_t* __restrict__ count) {
  kernel_begin();
  __shared__ uint32_t sm[TREE_THREADS / 32];
  __shared__ uint32_t tile[WORDS_TILE];
  uint32_t before = 0;
  for (uint32_t b = threadIdx.x; b < blockIdx.x; b += TREE_THREADS) before += ld_ca(sums + b);
  before = block_sum(before, sm);
  const uint32_t base = blockIdx.x * WORDS_TILE;
#pragma unroll
  for (int i = 0; i < WORDS_PER; ++i) {
    const uint32_t w = base + i * TREE_THREADS + threadIdx.x;
    tile[i * TREE_THREADS + threadIdx.x] = w < words ? inner_word(inner, w) : 0u;
  }
  __syncthreads();
  uint32_t mine = 0;
#pragma unroll
  for (int i = 0; i < WORDS_PER; ++i) mine += __popc(tile[threadIdx.x * WORDS_PER + i]);
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += t;
  }
  if (lane == 31u) sm[threadIdx.x >> 5] = incl;
  __syncthreads();
  uint32_t pre = before + incl - mine;
  for (uint32_t i = 0; i < (threadIdx.x >> 5); ++i) pre += sm[i];
#pragma unroll
  for (int i = 0; i < WORDS_PER; ++i) {
    const uint32_t at = threadIdx.x * WORDS_PER + i;
    const uint32_t bits = tile[at];
    if (base + at < words) iw[base + at] = make_uint2(bits, pre);
    pre += __popc(bits);
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == TREE_THREADS - 1) *count = pre;
}

// A vertex with children: its number.
__device__ __forceinline__ uint32_t number_of(uint2 w, uint32_t v) {
  return w.y + (uint32_t)__popc(w.x & ((1u << (v & 31)) - 1u));
}

// The records of the numbered vertices; vert: their vertices (the roots').
// report: the elements of the forest's Euler tour with a leaf's two edges as
// one (the vertices, and once more those with children that are not roots), the
// size a call reports for level 0, go to the status.
template <class P>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_records(const P* parent, uint32_t n,
                                                               const uint2* iw, Rulers rl,
                                                               uint32_t* __restrict__ rec,
                                                               uint32_t* __restrict__ vert, bool report,
                                                               DevStatus* st) {
  kernel_begin();
  const uint64_t tile_sz = (uint64_t)blockDim.x * TREE_REC_ITEMS;
  uint32_t downs = 0;
  for (uint64_t tile = (uint64_t)blockIdx.x * tile_sz; tile < n; tile += (uint64_t)gridDim.x * tile_sz) {
    uint64_t p[TREE_REC_ITEMS];
    uint2 own[TREE_REC_ITEMS], up[TREE_REC_ITEMS];
#pragma unroll
    for (int i = 0; i < TREE_REC_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      p[i] = parent_of(parent, v, n);
      own[i] = v < n ? ld_ca(iw + (v >> 5)) : make_uint2(0, 0);
    }
#pragma unroll
    for (int i = 0; i < TREE_REC_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      if (p[i] >= n) p[i] = v;
      if (!((own[i].x >> (v & 31)) & 1u)) p[i] = ~0ull;  // a leaf
      up[i] = p[i] < n ? ld_ca(iw + (p[i] >> 5)) : make_uint2(0, 0);
    }
#pragma unroll
    for (int i = 0; i < TREE_REC_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      if (p[i] >= n) continue;
      const uint32_t c = number_of(own[i], (uint32_t)v);
      uint32_t b = number_of(up[i], (uint32_t)p[i]), j;
      if (p[i] == v)
        vert[c] = (uint32_t)v;
      else
        ++downs, b |= rl.is(b, &j) ? REC8_RULER : 0u;
      rec[c] = b;
    }
  }
  if (!report) return;
  downs = __reduce_add_sync(0xffffffffu, downs);
  if ((threadIdx.x & 31u) == 0 && downs) atomicAdd(&st->counter[1], (unsigned long long)downs);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&st->counter[1], (unsigned long long)n);
}

// Every vertex's result from the numbered ones' (depth, root).  `parent` may be
// the sink's root array: a thread reads the parents of the vertices of its own
// step only, all before it writes their results.
template <class P, class Sink>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_leaves(const P* parent, uint32_t n,
                                                              const uint2* iw,
                                                              const uint2* out, Sink sink,
                                                              DevStatus* st, unsigned long long* status) {
  kernel_begin();
  const uint64_t tile_sz = (uint64_t)blockDim.x * TREE_OUT_ITEMS;
  for (uint64_t tile = (uint64_t)blockIdx.x * tile_sz; tile < n; tile += (uint64_t)gridDim.x * tile_sz) {
    uint64_t p[TREE_OUT_ITEMS];
    uint2 w[TREE_OUT_ITEMS], o[TREE_OUT_ITEMS];
    bool leaf[TREE_OUT_ITEMS];
#pragma unroll
    for (int i = 0; i < TREE_OUT_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      p[i] = parent_of(parent, v, n);
      w[i] = v < n ? ld_ca(iw + (v >> 5)) : make_uint2(0, 0);
    }
#pragma unroll
    for (int i = 0; i < TREE_OUT_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      if (p[i] >= n) p[i] = v;
      leaf[i] = !((w[i].x >> (v & 31)) & 1u);
      if (leaf[i] && p[i] != v) w[i] = ld_ca(iw + (p[i] >> 5));
    }
#pragma unroll
    for (int i = 0; i < TREE_OUT_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      o[i] = make_uint2(0, 0);
      if (p[i] != v) o[i] = ld_ca(out + number_of(w[i], leaf[i] ? (uint32_t)p[i] : (uint32_t)v));
    }
#pragma unroll
    for (int i = 0; i < TREE_OUT_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      if (v < n) sink.put((uint32_t)v, o[i].x + (leaf[i] ? 1u : 0u), o[i].y, p[i] == v);
    }
  }
  publish_status(st, status);
}

// ---------------------------------------------------------------------------
// Levels.
// ---------------------------------------------------------------------------
// Every ruler's walk to the next ruler or its root.  next.s == 0: the last
// level's rulers are the one-CTA ranker's.
template <class L, class N>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_chase(const typename L::R* rec, Extent ext,
                                                             Rulers rl, Extent next_ext,
                                                             const uint32_t* rootel,
                                                             typename N::R* __restrict__ nrec,
                                                             uint32_t* __restrict__ nroot, Rulers nrl,
                                                             uint32_t hop_cap, DevStatus* st) {
  kernel_begin();
  const uint32_t n = ext.get(), rulers = next_ext.get();
  if (nrl.s == 0) nrl = cta_rulers(rulers);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rulers; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t id = (uint32_t)i;
    const uint64_t x0 = rl.elem(id);
    uint64_t acc = 0;
    uint32_t next = id, k;
    if (x0 < n) {  // (the last block's ruler may lie beyond the elements)
      uint32_t x = (uint32_t)x0, hops = 0;
      while (true) {
        const Hop h = L::hop(rec + x);
        if (h.b == x) {
          if (L::kEndWeight) acc += h.w;
          nroot[id] = rootel ? ld_ca(rootel + x) : x;
          break;
        }
        acc += h.w;
        if (h.ruler) {
          next = rl.block_of(h.b);
          if (next == id) set_error(st, KASCADE_ERR_CYCLE, id);  // back at itself
          break;
        }
        x = h.b;
        if (++hops == hop_cap) {
          hops = 0;
          if (endless<L>(rec, x)) {
            set_error(st, KASCADE_ERR_CYCLE, id);
            break;
          }
        }
      }
    }
    N::put(nrec + id, acc, next, nrl.s == 1 || nrl.is(next, &k));
  }
}

// Every element's result: its ruler's, or the first ruler's on its path.
template <class L, class N, class Sink>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_propagate(const typename L::R* rec, Extent ext,
                                                                 Rulers rl, const uint32_t* rootel,
                                                                 const typename N::O* out, Sink sink,
                                                                 DevStatus* st, unsigned long long* status) {
  kernel_begin();
  const uint32_t n = ext.get();
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)v;
    Hop h = L::hop(rec + x);
    if (h.b == x) {
      sink.put(x, L::kEndWeight ? h.w : 0ull, rootel ? ld_ca(rootel + x) : x, true);
      continue;
    }
    uint32_t j;
    if (rl.is(x, &j)) {
      const Out o = N::out(out + j);
      sink.put(x, o.rank, o.root, false);
      continue;
    }
    uint64_t acc = h.w;
    uint32_t y = h.b, hops = 0, mark = x;
    while (!h.ruler) {
      h = L::hop(rec + y);
      if (h.b == y) break;
      acc += h.w;
      if (y == mark && hops) break;  // a cycle without rulers
      ++hops;
      if ((hops & (hops - 1)) == 0) mark = y;
      y = h.b;
    }
    if (h.ruler) {
      const Out o = N::out(out + rl.block_of(y));
      sink.put(x, acc + o.rank, o.root, false);
    } else if (h.b == y) {
      sink.put(x, L::kEndWeight ? acc + h.w : acc, rootel ? ld_ca(rootel + y) : y, false);
    } else {
      set_error(st, KASCADE_ERR_CYCLE, x);
    }
  }
  publish_status(st, status);
}

// Levels of n elements, or of as many of them as *count says.
TreeLevels plan_tree(uint32_t n, const uint32_t* count, const Params& p) {
  TreeLevels lv;
  const uint32_t base = std::max(1u, std::min(p.base_max, TREE_BASE));
  int k = 0;
  lv.ext[0].cap = n;
  lv.ext[0].count = count;
  while (lv.ext[k].cap > base && k < MAX_LEVELS) {
    const uint32_t given = k == 0 ? p.spacing_given : p.spacing_deep;
    const uint32_t s = given                        ? std::clamp(given, 2u, TREE_SPACING)
                       : lv.ext[k].cap > TREE_LARGE ? TREE_SPACING_LARGE
                                                    : TREE_SPACING;
    lv.rulers[k] = make_rulers(s, salt_for(p.seed, k));
    lv.ext[k + 1].cap = ruler_count(lv.ext[k].cap, lv.rulers[k]);
    lv.ext[k + 1].count = count;
    lv.ext[k + 1].div = (uint32_t)std::min<uint64_t>((uint64_t)lv.ext[k].div * lv.rulers[k].s, 0xFFFFFFFFu);
    ++k;
  }
  lv.last = k;
  lv.rulers[k].s = 0;
  return lv;
}

// Parameters without the caller's spacing, where that is not the trees'.
Params own_spacing(Params p) {
  p.spacing_given = p.spacing_deep = 0;
  return p;
}

template <class L, class N>
kascade_status tree_chase(kascade_ctx& ctx, const TreeLevels& lv, int k, const typename L::R* rec,
                          const uint32_t* rootel, typename N::R* nrec, uint32_t* nroot, cudaStream_t s) {
  ProfScope ps(ctx, "chase", s);
  KS_TRY(launch(ctx, k_tree_chase<L, N>, grid_for(ctx, lv.ext[k + 1].cap, TREE_THREADS, 8), TREE_THREADS, 0, s, rec,
                lv.ext[k], lv.rulers[k], lv.ext[k + 1], rootel, nrec, nroot, lv.rulers[k + 1], hop_cap(lv.rulers[k]),
                ctx.d_status));
  return KASCADE_OK;
}

template <class L, class N, class Sink>
kascade_status tree_propagate(kascade_ctx& ctx, const TreeLevels& lv, int k, const typename L::R* rec,
                              const uint32_t* rootel, const typename N::O* out, const Sink& sink, bool last,
                              cudaStream_t s) {
  ProfScope ps(ctx, "propagate", s);
  KS_TRY(launch(ctx, k_tree_propagate<L, N, Sink>, grid_for(ctx, lv.ext[k].cap, TREE_THREADS, 8), TREE_THREADS, 0, s,
                rec, lv.ext[k], lv.rulers[k], rootel, out, sink, ctx.d_status, status_host(ctx, last)));
  return KASCADE_OK;
}

template <class R, class O>
kascade_status alloc_rulers(kascade_ctx& ctx, const TreeLevels& lv, TreeRulers<R, O>* up) {
  for (int k = 1; k <= lv.last; ++k) {
    const uint64_t cap = lv.ext[k].cap;
    up->rec[k] = alloc<R>(ctx, cap);
    up->root[k] = alloc<uint32_t>(ctx, cap);
    up->out[k] = alloc<O>(ctx, cap);
    if (!up->rec[k] || !up->root[k] || !up->out[k]) return KASCADE_ERR_OOM;
  }
  return KASCADE_OK;
}

// Levels 0..last from level 0's records; there is at least one ruler level.
template <class L, class N, class SinkN, class Sink>
kascade_status rank_tree(kascade_ctx& ctx, const TreeLevels& lv, const typename L::R* rec, const uint32_t* rootel,
                         const TreeRulers<typename N::R, typename N::O>& up, const Sink& sink, bool last,
                         cudaStream_t s) {
  KS_TRY((tree_chase<L, N>(ctx, lv, 0, rec, rootel, up.rec[1], up.root[1], s)));
  for (int k = 1; k < lv.last; ++k)
    KS_TRY((tree_chase<N, N>(ctx, lv, k, up.rec[k], up.root[k], up.rec[k + 1], up.root[k + 1], s)));
  KS_TRY(rank_trees_one_cta(ctx, up.rec[lv.last], up.root[lv.last], lv.ext[lv.last], up.out[lv.last], s));
  for (int k = lv.last - 1; k >= 1; --k)
    KS_TRY((tree_propagate<N, N>(ctx, lv, k, up.rec[k], up.root[k], up.out[k + 1], SinkN{up.out[k]}, false, s)));
  return tree_propagate<L, N>(ctx, lv, 0, rec, rootel, up.out[1], sink, last, s);
}

uint32_t words_of(uint32_t n) { return (uint32_t)(((uint64_t)n + 31) / 32); }
uint32_t tiles_of(uint32_t n) { return (words_of(n) + WORDS_TILE - 1) / WORDS_TILE; }
uint64_t inner_bytes(const Forest& f) { return (f.bits ? 4ull : 32ull) * words_of(f.n); }

kascade_status alloc_forest_once(kascade_ctx& ctx, uint32_t n, bool bits, const Params& p, Forest* f) {
  *f = Forest{};
  f->n = n;
  f->bits = bits;
  if (n == 0) return KASCADE_OK;
  f->count = alloc<uint32_t>(ctx, 1);
  if (!f->count) return KASCADE_ERR_OOM;
  f->lv = plan_tree(n, f->count, p);
  if (f->lv.last == 0) return KASCADE_OK;
  f->inner = alloc<char>(ctx, inner_bytes(*f));
  f->sums = alloc<uint32_t>(ctx, tiles_of(n));
  f->iw = alloc<uint2>(ctx, words_of(n));
  f->rec = alloc<uint32_t>(ctx, n);
  f->vert = alloc<uint32_t>(ctx, n);
  f->out = alloc<uint2>(ctx, n);
  if (!f->inner || !f->sums || !f->iw || !f->rec || !f->vert || !f->out) return KASCADE_ERR_OOM;
  return alloc_rulers(ctx, f->lv, &f->up);
}

kascade_status alloc_forest(kascade_ctx& ctx, uint32_t n, bool bits, const Params& p, Forest* f) {
  return arena_try(ctx, [&] { return alloc_forest_once(ctx, n, bits, p, f); });
}

// Depths and roots of a forest of more than TREE_BASE vertices.
template <class P, class Sink>
kascade_status root_levels(kascade_ctx& ctx, const P* parent, const Forest& f, const Sink& sink, bool report, bool last,
                           cudaStream_t s) {
  const uint32_t n = f.n, words = words_of(n), tiles = tiles_of(n);
  {
    ProfScope ps(ctx, "prepare", s);
    KS_CUDA(cudaMemsetAsync(f.inner, 0, inner_bytes(f), s));
    const unsigned grid = grid_for(ctx, ((uint64_t)n + TREE_PREP_ITEMS - 1) / TREE_PREP_ITEMS, TREE_THREADS, 8);
    auto number = [&](auto* flags) {
      using I = std::remove_reference_t<decltype(*flags)>;
      KS_TRY(launch(ctx, k_tree_inner<P, I>, grid, TREE_THREADS, 0, s, parent, n, flags, ctx.d_status));
      if (tiles > 1) KS_TRY(launch(ctx, k_tree_count<I>, tiles, TREE_THREADS, 0, s, flags, words, f.sums));
      return launch(ctx, k_tree_number<I>, tiles, TREE_THREADS, 0, s, flags, words, f.sums, f.iw, f.count);
    };
    KS_TRY(f.bits ? number(reinterpret_cast<uint32_t*>(f.inner)) : number(reinterpret_cast<unsigned char*>(f.inner)));
    const unsigned rec_grid = grid_for(ctx, ((uint64_t)n + TREE_REC_ITEMS - 1) / TREE_REC_ITEMS, TREE_THREADS, 8);
    KS_TRY(launch(ctx, k_tree_records<P>, rec_grid, TREE_THREADS, 0, s, parent, n, f.iw, f.lv.rulers[0], f.rec, f.vert, report,
                  ctx.d_status));
  }
  KS_TRY((rank_tree<TreeUnit, Tree8, SinkOut8>(ctx, f.lv, f.rec, f.vert, f.up, SinkOut8{f.out}, false, s)));
  ProfScope ps(ctx, "leaves", s);
  const unsigned grid = grid_for(ctx, ((uint64_t)n + TREE_OUT_ITEMS - 1) / TREE_OUT_ITEMS, TREE_THREADS, 8);
  KS_TRY(launch(ctx, k_tree_leaves<P, Sink>, grid, TREE_THREADS, 0, s, parent, n, f.iw, f.out, sink, ctx.d_status,
                status_host(ctx, last)));
  return KASCADE_OK;
}

}  // namespace

kascade_status root_forest_impl(kascade_ctx& ctx, const uint64_t* parent, uint32_t n, uint64_t* root_out,
                                uint64_t* depth_out, int keep_roots, const Params& p, cudaStream_t s) {
  if (n == 0) return KASCADE_OK;
  const SinkPlain sink{root_out, depth_out, keep_roots};
  Forest f;
  KS_TRY(alloc_forest(ctx, n, n > TREE_BYTES_MAX, p, &f));
  if (f.lv.last == 0) return rank_arrays_one_cta(ctx, parent, WKind::Unit, nullptr, n, sink, CTA_ROOTING, s);
  ctx.last_levels.assign(1, n);
  for (int k = 1; k <= f.lv.last; ++k) ctx.last_levels.push_back(f.lv.ext[k].cap);
  return root_levels(ctx, parent, f, sink, true, true, s);
}

kascade_status alloc_forests(kascade_ctx& ctx, uint32_t n, const Params& p, Forest* f) {
  return alloc_forest(ctx, n, n > TREE_BYTES_MAX_BATCH, own_spacing(p), f);  // (a batch's spacing is its lists')
}

kascade_status root_forests(kascade_ctx& ctx, const uint32_t* parent, const Forest& f, const SinkBatch& sink, bool last,
                            cudaStream_t s) {
  if (f.n == 0) return KASCADE_OK;
  if (f.lv.last == 0) return rank_parents_one_cta(ctx, parent, f.n, sink, last, s);
  return root_levels(ctx, parent, f, sink, false, last, s);
}

kascade_status rank_forest_weighted(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                                    const SinkPlain& sink, const Params& p, cudaStream_t s) {
  const TreeLevels lv = plan_tree(n, nullptr, own_spacing(p));
  if (lv.last == 0) return rank_arrays_one_cta(ctx, succ, wk, w, n, sink, CTA_TREES, s);
  ctx.last_levels.assign(1, n);
  Level0 l0;  // F16x16, no stamps
  Rec* rec = nullptr;
  TreeRulers<Rec, Out> up;
  KS_TRY(arena_try(ctx, [&] {
    rec = alloc<Rec>(ctx, n);
    return rec ? alloc_rulers(ctx, lv, &up) : KASCADE_ERR_OOM;
  }));
  l0.rec = rec;
  KS_TRY(prepare_arrays(ctx, succ, wk, w, n, l0, lv.rulers[0], s));
  return rank_tree<Tree16, Tree16, SinkOut>(ctx, lv, rec, nullptr, up, sink, true, s);
}

}  // namespace ks
