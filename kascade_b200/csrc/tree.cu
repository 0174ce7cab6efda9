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
#include <vector>

#include "ranker.cuh"

namespace ks {

namespace {

constexpr int TREE_THREADS = 256;
constexpr int TREE_PREP_ITEMS = 8;
constexpr uint32_t TREE_SPACING = 3;
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
    const uint32_t v = __ldg(p);
    return Hop{1, v & ~REC8_RULER, (v & REC8_RULER) != 0u};
  }
};
// Deeper levels of one: depths in 32 bits.
struct Tree8 {
  using R = Rec8;
  using O = uint2;  // rank, root
  static constexpr bool kEndWeight = true;
  static __device__ __forceinline__ Hop hop(const R* p) {
    return Record8::unpack(__ldg(reinterpret_cast<const uint2*>(p)));
  }
  static __device__ __forceinline__ Out out(const O* p) {
    const uint2 v = __ldg(p);
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
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    return Hop{(uint64_t)v.x | ((uint64_t)v.y << 32), v.z, v.w != 0u};
  }
  static __device__ __forceinline__ Out out(const O* p) { return ld_out(p); }
  static __device__ __forceinline__ void put(R* p, uint64_t w, uint32_t b, bool ruler) {
    Record16::put(p, w, b, ruler);
  }
};

__device__ __forceinline__ bool bit_of(const uint32_t* bits, uint32_t x) {
  return (__ldg(bits + (x >> 5)) >> (x & 31)) & 1u;
}

// Level-0 records of a tree rooting, and a bit for every vertex with a child
// (zeroed by the caller): a ruler without one is on nobody's path.
__global__ void __launch_bounds__(TREE_THREADS) k_tree_prepare(const uint64_t* __restrict__ parent, uint32_t n,
                                                               Rulers rl, uint32_t* __restrict__ rec,
                                                               uint32_t* __restrict__ inner, DevStatus* st) {
  const uint64_t tile_sz = (uint64_t)blockDim.x * TREE_PREP_ITEMS;
  for (uint64_t tile = (uint64_t)blockIdx.x * tile_sz; tile < n; tile += (uint64_t)gridDim.x * tile_sz) {
    uint64_t p[TREE_PREP_ITEMS];
    uint32_t w[TREE_PREP_ITEMS];
#pragma unroll
    for (int i = 0; i < TREE_PREP_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      p[i] = v < n ? __ldcs(reinterpret_cast<const unsigned long long*>(parent) + v) : v;
    }
#pragma unroll
    for (int i = 0; i < TREE_PREP_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      w[i] = 0xFFFFFFFFu;
      if (v >= n) continue;
      if (p[i] >= n) {
        set_error(st, KASCADE_ERR_OUT_OF_RANGE, v);
        p[i] = v;
      }
      if (p[i] != v) w[i] = __ldcg(inner + (p[i] >> 5));  // a set bit is not set again: a star's root stays cheap
    }
#pragma unroll
    for (int i = 0; i < TREE_PREP_ITEMS; ++i) {
      const uint64_t v = tile + (uint64_t)i * blockDim.x + threadIdx.x;
      if (v >= n) continue;
      const uint32_t b = (uint32_t)p[i];
      if (!((w[i] >> (b & 31)) & 1u)) atomicOr(inner + (b >> 5), 1u << (b & 31));
      uint32_t j;
      rec[v] = b | (b != (uint32_t)v && rl.is(b, &j) ? REC8_RULER : 0u);
    }
  }
}

// Every ruler's walk to the next ruler or its root.  inner: level 0's vertices
// with a child (null: not known).
template <class L, class N>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_chase(const typename L::R* __restrict__ rec, uint32_t n,
                                                             Rulers rl, uint32_t rulers,
                                                             const uint32_t* __restrict__ inner,
                                                             const uint32_t* __restrict__ rootel,
                                                             typename N::R* __restrict__ nrec,
                                                             uint32_t* __restrict__ nroot, Rulers nrl,
                                                             uint32_t hop_cap, DevStatus* st) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rulers; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t id = (uint32_t)i;
    const uint64_t x0 = rl.elem(id);
    uint64_t acc = 0;
    uint32_t next = id, k;
    if (x0 < n && (!inner || bit_of(inner, (uint32_t)x0))) {
      uint32_t x = (uint32_t)x0, hops = 0;
      while (true) {
        const Hop h = L::hop(rec + x);
        if (h.b == x) {
          if (L::kEndWeight) acc += h.w;
          nroot[id] = rootel ? __ldg(rootel + x) : x;
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
// inner (level 0): the vertices with children are counted for the call's
// report of its tour's length.
template <class L, class N, class Sink>
__global__ void __launch_bounds__(TREE_THREADS) k_tree_propagate(const typename L::R* __restrict__ rec, uint32_t n,
                                                                 Rulers rl, const uint32_t* __restrict__ inner,
                                                                 const uint32_t* __restrict__ rootel,
                                                                 const typename N::O* __restrict__ out, Sink sink,
                                                                 DevStatus* st) {
  uint32_t downs = 0;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)v;
    Hop h = L::hop(rec + x);
    const bool in = !inner || bit_of(inner, x);
    if (h.b == x) {
      sink.put(x, L::kEndWeight ? h.w : 0ull, rootel ? __ldg(rootel + x) : x, true);
      continue;
    }
    if (inner && in) ++downs;
    uint32_t j;
    if (in && rl.is(x, &j)) {
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
      sink.put(x, L::kEndWeight ? acc + h.w : acc, rootel ? __ldg(rootel + y) : y, false);
    } else {
      set_error(st, KASCADE_ERR_CYCLE, x);
    }
  }
  if (inner) {
    downs = __reduce_add_sync(0xffffffffu, downs);
    if ((threadIdx.x & 31u) == 0 && downs) atomicAdd(&st->counter[1], (unsigned long long)downs);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&st->counter[1], (unsigned long long)n);
  }
}

struct TreeLevels {
  int last = 0;
  uint32_t n[MAX_LEVELS + 1];
  Rulers rulers[MAX_LEVELS + 1];
};

TreeLevels plan_tree(uint32_t n, const Params& p) {
  TreeLevels lv;
  const uint32_t base = std::max(1u, std::min(p.base_max, TREE_BASE));
  uint32_t m = n;
  int k = 0;
  lv.n[0] = n;
  while (m > base && k < MAX_LEVELS) {
    const uint32_t s = k == 0 ? (p.spacing_given ? p.spacing_given : TREE_SPACING)
                              : (p.spacing_deep ? p.spacing_deep : TREE_SPACING);
    lv.rulers[k] = make_rulers(s, salt_for(p.seed, k));
    m = ruler_count(m, lv.rulers[k]);
    lv.n[++k] = m;
  }
  lv.last = k;
  lv.rulers[k] = cta_rulers(m);
  return lv;
}

template <class L, class N>
kascade_status tree_chase(kascade_ctx& ctx, const TreeLevels& lv, int k, const typename L::R* rec,
                          const uint32_t* inner, const uint32_t* rootel, typename N::R* nrec, uint32_t* nroot,
                          cudaStream_t s) {
  ProfScope ps(ctx, "chase", s);
  k_tree_chase<L, N><<<grid_for(ctx, lv.n[k + 1], TREE_THREADS, 8), TREE_THREADS, 0, s>>>(
      rec, lv.n[k], lv.rulers[k], lv.n[k + 1], inner, rootel, nrec, nroot, lv.rulers[k + 1], hop_cap(lv.rulers[k]),
      ctx.d_status);
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

template <class L, class N, class Sink>
kascade_status tree_propagate(kascade_ctx& ctx, const TreeLevels& lv, int k, const typename L::R* rec,
                              const uint32_t* inner, const uint32_t* rootel, const typename N::O* out,
                              const Sink& sink, cudaStream_t s) {
  ProfScope ps(ctx, "propagate", s);
  k_tree_propagate<L, N, Sink><<<grid_for(ctx, lv.n[k], TREE_THREADS, 8), TREE_THREADS, 0, s>>>(
      rec, lv.n[k], lv.rulers[k], inner, rootel, out, sink, ctx.d_status);
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

// Levels 0..last from level 0's records; there is at least one ruler level.
template <class L, class N, class SinkN, class Sink>
kascade_status rank_tree(kascade_ctx& ctx, const TreeLevels& lv, const typename L::R* rec, const uint32_t* inner,
                         const Sink& sink, cudaStream_t s) {
  typename N::R* nrec[MAX_LEVELS + 1] = {};
  uint32_t* nroot[MAX_LEVELS + 1] = {};
  typename N::O* nout[MAX_LEVELS + 1] = {};
  for (int k = 1; k <= lv.last; ++k) {
    nrec[k] = alloc<typename N::R>(ctx, lv.n[k]);
    nroot[k] = alloc<uint32_t>(ctx, lv.n[k]);
    nout[k] = alloc<typename N::O>(ctx, lv.n[k]);
    if (!nrec[k] || !nroot[k] || !nout[k]) return KASCADE_ERR_OOM;
  }
  KS_TRY((tree_chase<L, N>(ctx, lv, 0, rec, inner, nullptr, nrec[1], nroot[1], s)));
  for (int k = 1; k < lv.last; ++k)
    KS_TRY((tree_chase<N, N>(ctx, lv, k, nrec[k], nullptr, nroot[k], nrec[k + 1], nroot[k + 1], s)));
  KS_TRY(rank_trees_one_cta(ctx, nrec[lv.last], nroot[lv.last], lv.n[lv.last], nout[lv.last], s));
  for (int k = lv.last - 1; k >= 1; --k)
    KS_TRY((tree_propagate<N, N>(ctx, lv, k, nrec[k], nullptr, nroot[k], nout[k + 1], SinkN{nout[k]}, s)));
  return tree_propagate<L, N>(ctx, lv, 0, rec, inner, nullptr, nout[1], sink, s);
}

}  // namespace

kascade_status root_forest_impl(kascade_ctx& ctx, const uint64_t* parent, uint32_t n, uint64_t* root_out,
                                uint64_t* depth_out, int keep_roots, const Params& p, cudaStream_t s) {
  if (n == 0) return KASCADE_OK;
  const SinkPlain sink{root_out, depth_out, keep_roots};
  const TreeLevels lv = plan_tree(n, p);
  if (lv.last == 0) return rank_arrays_one_cta(ctx, parent, WKind::Unit, nullptr, n, sink, CTA_ROOTING, s);
  ctx.last_levels.assign(lv.n, lv.n + lv.last + 1);
  const uint32_t words = (uint32_t)(((uint64_t)n + 31) / 32);
  uint32_t* rec = alloc<uint32_t>(ctx, n);
  uint32_t* inner = alloc<uint32_t>(ctx, words);
  if (!rec || !inner) return KASCADE_ERR_OOM;
  {
    ProfScope ps(ctx, "prepare", s);
    KS_CUDA(cudaMemsetAsync(inner, 0, sizeof(uint32_t) * (size_t)words, s));
    const unsigned grid =
        grid_for(ctx, ((uint64_t)n + TREE_PREP_ITEMS - 1) / TREE_PREP_ITEMS, TREE_THREADS, 8);
    k_tree_prepare<<<grid, TREE_THREADS, 0, s>>>(parent, n, lv.rulers[0], rec, inner, ctx.d_status);
    KS_CHECK_LAUNCH();
  }
  return rank_tree<TreeUnit, Tree8, SinkOut8>(ctx, lv, rec, inner, sink, s);
}

kascade_status rank_forest_weighted(kascade_ctx& ctx, const uint64_t* succ, WKind wk, const void* w, uint32_t n,
                                    const SinkPlain& sink, const Params& p, cudaStream_t s) {
  const TreeLevels lv = plan_tree(n, p);
  if (lv.last == 0) return rank_arrays_one_cta(ctx, succ, wk, w, n, sink, CTA_TREES, s);
  ctx.last_levels.assign(1, n);
  Level0 l0;  // F16x16, no stamps
  Rec* rec = alloc<Rec>(ctx, n);
  if (!rec) return KASCADE_ERR_OOM;
  l0.rec = rec;
  KS_TRY(prepare_arrays(ctx, succ, wk, w, n, l0, lv.rulers[0], s));
  return rank_tree<Tree16, Tree16, SinkOut>(ctx, lv, rec, nullptr, sink, s);
}

}  // namespace ks
