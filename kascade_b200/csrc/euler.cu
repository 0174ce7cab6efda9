// The Euler tour of a forest in the reference's numbering.
//
// Reference: compute_euler_tour / compute_euler_tour_impl
// (lib/kascade/eulertour.cpp:33-127, 379-392) on the forest built by
// reverse_rooted_tree + make_graph (lib/kascade/successor_utils.cpp:236-300).
// The children are sorted by parent; ranking a forest (rank_via_euler_tour,
// eulertour.cpp:337-377) needs no tour (tree.cu).
#include <algorithm>

#include "ranker.cuh"
#include "sort.cuh"

namespace ks {

namespace {

inline int bits_for(uint64_t n) {
  int b = 1;
  while (b < 63 && (1ull << b) < n) b++;
  return b;
}

// seg[v] = [start, end) of v's entries in the sorted children array
__global__ void __launch_bounds__(256) k_seg_bounds(const uint32_t* __restrict__ keys, uint32_t n,
                                                    uint2* __restrict__ seg) {
  for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t k = keys[q];
    if (q == 0 || keys[q - 1] != k) seg[k].x = (uint32_t)q;
    if (q + 1 == n || keys[q + 1] != k) seg[k].y = (uint32_t)(q + 1);
  }
}

// ---------------------------------------------------------------------------
// compute_euler_tour in the reference's numbering (one rank).
// ---------------------------------------------------------------------------
// deg[v] = #children + (v not a root); droot[v] = 1 for roots with deg > 0
__global__ void __launch_bounds__(256) k_ref_degrees(const uint64_t* __restrict__ parent, uint32_t n,
                                                     const uint2* __restrict__ seg, uint32_t* __restrict__ deg,
                                                     uint32_t* __restrict__ droot) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const bool root = parent[v] == v;
    const uint2 sg = seg[v];
    const uint32_t children = (sg.y - sg.x) - (root ? 1u : 0u);
    const uint32_t d = children + (root ? 0u : 1u);
    deg[v] = d;
    droot[v] = (root && d > 0) ? 1u : 0u;
  }
}

__global__ void __launch_bounds__(256) k_iota64(uint64_t* __restrict__ out, uint64_t m) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = i;
}

// Per sorted child entry (p, c): the element (c, p) and the element (p, c).
// A vertex v's neighbours in the reference CSR are ordered by decreasing key,
// with key(child) = child id and key(parent) = v (successor_utils.cpp:281-293
// appends (i, parent) then (parent, i) for i ascending; make_graph fills each
// segment from its end).
__global__ void __launch_bounds__(256) k_ref_tour(const uint64_t* __restrict__ parent, const uint32_t* __restrict__ keys,
                                                  const uint32_t* __restrict__ vals, uint32_t n,
                                                  const uint2* __restrict__ seg, const uint32_t* __restrict__ deg,
                                                  const uint32_t* __restrict__ xadj, const uint32_t* __restrict__ didx,
                                                  uint32_t num_edges, uint64_t* __restrict__ tour) {
  for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t p = keys[q], c = vals[q];
    if (p == c) continue;
    const bool proot = parent[p] == p;
    const uint2 sp = seg[p], sc = seg[c];
    const uint32_t cc_p = (sp.y - sp.x) - (proot ? 1u : 0u);
    // index of c among p's children in increasing id order
    uint32_t j = (uint32_t)q - sp.x;
    if (proot && p < c) j -= 1;  // p's own entry sits before c
    const uint32_t pos_c_in_p = (cc_p - 1 - j) + ((!proot && p > c) ? 1u : 0u);
    // number of c's children with id > c (c is not a root: no own entry)
    uint32_t lo = sc.x, hi = sc.y;
    while (lo < hi) {
      uint32_t mid = (lo + hi) >> 1;
      if (vals[mid] <= c)
        lo = mid + 1;
      else
        hi = mid;
    }
    const uint32_t pos_p_in_c = sc.y - lo;
    const uint32_t dp = deg[p], dc = deg[c];
    const uint32_t id_up = xadj[c] + pos_p_in_c;
    const uint32_t id_down = xadj[p] + pos_c_in_p;
    // succ of (c, p): (p, nbr_p[(pos_c_in_p + 1) mod deg p]), or p's dummy
    uint32_t k = (pos_c_in_p + 1) % dp;
    tour[id_up] = (proot && k == 0) ? (uint64_t)num_edges + didx[p] : (uint64_t)xadj[p] + k;
    // succ of (p, c): (c, nbr_c[(pos_p_in_c + 1) mod deg c])
    k = (pos_p_in_c + 1) % dc;
    tour[id_down] = (uint64_t)xadj[c] + k;
  }
}

// The reference-numbered tour's children array: (parent, child) pairs
// sorted by parent (stable, so children in increasing id), and each
// vertex's segment of it.
kascade_status sort_children(kascade_ctx& ctx, const uint64_t* parent, uint32_t n, uint32_t** keys, uint32_t** vals,
                             uint2** seg, cudaStream_t s) {
  SortSource src;
  src.parent = parent;
  KS_TRY(radix_sort_pairs(ctx, src, n, bits_for(n), keys, vals, s));
  *seg = alloc<uint2>(ctx, n);
  if (!*seg) return KASCADE_ERR_OOM;
  KS_CUDA(cudaMemsetAsync(*seg, 0, sizeof(uint2) * (size_t)n, s));
  ProfScope ps(ctx, "seg_bounds", s);
  k_seg_bounds<<<grid_for(ctx, n, 256, 8), 256, 0, s>>>(*keys, n, *seg);
  KS_CHECK_LAUNCH();
  return KASCADE_OK;
}

}  // namespace

kascade_status compute_euler_tour_impl(kascade_ctx& ctx, const uint64_t* parent, uint32_t n, uint64_t* tour,
                                       uint64_t* m_out, cudaStream_t s) {
  *m_out = 0;
  if (n == 0) return KASCADE_OK;
  uint32_t *keys, *vals;
  uint2* seg;
  KS_TRY(sort_children(ctx, parent, n, &keys, &vals, &seg, s));
  uint32_t* deg = alloc<uint32_t>(ctx, n);
  uint32_t* droot = alloc<uint32_t>(ctx, n);
  uint32_t* xadj = alloc<uint32_t>(ctx, n);
  uint32_t* tot = alloc<uint32_t>(ctx, 2);
  if (!deg || !droot || !xadj || !tot) return KASCADE_ERR_OOM;
  const unsigned grid = grid_for(ctx, n, 256, 8);
  k_ref_degrees<<<grid, 256, 0, s>>>(parent, n, seg, deg, droot);
  KS_CHECK_LAUNCH();
  KS_TRY(exclusive_scan_u32(ctx, deg, xadj, n, tot, s));
  KS_TRY(exclusive_scan_u32(ctx, droot, droot, n, tot + 1, s));
  uint32_t num_edges = 0;
  KS_TRY(read_u32(ctx, tot, &num_edges, s));
  // m = num_edges + #roots; #roots = n - num_edges / 2
  const uint64_t roots = (uint64_t)n - num_edges / 2;
  const uint64_t m = (uint64_t)num_edges + roots;
  k_iota64<<<grid_for(ctx, m, 256, 8), 256, 0, s>>>(tour, m);
  KS_CHECK_LAUNCH();
  {
    ProfScope ps(ctx, "ref_tour", s);
    k_ref_tour<<<grid, 256, 0, s>>>(parent, keys, vals, n, seg, deg, xadj, droot, num_edges, tour);
    KS_CHECK_LAUNCH();
  }
  *m_out = m;
  return KASCADE_OK;
}

}  // namespace ks
