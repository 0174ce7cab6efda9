// Shared device-side definitions of the B200 list-ranking library.
//
// An element's record holds its weight and successor, so that a dependent hop of
// the ruler chase is one aligned load of 8 or 16 B; the formats of a level are
// described below, after the loads.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/kascade_b200.h"

namespace ks {

// ---------------------------------------------------------------------------
// 16 B record.
//   a : weight, as 64-bit two's complement; in a record that is stamped, the
//       distance from the element's ruler
//   b : successor index (every state keeps it)
//   c : by format: whether the successor is a ruler (Record16), that and the
//       stamp's ruler id (F16i), or, in a shard, the tag TAG_UNREACHED,
//       TAG_RULER | ruler id, or a ruler id (reached)
// ---------------------------------------------------------------------------
struct __align__(16) Rec {
  uint64_t a;
  uint32_t b;
  uint32_t c;
};
static_assert(sizeof(Rec) == 16, "record must be 16 bytes");

constexpr uint32_t TAG_UNREACHED = 0xFFFFFFFFu;
constexpr uint32_t TAG_RULER = 0x80000000u;
constexpr uint32_t MAX_ELEMS = 0xFFFFFFFEu;   // element indices fit in 32 bits

__host__ __device__ __forceinline__ bool tag_unreached(uint32_t c) { return c == TAG_UNREACHED; }
__host__ __device__ __forceinline__ bool tag_ruler(uint32_t c) {
  return (c & TAG_RULER) != 0u && c != TAG_UNREACHED;
}
__host__ __device__ __forceinline__ uint32_t tag_id(uint32_t c) { return c & 0x7FFFFFFFu; }

// Result of a deeper level for one of its elements: rank (distance to root)
// and the root as a level-0 element index.
struct __align__(16) Out {
  uint64_t rank;
  uint32_t root;
  uint32_t pad;
};
static_assert(sizeof(Out) == 16, "Out must be 16 bytes");

// Pointer-doubling record (double-buffered jump kernel).
struct __align__(16) PdRec {
  uint64_t rank;
  uint32_t succ;
  uint32_t done;  // 1 once succ is a root
};

// ---------------------------------------------------------------------------
// Device status word: the first error wins; kernels never trap.
// ---------------------------------------------------------------------------
struct DevStatus {
  unsigned int code;
  unsigned int blocks;  // of a call's last kernel: done so far
  unsigned long long info;
  // [1]: level 0's size, when only the device knows it; [2], [3]: elements
  // stamped by chains / found stamped (more of the former: two chains met)
  unsigned long long counter[6];
  unsigned int work[32];          // per level: rulers handed out beyond the warps' first shares
};

__device__ __forceinline__ void set_error(DevStatus* st, unsigned int code, unsigned long long info) {
  if (atomicCAS(&st->code, 0u, code) == 0u) st->info = info;
}

// The beginning of a kernel that `launch` starts: its blocks may be in place
// while the kernel ahead in the stream still runs, and wait here until that
// has ended and its stores are visible.  Then the next kernel's may come.
__device__ __forceinline__ void kernel_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------------------
// Counter hash used for ruler sampling (the "lowbias32" integer mixer,
// a public-domain construction by C. Wellons).
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

__device__ __forceinline__ bool sampled(uint32_t x, uint32_t salt, uint32_t thresh) {
  return mix32(x ^ salt) < thresh;
}

// ---------------------------------------------------------------------------
// Loads of what the kernel ahead may still be storing.  A kernel that `launch`
// starts is in place while that one runs.  Its loads may not be of the
// non-coherent kind (__ldg, or what the compiler makes of a const __restrict__
// pointer): that takes the data as unchanging for as long as the kernel is
// resident.  Nor may they move above kernel_begin's wait: ld_cg and ld_cs are
// volatile, as the wait is, and ld_ca is a plain read, which the wait's memory
// clobber holds back (as a volatile load it cost the forests' walks 1 to 4%:
// 4.2e6 vertices 232 us, plain 222; by __ldg, each kernel started after the one
// ahead had ended, 249 against 251, pointer doubling of 1e6 184 against 189).
//   ld_ca  through L1 (what neighbours or later loads read again)
//   ld_cg  from L2 (random hops, which never hit L1; what other SMs write)
//   ld_cs  streaming, evict-first
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T ld_ca(const T* p) {
  return *p;
}
#define KS_LOADS(name, op)                                                                                  \
  __device__ __forceinline__ uint32_t name(const uint32_t* p) {                                             \
    uint32_t v;                                                                                             \
    asm volatile("ld.global." op ".u32 %0, [%1];" : "=r"(v) : "l"(p));                                      \
    return v;                                                                                               \
  }                                                                                                         \
  __device__ __forceinline__ uint64_t name(const uint64_t* p) {                                             \
    uint64_t v;                                                                                             \
    asm volatile("ld.global." op ".u64 %0, [%1];" : "=l"(v) : "l"(p));                                      \
    return v;                                                                                               \
  }                                                                                                         \
  __device__ __forceinline__ unsigned long long name(const unsigned long long* p) {                         \
    unsigned long long v;                                                                                   \
    asm volatile("ld.global." op ".u64 %0, [%1];" : "=l"(v) : "l"(p));                                      \
    return v;                                                                                               \
  }                                                                                                         \
  __device__ __forceinline__ uint2 name(const uint2* p) {                                                   \
    uint2 v;                                                                                                \
    asm volatile("ld.global." op ".v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));                \
    return v;                                                                                               \
  }                                                                                                         \
  __device__ __forceinline__ uint4 name(const uint4* p) {                                                   \
    uint4 v;                                                                                                \
    asm volatile("ld.global." op ".v4.u32 {%0, %1, %2, %3}, [%4];"                                          \
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)                                               \
                 : "l"(p));                                                                                 \
    return v;                                                                                               \
  }
KS_LOADS(ld_cg, "cg")
KS_LOADS(ld_cs, "cs")
#undef KS_LOADS

// The words of a status that the host reads.
constexpr uint32_t STATUS_WORDS = 8;
static_assert(offsetof(DevStatus, work) == STATUS_WORDS * 8 && sizeof(DevStatus) % 8 == 0, "status words");

// The end of a call's last kernel: its last block to finish copies the status
// to the host's pinned words (host == nullptr: not here) and clears it for the
// next call.  A call of one launch is then that launch: with a memset ahead of
// it and a copy behind it 1000 elements took 38.7 us instead of 30.
// Called by all threads of every block.
__device__ __forceinline__ void publish_status(DevStatus* st, unsigned long long* host) {
  if (!host) return;
  __syncthreads();
  if (threadIdx.x >= 32u) return;
  uint32_t last = 1;
  if (threadIdx.x == 0) {
    __threadfence();
    if (gridDim.x > 1) last = atomicAdd(&st->blocks, 1u) == gridDim.x - 1 ? 1u : 0u;
    __threadfence();
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  unsigned long long* w = reinterpret_cast<unsigned long long*>(st);
  if (threadIdx.x < STATUS_WORDS) *(volatile unsigned long long*)(host + threadIdx.x) = ld_cg(w + threadIdx.x);
  if (threadIdx.x < sizeof(DevStatus) / 8) __stcg(w + threadIdx.x, 0ull);
}

__device__ __forceinline__ Rec ld_rec_cg(const Rec* p) {
  uint4 v = ld_cg(reinterpret_cast<const uint4*>(p));
  Rec r;
  r.a = (uint64_t)v.x | ((uint64_t)v.y << 32);
  r.b = v.z;
  r.c = v.w;
  return r;
}
__device__ __forceinline__ Rec ld_rec_cs(const Rec* p) {
  uint4 v = ld_cs(reinterpret_cast<const uint4*>(p));
  Rec r;
  r.a = (uint64_t)v.x | ((uint64_t)v.y << 32);
  r.b = v.z;
  r.c = v.w;
  return r;
}
__device__ __forceinline__ void st_rec_cg(Rec* p, Rec r) {
  uint4 v = make_uint4((uint32_t)r.a, (uint32_t)(r.a >> 32), r.b, r.c);
  __stcg(reinterpret_cast<uint4*>(p), v);
}
__device__ __forceinline__ void st_rec_cs(Rec* p, Rec r) {
  uint4 v = make_uint4((uint32_t)r.a, (uint32_t)(r.a >> 32), r.b, r.c);
  __stcs(reinterpret_cast<uint4*>(p), v);
}
// ---------------------------------------------------------------------------
// Record formats of a level.  A record holds an element's weight and
// successor and is only ever read while chains run: both halves of the L2
// keep copies, and a dependent hop costs 0.15-0.22 us; with the stamp stored
// into the record it had just been read from, every hop paid the cross-die
// coherence (0.26-0.44 us).  Stamps (ruler id, distance) have an array of
// their own.
// A record also says whether its successor is a ruler, so that a hop needs no
// index arithmetic (it was a third of the chase's instructions) and a chain
// knows that it ends before it asks for another record.  8 B records keep that
// bit in the successor word: at most 2^31 elements.
//   F8x8   unit weights (a chain is shorter than 2^32), 8 B stamps
//   F8x16  32-bit weights, 64-bit distances
//   F16x16 64-bit weights (in-place calls, every deeper level)
//   F16i   any weights, the stamp stored into the record: half the memory of
//          F16x16, for sizes at which that decides what stays in L2
// ---------------------------------------------------------------------------
struct __align__(8) Rec8 {
  uint32_t b;  // successor | REC8_RULER when that is a ruler
  uint32_t w;  // weight
};
constexpr uint32_t REC8_RULER = 0x80000000u;
constexpr uint64_t REC8_MAX = 0x80000000ull;  // elements
struct Hop {
  uint64_t w;
  uint32_t b;
  bool ruler;  // whether b is one
};
struct Stamp {
  uint32_t id;  // TAG_UNREACHED: none
  uint64_t dist;
};
struct Stamp8 {
  using S = uint2;
  static __device__ __forceinline__ void put(S* p, uint32_t id, uint64_t dist) {
    __stcg(p, make_uint2(id, (uint32_t)dist));
  }
  static __device__ __forceinline__ void clear(S* p) { __stcg(p, make_uint2(TAG_UNREACHED, 0u)); }
  static __device__ __forceinline__ Stamp get_stream(const S* p) {
    const uint2 v = ld_cs(p);
    return Stamp{v.x, v.y};
  }
  static __device__ __forceinline__ Stamp get(const S* p) {
    const uint2 v = ld_cg(p);
    return Stamp{v.x, v.y};
  }
};
struct Stamp16 {
  using S = uint4;
  static __device__ __forceinline__ void put(S* p, uint32_t id, uint64_t dist) {
    __stcg(p, make_uint4((uint32_t)dist, (uint32_t)(dist >> 32), id, 0u));
  }
  static __device__ __forceinline__ void clear(S* p) { __stcg(p, make_uint4(0u, 0u, TAG_UNREACHED, 0u)); }
  static __device__ __forceinline__ Stamp get_stream(const S* p) {
    const uint4 v = ld_cs(p);
    return Stamp{v.z, (uint64_t)v.x | ((uint64_t)v.y << 32)};
  }
  static __device__ __forceinline__ Stamp get(const S* p) {
    const uint4 v = ld_cg(p);
    return Stamp{v.z, (uint64_t)v.x | ((uint64_t)v.y << 32)};
  }
};
struct Record8 {
  using R = Rec8;
  static constexpr uint64_t kMaxElems = REC8_MAX;
  static __device__ __forceinline__ Hop unpack(uint2 v) {
    return Hop{v.y, v.x & ~REC8_RULER, (v.x & REC8_RULER) != 0u};
  }
  static __device__ __forceinline__ Hop hop(const R* p) { return unpack(ld_cg(reinterpret_cast<const uint2*>(p))); }
  static __device__ __forceinline__ void put(R* p, uint64_t w, uint32_t b, bool ruler) {
    __stcg(reinterpret_cast<uint2*>(p), make_uint2(b | (ruler ? REC8_RULER : 0u), (uint32_t)w));
  }
};
struct Record16 {
  using R = Rec;
  static __device__ __forceinline__ Hop hop(const R* p) {
    const Rec r = ld_rec_cg(p);
    return Hop{r.a, r.b, r.c != 0u};
  }
  static __device__ __forceinline__ void put(R* p, uint64_t w, uint32_t b, bool ruler) {
    Rec r;
    r.a = w;
    r.b = b;
    r.c = ruler ? 1u : 0u;
    st_rec_cg(p, r);
  }
};
template <class Record, class StampT>
struct Split : Record, StampT {
  static constexpr bool kInPlace = false;
  using Record::put;
  static __device__ __forceinline__ void stamp(typename StampT::S* p, uint32_t id, uint64_t d, const Hop&) {
    StampT::put(p, id, d);
  }
};
using F8x8 = Split<Record8, Stamp8>;
using F8x16 = Split<Record8, Stamp16>;
using F16x16 = Split<Record16, Stamp16>;
struct F16i {
  static constexpr bool kInPlace = true;
  using R = Rec;
  using S = Rec;  // the records themselves
  static constexpr uint32_t NONE = 0x7FFFFFFFu, RULER = 0x80000000u;  // word c: ruler id or NONE, successor's bit
  static __device__ __forceinline__ Hop hop(const R* p) {
    const Rec r = ld_rec_cg(p);
    return Hop{r.a, r.b, (r.c & RULER) != 0u};
  }
  static __device__ __forceinline__ void put(R* p, uint64_t w, uint32_t b, bool ruler) {
    Rec r;
    r.a = w;
    r.b = b;
    r.c = NONE | (ruler ? RULER : 0u);
    st_rec_cg(p, r);
  }
  static __device__ __forceinline__ void stamp(S* p, uint32_t id, uint64_t d, const Hop& h) {
    Rec r;
    r.a = d;
    r.b = h.b;
    r.c = id | (h.ruler ? RULER : 0u);
    st_rec_cg(p, r);
  }
  static __device__ __forceinline__ void clear(S*) {}  // part of put
  static __device__ __forceinline__ Stamp unpack(const Rec& r) {
    const uint32_t id = r.c & ~RULER;
    return Stamp{id == NONE ? TAG_UNREACHED : id, r.a};
  }
  static __device__ __forceinline__ Stamp get_stream(const S* p) { return unpack(ld_rec_cs(p)); }
  static __device__ __forceinline__ Stamp get(const S* p) { return unpack(ld_rec_cg(p)); }
};
enum class Format { F8x8, F8x16, F16x16, F16i };

__device__ __forceinline__ Out ld_out(const Out* p) {
  uint4 v = ld_cg(reinterpret_cast<const uint4*>(p));
  Out o;
  o.rank = (uint64_t)v.x | ((uint64_t)v.y << 32);
  o.root = v.z;
  o.pad = v.w;
  return o;
}
// The same load, with the line kept in L2 ahead of streaming traffic: for
// small tables read at random by every element (a level's ruler results).
__device__ __forceinline__ uint64_t l2_keep_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
// Through the read-only (L1) path with the same L2 hint: for lookups whose
// neighbours in a warp's stream tend to repeat (log entries of one chain).
// Non-coherent: for kernels that start after the kernel ahead has ended.
__device__ __forceinline__ Out ld_out_nc_keep(const Out* p, uint64_t pol) {
  uint32_t a, b, c, d;
  asm volatile("ld.global.nc.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
               : "l"(p), "l"(pol));
  Out o;
  o.rank = (uint64_t)a | ((uint64_t)b << 32);
  o.root = c;
  o.pad = d;
  return o;
}
__device__ __forceinline__ Out ld_out_keep(const Out* p, uint64_t pol) {
  uint32_t a, b, c, d;
  asm volatile("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
               : "l"(p), "l"(pol));
  Out o;
  o.rank = (uint64_t)a | ((uint64_t)b << 32);
  o.root = c;
  o.pad = d;
  return o;
}
__device__ __forceinline__ void st_out(Out* p, uint64_t rank, uint32_t root) {
  __stcg(reinterpret_cast<uint4*>(p), make_uint4((uint32_t)rank, (uint32_t)(rank >> 32), root, 0u));
}

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Block-wide exclusive scan of one uint32 per thread; returns the prefix and
// writes the block total to *total.  `smem` needs blockDim/32 + 1 words.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = (lane < nwarps) ? smem[lane] : 0u;
    uint32_t t = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nwarps) smem[lane] = t - w;
    if (lane == nwarps - 1) smem[32] = t;
  }
  __syncthreads();
  uint32_t res = smem[warp] + x - v;
  *total = smem[32];
  __syncthreads();
  return res;
}

// Segments of an element range and where their outputs go: a batch's list or
// forest elements, instance after instance, are numbered densely; outputs are
// at the instances' places in the caller's arrays, roots relative to their
// instance.  At most 2^32 elements: offsets wrap.
struct SegMap {
  const uint32_t* base = nullptr;   // n + 1: the segments' first elements, non-decreasing; then the end
  const uint32_t* delta = nullptr;  // element + delta: its place in the outputs
  const uint32_t* hint = nullptr;   // [k]: the segment of element 4096 k, and one more for the end
  uint32_t n = 0;                   // 0: one instance, in place
  __device__ __forceinline__ uint32_t find(uint32_t x) const {  // the last j with base[j] <= x
    uint32_t lo = ld_ca(hint + (x >> 12)), hi = min(ld_ca(hint + (x >> 12) + 1) + 1, n);
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (ld_ca(base + mid) <= x)
        lo = mid;
      else
        hi = mid;
    }
    return lo;
  }
};

}  // namespace ks
