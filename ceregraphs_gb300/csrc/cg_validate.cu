// Graph500 result validation on the device: the five tree checks for k
// searches, 16 of them per pass over the resident graph, instead of the host-side
// scipy cross-check and invalid_parents walk the reference runs per search
// (run_graph500.py:383-395, bfs/plots/bfs_tree_plot.py:140-152), which
// dominates wall time for 64 searches at scale 23 and above.
//
// Checks (each search has a root, levels[n] and parents[n]; -1 = unreached):
//   ROOT       parent[root] == root and level[root] == 0
//   TREE       every reached v != root has a parent p in [0, n), level[v] >= 1
//              and level[p] == level[v] - 1 (levels fall by one along every
//              parent pointer, so the pointers form a tree into the root)
//   EDGES      every stored edge u -> v with u reached has v reached and
//              level[v] <= level[u] + 1 (for symmetric graphs both
//              orientations are stored, giving |level[u] - level[v]| <= 1)
//   SPAN       level[v] >= 0 exactly when parent[v] >= 0; with TREE and EDGES
//              the reached set is closed under out-edges and every reached
//              vertex leads to the root, so it is the reachable set
//   TREE_EDGE  parent[v] -> v is an edge (parent[v] is in v's in-list)
//   LOWEST     parent[v] is the lowest-index in-neighbour at level[v] - 1
//              (this engine's parent rule; not a Graph500 requirement)
// Inputs are treated as untrusted: a parent outside [0, n) is counted, never
// dereferenced.
#include <cuda_runtime.h>
#include <stdint.h>

#include <new>

#include "cg_internal.cuh"

namespace cg {
namespace {

constexpr int kChecks = CG_CHECKS;
constexpr int kBlock = 256;
constexpr int kEdgesPerWarp = 32 * 64;

struct Tally {  // per search, device side
  unsigned long long fail[kChecks];
  unsigned long long first[kChecks];  // lowest failing vertex, ~0 if none
};

__device__ __forceinline__ void flag(Tally *t, int check, int64_t v) {
  atomicAdd(&t->fail[check], 1ull);
  atomicMin(&t->first[check], (unsigned long long)v);
}

// Binary search for u in the sorted list idx[b, e).
__device__ __forceinline__ bool contains(const int32_t *__restrict__ idx, int64_t b, int64_t e,
                                         int32_t u) {
  while (b < e) {
    const int64_t mid = (b + e) >> 1;
    const int32_t x = idx[mid];
    if (x == u) return true;
    if (x < u)
      b = mid + 1;
    else
      e = mid;
  }
  return false;
}

// ---- up to 16 searches at once, levels below 126 ------------------------------
// The graph is read once for a group of 4 * NW searches instead of once per
// search.  A packing pass turns the group's levels into one byte per (vertex,
// search), b = level + 1, or 127 for an unreached vertex, stored vertex-major:
// one 4 * NW byte load per list entry gives its level in every search.  With
// t = level(v) for a reached v and 127 for an unreached one, an entry u -> v
//   breaks EDGES exactly when          b(u) <  t,
//   is one level above v exactly when  b(u) == t   (v reached),
// and both compares run on four searches per instruction: bytes are at most
// 127, so (t | 0x80) - b keeps bit 7 of a byte exactly when b <= t, without a
// borrow into the next byte.  A level above 125 does not fit: the packing pass
// then raises a flag, these kernels return and the per-search kernels below
// run instead (they return at once when the flag is down).
//
// Bound by instruction issue (1.7 of 4 per clock at 22 warps an SM: about 30
// instructions per 32 entries and 16 searches, and lists of uneven lengths in a
// warp) and by the latency of the 4 * NW byte gathers, which the L2 serves.
// R-MAT scale 20, 16 searches, device time: 6670 us for the two per-search
// kernels, 510 us for these (packing 12, vertices 417, long lists 81).
constexpr uint32_t kHigh = 0x80808080u, kOnes = 0x01010101u;
constexpr int kUnreached = 127, kMaxLevel = 125;
constexpr int kGroup = 16;          // searches of a group at most
constexpr int64_t kLaneList = 32;   // in-lists up to this: one thread
// Lists up to warp_list: the warp that owns the vertex; longer ones in chunks of
// 1 << chunk_bits entries, a warp each.  Large graphs have warps enough for
// longer pieces, whose set-up then counts less (16 searches, R-MAT, us with 128 and
// 512 / 512 and 1024: 1 M 693 / 658, degree 32 693 / 601, 256 K 369 / 371, 16 K 198 /
// 230).
constexpr int64_t kWarpList = 128, kWarpListLarge = 512;
constexpr int kChunkBits = 9, kChunkBitsLarge = 10;
constexpr int64_t kLargeGraph = 1 << 19;

// A vertex whose in-list is scanned in chunks: `base` is its first chunk.
struct LongVertex {
  int32_t v;
  uint32_t base;
};

struct GroupArgs {
  int64_t n;
  const int64_t *in_off;
  const int32_t *in_idx;
  const int64_t *roots;      // of the group's searches
  const int32_t *levels;     // [searches][n]
  const int32_t *parents;
  int searches;              // 1 .. 4 * NW
  Tally *tally;
  uint32_t *lv;              // [n][NW] level bytes
  int *wide;                 // set: some level does not fit a byte
  unsigned long long *nlong; // (vertices << 32) | chunks of the list below
  LongVertex *longs;
  uint32_t *pend;            // [longs][NW] searches whose parent is still to be checked
  uint32_t *bad;             // [longs][NW] searches already counted as LOWEST failures
  int64_t warp_list;
  int chunk_bits;
};

template <int NW>
__device__ __forceinline__ void ld_words(const uint32_t *lv, int64_t v, uint32_t (&x)[NW]) {
  if constexpr (NW == 4) {
    const uint4 q = __ldg(reinterpret_cast<const uint4 *>(lv) + v);
    x[0] = q.x, x[1] = q.y, x[2] = q.z, x[3] = q.w;
  } else if constexpr (NW == 2) {
    const uint2 q = __ldg(reinterpret_cast<const uint2 *>(lv) + v);
    x[0] = q.x, x[1] = q.y;
  } else {
    x[0] = __ldg(lv + v);
  }
}

// t | 0x80 per byte, from a vertex's level bytes: level, or 127 if unreached.
__device__ __forceinline__ uint32_t bound_of(uint32_t b) {
  const uint32_t unreached = ((b + kOnes) & kHigh) >> 7;
  return (b - kOnes + unreached) | kHigh;
}

// The low four bits of m as bit 7 of a byte each.
__device__ __forceinline__ uint32_t byte_flags(unsigned m) {
  return ((m & 0xfu) * 0x00204081u & kOnes) << 7;
}

template <int NW>
__device__ __forceinline__ void pack_levels(const GroupArgs &a) {
  const int64_t v = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  if (v >= a.n) return;
  uint32_t x[NW];
  bool wide = false;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    x[w] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int s = 4 * w + j;
      const int32_t l = s < a.searches ? __ldg(a.levels + (int64_t)s * a.n + v) : -1;
      wide |= l > kMaxLevel;
      x[w] |= (uint32_t)(l < 0 || l > kMaxLevel ? kUnreached : l + 1) << (8 * j);
    }
  }
#pragma unroll
  for (int w = 0; w < NW; ++w) a.lv[v * NW + w] = x[w];
  if (wide) *a.wide = 1;
}

// Failing searches of one list entry (bit 7 of each byte of m): EDGES at v.
template <int NW>
__device__ __noinline__ void flag_edges(const GroupArgs &a, const uint32_t (&m)[NW], int64_t v) {
  for (int s = 0; s < a.searches; ++s)
    if ((m[s >> 2] >> (8 * (s & 3) + 7)) & 1u) flag(a.tally + s, CG_CHECK_EDGES, v);
}

// Searches in which v is reached, below its root (bit 7 of each byte), from
// bound_of: t is 1 .. 126.
__device__ __forceinline__ uint32_t below_root(uint32_t th) {
  const uint32_t t = th & ~kHigh;
  return (t + ~kHigh) & ~(t + kOnes) & kHigh;
}

// v's t (level, or 127) in search s, s the lane's own.
template <int NW>
__device__ __forceinline__ int level_of(const uint32_t (&th)[NW], int s) {
  uint32_t x = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w)
    if ((s >> 2) == w) x = th[w];
  return (int)((x >> (8 * (s & 3))) & 0x7fu);
}

// The checks of v's own level t and parent p in search s (SPAN, ROOT and what
// TREE needs no other vertex for).  True if p is a vertex to look for among v's
// in-neighbours.
__device__ __forceinline__ bool check_vertex(const GroupArgs &a, int s, int64_t v, int t,
                                             int32_t p) {
  const bool reached = t != kUnreached;
  if (reached != (p >= 0)) flag(a.tally + s, CG_CHECK_SPAN, v);
  if (v == __ldg(a.roots + s)) {
    if (p != (int32_t)v || t != 0) flag(a.tally + s, CG_CHECK_ROOT, v);
    return false;
  }
  if (p >= 0 && reached && t > 0 && p < a.n) return true;
  if (p >= 0 || p < -1) flag(a.tally + s, CG_CHECK_TREE, v);
  return false;
}

// p is one level up from v in search s (TREE).
template <int NW>
__device__ __forceinline__ bool one_up(const GroupArgs &a, int s, int64_t v, int t, int32_t p) {
  if (__ldg(reinterpret_cast<const uint8_t *>(a.lv) + (int64_t)p * (4 * NW) + s) == t) return true;
  flag(a.tally + s, CG_CHECK_TREE, v);
  return false;
}

// The first in-neighbour of v one level up in search s is u (-1: none), its
// parent is p: where they are the same, p is one level up, in the list and the
// lowest, and its level is not read.
template <int NW>
__device__ __forceinline__ void check_first(const GroupArgs &a, int s, int64_t v, int64_t b,
                                            int64_t e, int t, int32_t u, int32_t p) {
  if (u == p || !one_up<NW>(a, s, v, t, p)) return;
  flag(a.tally + s, CG_CHECK_LOWEST, v);
  if (!contains(a.in_idx, b, e, p)) flag(a.tally + s, CG_CHECK_TREE_EDGE, v);
}

// Entries [j0, j1) of v's in-list by the whole warp, 128 a step, no lane
// diverging: a search of `pend` with an entry one level up leaves pend, and
// lane s (its search's number) returns the first such entry, or -1.
template <int NW>
__device__ __forceinline__ int32_t warp_entries(const GroupArgs &a, int64_t v, int64_t j0,
                                                int64_t j1, const uint32_t (&th)[NW],
                                                uint32_t (&pend)[NW]) {
  constexpr int Q = 4;
  const int lane = threadIdx.x & 31;
  int32_t first = -1;
  uint32_t open = 0;  // some search of pend is left (the same in every lane)
#pragma unroll
  for (int w = 0; w < NW; ++w) open |= pend[w];
  for (int64_t j = j0; j < j1; j += 32 * Q) {
    int32_t u[Q];
    uint32_t x[Q][NW];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int64_t i = j + 32 * q + lane;
      u[q] = i < j1 ? __ldg(a.in_idx + i) : -1;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (u[q] >= 0) {
        ld_words<NW>(a.lv, u[q], x[q]);
      } else {
#pragma unroll
        for (int w = 0; w < NW; ++w) x[q][w] = (uint32_t)kUnreached * kOnes;
      }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      uint32_t lt[NW], eq[NW], any_lt = 0, any_eq = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const uint32_t d = th[w] - x[q][w];
        lt[w] = (d - kOnes) & kHigh;
        eq[w] = d & ~lt[w] & pend[w];
        any_lt |= lt[w];
        any_eq |= eq[w];
      }
      if (any_lt) flag_edges<NW>(a, lt, v);
      if (!open || !__any_sync(0xffffffffu, any_eq != 0)) continue;
      open = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        uint32_t m = __reduce_or_sync(0xffffffffu, eq[w]);
        pend[w] &= ~m;
        open |= pend[w];
        while (m) {
          const int bit = __ffs(m) - 1;
          m &= m - 1;
          const unsigned who = __ballot_sync(0xffffffffu, (eq[w] >> bit) & 1u);
          const int32_t uu = __shfl_sync(0xffffffffu, u[q], __ffs(who) - 1);
          if (lane == 4 * w + (bit >> 3)) first = uu;
        }
      }
    }
  }
  return first;
}

// Every check of the group's searches, one warp per 32 consecutive vertices:
// short in-lists by their lane (four entries' loads in flight), middling ones by
// the warp; long ones go on a list for check_long_kernel.  Parents are read
// once, after the list: the level of one that is the list's first vertex a level
// up needs no look (16 M byte gathers less, 338 -> 330 us).
template <int NW>
__device__ __forceinline__ void check_vertices(const GroupArgs &a) {
  if (*(volatile int *)a.wide) return;
  const int lane = threadIdx.x & 31;
  const int64_t v = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  uint32_t th[NW], pend[NW];
  int64_t b = 0, e = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) th[w] = ~0u, pend[w] = 0;
  if (v < a.n) {
    uint32_t mine[NW];
    ld_words<NW>(a.lv, v, mine);
    b = __ldg(a.in_off + v);
    e = __ldg(a.in_off + v + 1);
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      th[w] = bound_of(mine[w]);
      pend[w] = below_root(th[w]);
    }
  }
  const int64_t deg = e - b;
  if (deg <= kLaneList) {
    // each search's first entry one level up, as a list position in its byte
    // (no branch: every lane would take it at an entry of its own)
    uint32_t at[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) at[w] = 0;
    for (int64_t j = b; j < e; j += 4) {
      int32_t u[4];
      uint32_t x[4][NW];
#pragma unroll
      for (int q = 0; q < 4; ++q) u[q] = j + q < e ? __ldg(a.in_idx + j + q) : -1;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (u[q] >= 0) {
          ld_words<NW>(a.lv, u[q], x[q]);
        } else {
#pragma unroll
          for (int w = 0; w < NW; ++w) x[q][w] = (uint32_t)kUnreached * kOnes;
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t lt[NW], eq[NW], any_lt = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          const uint32_t d = th[w] - x[q][w];
          lt[w] = (d - kOnes) & kHigh;
          eq[w] = d & ~lt[w] & pend[w];
          any_lt |= lt[w];
        }
        if (any_lt) flag_edges<NW>(a, lt, v);
        const uint32_t pos = (uint32_t)(j - b) + q;  // < 32
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          at[w] += (eq[w] >> 7) * pos;
          pend[w] &= ~eq[w];
        }
      }
    }
    if (v < a.n) {
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const uint32_t found = below_root(th[w]) & ~pend[w];
        int32_t p[4], u[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int s = 4 * w + j;
          p[j] = s < a.searches ? __ldg(a.parents + (int64_t)s * a.n + v) : -1;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          u[j] = (found >> (8 * j + 7)) & 1u
                     ? __ldg(a.in_idx + b + ((at[w] >> (8 * j)) & 0xffu))
                     : -1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int s = 4 * w + j;
          const int t = (int)((th[w] >> (8 * j)) & 0x7fu);
          if (s < a.searches && check_vertex(a, s, v, t, p[j]))
            check_first<NW>(a, s, v, b, e, t, u[j], p[j]);
        }
      }
    }
  }
  // lists of kLaneList + 1 .. warp_list entries: the whole warp, one at a time
  unsigned todo = __ballot_sync(0xffffffffu, deg > kLaneList && deg <= a.warp_list);
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const int64_t vb = __shfl_sync(0xffffffffu, b, src), ve = __shfl_sync(0xffffffffu, e, src);
    const int64_t vv = v - lane + src;
    uint32_t sth[NW], sp[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      sth[w] = __shfl_sync(0xffffffffu, th[w], src);
      sp[w] = __shfl_sync(0xffffffffu, pend[w], src);
    }
    // lane s: search s's parent
    const int32_t p = lane < a.searches ? __ldg(a.parents + (int64_t)lane * a.n + vv) : -1;
    const int32_t u = warp_entries<NW>(a, vv, vb, ve, sth, sp);
    const int t = level_of<NW>(sth, lane);
    if (lane < a.searches && check_vertex(a, lane, vv, t, p))
      check_first<NW>(a, lane, vv, vb, ve, t, u, p);
  }
  const unsigned ml = __ballot_sync(0xffffffffu, deg > a.warp_list);
  // long lists: lane s checks search s's parent, in the list or not; the chunks
  // then only look for a lower one
  for (unsigned m = ml; m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const int64_t vb = __shfl_sync(0xffffffffu, b, src), ve = __shfl_sync(0xffffffffu, e, src);
    const int64_t vv = v - lane + src;
    uint32_t sth[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) sth[w] = __shfl_sync(0xffffffffu, th[w], src);
    bool want = false;
    if (lane < a.searches) {
      const int32_t p = __ldg(a.parents + (int64_t)lane * a.n + vv);
      const int t = level_of<NW>(sth, lane);
      want = check_vertex(a, lane, vv, t, p) && one_up<NW>(a, lane, vv, t, p);
      if (want && !contains(a.in_idx, vb, ve, p)) {
        flag(a.tally + lane, CG_CHECK_LOWEST, vv);
        flag(a.tally + lane, CG_CHECK_TREE_EDGE, vv);
        want = false;
      }
    }
    const unsigned wanted = __ballot_sync(0xffffffffu, want);
    if (lane == src) {
#pragma unroll
      for (int w = 0; w < NW; ++w) pend[w] = byte_flags(wanted >> (4 * w));
    }
  }
  if (deg > a.warp_list) {
    const unsigned chunks = (unsigned)((deg - 1) >> a.chunk_bits) + 1u;
    // one packed add gives the entry's place and its first chunk, so the list
    // is sorted by first chunk
    const unsigned long long old = atomicAdd(a.nlong, (1ull << 32) | chunks);
    const unsigned at = (unsigned)(old >> 32);
    a.longs[at] = LongVertex{(int32_t)v, (uint32_t)old};
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      a.pend[(int64_t)at * NW + w] = pend[w];
      a.bad[(int64_t)at * NW + w] = 0;
    }
  }
}

// The listed vertices' in-lists, a warp per chunk.  The
// parents are known to be in the lists, so LOWEST fails exactly when a chunk
// holds an entry one level up below the parent; `bad` counts it once.
template <int NW>
__device__ __forceinline__ void check_long(const GroupArgs &a) {
  if (*(volatile int *)a.wide) return;
  const unsigned long long total = *(volatile unsigned long long *)a.nlong;
  const unsigned nv = (unsigned)(total >> 32), nchunks = (unsigned)total;
  const unsigned nwarps = gridDim.x * (kBlock / 32);
  const int lane = threadIdx.x & 31;
  for (unsigned c = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); c < nchunks; c += nwarps) {
    unsigned lo = 0, hi = nv - 1;  // the last entry whose first chunk is <= c
    while (lo < hi) {
      const unsigned mid = (lo + hi + 1) >> 1;
      if (a.longs[mid].base <= c)
        lo = mid;
      else
        hi = mid - 1;
    }
    const int64_t v = a.longs[lo].v;
    const int64_t b = __ldg(a.in_off + v) + ((int64_t)(c - a.longs[lo].base) << a.chunk_bits);
    const int64_t end = __ldg(a.in_off + v + 1);
    const int64_t e = min(b + ((int64_t)1 << a.chunk_bits), end);
    uint32_t th[NW], pend[NW];
    ld_words<NW>(a.lv, v, th);
    // lane s holds search s's parent; only the chunks that start below it can
    // hold a lower entry (a list's first ones, mostly)
    const int32_t par = lane < a.searches ? __ldg(a.parents + (int64_t)lane * a.n + v) : -1;
    const unsigned below = __ballot_sync(0xffffffffu, __ldg(a.in_idx + b) < par);
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      th[w] = bound_of(th[w]);
      pend[w] = a.pend[(int64_t)lo * NW + w] & byte_flags(below >> (4 * w));
    }
    const int32_t u = warp_entries<NW>(a, v, b, e, th, pend);
    if (u < 0 || u >= par) continue;
    const uint32_t bit = 0x80u << (8 * (lane & 3));
    if (!(atomicOr(a.bad + (int64_t)lo * NW + (lane >> 2), bit) & bit))
      flag(a.tally + lane, CG_CHECK_LOWEST, v);
  }
}

template <int NW>
__global__ void __launch_bounds__(kBlock) pack_levels_kernel(GroupArgs a) { pack_levels<NW>(a); }
template <int NW>
__global__ void __launch_bounds__(kBlock, 4) check_vertices_kernel(GroupArgs a) {
  check_vertices<NW>(a);
}
template <int NW>
__global__ void __launch_bounds__(kBlock, 4) check_long_kernel(GroupArgs a) { check_long<NW>(a); }

// The same for full groups side by side, group `a` + blockIdx.y; long_cap: entries
// of each one's longs, pend and bad.
__device__ __forceinline__ GroupArgs beside(const GroupArgs &first, int64_t long_cap) {
  GroupArgs a = first;
  const int64_t y = blockIdx.y;
  a.roots += y * kGroup;
  a.levels += y * kGroup * a.n;
  a.parents += y * kGroup * a.n;
  a.tally += y * kGroup;
  a.wide += y;
  a.nlong += y;
  a.lv += y * a.n * (kGroup / 4);
  a.longs += y * long_cap;
  a.pend += y * long_cap * (kGroup / 4);
  a.bad += y * long_cap * (kGroup / 4);
  return a;
}
__global__ void __launch_bounds__(kBlock) pack_levels_beside_kernel(GroupArgs a, int64_t long_cap) {
  pack_levels<kGroup / 4>(beside(a, long_cap));
}
__global__ void __launch_bounds__(kBlock, 4) check_vertices_beside_kernel(GroupArgs a,
                                                                          int64_t long_cap) {
  check_vertices<kGroup / 4>(beside(a, long_cap));
}
__global__ void __launch_bounds__(kBlock, 4) check_long_beside_kernel(GroupArgs a,
                                                                      int64_t long_cap) {
  check_long<kGroup / 4>(beside(a, long_cap));
}

// ---- one search at a time, any level ------------------------------------------
// Per-vertex checks (ROOT, TREE, SPAN, TREE_EDGE, LOWEST).  Each warp takes 32
// consecutive vertices; a lane scans its own in-list for the lowest parent
// when it is short, and the warp scans the long ones together.  `wide`, if
// given: run only when it is set.
__global__ void __launch_bounds__(kBlock) vertex_checks_kernel(
    int64_t n, const int64_t *__restrict__ in_off, const int32_t *__restrict__ in_idx,
    const int64_t *__restrict__ roots, int k, const int32_t *__restrict__ levels_all,
    const int32_t *__restrict__ parents_all, const int *wide, Tally *tallies) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (kBlock / 32);
  for (int s = blockIdx.y; s < k; s += gridDim.y) {
    if (wide && !wide[s / kGroup]) continue;
    const int32_t *__restrict__ level = levels_all + (int64_t)s * n;
    const int32_t *__restrict__ parent = parents_all + (int64_t)s * n;
    const int64_t root = roots[s];
    Tally *t = tallies + s;
    for (int64_t base = ((int64_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * 32; base < n;
         base += warps * 32) {
      const int64_t v = base + lane;
      bool long_scan = false, checked = false;
      int32_t want_level = 0, p = -1, low = -1;
      int64_t b = 0, e = 0;
      if (v < n) {
        const int32_t lv = level[v];
        p = parent[v];
        if ((lv >= 0) != (p >= 0)) flag(t, CG_CHECK_SPAN, v);
        if (v == root) {
          if (p != (int32_t)root || lv != 0) flag(t, CG_CHECK_ROOT, v);
        } else if (p >= 0) {
          if (p >= n || lv < 1 || level[p] != lv - 1) {
            flag(t, CG_CHECK_TREE, v);
          } else {
            checked = true;
            b = in_off[v];
            e = in_off[v + 1];
            want_level = lv - 1;
            if (e - b <= 32) {
              for (int64_t j = b; j < e; ++j) {
                const int32_t u = in_idx[j];
                if (level[u] == want_level) {
                  low = u;
                  break;
                }
              }
            } else {
              long_scan = true;
            }
          }
        } else if (p < -1) {
          flag(t, CG_CHECK_TREE, v);
        }
      }
      // long in-lists: the whole warp scans one list at a time, 32 entries per step
      unsigned pending = __ballot_sync(0xffffffffu, long_scan);
      while (pending) {
        const int src = __ffs(pending) - 1;
        pending &= pending - 1;
        const int64_t sb = __shfl_sync(0xffffffffu, b, src);
        const int64_t se = __shfl_sync(0xffffffffu, e, src);
        const int32_t sl = __shfl_sync(0xffffffffu, want_level, src);
        int32_t first = -1;
        for (int64_t j = sb; j < se; j += 32) {
          const int64_t jj = j + lane;
          const bool hit = jj < se && level[in_idx[jj]] == sl;
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          if (m) {
            first = __shfl_sync(0xffffffffu, jj < se ? in_idx[jj] : -1, __ffs(m) - 1);
            break;
          }
        }
        if (lane == src) low = first;
      }
      // the parent is one level up: it is the first such entry, or it is not
      // in the list, or a lower one precedes it
      if (checked && low != p) {
        flag(t, CG_CHECK_LOWEST, v);
        if (!contains(in_idx, b, e, p)) flag(t, CG_CHECK_TREE_EDGE, v);
      }
    }
  }
}

// EDGES over every stored entry, balanced by entries: each warp owns
// kEdgesPerWarp consecutive entries, lanes stride by 32 and track their row.
__global__ void __launch_bounds__(kBlock) edge_checks_kernel(
    int64_t n, int64_t nnz, const int64_t *__restrict__ in_off, const int32_t *__restrict__ in_idx,
    int k, const int32_t *__restrict__ levels_all, const int *wide, Tally *tallies) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (kBlock / 32);
  for (int s = blockIdx.y; s < k; s += gridDim.y) {
    if (wide && !wide[s / kGroup]) continue;
    const int32_t *__restrict__ level = levels_all + (int64_t)s * n;
    Tally *t = tallies + s;
    for (int64_t w0 = ((int64_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * kEdgesPerWarp;
         w0 < nnz; w0 += warps * kEdgesPerWarp) {
      int64_t e = w0 + lane;
      if (e >= nnz) continue;
      // row r with in_off[r] <= e < in_off[r + 1]
      int64_t lo = 0, hi = n;
      while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (in_off[mid] <= e)
          lo = mid;
        else
          hi = mid - 1;
      }
      int64_t r = lo, r_end = in_off[r + 1];
      int32_t lr = level[r];
      const int64_t stop = min(w0 + (int64_t)kEdgesPerWarp, nnz);
      for (; e < stop; e += 32) {
        while (e >= r_end) {
          ++r;
          r_end = in_off[r + 1];
          lr = level[r];
        }
        const int32_t lu = level[in_idx[e]];
        if (lu >= 0 && (lr < 0 || (int64_t)lr > (int64_t)lu + 1)) flag(t, CG_CHECK_EDGES, r);
      }
    }
  }
}

__global__ void tally_init_kernel(Tally *t, int k) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < k * kChecks) {
    t[i / kChecks].fail[i % kChecks] = 0ull;
    t[i / kChecks].first[i % kChecks] = ~0ull;
  }
}

constexpr size_t round256(size_t x) { return (x + 255) & ~(size_t)255; }

// In-lists longer than kWarpList, at most.
int64_t long_capacity(const cg_graph *g) {
  const int64_t c = g->nnz / (kWarpList + 1) + 1;
  return c < g->n ? c : g->n;
}

// Full groups side by side: as many as fill the GPU, 8 blocks an SM, one vertex a
// thread.
int groups_beside(const cg_graph *g, int full) {
  const int64_t blocks = (g->n + kBlock - 1) / kBlock, most = (int64_t)g->num_sms * 8 / blocks;
  const int64_t side = most < full ? most : full;
  return side < 1 ? 1 : (int)side;
}

// The handle's workspace for `groups` groups of `nw` level words per vertex (kept
// for later calls, freed with the handle); false when it cannot be had, and the
// per-search kernels, which need none, do the work.
bool check_workspace(cg_graph *g, int nw, int groups, GroupArgs *a) {
  const size_t nl = (size_t)long_capacity(g) * groups;
  const size_t lv = round256(sizeof(uint32_t) * nw * (size_t)g->n * groups);
  const size_t longs = round256(sizeof(LongVertex) * nl), mask = round256(sizeof(uint32_t) * nw * nl);
  const size_t bytes = lv + longs + 2 * mask;
  if (g->check_bytes < bytes) {
    cudaFree(g->check_ws);  // earlier calls have waited for their kernels
    g->check_ws = nullptr;
    g->device_bytes -= (int64_t)g->check_bytes;
    g->check_bytes = 0;
    if (cudaMalloc(&g->check_ws, bytes) != cudaSuccess) {
      cudaGetLastError();
      g->check_ws = nullptr;
      return false;
    }
    g->check_bytes = bytes;
    g->device_bytes += (int64_t)bytes;
  }
  unsigned char *p = static_cast<unsigned char *>(g->check_ws);
  a->lv = reinterpret_cast<uint32_t *>(p);
  a->longs = reinterpret_cast<LongVertex *>(p + lv);
  a->pend = reinterpret_cast<uint32_t *>(p + lv + longs);
  a->bad = reinterpret_cast<uint32_t *>(p + lv + longs + mask);
  return true;
}

template <int NW>
void launch_group(const cg_graph *g, const GroupArgs &a) {
  const unsigned vb = (unsigned)((g->n + kBlock - 1) / kBlock);
  pack_levels_kernel<NW><<<vb, kBlock, 0, g->stream>>>(a);
  check_vertices_kernel<NW><<<vb, kBlock, 0, g->stream>>>(a);
  check_long_kernel<NW><<<(unsigned)g->num_sms * 6, kBlock, 0, g->stream>>>(a);
}

// Groups a .. a + groups - 1, 16 searches each, at once: a small graph's group
// leaves most of the GPU idle (64 searches of R-MAT scale 12: 553 us a call with the
// groups in turn, 288 so; scale 16: 597 and 366).
void launch_groups(const cg_graph *g, const GroupArgs &a, int groups) {
  const dim3 vb((unsigned)((g->n + kBlock - 1) / kBlock), (unsigned)groups);
  const int64_t cap = long_capacity(g);
  pack_levels_beside_kernel<<<vb, kBlock, 0, g->stream>>>(a, cap);
  check_vertices_beside_kernel<<<vb, kBlock, 0, g->stream>>>(a, cap);
  const dim3 lb((unsigned)((g->num_sms * 6 + groups - 1) / groups), (unsigned)groups);
  check_long_beside_kernel<<<lb, kBlock, 0, g->stream>>>(a, cap);
}

// Grid of a per-search kernel, one search filling `blocks` blocks: at most 8
// blocks an SM for a search, and searches side by side (blockIdx.y, the rest in
// turn) up to four times that, k / 8 times from 32 searches on.  One after another,
// the searches of a small deep graph leave the GPU idle: 64 of a 200^2 grid took
// 2,960 us a call, 302 so; of a caterpillar of 3,000 vertices with 30 leaves each
// 9,760 and 460.  No more, so that the launch stays short where the groups have done
// all of it (16 searches of R-MAT scale 20, 665 us: 8 us longer with 16 times).
dim3 search_grid(const cg_graph *g, int64_t blocks, int k) {
  const int64_t cap = (int64_t)g->num_sms * 8;
  const int64_t x = blocks < cap ? blocks : cap;
  const int64_t side = ((k / 8 > 4 ? k / 8 : 4) * cap + x - 1) / x;
  return dim3((unsigned)x, (unsigned)(side < k ? side : k));
}

}  // namespace
}  // namespace cg

using namespace cg;

extern "C" int cg_validate_device(cg_graph *g, const int64_t *roots, int32_t k,
                                  const int32_t *d_levels, const int32_t *d_parents,
                                  cg_validation *out) {
  if (g) {
    if (int r = refuse_reordered(g, "cg_validate_device")) return r;
  }
  if (!g || !roots || k <= 0 || k > 65535 || !d_levels || !d_parents || !out)
    return CG_ERR_INVALID_ARG;
  for (int32_t i = 0; i < k; ++i)
    if (roots[i] < 0 || roots[i] >= g->n) return CG_ERR_INVALID_ARG;
  CG_CUDA(cudaSetDevice(g->device));
  // one block of scratch: tallies, roots, then per group of searches the count
  // of its long in-lists and its `wide` flag (the last two start at zero)
  const int groups = (k + kGroup - 1) / kGroup;
  const size_t t_bytes = round256(sizeof(Tally) * (size_t)k);
  const size_t r_bytes = round256(sizeof(int64_t) * (size_t)k);
  const size_t z_bytes = (sizeof(unsigned long long) + sizeof(int)) * (size_t)groups;
  unsigned char *scratch = nullptr;
  if (int r = call_scratch(g, t_bytes + r_bytes + z_bytes, (void **)&scratch)) return r;
  Tally *d_t = reinterpret_cast<Tally *>(scratch);
  int64_t *d_roots = reinterpret_cast<int64_t *>(scratch + t_bytes);
  unsigned long long *d_nlong =
      reinterpret_cast<unsigned long long *>(scratch + t_bytes + r_bytes);
  int *d_wide = reinterpret_cast<int *>(d_nlong + groups);
  int rc = CG_OK;
  Tally *h_t = new (std::nothrow) Tally[k];
  do {
    if (!h_t) { rc = CG_ERR_OUT_OF_MEMORY; break; }
    cudaError_t e = cudaMemcpyAsync(d_roots, roots, sizeof(int64_t) * (size_t)k,
                                    cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_nlong, 0, z_bytes, g->stream);
    if (e != cudaSuccess) { rc = cuda_fail(e, "validate roots"); break; }
    tally_init_kernel<<<(k * kChecks + 255) / 256, 256, 0, g->stream>>>(d_t, k);
    GroupArgs a{};
    const int most = k < kGroup ? k : kGroup;
    const int side = groups_beside(g, k / kGroup);
    const bool grouped = check_workspace(g, most <= 4 ? 1 : (most <= 8 ? 2 : 4), side, &a);
    if (grouped) {
      a.n = g->n;
      a.in_off = g->in_off;
      a.in_idx = g->in_idx;
      a.warp_list = g->n >= kLargeGraph ? kWarpListLarge : kWarpList;
      a.chunk_bits = g->n >= kLargeGraph ? kChunkBitsLarge : kChunkBits;
      for (int i = 0, now; i < groups; i += now) {
        const int64_t s0 = (int64_t)i * kGroup;
        a.roots = d_roots + s0;
        a.levels = d_levels + s0 * g->n;
        a.parents = d_parents + s0 * g->n;
        a.searches = (int)(k - s0 < kGroup ? k - s0 : kGroup);
        a.tally = d_t + s0;
        a.wide = d_wide + i;
        a.nlong = d_nlong + i;
        now = 1;
        if (side > 1 && a.searches == kGroup) {
          now = k / kGroup - i < side ? k / kGroup - i : side;
          launch_groups(g, a, now);
        } else if (a.searches <= 4) {
          launch_group<1>(g, a);
        } else if (a.searches <= 8) {
          launch_group<2>(g, a);
        } else {
          launch_group<4>(g, a);
        }
      }
    }
    // the searches the groups left (levels past a byte), or all of them
    const int *wide = grouped ? d_wide : nullptr;
    vertex_checks_kernel<<<search_grid(g, (g->n + kBlock - 1) / kBlock, k), kBlock, 0,
                           g->stream>>>(g->n, g->in_off, g->in_idx, d_roots, k, d_levels,
                                        d_parents, wide, d_t);
    if (g->nnz > 0) {
      const int64_t per_block = (int64_t)kEdgesPerWarp * (kBlock / 32);
      edge_checks_kernel<<<search_grid(g, (g->nnz + per_block - 1) / per_block, k), kBlock, 0,
                           g->stream>>>(g->n, g->nnz, g->in_off, g->in_idx, k, d_levels, wide,
                                        d_t);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(h_t, d_t, sizeof(Tally) * (size_t)k, cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    if (e != cudaSuccess) { rc = cuda_fail(e, "cg_validate_device"); break; }
    for (int32_t i = 0; i < k; ++i) {
      for (int c = 0; c < kChecks; ++c) {
        out[i].failures[c] = (int64_t)h_t[i].fail[c];
        out[i].first[c] = h_t[i].first[c] == ~0ull ? -1 : (int64_t)h_t[i].first[c];
      }
    }
  } while (0);
  if (rc) cudaStreamSynchronize(g->stream);
  delete[] h_t;
  return rc;
}
