// FIFO parents: the parent rule of scipy's breadth_first_order, the host BFS
// the reference's driver checks its searches against (run_graph500.py:383-395,
// run_bfs.py:517-527).  That search pops its queue in order and gives every
// out-neighbour it has not seen yet (in ascending id order) the popped vertex
// as predecessor.  So the parent of a vertex at level L+1 is its level-L
// in-neighbour of smallest queue rank, and level L+1 is queued in order of
// (rank of the parent, vertex id).
//
// Given the levels of a finished search, this pass recomputes the parents
// level by level.  The vertices are first listed by level, each level in id order
// (fifo_list_kernel).  Level L's ranks reach level L+1
// from whichever side has fewer list entries -- each vertex takes the minimum
// over its in-list of a 4-byte rank map, or level L's out-lists push their ranks
// by atomicMin -- and a stable sort of level L+1 by parent rank, as few bits as
// level L has ranks, is its queue order.  After a level of one vertex nothing
// is left to do: the search's parents stand and id order is queue order.  The
// level sizes steer this from the host, so the pass synchronises with the
// stream (and is refused inside a graph capture).
//
// Bound by the dependent launches of a level (about nine, 3 to 10 us each) and
// by the rank gathers of the widest levels.  R-MAT scale 20, a call with its
// search: 1,296 us with a warp per vertex, 64-bit sorts and one block for levels of
// few vertices but long lists, 414 us now.
#include <cuda_runtime.h>
#include <stdint.h>

#include <new>
#include <vector>

#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>

#include "cg_internal.cuh"

namespace cg {

constexpr int kFifoSums = 64;  // levels whose list entries are counted

struct FifoSums {
  int maxlevel;
  unsigned counts[kFifoSums];
  unsigned long long out[kFifoSums], in[kFifoSums];  // degrees summed
};

struct FifoLong {  // a long list: its first chunk, the vertex, its rank (out-lists)
  uint32_t base;
  int32_t v;
  uint32_t rank;
};

struct FifoState {
  int64_t n = 0;
  unsigned char *base = nullptr;  // the one allocation of what follows
  FifoSums *sums = nullptr;
  unsigned long long *nlong = nullptr;  // (lists << 32) | chunks of `longs`
  int32_t *order = nullptr;       // [n] vertices sorted by (level, id)
  uint32_t *rk = nullptr;         // [n] rank of the level being read, ~0 elsewhere
  uint32_t *best = nullptr;       // [n] smallest parent rank of a vertex, ~0 none yet
  uint32_t *key[2] = {nullptr, nullptr};  // [n] sort keys
  int32_t *queue[3] = {nullptr, nullptr, nullptr};  // [n] a level in queue order, and sort values
  unsigned *counts = nullptr;     // [n + 1] vertices per level
  unsigned *block_counts = nullptr;  // [kListDigits][list_blocks + 1] of the listing passes
  FifoLong *longs = nullptr;
  void *temp = nullptr;           // radix sort scratch
  size_t temp_bytes = 0;
  // runs of small levels: the ranks, and (level << 32) | rank and (level << 32)
  // | FIFO parent of the vertices ranked so far in this pass (-1 elsewhere)
  int32_t *rank = nullptr;                      // [n]
  unsigned long long *lr = nullptr, *pl = nullptr;  // [n]
  unsigned *offs = nullptr;       // [n + 2] first slot of each level in order
};

namespace {

constexpr int kFifoBlock = 256;
constexpr unsigned kAll = 0xffffffffu;
constexpr uint32_t kNoRank = 0xffffffffu;
constexpr int64_t kFifoLane = 32;    // in-lists up to this: one thread
constexpr int64_t kFifoWarp = 1024;  // lists up to this: the warp that meets them; above: chunks
constexpr int64_t kFifoChunk = 512;

// A listing pass's blocks have a run of items each, of the graph's vertices 4 blocks
// an SM.
constexpr int kListDigits = 256;
static_assert(kFifoSums <= kListDigits && kFifoBlock == kListDigits, "a thread per digit");
int64_t list_run(int64_t n, int sms) {
  const int64_t run = (n + 4 * (int64_t)sms - 1) / (4 * (int64_t)sms);
  return (run + kFifoBlock - 1) / kFifoBlock * kFifoBlock;
}
unsigned list_blocks(int64_t items, int64_t run) { return (unsigned)((items + run - 1) / run); }

// Vertices per level (levels >= 0), their degrees summed (the first kFifoSums
// levels), and the deepest level; block_counts: the first kFifoSums levels' counts
// by block, for fifo_list_kernel (the same grid and run).  One round of shared atomics per level
// present in a warp, then one global atomic a block and value: a maximum from
// each of 9,700 warps to one address, and the sums of 2,400 blocks, were most of its
// 20 us on R-MAT scale 20 (the whole call 294 -> 282 us with 4 blocks an SM; 286 with
// 2, 288 with 8 or 16).
__global__ void __launch_bounds__(kFifoBlock) fifo_hist_kernel(
    int64_t n, int64_t run, const int32_t *__restrict__ levels,
    const int64_t *__restrict__ in_off, const int64_t *__restrict__ out_off, unsigned *counts,
    unsigned *block_counts, FifoSums *sums) {
  __shared__ unsigned s_count[kFifoSums];
  __shared__ unsigned long long s_out[kFifoSums], s_in[kFifoSums];
  __shared__ int s_max;
  if (threadIdx.x == 0) s_max = -1;
  for (int i = threadIdx.x; i < kFifoSums; i += blockDim.x) s_count[i] = s_out[i] = s_in[i] = 0;
  __syncthreads();
  const int lane = lane_id();
  int mx = -1;
  const int64_t end = min(n, (blockIdx.x + 1) * run);
  for (int64_t base = blockIdx.x * run + (threadIdx.x & ~31u); base < end; base += kFifoBlock) {
    const int64_t v = base + lane;
    const int L = v < end ? levels[v] : -1;
    unsigned din = 0, dout = 0;
    if (L >= 0 && L < kFifoSums) {
      din = (unsigned)(__ldg(in_off + v + 1) - __ldg(in_off + v));
      dout = out_off == in_off ? din : (unsigned)(__ldg(out_off + v + 1) - __ldg(out_off + v));
    }
    mx = max(mx, L);
    unsigned todo = __ballot_sync(kAll, L >= 0);
    while (todo) {
      const int l = __shfl_sync(kAll, L, __ffs(todo) - 1);
      const unsigned m = __ballot_sync(kAll, L == l);
      todo &= ~m;
      if (l >= kFifoSums) {
        if (lane == 0) atomicAdd(&counts[l], (unsigned)__popc(m));
        continue;
      }
      const unsigned i = __reduce_add_sync(kAll, L == l ? din : 0u);
      const unsigned o = out_off == in_off ? i : __reduce_add_sync(kAll, L == l ? dout : 0u);
      if (lane == 0) {
        atomicAdd(&s_count[l], (unsigned)__popc(m));
        atomicAdd(&s_in[l], (unsigned long long)i);
        atomicAdd(&s_out[l], (unsigned long long)o);
      }
    }
  }
  mx = __reduce_max_sync(kAll, mx);
  if (lane == 0 && mx >= 0) atomicMax(&s_max, mx);
  __syncthreads();
  if (threadIdx.x == 0 && s_max >= 0) atomicMax(&sums->maxlevel, s_max);
  for (int i = threadIdx.x; i < kFifoSums; i += blockDim.x) {
    block_counts[i * gridDim.x + blockIdx.x] = s_count[i];
    if (s_count[i]) {
      atomicAdd(&counts[i], s_count[i]);
      atomicAdd(&sums->counts[i], s_count[i]);
      atomicAdd(&sums->in[i], s_in[i]);
      atomicAdd(&sums->out[i], s_out[i]);
    }
  }
}

// One pass of the listing: the items (in[0 .. count), or all vertices below `count`
// that were reached) in the order of digit (level >> shift) & 255, items of one
// digit in the order they came in.  Up to kFifoSums levels fifo_hist_kernel has
// counted the blocks' digits and one pass lists them; deeper searches take a pass
// per 8 bits of the level, lowest first, with fifo_digits_kernel and
// fifo_scan_kernel before each.
__device__ __forceinline__ int list_digit(const int32_t *__restrict__ in,
                                          const int32_t *__restrict__ levels, int shift, int64_t i,
                                          int64_t end, int32_t &v) {
  v = i < end ? (in ? __ldg(in + i) : (int32_t)i) : -1;
  const int L = v >= 0 ? __ldg(levels + v) : -1;
  return L < 0 ? -1 : (L >> shift) & (kListDigits - 1);
}

__global__ void __launch_bounds__(kFifoBlock) fifo_digits_kernel(
    int64_t count, int64_t run, const int32_t *__restrict__ in,
    const int32_t *__restrict__ levels, int shift, unsigned *__restrict__ block_counts) {
  __shared__ unsigned s[kListDigits];
  s[threadIdx.x] = 0;
  __syncthreads();
  const int64_t end = min(count, (blockIdx.x + 1) * run);
  const int lane = lane_id();
  for (int64_t base = blockIdx.x * run + (threadIdx.x & ~31u); base < end; base += kFifoBlock) {
    int32_t v;
    const int d = list_digit(in, levels, shift, base + lane, end, v);
    const unsigned peers = __match_any_sync(kAll, d);
    if (d >= 0 && lane == __ffs(peers) - 1) atomicAdd(&s[d], (unsigned)__popc(peers));
  }
  __syncthreads();
  block_counts[threadIdx.x * gridDim.x + blockIdx.x] = s[threadIdx.x];
}

// Each digit's counts become the items of that digit in the blocks before; totals:
// in all of them.  A warp per digit.
__global__ void __launch_bounds__(kFifoBlock) fifo_scan_kernel(unsigned blocks, int digits,
                                                               unsigned *block_counts,
                                                               unsigned *__restrict__ totals) {
  const int lane = lane_id(), d = (int)warp_id_global();
  if (d >= digits) return;
  unsigned *row = block_counts + d * blocks, carry = 0;
  for (unsigned b0 = 0; b0 < blocks; b0 += 32) {
    const unsigned b = b0 + lane, mine = b < blocks ? row[b] : 0u;
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned x = __shfl_up_sync(kAll, incl, o);
      if (lane >= o) incl += x;
    }
    if (b < blocks) row[b] = carry + incl - mine;
    carry += __shfl_sync(kAll, incl, 31);
  }
  if (lane == 0) totals[d] = carry;
}

// A warp has a run of items of its own: it counts their digits, learns where each
// digit's items of this block begin (after those of lower digits, and of the same
// digit in the blocks before: totals and block_counts after fifo_scan_kernel, or, for
// few digits, `totals` null, each block sums the counts for itself), and goes through
// its items again.  digits: that occur, at most.  Bound by its chain of dependent
// steps and the scattered stores: R-MAT scale 20 (1 M vertices, 8 levels) 12 us, where
// a radix sort of (level, id) pairs took 27; 93,000 vertices on 1,552 levels, two
// passes of three kernels, 27 us for 30.
__global__ void __launch_bounds__(kFifoBlock) fifo_list_kernel(
    int64_t count, int64_t run, const int32_t *__restrict__ in,
    const int32_t *__restrict__ levels, int shift, int digits,
    const unsigned *__restrict__ block_counts, const unsigned *__restrict__ totals,
    int32_t *__restrict__ out) {
  constexpr int kWarps = kFifoBlock / 32;
  __shared__ unsigned s_at[kWarps][kListDigits];
  __shared__ unsigned s_all[kListDigits], s_before[kListDigits], s_warp[kWarps];
  const int lane = lane_id(), wib = threadIdx.x >> 5, t = threadIdx.x;
  for (int d = lane; d < digits; d += 32) s_at[wib][d] = 0;
  __syncwarp();
  const int64_t first = blockIdx.x * run + wib * (run / kWarps);
  const int64_t end = min(count, first + run / kWarps);
  for (int64_t base = first; base < end; base += 32) {
    int32_t v;
    const int d = list_digit(in, levels, shift, base + lane, end, v);
    const unsigned peers = __match_any_sync(kAll, d);
    if (d >= 0 && lane == __ffs(peers) - 1) s_at[wib][d] += (unsigned)__popc(peers);
    __syncwarp();
  }
  if (totals) {
    if (t < digits) {
      s_all[t] = __ldg(totals + t);
      s_before[t] = __ldg(block_counts + t * gridDim.x + blockIdx.x);
    }
  } else {
    for (int d = wib; d < digits; d += kWarps) {
      unsigned all = 0, before = 0;
      for (unsigned b0 = lane; b0 < gridDim.x; b0 += 128) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {  // in flight at once
          const unsigned b = b0 + 32 * h;
          const unsigned x = b < gridDim.x ? __ldg(block_counts + d * gridDim.x + b) : 0u;
          all += x;
          before += b < blockIdx.x ? x : 0u;
        }
      }
      all = __reduce_add_sync(kAll, all);
      before = __reduce_add_sync(kAll, before);
      if (lane == 0) {
        s_all[d] = all;
        s_before[d] = before;
      }
    }
  }
  __syncthreads();
  {  // a thread per digit: its first place, and each warp's
    const unsigned mine = t < digits ? s_all[t] : 0u;
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned x = __shfl_up_sync(kAll, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) s_warp[wib] = incl;
    __syncthreads();
    unsigned at = incl - mine;
    for (int w = 0; w < wib; ++w) at += s_warp[w];
    if (t < digits) {
      at += s_before[t];
      for (int w = 0; w < kWarps; ++w) {
        const unsigned x = s_at[w][t];
        s_at[w][t] = at;
        at += x;
      }
    }
  }
  __syncthreads();
  for (int64_t base = first; base < end; base += 32) {
    int32_t v;
    const int d = list_digit(in, levels, shift, base + lane, end, v);
    const unsigned peers = __match_any_sync(kAll, d);
    const int leader = __ffs(peers) - 1;
    unsigned at = 0;
    if (d >= 0 && lane == leader) {
      at = s_at[wib][d];
      s_at[wib][d] = at + (unsigned)__popc(peers);
    }
    at = __shfl_sync(kAll, at, leader);
    if (d >= 0) out[at + __popc(peers & ((1u << lane) - 1u))] = v;
    __syncwarp();
  }
}

// The rank map of level L (rk is ~0 elsewhere).
__global__ void fifo_ranks_kernel(const int32_t *__restrict__ queue, unsigned count,
                                  uint32_t *rk) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    rk[queue[i]] = i;
}

__device__ __forceinline__ void fifo_list_long(bool is_long, int32_t v, uint32_t rank, int64_t deg,
                                               FifoLong *longs, unsigned long long *nlong) {
  if (!is_long) return;
  const unsigned chunks = (unsigned)((deg + kFifoChunk - 1) / kFifoChunk);
  const unsigned long long old = atomicAdd(nlong, (1ull << 32) | chunks);
  longs[old >> 32] = FifoLong{(uint32_t)old, v, rank};
}

// Pull: level L+1's vertices (seg) take the smallest rank over their in-lists.
// A warp has 32 of them: short lists by a lane each (four entries' ranks in
// flight), longer ones by the warp (128 entries in flight), the longest listed.
__global__ void __launch_bounds__(kFifoBlock) fifo_pull_kernel(
    const int64_t *__restrict__ in_off, const int32_t *__restrict__ in_idx,
    const uint32_t *__restrict__ rk, const int32_t *__restrict__ seg, unsigned count,
    uint32_t *__restrict__ best, FifoLong *longs, unsigned long long *nlong) {
  const int lane = lane_id();
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = (int64_t)warp_id_global() * 32; base < count; base += nwarps * 32) {
    int32_t v = 0;
    int64_t b = 0, e = 0;
    if (base + lane < count) {
      v = seg[base + lane];
      b = __ldg(in_off + v);
      e = __ldg(in_off + v + 1);
    }
    const int64_t deg = e - b;
    uint32_t low = kNoRank;
    if (deg <= kFifoLane) {
      for (int64_t j = b; j < e; j += 4) {
        int32_t u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) u[q] = j + q < e ? __ldg(in_idx + j + q) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (u[q] >= 0) low = min(low, __ldg(rk + u[q]));
      }
    }
    unsigned todo = __ballot_sync(kAll, deg > kFifoLane && deg <= kFifoWarp);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const int64_t sb = __shfl_sync(kAll, b, src), se = __shfl_sync(kAll, e, src);
      uint32_t x = kNoRank;
      for (int64_t j = sb + lane; j < se; j += 128) {
        int32_t u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) u[q] = j + 32 * q < se ? __ldg(in_idx + j + 32 * q) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (u[q] >= 0) x = min(x, __ldg(rk + u[q]));
      }
      x = __reduce_min_sync(kAll, x);
      if (lane == src) low = x;
    }
    if (base + lane < count && deg <= kFifoWarp) best[v] = low;
    fifo_list_long(deg > kFifoWarp, v, 0u, deg, longs, nlong);
  }
}

__device__ __forceinline__ void fifo_offer(const int32_t *__restrict__ levels, int32_t v, int L,
                                           uint32_t rank, uint32_t *best) {
  // a read first: a hub's rank is low, and most targets have it already
  if (__ldg(levels + v) == L + 1 && __ldcg(best + v) > rank) atomicMin(best + v, rank);
}

// Push: level L's vertices offer their rank to their level-(L+1)
// out-neighbours.  A warp spreads the edges of 32 vertices over its lanes, of
// fewer when there are not 32 for every warp, four edges a lane in flight (110
// hubs' neighbours at R-MAT scale 20: 339 us on 4 warps, 24 us on 110); the
// longest lists go on the list.
__global__ void __launch_bounds__(kFifoBlock) fifo_push_kernel(
    const int64_t *__restrict__ out_off, const int32_t *__restrict__ out_idx,
    const int32_t *__restrict__ levels, const int32_t *__restrict__ queue, unsigned count, int L,
    uint32_t *best, FifoLong *longs, unsigned long long *nlong) {
  __shared__ uint32_t s_first[kFifoBlock / 32][32];
  __shared__ int64_t s_start[kFifoBlock / 32][32];
  const int lane = lane_id();
  uint32_t *first = s_first[threadIdx.x >> 5];
  int64_t *start = s_start[threadIdx.x >> 5];
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int group = 1;
  while (group < 32 && (int64_t)count > group * nwarps) group <<= 1;
  for (int64_t base = (int64_t)warp_id_global() * group; base < count; base += nwarps * group) {
    int64_t b = 0, deg = 0;
    int32_t u = 0;
    if (lane < group && base + lane < count) {
      u = queue[base + lane];
      b = __ldg(out_off + u);
      deg = __ldg(out_off + u + 1) - b;
    }
    fifo_list_long(deg > kFifoWarp, u, (uint32_t)(base + lane), deg, longs, nlong);
    const uint32_t d = deg > kFifoWarp ? 0u : (uint32_t)deg;
    uint32_t incl = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kAll, incl, o);
      if (lane >= o) incl += t;
    }
    const uint32_t total = __shfl_sync(kAll, incl, 31);
    first[lane] = incl - d;
    start[lane] = b;
    __syncwarp();
    for (uint32_t t0 = lane; t0 < total; t0 += 128) {
      int lo[4];
      int32_t v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t t = t0 + 32 * q;
        lo[q] = 0;  // the last of the 32 whose prefix is <= t
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (first[lo[q] + step] <= t) lo[q] += step;
        v[q] = t < total ? __ldg(out_idx + start[lo[q]] + (t - first[lo[q]])) : -1;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (v[q] >= 0) fifo_offer(levels, v[q], L, (uint32_t)(base + lo[q]), best);
    }
    __syncwarp();
  }
}

// The listed long lists, a warp per chunk.
template <bool Push>
__global__ void __launch_bounds__(kFifoBlock) fifo_long_kernel(
    const int64_t *__restrict__ off, const int32_t *__restrict__ idx,
    const int32_t *__restrict__ levels, const uint32_t *__restrict__ rk, int L, uint32_t *best,
    const FifoLong *__restrict__ longs, const unsigned long long *nlong) {
  const unsigned long long all = *nlong;
  const unsigned lists = (unsigned)(all >> 32), chunks = (unsigned)all;
  const int lane = lane_id();
  const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
  for (unsigned c = (unsigned)warp_id_global(); c < chunks; c += nwarps) {
    unsigned lo = 0, hi = lists - 1;
    while (lo < hi) {
      const unsigned mid = (lo + hi + 1) >> 1;
      if (longs[mid].base <= c)
        lo = mid;
      else
        hi = mid - 1;
    }
    const FifoLong x = longs[lo];
    const int64_t b = __ldg(off + x.v) + (int64_t)(c - x.base) * kFifoChunk;
    const int64_t e = min(b + kFifoChunk, __ldg(off + x.v + 1));
    uint32_t low = kNoRank;
    for (int64_t j = b + lane; j < e; j += 128) {
      int32_t u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) u[q] = j + 32 * q < e ? __ldg(idx + j + 32 * q) : -1;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (u[q] >= 0) {
          if (Push)
            fifo_offer(levels, u[q], L, x.rank, best);
          else
            low = min(low, __ldg(rk + u[q]));
        }
    }
    if (!Push) {
      low = __reduce_min_sync(kAll, low);
      if (lane == 0 && low != kNoRank) atomicMin(best + x.v, low);
    }
  }
}

// Level L+1 (seg) takes its parents; the sort's keys (parent ranks) and values.
// `clear`: rk's entries of level L go back to ~0.
__global__ void fifo_finish_kernel(const int32_t *__restrict__ seg, unsigned count,
                                   const uint32_t *__restrict__ best,
                                   const int32_t *__restrict__ queue, unsigned parents_count,
                                   int clear, uint32_t *rk, uint32_t *__restrict__ keys,
                                   int32_t *__restrict__ vals, int32_t *__restrict__ parents,
                                   unsigned long long *nlong) {
  const unsigned t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  if (t0 == 0) *nlong = 0;
  for (unsigned i = t0; i < count; i += step) {
    const int32_t v = seg[i];
    const uint32_t r = best[v];
    parents[v] = r == kNoRank ? -1 : queue[r];
    keys[i] = r;
    vals[i] = v;
  }
  if (clear)
    for (unsigned i = t0; i < parents_count; i += step) rk[queue[i]] = kNoRank;
}

// Into and out of a run of small levels: level L's ranks from its queue, and
// its queue from its ranks (seg: its vertices).
__global__ void fifo_enter_kernel(const int32_t *__restrict__ queue, unsigned count, int level,
                                  int32_t *rank, unsigned long long *lr) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += gridDim.x * blockDim.x) {
    rank[queue[i]] = (int32_t)i;
    lr[queue[i]] = ((unsigned long long)level << 32) | i;
  }
}
__global__ void fifo_leave_kernel(const int32_t *__restrict__ seg, unsigned count,
                                  const int32_t *__restrict__ rank, int32_t *queue) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    queue[rank[seg[i]]] = seg[i];
}

// Runs of levels of at most kSmallLevel vertices and kSmallEdges list entries
// (counted for the first kFifoSums levels only; the vertices bound those behind)
// are handled by one block, many levels to a launch, with no sort: level L+1's queue is level L's queue in
// order with each vertex's children (the out-neighbours whose FIFO parent it
// is) appended in out-list order, which is ascending -- the same order the
// sort of (parent rank, id) gives.  Per level: (1) every child picks its
// parent, the level-L in-neighbour of smallest rank (one 8-byte load of
// (level, rank) per in-list entry), records (level + 1, parent) for the
// parent's scan and counts itself in its parent's shared-memory counter;
// (2) a block scan of the counts in rank order gives each parent its first
// child's rank; (3) every parent with children walks its out-list handing
// out ranks to the entries recorded as its children.  Long lists go to a
// warp.  One SM's load pipeline bounds this, so each list entry costs one
// load.  On deep graphs launches would otherwise dominate (a 4096 x 4096 grid
// has ~8000 levels).
constexpr int kSmallThreads = 1024;
constexpr int kSmallPer = 8;                                // counts a thread scans
constexpr int kSmallLevel = kSmallThreads * kSmallPer;     // vertices per level, at most
constexpr uint64_t kSmallEdges = 1 << 15;  // out-edges of level L, in-edges of level L + 1
constexpr int kSmallRun = 3;    // levels worth a run: it sets up 16 bytes a vertex
constexpr int kHeavyList = 64;  // list length above which a warp scans
using SmallScan = cub::BlockScan<unsigned, kSmallThreads>;
struct SmallSmem {
  int32_t queue[2][kSmallLevel];     // levels L and L+1 in queue (rank) order
  unsigned cnt[kSmallLevel + 1];     // children per parent rank, then first ranks
  int32_t heavy[kSmallLevel];        // positions whose lists a warp scans
  unsigned nheavy;
  typename SmallScan::TempStorage scan;
};

__device__ __forceinline__ unsigned long long warp_min64(unsigned long long x) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, x, d);
    x = o < x ? o : x;
  }
  return x;
}

// Over in-list entries [s, e) (lanes lane, lane + step, ...), the smallest
// (rank << 32) | u of a level-L in-neighbour u; lr is written by this block at
// earlier levels, so it is read with ordinary loads, never the read-only path.
__device__ __forceinline__ unsigned long long fifo_best(const int32_t *__restrict__ in_idx,
                                                        const unsigned long long *lr, int64_t s,
                                                        int64_t e, int L, int lane, int step) {
  unsigned long long best = ~0ull;
  for (int64_t j = s + lane; j < e; j += step) {
    const int32_t u = __ldg(in_idx + j);
    const unsigned long long x = lr[u];
    if ((unsigned)(x >> 32) == (unsigned)L) {
      const unsigned long long k = ((x & 0xffffffffull) << 32) | (uint32_t)u;
      best = k < best ? k : best;
    }
  }
  return best;
}

// Level L+1 vertex w takes parent u (rank r among level L).
__device__ __forceinline__ void fifo_adopt(int32_t w, unsigned long long best, int L,
                                           int32_t *parents, unsigned long long *pl,
                                           unsigned *cnt) {
  if (best == ~0ull) return;  // no level-L in-neighbour: not a level-(L+1) vertex
  const int32_t u = (int32_t)(uint32_t)best;
  parents[w] = u;
  pl[w] = ((unsigned long long)(L + 1) << 32) | (uint32_t)u;
  atomicAdd(&cnt[best >> 32], 1u);
}

// One block: levels L0 .. L1-1 in turn; for each, level L has counts[L] and
// level L+1 counts[L+1] vertices, both at most kSmallLevel; order[offs[L+1] ..]
// lists level L+1 in no particular order.
__global__ void __launch_bounds__(kSmallThreads) fifo_small_levels_kernel(
    const int64_t *__restrict__ in_off, const int32_t *__restrict__ in_idx,
    const int64_t *__restrict__ out_off, const int32_t *__restrict__ out_idx, int32_t *rank,
    unsigned long long *lr, unsigned long long *pl, const int32_t *__restrict__ order,
    const unsigned *__restrict__ counts, const unsigned *__restrict__ offs, int L0, int L1,
    int32_t root, int32_t *parents) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  SmallSmem &S = *reinterpret_cast<SmallSmem *>(s_raw);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  constexpr int kWarps = kSmallThreads / 32;
  int cur = 0;
  // level L0 in queue order, from the ranks already assigned
  if (L0 == 0) {
    if (t == 0) S.queue[0][0] = root;
  } else {
    for (unsigned i = t; i < counts[L0]; i += kSmallThreads) {
      const int32_t u = order[offs[L0] + i];
      S.queue[0][rank[u]] = u;
    }
  }
  for (int L = L0; L < L1; ++L) {
    const unsigned c = counts[L + 1], p = counts[L];
    const unsigned base = offs[L + 1];
    int32_t *qL = S.queue[cur];
    int32_t *qN = S.queue[cur ^ 1];
    for (unsigned r = t; r < p; r += kSmallThreads) S.cnt[r] = 0;
    if (t == 0) S.nheavy = 0;
    __syncthreads();
    // (1) parents of level L+1
    for (unsigned pos = t; pos < c; pos += kSmallThreads) {
      const int32_t w = order[base + pos];
      const int64_t s = __ldg(in_off + w), e = __ldg(in_off + w + 1);
      if (e - s > kHeavyList)
        S.heavy[atomicAdd(&S.nheavy, 1u)] = w;
      else
        fifo_adopt(w, fifo_best(in_idx, lr, s, e, L, 0, 1), L, parents, pl, S.cnt);
    }
    __syncthreads();
    for (unsigned h = warp; h < S.nheavy; h += kWarps) {
      const int32_t w = S.heavy[h];
      const unsigned long long best =
          warp_min64(fifo_best(in_idx, lr, __ldg(in_off + w), __ldg(in_off + w + 1), L, lane, 32));
      if (lane == 0) fifo_adopt(w, best, L, parents, pl, S.cnt);
    }
    __syncthreads();  // every warp is done with the list before it is reset
    // (2) first rank of each parent's children: exclusive scan in rank order
    {
      unsigned v[kSmallPer], sum = 0;
#pragma unroll
      for (int i = 0; i < kSmallPer; ++i) {
        const unsigned r = t * kSmallPer + i;
        v[i] = r < p ? S.cnt[r] : 0u;
        sum += v[i];
      }
      unsigned before = 0;
      SmallScan(S.scan).ExclusiveSum(sum, before);
      __syncthreads();
#pragma unroll
      for (int i = 0; i < kSmallPer; ++i) {
        const unsigned r = t * kSmallPer + i;
        if (r < p) S.cnt[r] = before;
        before += v[i];
      }
      if (t == 0) {
        S.cnt[p] = c;
        S.nheavy = 0;
      }
    }
    __syncthreads();
    // (3) ranks of level L+1: parents with children walk their out-lists
    const unsigned long long tag = (unsigned long long)(L + 1) << 32;
    for (unsigned r = t; r < p; r += kSmallThreads) {
      unsigned at = S.cnt[r];
      const unsigned end = S.cnt[r + 1];
      if (at == end) continue;
      const int32_t u = qL[r];
      const int64_t s = __ldg(out_off + u), e = __ldg(out_off + u + 1);
      if (e - s > kHeavyList) {
        S.heavy[atomicAdd(&S.nheavy, 1u)] = (int32_t)r;
        continue;
      }
      const unsigned long long mine = tag | (uint32_t)u;
      for (int64_t j = s; j < e && at < end; ++j) {
        const int32_t w = __ldg(out_idx + j);
        if (pl[w] == mine) {
          rank[w] = (int32_t)at;
          lr[w] = tag | at;
          qN[at++] = w;
        }
      }
    }
    __syncthreads();
    for (unsigned h = warp; h < S.nheavy; h += kWarps) {
      const unsigned r = (unsigned)S.heavy[h];
      const int32_t u = qL[r];
      const unsigned long long mine = tag | (uint32_t)u;
      const int64_t s = __ldg(out_off + u), e = __ldg(out_off + u + 1);
      unsigned at = S.cnt[r];
      for (int64_t j0 = s; j0 < e; j0 += 32) {
        const int64_t j = j0 + lane;
        int32_t w = 0;
        bool child = false;
        if (j < e) {
          w = __ldg(out_idx + j);
          child = pl[w] == mine;
        }
        const unsigned m = __ballot_sync(0xffffffffu, child);
        if (child) {
          const unsigned k = at + __popc(m & ((1u << lane) - 1u));
          rank[w] = (int32_t)k;
          lr[w] = tag | k;
          qN[k] = w;
        }
        at += __popc(m);
      }
    }
    __syncthreads();
    cur ^= 1;
  }
}

// Bits needed for the values 0 .. x (at least 1).
int bits_for(uint64_t x) {
  int b = 1;
  while (b < 64 && (x >> b)) ++b;
  return b;
}

unsigned grid_for(int64_t items, int per_block, int sms) {
  int64_t b = (items + per_block - 1) / per_block;
  const int64_t cap = (int64_t)sms * 16;
  if (b > cap) b = cap;
  return (unsigned)(b > 0 ? b : 1);
}

int fifo_state(cg_graph *g, FifoState **out) {
  if (g->fifo) {
    *out = g->fifo;
    return CG_OK;
  }
  FifoState *f = new (std::nothrow) FifoState();
  if (!f) return CG_ERR_OUT_OF_MEMORY;
  f->n = g->n;
  const size_t n = (size_t)g->n;
  {
    cub::DoubleBuffer<uint32_t> k(nullptr, nullptr);
    cub::DoubleBuffer<int32_t> v(nullptr, nullptr);
    cub::DeviceRadixSort::SortPairs(nullptr, f->temp_bytes, k, v, (int64_t)n, 0, 32, g->stream);
  }
  const size_t nlongs = (size_t)(g->nnz / (kFifoWarp + 1) + 1);
  size_t bytes = 0;
  auto piece = [&](size_t size) {
    const size_t at = bytes;
    bytes = (bytes + size + 255) & ~(size_t)255;
    return at;
  };
  // (what a call clears together lies together: sums, nlong and counts; lr and
  // pl; rk and best)
  const size_t at_sums = piece(sizeof(FifoSums)), at_nlong = piece(sizeof(unsigned long long)),
               at_counts = piece(sizeof(unsigned) * (n + 1)),
               at_longs = piece(sizeof(FifoLong) * nlongs), at_temp = piece(f->temp_bytes),
               at_offs = piece(sizeof(unsigned) * (n + 2)), at_lr = piece(8 * n),
               at_pl = piece(8 * n),
               at_blocks = piece(sizeof(unsigned) * kListDigits *
                                 (list_blocks((int64_t)n, list_run((int64_t)n, g->num_sms)) + 1));
  size_t at4[9];  // 4 bytes a vertex each
  for (size_t &x : at4) x = piece(4 * n);
  if (cudaMalloc(&f->base, bytes) != cudaSuccess ||
      cudaFuncSetAttribute(fifo_small_levels_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(SmallSmem)) != cudaSuccess) {
    cudaGetLastError();
    fifo_free(f);
    return CG_ERR_OUT_OF_MEMORY;
  }
  f->sums = reinterpret_cast<FifoSums *>(f->base + at_sums);
  f->nlong = reinterpret_cast<unsigned long long *>(f->base + at_nlong);
  f->longs = reinterpret_cast<FifoLong *>(f->base + at_longs);
  f->temp = f->base + at_temp;
  f->counts = reinterpret_cast<unsigned *>(f->base + at_counts);
  f->block_counts = reinterpret_cast<unsigned *>(f->base + at_blocks);
  f->offs = reinterpret_cast<unsigned *>(f->base + at_offs);
  f->lr = reinterpret_cast<unsigned long long *>(f->base + at_lr);
  f->pl = reinterpret_cast<unsigned long long *>(f->base + at_pl);
  f->order = reinterpret_cast<int32_t *>(f->base + at4[0]);
  f->rk = reinterpret_cast<uint32_t *>(f->base + at4[1]);
  f->best = reinterpret_cast<uint32_t *>(f->base + at4[2]);
  f->rank = reinterpret_cast<int32_t *>(f->base + at4[3]);
  for (int i = 0; i < 2; ++i) f->key[i] = reinterpret_cast<uint32_t *>(f->base + at4[4 + i]);
  for (int i = 0; i < 3; ++i) f->queue[i] = reinterpret_cast<int32_t *>(f->base + at4[6 + i]);
  g->device_bytes += (int64_t)bytes;
  g->fifo = f;
  *out = f;
  return CG_OK;
}

}  // namespace

void fifo_free(FifoState *f) {
  if (!f) return;
  cudaFree(f->base);
  delete f;
}

int fifo_parents(cg_graph *g, int64_t root, const int32_t *d_levels, int32_t *d_parents) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CG_CUDA(cudaStreamIsCapturing(g->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) {
    set_error_text("the FIFO parent rule synchronises with the stream: not capturable");
    return CG_ERR_NOT_SUPPORTED;
  }
  FifoState *f = nullptr;
  int rc = fifo_state(g, &f);
  if (rc) return rc;
  const int64_t n = g->n;
  const int sms = g->num_sms;
  cudaStream_t st = g->stream;
  auto fill = [&](void *first, void *last, size_t last_bytes, int value) {
    return cudaMemsetAsync(first, value,
                           (size_t)(static_cast<unsigned char *>(last) -
                                    static_cast<unsigned char *>(first)) + last_bytes, st);
  };
  CG_CUDA(fill(f->sums, f->counts, sizeof(unsigned) * (size_t)(n + 1), 0));
  const int64_t run = list_run(n, sms);
  fifo_hist_kernel<<<list_blocks(n, run), kFifoBlock, 0, st>>>(
      n, run, d_levels, g->in_off, g->out_off, f->counts, f->block_counts, f->sums);
  CG_CUDA(cudaGetLastError());
  FifoSums sums;
  CG_CUDA(cudaMemcpyAsync(&sums, f->sums, sizeof(sums), cudaMemcpyDeviceToHost, st));
  CG_CUDA(cudaStreamSynchronize(st));
  const int maxlevel = sums.maxlevel;
  if (maxlevel <= 0) return CG_OK;  // only the root: its parent is itself already
  std::vector<unsigned> counts(sums.counts, sums.counts + kFifoSums);
  counts.resize((size_t)maxlevel + 1);
  if (maxlevel >= kFifoSums) {
    CG_CUDA(cudaMemcpyAsync(counts.data(), f->counts, sizeof(unsigned) * counts.size(),
                            cudaMemcpyDeviceToHost, st));
    CG_CUDA(cudaStreamSynchronize(st));
  }
  std::vector<unsigned> offs((size_t)maxlevel + 2, 0u);
  for (int L = 0; L <= maxlevel; ++L) offs[(size_t)L + 1] = offs[(size_t)L] + counts[(size_t)L];
  // the reached vertices by level, in id order within one
  if (maxlevel < kFifoSums) {
    fifo_list_kernel<<<list_blocks(n, run), kFifoBlock, 0, st>>>(
        n, run, nullptr, d_levels, 0, maxlevel + 1, f->block_counts, nullptr, f->order);
  } else {
    const int passes = (bits_for((uint64_t)maxlevel) + 7) / 8;
    const int32_t *in = nullptr;
    for (int q = 0; q < passes; ++q) {
      const int64_t items = q ? (int64_t)offs.back() : n;
      const unsigned blocks = list_blocks(items, run);
      const int top = maxlevel >> (8 * q), digits = top < kListDigits ? top + 1 : kListDigits;
      unsigned *totals = f->block_counts + (size_t)kListDigits * blocks;
      int32_t *out = (passes - q) & 1 ? f->order : f->queue[0];
      fifo_digits_kernel<<<blocks, kFifoBlock, 0, st>>>(items, run, in, d_levels, 8 * q,
                                                        f->block_counts);
      fifo_scan_kernel<<<(digits + 7) / 8, kFifoBlock, 0, st>>>(blocks, digits, f->block_counts,
                                                                totals);
      fifo_list_kernel<<<blocks, kFifoBlock, 0, st>>>(items, run, in, d_levels, 8 * q, digits,
                                                      f->block_counts, totals, out);
      in = out;
    }
  }
  CG_CUDA(cudaGetLastError());
  CG_CUDA(fill(f->rk, f->best, sizeof(uint32_t) * (size_t)n, 0xff));
  auto small = [&](int L) {  // level L to L + 1 suits a run of small levels
    return counts[(size_t)L] <= (unsigned)kSmallLevel &&
           counts[(size_t)L + 1] <= (unsigned)kSmallLevel && counts[(size_t)L + 1] > 0 &&
           (L + 1 >= kFifoSums || (sums.out[L] <= kSmallEdges && sums.in[L + 1] <= kSmallEdges));
  };
  bool small_ready = false;
  const int32_t *queue = f->order;  // level L in queue order: level 0 is the root alone
  int at = 0;                       // f->queue[at], at + 1, at + 2 (mod 3): queue, free, free
  for (int L = 0; L < maxlevel; ++L) {
    const unsigned c = counts[(size_t)L + 1], p = counts[(size_t)L];
    if (c == 0) break;
    const int32_t *seg = f->order + offs[(size_t)L + 1];
    int L1 = L;
    while (L1 < maxlevel && small(L1)) ++L1;
    if (L1 - L >= kSmallRun) {
      // levels L .. L1 in one launch of one block
      if (!small_ready) {
        CG_CUDA(fill(f->lr, f->pl, sizeof(unsigned long long) * (size_t)n, 0xff));
        CG_CUDA(cudaMemcpyAsync(f->offs, offs.data(), sizeof(unsigned) * offs.size(),
                                cudaMemcpyHostToDevice, st));
        small_ready = true;
      }
      fifo_enter_kernel<<<grid_for(p, kFifoBlock, sms), kFifoBlock, 0, st>>>(queue, p, L, f->rank,
                                                                             f->lr);
      fifo_small_levels_kernel<<<1, kSmallThreads, sizeof(SmallSmem), st>>>(
          g->in_off, g->in_idx, g->out_off, g->out_idx, f->rank, f->lr, f->pl, f->order,
          f->counts, f->offs, L, L1, (int32_t)root, d_parents);
      CG_CUDA(cudaGetLastError());
      if (L1 < maxlevel) {
        int32_t *next = f->queue[(at + 1) % 3];
        const unsigned c1 = counts[(size_t)L1];
        fifo_leave_kernel<<<grid_for(c1, kFifoBlock, sms), kFifoBlock, 0, st>>>(
            f->order + offs[(size_t)L1], c1, f->rank, next);
        queue = next;
        at = (at + 1) % 3;
      }
      L = L1 - 1;
      continue;
    }
    if (p == 1) {
      // one possible parent, the search's own; queue order is id order
      queue = seg;
      continue;
    }
    // atomics count double
    const bool push = L + 1 < kFifoSums && 2 * sums.out[L] < sums.in[L + 1];
    if (push) {
      fifo_push_kernel<<<grid_for((int64_t)p * 32, kFifoBlock, sms), kFifoBlock, 0, st>>>(
          g->out_off, g->out_idx, d_levels, queue, p, L, f->best, f->longs, f->nlong);
      fifo_long_kernel<true><<<sms * 8, kFifoBlock, 0, st>>>(g->out_off, g->out_idx, d_levels,
                                                             f->rk, L, f->best, f->longs, f->nlong);
    } else {
      fifo_ranks_kernel<<<grid_for(p, kFifoBlock, sms), kFifoBlock, 0, st>>>(queue, p, f->rk);
      fifo_pull_kernel<<<grid_for(c, kFifoBlock, sms), kFifoBlock, 0, st>>>(
          g->in_off, g->in_idx, f->rk, seg, c, f->best, f->longs, f->nlong);
      fifo_long_kernel<false><<<sms * 8, kFifoBlock, 0, st>>>(g->in_off, g->in_idx, d_levels, f->rk,
                                                              L, f->best, f->longs, f->nlong);
    }
    int32_t *vals[2] = {f->queue[(at + 1) % 3], f->queue[(at + 2) % 3]};
    fifo_finish_kernel<<<grid_for(c > p ? c : p, kFifoBlock, sms), kFifoBlock, 0, st>>>(
        seg, c, f->best, queue, p, push ? 0 : 1, f->rk, f->key[0], vals[0], d_parents, f->nlong);
    CG_CUDA(cudaGetLastError());
    if (L + 1 == maxlevel) break;  // the last level's order is not needed
    cub::DoubleBuffer<uint32_t> kb(f->key[0], f->key[1]);
    cub::DoubleBuffer<int32_t> vb(vals[0], vals[1]);
    size_t tb = f->temp_bytes;
    CG_CUDA(cub::DeviceRadixSort::SortPairs(f->temp, tb, kb, vb, (int64_t)c, 0, bits_for(p - 1),
                                            st));
    queue = vb.Current();
    at = vb.Current() == vals[0] ? (at + 1) % 3 : (at + 2) % 3;
  }
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

}  // namespace cg
