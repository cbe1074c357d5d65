// Per-root direction-optimizing BFS: one persistent cooperative kernel that
// runs every round of a search on the device, with one grid-wide wait per round.
//
// Reference mapping (bfs/implementation/src/bool_pe.csl):
//   start_spmv (:673-729)          -> phase 0 of bfs_persistent (state reset, seed)
//   compute_topdown (:865-887)     -> push_round_*: frontier queue (or bitmap),
//                                     out-lists, atomicOr into the next frontier
//   compute_bottomup (:899-921)    -> pull_round: unvisited vertices scan their
//                                     ascending in-lists, stop at the first
//                                     frontier source
//   reduce_or + reduce_done        -> the shared bitmaps make the OR-reduce
//     (:923-1004, collectives_2d     implicit; the visited set is vis | F_L, and
//      pe.csl:319-349)                 vis |= F_L is folded into round L's work;
//                                     per-round counters give nf = popcount
//   termination relay (:1003-1046)  -> every block reads nf from the round
//                                     record after the grid-wide wait; nf == 0 ends
//   direction switch (:1078-1088)   -> next_direction(): Beamer's alpha/beta rule,
//                                     or the reference's one-way tau rule
//   reduce_select_any (:1145-1154)  -> not needed: every parent is final when it
//                                     is written (lowest-index rule below)
//
// Parent rule: the lowest-numbered in-neighbour one level closer
// (bfs/README.md:208-224).  A push round applies atomicMin over every
// frontier source of a newly reached vertex (the visited set is frozen during
// the round, so all of them are seen); a pull round takes the first frontier
// source of an ascending in-list, which is the minimum.  Parents start at
// 0xFFFFFFFF, the reference's PARENT_NONE (device_io.py:157), which reads back
// as -1 through int32 without a conversion pass.
//
// Bitmaps: vis holds the vertices of F_0 .. F_{L-1}, the frontier F_L is
// fr[L % 3], the next frontier is written into fr[(L+1) % 3] and fr[(L+2) % 3]
// (F_{L-1}) is cleared during round L.  "Visited" is tested as vis | F_L, so
// merging F_L into vis during round L races with nothing.
#include <cuda_runtime.h>

#include <type_traits>

#include "cg_internal.cuh"

namespace cg {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kPush = 0, kPull = 1;
constexpr int kBfsBlock = 512;
// Pull rounds: in-list entries a thread loads at once (all in flight before
// any is tested), and how many entries of its vertex's list a thread scans
// before the whole warp takes over the rest of it.
constexpr int kPullThreadScan = 4;
constexpr unsigned kPullLaneMax = 32;
constexpr int kBfsWarps = kBfsBlock / 32;
// Per-warp shared memory of the bitmap-wide rounds: a staged tile (its words
// and the exclusive prefix of their popcounts, so that a lane can select the
// k-th set bit) and the tile's next-frontier words found by a pull round.
struct __align__(16) WarpTile {  // 16-byte vector accesses to every member
  uint32_t m[kTileWords];
  uint32_t pre[kTileWords];
  uint32_t found[kTileWords];
};
static_assert(sizeof(WarpTile) % 16 == 0 && kTileWords % 4 == 0, "16-byte tile rows");
// Per-warp shared memory of a push round (a pull round keeps the vertices whose
// first in-neighbour was no parent here): the edge spreading of gather_expand
// (a resident graph's list starts and prefix counts fit 32 bits, its nnz being
// below 2^32; larger ones: s_start_high), and the
// light vertices claimed and not queued yet.  Big ones wait in the tile's
// `found` words, which push rounds do not use.
struct WarpExpand {
  int32_t u[32];
  uint32_t s[32];
  uint32_t x[32];
  int32_t light[64];
};
struct BigClaims {
  int32_t v[64];
  uint32_t deg[64];
};
static_assert(sizeof(BigClaims) == sizeof(uint32_t) * kTileWords, "fits WarpTile::found");

// Graphs of 2^32 - 2^16 list entries and more (kWide: only a caller's own arrays
// can be so large, cg_bfs_noalloc): list starts take 64 bits, their high words
// here, and a round record's `big` has its count from bit 43 on (at most 2^20 big
// vertices there).  A frontier of kEdges32 big edges or more is expanded from the
// bitmap, where edges are counted per 32 vertices.
__shared__ uint32_t s_start_high[kBfsWarps][32];
constexpr unsigned long long kEdges32 = (1ull << 32) - (1ull << 16);
template <bool kWide>
struct BigWord {
  static constexpr int kShift = kWide ? 43 : 32;
  static constexpr unsigned long long kEdges = (1ull << kShift) - 1ull;
  static __device__ __forceinline__ unsigned long long pack(unsigned count, unsigned edges) {
    return ((unsigned long long)count << kShift) | edges;
  }
};

// Shared memory of block 0's runs of small rounds (solo_rounds): the frontier
// and the next one (vertex, list start, out-degree), and the prefix of the
// frontier's degrees.
constexpr int kSoloMax = 1280;             // vertices of a frontier kept here
constexpr unsigned kSoloEdges = 4096;      // edges of a round run by one block
constexpr unsigned kSoloEnter = 2048;      // edges of the first round of a run
// A run that goes on above kTeamEnter edges a round is taken by a team of
// blocks (team_rounds) in the kernel for graphs where that happens.
constexpr int kTeamBlock = 384;            // threads of a block of that kernel, at most
constexpr unsigned kTeam = 16;             // blocks
constexpr unsigned kTeamEdges = 32768;     // edges of a round of the team
constexpr unsigned kTeamEnter = 1024, kTeamLeave = 512;
constexpr int64_t kTeamVertices = 1 << 16; // of a graph, at least
constexpr int64_t kTeamDegree = 8;         // in-degree that all but 1/1024 of the entries keep to
constexpr int kTeamAfter = 4;              // rounds above kTeamEnter before the hand-over
constexpr int kTeamSession = 64;           // rounds of one hand-over, at most
struct SoloShared {
  int32_t v[2][kSoloMax];
  uint32_t s[2][kSoloMax];
  uint32_t d[2][kSoloMax];
  uint32_t x[kSoloMax];
  uint32_t warp_total[kBfsWarps];
  unsigned n, mf;                          // the next frontier's vertices and edges
  unsigned payload;
};
struct GridShared {
  WarpTile tiles[kBfsWarps];
  WarpExpand expand[kBfsWarps];
};
// One round at a time uses it, one way or the other.
union __align__(16) RoundShared {
  GridShared grid;
  SoloShared solo;
};
__shared__ RoundShared s_round;
__shared__ unsigned s_commands;  // the team lead's commands that this block has served
#define s_tiles s_round.grid.tiles
#define s_expand s_round.grid.expand

__device__ __forceinline__ uint4 ld4(const uint32_t *a) {
  return *reinterpret_cast<const uint4 *>(a);
}
// Non-coherent (read-only path) load: only for data no thread writes while
// the kernel runs (the dead-vertex map).  Bitmaps that earlier rounds wrote are
// read with ordinary loads, which the grid waits' acquire makes current.
__device__ __forceinline__ uint4 ldg4(const uint32_t *a) {
  return __ldg(reinterpret_cast<const uint4 *>(a));
}
__device__ __forceinline__ void st4(uint32_t *a, uint4 v) { *reinterpret_cast<uint4 *>(a) = v; }
__device__ __forceinline__ bool any4(uint4 v) { return (v.x | v.y | v.z | v.w) != 0u; }

// Original id of resident vertex v (the identity unless the graph was
// relabelled): the output position and the parent value outputs use.
__device__ __forceinline__ int32_t orig_id(const BfsParams &p, int64_t v) {
  return p.orig ? __ldg(p.orig + v) : (int32_t)v;
}

// Bits of word `wi` that stand for vertices < n.
__device__ __forceinline__ uint32_t valid_bits(int64_t wi, int64_t n) {
  const int64_t lo = wi * 32;
  if (lo + 32 <= n) return kFull;
  if (lo >= n) return 0u;
  return (1u << (unsigned)(n - lo)) - 1u;
}

// Stages the tile's 128 words (4 per lane, lane order) in shared memory with
// the exclusive prefix of their popcounts; returns the tile's total number of
// set bits (the same in every lane).  All 32 lanes call.
__device__ __forceinline__ unsigned stage_tile(uint4 m, WarpTile &T) {
  const int lane = lane_id();
  const unsigned c0 = __popc(m.x), c1 = __popc(m.y), c2 = __popc(m.z), c3 = __popc(m.w);
  const unsigned cnt = c0 + c1 + c2 + c3;
  unsigned incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  const unsigned base = incl - cnt;
  st4(T.m + 4 * lane, m);
  st4(T.pre + 4 * lane, make_uint4(base, base + c0, base + c0 + c1, base + c0 + c1 + c2));
  __syncwarp();
  return __shfl_sync(kFull, incl, 31);
}

// The k-th set bit (k below the staged total) of the staged tile: word j of
// the tile and bit b of that word.  The last word whose prefix is <= k holds it.
__device__ __forceinline__ void select_bit(const WarpTile &T, unsigned k, int &j, int &b) {
  int lo = 0;
#pragma unroll
  for (int step = kTileWords / 2; step > 0; step >>= 1)
    if (T.pre[lo + step] <= k) lo += step;
  j = lo;
  b = (int)__fns(T.m[lo], 0, (int)(k - T.pre[lo]) + 1);
}

// A thread's discoveries in one round: vertices, and the sum of their
// out-degrees / in-degrees.  32 bits suffice: a round discovers at most n
// vertices and their degrees sum to at most nnz < 2^32 (checked at upload).
struct Acc {
  unsigned nf = 0, mf = 0, visdeg = 0;
};

// Appends the discoveries of one warp-wide step to the next frontier's queue:
// light vertices at the front; big ones at the back, each with the prefix
// offset of its edge list among the big vertices (one packed 64-bit atomic per
// warp: count in the high word, edges in the low word).  All 32 lanes call.
__device__ __forceinline__ void enqueue_claims(const BfsParams &p, bool claimed, int32_t v,
                                               int64_t deg, int next_parity, RoundRec *Rn,
                                               Acc &acc) {
  const int lane = lane_id();
  if (!__ballot_sync(kFull, claimed)) return;
  int32_t *q = next_parity ? p.queue1 : p.queue0;
  const bool light = claimed && deg <= kLightMax;
  const bool big = claimed && deg > kLightMax;
  const unsigned below = (1u << lane) - 1u;
  const unsigned ml = __ballot_sync(kFull, light);
  if (ml) {
    const int leader = __ffs(ml) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(&Rn->nlight, (unsigned)__popc(ml));
    base = __shfl_sync(kFull, base, leader);
    if (light) q[base + __popc(ml & below)] = v;
  }
  const unsigned mb = __ballot_sync(kFull, big);
  if (mb) {
    const unsigned d = big ? (unsigned)deg : 0u;
    unsigned incl = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    const unsigned total = __shfl_sync(kFull, incl, 31);
    unsigned long long old = 0;
    if (lane == 0)
      old = atomicAdd(&Rn->big, ((unsigned long long)__popc(mb) << 32) | total);
    old = __shfl_sync(kFull, old, 0);
    if (big) {
      const unsigned idx = (unsigned)(old >> 32) + __popc(mb & below);
      q[p.n - 1 - (int64_t)idx] = v;
      (next_parity ? p.bigoff1 : p.bigoff0)[idx] = (unsigned)(old & 0xffffffffu) + incl - d;
    }
  }
  if (claimed) {
    acc.nf += 1;
    acc.mf += (unsigned)deg;
    acc.visdeg += (unsigned)deg;
  }
}

// Claimed vertices on their way to the next frontier's queue.  A returning
// atomic on one address takes about 2 ns however many blocks make them, and a
// round that made one per step with claims, or one per warp at its end, was
// bound by them.  So a warp keeps its claims in shared memory, light and big
// ones apart, queues 32 of a kind with one atomic, and the block queues what its
// warps have left together at the round's end.  Rounds of 61,564 claims (R-MAT n
// = 100,003, top-down): 37 -> 28 us; of 202,765 (directed ER): 33 -> 24 us; of 862,250 (R-MAT
// scale 23): 173 -> 92 us.
struct Claims {
  WarpExpand &X;
  BigClaims &B;
  unsigned nl = 0, nb = 0;  // waiting (the same in every lane), < 32 between steps
};

// Big vertices B[from .. from + n), n <= 32, at queue index `idx` with edge
// offset `edges` among the big vertices' lists.  All 32 lanes call.
__device__ __forceinline__ void put_big(const BfsParams &p, const BigClaims &B, unsigned from,
                                        unsigned n, unsigned idx, unsigned edges,
                                        int next_parity) {
  const int lane = lane_id();
  const bool has = (unsigned)lane < n;
  const uint32_t d = has ? B.deg[from + lane] : 0u;
  uint32_t incl = d;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  if (!has) return;
  (next_parity ? p.queue1 : p.queue0)[p.n - 1 - (int64_t)(idx + lane)] = B.v[from + lane];
  (next_parity ? p.bigoff1 : p.bigoff0)[idx + lane] = edges + incl - d;
}

// The claims of one warp-wide step.  All 32 lanes call.
template <bool kWide>
__device__ __forceinline__ void keep_claims(const BfsParams &p, bool claimed, int32_t v,
                                            uint32_t deg, int next_parity, RoundRec *Rn, Claims &C,
                                            Acc &acc) {
  const int lane = lane_id();
  const unsigned below = (1u << lane) - 1u;
  const unsigned m = __ballot_sync(kFull, claimed);
  if (!m) return;
  if (claimed) {
    acc.nf += 1;
    acc.mf += deg;
    acc.visdeg += deg;
  }
  const bool big = claimed && deg > (uint32_t)kLightMax;
  const unsigned mb = __ballot_sync(kFull, big), ml = m & ~mb;
  if (big) {
    const unsigned at = C.nb + __popc(mb & below);
    C.B.v[at] = v;
    C.B.deg[at] = deg;
  } else if (claimed) {
    C.X.light[C.nl + __popc(ml & below)] = v;
  }
  C.nb += __popc(mb);
  C.nl += __popc(ml);
  __syncwarp();
  // full groups: the last 32, the entries below keep their places
  if (C.nl >= 32) {
    C.nl -= 32;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&Rn->nlight, 32u);
    base = __shfl_sync(kFull, base, 0);
    (next_parity ? p.queue1 : p.queue0)[base + lane] = C.X.light[C.nl + lane];
    __syncwarp();
  }
  if (C.nb >= 32) {
    C.nb -= 32;
    const uint32_t edges = __reduce_add_sync(kFull, C.B.deg[C.nb + lane]);
    unsigned long long old = 0;
    if (lane == 0) old = atomicAdd(&Rn->big, BigWord<kWide>::pack(32, edges));
    old = __shfl_sync(kFull, old, 0);
    put_big(p, C.B, C.nb, 32, (unsigned)(old >> BigWord<kWide>::kShift), (unsigned)old,
            next_parity);
    __syncwarp();
  }
}

// What the block's warps have left, one atomic of a kind.  All threads call.
template <bool kWide>
__device__ __forceinline__ void queue_rest(const BfsParams &p, Claims &C, int next_parity,
                                           RoundRec *Rn) {
  __shared__ unsigned s_nl[kBfsWarps], s_nb[kBfsWarps], s_edges[kBfsWarps];
  const int lane = lane_id(), wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t edges = __reduce_add_sync(kFull, (unsigned)lane < C.nb ? C.B.deg[lane] : 0u);
  if (lane == 0) {
    s_nl[wib] = C.nl;
    s_nb[wib] = C.nb;
    s_edges[wib] = edges;
  }
  __syncthreads();
  if (wib == 0) {  // exclusive prefixes, from the queue's own counts
    const unsigned l = lane < nw ? s_nl[lane] : 0u, b = lane < nw ? s_nb[lane] : 0u,
                   e = lane < nw ? s_edges[lane] : 0u;
    unsigned il = l, ib = b, ie = e;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned tl = __shfl_up_sync(kFull, il, o), tb = __shfl_up_sync(kFull, ib, o),
                     te = __shfl_up_sync(kFull, ie, o);
      if (lane >= o) il += tl, ib += tb, ie += te;
    }
    unsigned long long old = 0;
    if (lane == 31 && il) old = atomicAdd(&Rn->nlight, il);
    const unsigned base_l = (unsigned)__shfl_sync(kFull, old, 31);
    if (lane == 31) old = ib ? atomicAdd(&Rn->big, BigWord<kWide>::pack(ib, ie)) : 0ull;
    old = __shfl_sync(kFull, old, 31);
    if (lane < nw) {
      s_nl[lane] = base_l + il - l;
      s_nb[lane] = (unsigned)(old >> BigWord<kWide>::kShift) + ib - b;
      s_edges[lane] = (unsigned)old + ie - e;
    }
  }
  __syncthreads();
  if ((unsigned)lane < C.nl)
    (next_parity ? p.queue1 : p.queue0)[s_nl[wib] + lane] = C.X.light[lane];
  if (C.nb) put_big(p, C.B, 0, C.nb, s_nb[wib], s_edges[wib], next_parity);
}

// Position of a list entry; all bits set for none.
template <bool kWide>
using EdgePos = std::conditional_t<kWide, uint64_t, uint32_t>;
template <bool kWide>
constexpr EdgePos<kWide> kNoEdge = ~EdgePos<kWide>(0);

// Edge u -> out_idx[e] per lane of a push round (e = kNoEdge for none).  A
// target claimed already gets a read before its atomicMin: most of a big
// round's edges lead to vertices that a lower source has reached, and a read
// costs the L2 less.
template <bool kWide>
__device__ __forceinline__ void push_step(const BfsParams &p, const uint32_t *cur, uint32_t *nxt,
                                          int32_t u, EdgePos<kWide> e, int L, int next_parity,
                                          RoundRec *Rn, Claims &C, Acc &acc) {
  const int32_t v = e != kNoEdge<kWide> ? __ldg(p.out_idx + e) : -1;
  bool open = false, mine = false;  // not visited; nor claimed by another edge before
  if (v >= 0) {
    const uint32_t w = (uint32_t)v >> 5, bit = 1u << (v & 31);
    // the three words in one round trip: a claim bit seen set stays set (the
    // L1's copy may lack it: reading the hot words from the L2 took 140 us where
    // this takes 92, R-MAT n = 100,003, top-down)
    const uint32_t seen = p.vis[w] | cur[w], claimed = nxt[w];
    open = !(seen & bit);
    mine = open && !(claimed & bit);
  }
  bool claimed = false;
  uint32_t deg = 0;
  if (open) {
    const int32_t ov = orig_id(p, v);
    const unsigned ou = (unsigned)orig_id(p, u);
    unsigned *par = reinterpret_cast<unsigned *>(p.parents) + ov;
    if (mine) {
      atomicMin(par, ou);
      // the target's list bounds go out with its claim
      const int64_t o = __ldg(p.out_off + v);
      deg = (uint32_t)(__ldg(p.out_off + v + 1) - o);
      const uint32_t bit = 1u << (v & 31);
      claimed = !(atomicOr(nxt + ((uint32_t)v >> 5), bit) & bit);
      if (claimed) p.levels[ov] = L + 1;
    } else if (__ldcg(par) > ou) {
      atomicMin(par, ou);
    }
  }
  keep_claims<kWide>(p, claimed, v, deg, next_parity, Rn, C, acc);
}

// Expands up to 32 frontier vertices (one per lane, u < 0 for none) with the
// warp's combined edge list spread evenly over its lanes.
template <bool kWide>
__device__ __forceinline__ void gather_expand(const BfsParams &p, const uint32_t *cur,
                                              uint32_t *nxt, int32_t u, int L, int next_parity,
                                              RoundRec *Rn, Claims &C, Acc &acc) {
  const int lane = lane_id();
  WarpExpand &X = C.X;
  EdgePos<kWide> s = 0;
  uint32_t d = 0;
  if (u >= 0) {
    const int64_t o = __ldg(p.out_off + u);
    s = (EdgePos<kWide>)o;
    d = (uint32_t)(__ldg(p.out_off + u + 1) - o);
  }
  uint32_t incl = d;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  if (total == 0) return;
  X.u[lane] = u;
  X.s[lane] = (uint32_t)s;
  if constexpr (kWide) s_start_high[threadIdx.x >> 5][lane] = (uint32_t)(s >> 32);
  X.x[lane] = incl - d;
  __syncwarp();
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t t = base + lane;
    int lo = 0;  // the last of the 32 whose prefix is <= t
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (X.x[lo + step] <= t) lo += step;
    EdgePos<kWide> e = kNoEdge<kWide>;
    if (t < total && t >= base) {
      e = X.s[lo];
      if constexpr (kWide) e |= (uint64_t)s_start_high[threadIdx.x >> 5][lo] << 32;
      e += t - X.x[lo];
    }
    push_step<kWide>(p, cur, nxt, X.u[lo], e, L, next_parity, Rn, C, acc);
    if (base + 32 < base) break;  // total within a step of 2^32
  }
  __syncwarp();
}

// Expands frontier F_L from its queue (parity L & 1): edge-balanced chunks of
// the big vertices' combined edge list, then the light vertices, up to 32 to
// a warp.  A frontier of fewer light vertices than 32 a warp is spread over
// more warps (`group` each): a warp's steps run one after the other, about 2.6
// us each with cold lists, so 415 vertices of degree 8 took 8 steps on 13
// warps where one step on 415 does (29 -> 11 us a round; 26,618 vertices: 50 ->
// 16 us).  Item i goes to warp i first; warps that finish take the rest from a counter.
// bigw / nlight: F_L's queue sizes ((big count << 32) | big edges, light
// count), handed over with the barrier that ended round L - 1.
template <bool kWide>
__device__ void push_round_queue(const BfsParams &p, const uint32_t *cur, uint32_t *nxt, int L,
                                 RoundRec *Rc, RoundRec *Rn, unsigned long long bigw,
                                 unsigned nlight, Acc &acc) {
  const int lane = lane_id();
  const int wib = threadIdx.x >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int parity = L & 1, next_parity = parity ^ 1;
  const int32_t *q = parity ? p.queue1 : p.queue0;
  const uint32_t *boff = parity ? p.bigoff1 : p.bigoff0;

  const unsigned nbig = (unsigned)(bigw >> 32);
  const unsigned big_edges = (unsigned)(bigw & 0xffffffffu);
  // chunks of 32 .. kPushChunk edges: small frontiers still spread over the grid
  unsigned chunk = ((big_edges / (unsigned)nwarps) + 31u) & ~31u;
  chunk = chunk < 32u ? 32u : (chunk > (unsigned)kPushChunk ? (unsigned)kPushChunk : chunk);
  const unsigned nchunks = (big_edges + chunk - 1) / chunk;
  unsigned group = 1;
  while (group < 32u && nlight > group * (unsigned)nwarps) group <<= 1;
  const unsigned nitems = nchunks + (nlight + group - 1) / group;
  Claims C{s_expand[wib], reinterpret_cast<BigClaims &>(s_tiles[wib].found)};
  unsigned item = (unsigned)warp_id_global();
  while (item < nitems) {
    // the next item is claimed before this one is worked, hiding the atomic;
    // with no more items than warps there is none
    unsigned nextitem = nitems;
    if (nitems > (unsigned)nwarps && lane == 0)
      nextitem = (unsigned)nwarps + atomicAdd(&Rc->work, 1u);
    if (item < nchunks) {
      const unsigned x0 = item * chunk;
      const unsigned x1 = min(x0 + chunk, big_edges);
      // big vertex j holding edge position x0: the last j with boff[j] <= x0
      unsigned lo = 0, hi = nbig - 1;
      while (lo < hi) {
        const unsigned mid = (lo + hi + 1) >> 1;
        if (boff[mid] <= x0)
          lo = mid;
        else
          hi = mid - 1;
      }
      unsigned j = lo;
      int32_t vj = q[p.n - 1 - (int64_t)j];
      EdgePos<kWide> sj = (EdgePos<kWide>)__ldg(p.out_off + vj);
      unsigned oj = boff[j];
      unsigned endj = oj + (uint32_t)((EdgePos<kWide>)__ldg(p.out_off + vj + 1) - sj);
      for (unsigned base = x0; base < x1; base += 32) {
        while (base >= endj) {  // the next big vertex (degrees exceed 32)
          ++j;
          vj = q[p.n - 1 - (int64_t)j];
          sj = (EdgePos<kWide>)__ldg(p.out_off + vj);
          oj = boff[j];
          endj = oj + (uint32_t)((EdgePos<kWide>)__ldg(p.out_off + vj + 1) - sj);
        }
        const unsigned x = base + lane;
        const bool valid = x < x1;
        int32_t u = vj;
        EdgePos<kWide> e = valid ? sj + (x - oj) : kNoEdge<kWide>;
        if (__ballot_sync(kFull, valid && x >= endj)) {  // lanes past vertex j's end
          const int32_t vn = q[p.n - 1 - (int64_t)(j + 1)];
          if (valid && x >= endj) {
            u = vn;
            e = (EdgePos<kWide>)__ldg(p.out_off + vn) + (x - endj);
          }
        }
        push_step<kWide>(p, cur, nxt, u, e, L, next_parity, Rn, C, acc);
      }
    } else {
      const unsigned idx = (item - nchunks) * group + lane;
      gather_expand<kWide>(p, cur, nxt, (unsigned)lane < group && idx < nlight ? q[idx] : -1, L,
                           next_parity, Rn, C, acc);
    }
    item = __shfl_sync(kFull, nextitem, 0);
  }
  queue_rest<kWide>(p, C, next_parity, Rn);
}

// Work items of a bitmap-wide round: (tile, slot) pairs; a tile holds 4096
// vertices (there are fewer tiles than warps below ~30M vertices) and its S
// slots split its set bits into S even ranges.  A heavy round (enough work for
// every warp) hands out about two items per warp, item i to warp i first and
// the rest from the round record's counter: its work crowds into the low
// tiles, where the unvisited vertices with in-edges are.  A light round takes
// S = warps / tiles and item i to warp i, with no counter for the grid's warps
// to queue on when they all finish at once.
__device__ __forceinline__ unsigned tile_slots(int64_t tiles, int nwarps, bool heavy) {
  const int64_t s = heavy ? (2 * (int64_t)nwarps + tiles - 1) / tiles : (int64_t)nwarps / tiles;
  return (unsigned)(s < 1 ? 1 : (s > 64 ? 64 : s));
}

__device__ __forceinline__ int64_t next_item(int64_t item, int nwarps, RoundRec *Rc, bool heavy) {
  if (!heavy) return item + nwarps;
  unsigned nextitem = 0;
  if (lane_id() == 0) nextitem = (unsigned)nwarps + atomicAdd(&Rc->work, 1u);
  return (int64_t)__shfl_sync(kFull, nextitem, 0);
}

// Push round right after a pull round: the frontier is only in the bitmap, so
// warps stage it a tile at a time (one 16-byte load per lane) and expand its
// set bits 32 at a time (lane i takes the i-th bit of its batch).
template <bool kWide>
__device__ void push_round_bitmap(const BfsParams &p, const uint32_t *cur, uint32_t *nxt, int L,
                                  RoundRec *Rc, RoundRec *Rn, bool heavy, Acc &acc) {
  const int lane = lane_id();
  const int wib = threadIdx.x >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int next_parity = (L + 1) & 1;
  WarpTile &T = s_tiles[wib];
  Claims C{s_expand[wib], reinterpret_cast<BigClaims &>(s_tiles[wib].found)};
  const unsigned S = tile_slots(p.tiles, nwarps, heavy);
  const int64_t items = p.tiles * S;
  for (int64_t item = warp_id_global(); item < items; item = next_item(item, nwarps, Rc, heavy)) {
    const int64_t t = item % p.tiles;
    const unsigned slot = (unsigned)(item / p.tiles);
    const uint4 c = ld4(cur + t * kTileWords + 4 * lane);
    const unsigned total = stage_tile(c, T);
    const unsigned k1 = (unsigned)((unsigned long long)total * (slot + 1) / S);
    for (unsigned b = (unsigned)((unsigned long long)total * slot / S); b < k1; b += 32) {
      int32_t u = -1;
      if (b + lane < k1) {
        int j, bit;
        select_bit(T, b + lane, j, bit);
        u = (int32_t)((t * kTileWords + j) * 32 + bit);
      }
      gather_expand<kWide>(p, cur, nxt, u, L, next_parity, Rn, C, acc);
    }
    __syncwarp();  // T is restaged by the next item
  }
  queue_rest<kWide>(p, C, next_parity, Rn);
}

// Bottom-up round: every unvisited vertex scans its ascending in-list and
// stops at the first source in F_L, which is its lowest-index parent.
// Work items are (tile, slot) pairs of 4096-vertex bitmap tiles: one 16-byte
// load per lane of each of vis, F_L and the map of vertices without in-edges
// gives the tile's unvisited set, staged in shared memory, and the slot takes
// an even range of it.
//
// First the heads: a vertex's first in-neighbour and in-degree lie together in
// an array by vertex (`head`), so a test of the first entry -- on R-MAT graphs,
// a hub, the one that most vertices resolve at -- takes one coalesced 8-byte
// load and one bit, where the list bounds and then the list are two dependent,
// scattered trips.  An SM's scattered accesses, about 1.4 a ns, bound the big
// pull rounds: R-MAT scale 23, 3.6 M vertices found, 78 -> 55 us.  Light rounds,
// bound by the length of the chain, do without (n = 4096: 0.7 us a search).
//
// The misses are staged anew and scanned from their second entry on: each lane
// works on one vertex of the range at a time, an aligned block of
// kPullThreadScan entries of its list a step (one 16-byte load; all bit tests
// in flight at once); a lane whose vertex is done (found, or its list
// exhausted) takes the range's next vertex at once, so lanes do not wait for
// the slowest list of a batch.  A list still unresolved after kPullLaneMax
// entries is finished by the whole warp, 32 entries a step.  Found vertices set
// their bit in the warp's shared copy of the tile's next-frontier words, ORed
// into F_{L+1} at the end of the item.  Slot 0 of each tile also merges F_L into
// vis (the union vis | F_L that other slots test is unchanged by it) and clears
// F_{L-1} (the next round's output bitmap), so pull rounds need no sweep.
// Without heads (graphs without hubs, see bfs_prepare; cg_bfs_noalloc, whose
// arrays need not be aligned either; no memory for them) every vertex is scanned
// from its first entry.
__device__ void pull_round(const BfsParams &p, const uint32_t *cur, uint32_t *nxt, uint32_t *old,
                           int L, RoundRec *Rc, bool heavy, Acc &acc) {
  const int lane = lane_id();
  const unsigned lt_mask = (1u << lane) - 1u;
  const int wib = threadIdx.x >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  WarpTile &T = s_tiles[wib];
  const unsigned S = tile_slots(p.tiles, nwarps, heavy);
  const int64_t items = p.tiles * S;
  for (int64_t item = warp_id_global(); item < items; item = next_item(item, nwarps, Rc, heavy)) {
    const int64_t t = item % p.tiles;
    const unsigned slot = (unsigned)(item / p.tiles);
    const int64_t w0 = t * kTileWords + 4 * lane;
    const uint4 vi = ld4(p.vis + w0);
    const uint4 cu = ld4(cur + w0);
    uint4 dd;
    if (p.dead) {
      dd = ldg4(p.dead + w0);
    } else {
      dd = make_uint4(~valid_bits(w0, p.n), ~valid_bits(w0 + 1, p.n), ~valid_bits(w0 + 2, p.n),
                      ~valid_bits(w0 + 3, p.n));
    }
    if (slot == 0) {
      if (any4(cu))
        st4(p.vis + w0, make_uint4(vi.x | cu.x, vi.y | cu.y, vi.z | cu.z, vi.w | cu.w));
      st4(old + w0, make_uint4(0u, 0u, 0u, 0u));
    }
    const uint4 un = make_uint4(~(vi.x | cu.x | dd.x), ~(vi.y | cu.y | dd.y),
                                ~(vi.z | cu.z | dd.z), ~(vi.w | cu.w | dd.w));
    st4(T.found + 4 * lane, make_uint4(0u, 0u, 0u, 0u));
    unsigned total = stage_tile(un, T);
    unsigned k1 = (unsigned)((unsigned long long)total * (slot + 1) / S);
    unsigned cursor = (unsigned)((unsigned long long)total * slot / S);
    const int64_t v0 = t * kTileWords * 32;  // the tile's first vertex
    if (heavy && p.head) {
      constexpr int U = 2;  // batches of 32 vertices in flight
      uint32_t *miss = reinterpret_cast<uint32_t *>(&s_expand[wib]);
      static_assert(sizeof(WarpExpand) >= 4 * kTileWords && sizeof(WarpExpand) % 16 == 0, "miss");
      st4(miss + 4 * lane, make_uint4(0u, 0u, 0u, 0u));
      __syncwarp();
      for (unsigned b0 = cursor; b0 < k1; b0 += 32 * U) {
        int at[U];   // vertex of the tile
        uint2 h[U];  // its first in-neighbour and in-degree
#pragma unroll
        for (int q = 0; q < U; ++q) {
          const unsigned k = b0 + 32 * q + lane;
          at[q] = -1;
          h[q] = make_uint2(0u, 0u);
          if (k < k1) {
            int j, bit;
            select_bit(T, k, j, bit);
            at[q] = 32 * j + bit;
            h[q] = __ldg(p.head + v0 + at[q]);
          }
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
          if (at[q] < 0) continue;
          const uint32_t b = 1u << (at[q] & 31);
          if ((cur[h[q].x >> 5] >> (h[q].x & 31)) & 1u) {
            const int32_t ov = orig_id(p, v0 + at[q]);
            p.parents[ov] = orig_id(p, (int32_t)h[q].x);
            p.levels[ov] = L + 1;
            atomicOr(&T.found[at[q] >> 5], b);
            acc.nf += 1;
            acc.visdeg += h[q].y;
          } else if (h[q].y > 1) {
            atomicOr(&miss[at[q] >> 5], b);
          }
        }
      }
      __syncwarp();
      const uint4 m = ld4(miss + 4 * lane);
      total = stage_tile(m, T);
      cursor = 0;
      k1 = total;
    }
    // lane state: the vertex it works on (v, word j / bit of the tile), its
    // list [s, s + deg) and the next entry to scan
    bool has = false;
    int j = 0, bit = 0;
    int64_t s = 0;
    unsigned deg = 0, pos = 0;
    bool refill = true;  // some lane has no vertex (warp-uniform)
    while (true) {
      if (refill) {
        const unsigned need = __ballot_sync(kFull, !has);
        if (!has) {
          const unsigned k = cursor + __popc(need & lt_mask);
          if (k < k1) {
            has = true;
            select_bit(T, k, j, bit);
            const int64_t v = v0 + j * 32 + bit;
            s = __ldg(p.in_off + v);
            deg = (unsigned)(__ldg(p.in_off + v + 1) - s);
            pos = heavy && p.head ? 1 : 0;
          }
        }
        cursor += __popc(need);
      }
      if (!__any_sync(kFull, has)) break;
      bool found = false;
      if (has && pos < kPullLaneMax) {
        // the entries of the aligned block that holds entry pos (arrays of the
        // library's own), or the next kPullThreadScan ones
        int32_t u[kPullThreadScan];
        const int64_t e0 = s + pos;
        unsigned skip = p.head ? (unsigned)e0 & 3u : 0u;
        static_assert(kPullThreadScan == 4, "a 16-byte block");
        if (p.head && e0 - skip + 4 <= p.nnz) {
          const int4 x = __ldg(reinterpret_cast<const int4 *>(p.in_idx + (e0 - skip)));
          u[0] = x.x, u[1] = x.y, u[2] = x.z, u[3] = x.w;
#pragma unroll
          for (int k = 0; k < kPullThreadScan; ++k)
            if ((unsigned)k < skip || pos - skip + k >= deg) u[k] = -1;
        } else {
          skip = 0;
#pragma unroll
          for (int k = 0; k < kPullThreadScan; ++k)
            u[k] = pos + k < deg ? __ldg(p.in_idx + e0 + k) : -1;
        }
        uint32_t hit = 0;
#pragma unroll
        for (int k = 0; k < kPullThreadScan; ++k)
          if (u[k] >= 0 && ((cur[(uint32_t)u[k] >> 5] >> (u[k] & 31)) & 1u)) hit |= 1u << k;
        if (hit) {
          const int k = __ffs(hit) - 1;  // ascending list: the lowest hit is the minimum
          int32_t uk = u[0];
#pragma unroll
          for (int q = 1; q < kPullThreadScan; ++q)
            if (q == k) uk = u[q];
          const int32_t ov = orig_id(p, v0 + j * 32 + bit);
          p.parents[ov] = orig_id(p, uk);
          p.levels[ov] = L + 1;
          found = true;
        }
        pos += kPullThreadScan - skip;
      }
      // lists still open after kPullLaneMax entries: the whole warp scans the
      // rest, one vertex at a time
      unsigned rest = __ballot_sync(kFull, has && !found && pos >= kPullLaneMax && pos < deg);
      while (rest) {
        const int jl = __ffs(rest) - 1;
        rest &= rest - 1;
        const int64_t sj = __shfl_sync(kFull, s, jl);
        const unsigned pj = __shfl_sync(kFull, pos, jl);
        const unsigned dj = __shfl_sync(kFull, deg, jl);
        const int64_t vj = v0 + __shfl_sync(kFull, j * 32 + bit, jl);
        bool got = false;
        for (unsigned base = pj; base < dj; base += 32) {
          const unsigned i = base + lane;
          int32_t u = 0;
          bool hit = false;
          if (i < dj) {
            u = __ldg(p.in_idx + sj + i);
            hit = (cur[(uint32_t)u >> 5] >> (u & 31)) & 1u;
          }
          const unsigned who = __ballot_sync(kFull, hit);
          if (who) {
            if (lane == __ffs(who) - 1) {
              const int32_t ovj = orig_id(p, vj);
              p.parents[ovj] = orig_id(p, u);
              p.levels[ovj] = L + 1;
            }
            got = true;
            break;
          }
        }
        if (lane == jl) {
          found = got;
          pos = deg;  // scanned to the end (or found)
        }
      }
      if (found) {
        atomicOr(&T.found[j], 1u << bit);
        acc.nf += 1;
        acc.visdeg += deg;
      }
      const bool done = has && (found || pos >= deg);
      if (done) has = false;
      refill = __any_sync(kFull, done) && cursor < k1;
    }
    __syncwarp();
    const uint4 f = ld4(T.found + 4 * lane);
    if (f.x) atomicOr(nxt + w0, f.x);
    if (f.y) atomicOr(nxt + w0 + 1, f.y);
    if (f.z) atomicOr(nxt + w0 + 2, f.z);
    if (f.w) atomicOr(nxt + w0 + 3, f.w);
    __syncwarp();  // T is restaged by the next item
  }
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFull, x, o);
  return x;
}

// Block totals of the per-thread counters (all threads call; thread 0 gets
// the sums) -- the one __syncthreads of a round's end before the wait.
__device__ void block_totals(Acc &acc, unsigned long long &a, unsigned long long &b,
                             unsigned long long &c) {
  __shared__ unsigned long long s_red[3][kBfsBlock / 32];
  const int lane = lane_id(), wib = threadIdx.x >> 5;
  a = warp_sum(acc.nf);
  b = warp_sum(acc.mf);
  c = warp_sum(acc.visdeg);
  if (lane == 0) {
    s_red[0][wib] = a;
    s_red[1][wib] = b;
    s_red[2][wib] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    a = b = c = 0;
    for (int i = 0; i < nw; ++i) {
      a += s_red[0][i];
      b += s_red[1][i];
      c += s_red[2][i];
    }
  }
  acc = Acc();
}

__device__ __forceinline__ int next_direction(const BfsParams &p, int dir, unsigned long long nf,
                                              unsigned long long prev_nf,
                                              unsigned long long mf,
                                              unsigned long long explored) {
  switch (p.direction) {
    case CG_DIR_TOPDOWN:
      return kPush;
    case CG_DIR_BOTTOMUP:
      return kPull;
    case CG_DIR_TAU:
      // bool_pe.csl:1078-1088: one way only, once nf exceeds tau
      return (dir == kPull || (long long)nf > p.tau) ? kPull : kPush;
    default: {
      if (dir == kPush) {
        // Beamer's rule, plus a floor: a pull round walks every vertex's
        // visited word, so a frontier whose edges are fewer than n / 8 stays
        // push (near the end "unexplored" counts only unreachable edges)
        const double unexplored = (double)p.nnz - (double)explored;
        return ((double)mf > unexplored / (double)p.alpha && (double)mf > (double)p.n / 8.0)
                   ? kPull
                   : kPush;
      }
      const bool shrinking = nf < prev_nf;
      return (shrinking && (double)nf < (double)p.n / (double)p.beta) ? kPush : kPull;
    }
  }
}

// Payload of a round's grid-wide barrier: the search ended; the next round
// pulls; the next round is heavy (enough work for every warp of the grid).
constexpr unsigned kDone = 1u, kNextPull = 2u, kHeavy = 4u;
// ... is small enough for one block (solo_rounds)
constexpr unsigned kSolo = 8u;
// ... or for a team
constexpr unsigned kHandOver = 16u;
// ... expands its frontier from the bitmap, although it was queued (kWide)
constexpr unsigned kUnqueued = 32u;
__device__ __forceinline__ unsigned team_size() { return gridDim.x >= 2 * kTeam ? kTeam : 0u; }

// Flat grid-wide barrier of the per-root kernel, called by thread 0 of each
// block after a __syncthreads: one fire-and-forget release add on the launch's
// 64-bit arrival count, relaxed polls until the count reaches `target` (the
// b-th barrier of a launch waits for (b + 1) * gridDim.x arrivals; the count is
// zeroed before every launch), then one acquire fence, which makes every
// block's writes before its arrival visible.  Relaxed polls leave the SM's L1
// alone (an acquire load invalidates it while blocks of the same SM may still
// be working).  Bounded: after timeout_ns, or once another block has flagged
// an error, the thread records CG_ERR_TIMEOUT and returns false, so a barrier
// that cannot complete ends the kernel instead of spinning.
__device__ __forceinline__ void flat_arrive(unsigned long long *count) {
  asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(count) : "memory");
}

// The wait alone; `sleep_ns` between polls for a wait that may last (the polls
// of 455 blocks would share the L2 with the one block that works).
__device__ __forceinline__ bool flat_wait(unsigned long long *count, unsigned long long target,
                                          int *status, long long timeout_ns,
                                          unsigned sleep_ns = 0) {
  long long t0 = 0;
  unsigned spins = 0;
  while (true) {
    unsigned long long c;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(count) : "memory");
    if (c >= target) break;
    if (sleep_ns) __nanosleep(sleep_ns);
    if ((++spins & 255u) == 0) {
      if (t0 == 0) t0 = global_ns();
      if (*(volatile int *)status != 0 || global_ns() - t0 > timeout_ns) {
        atomicCAS(status, 0, (int)CG_ERR_TIMEOUT);
        return false;
      }
    }
  }
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  return true;
}

__device__ __forceinline__ bool flat_barrier(unsigned long long *count, unsigned long long target,
                                             int *status, long long timeout_ns) {
  flat_arrive(count);
  return flat_wait(count, target, status, timeout_ns);
}

// The search-wide bookkeeping of bool_pe.csl:947-1100 (visited total,
// explored edges, previous frontier size, pull rounds, direction switches).
// Every block keeps its own copy (thread 0) and updates it from the same round
// totals, so all blocks take the same decision without a second barrier.
struct SearchState {
  unsigned long long visited, prev_nf, explored;
  int pull_rounds, switches;
  long long t_mark;  // block 0: end of the previous round on the device clock
  long long t_session;  // team lead: when the other blocks began their bounded wait
  unsigned long long next_big;  // the next frontier's queue sizes (record big, nlight)
  unsigned next_light;
};

// End of round L: the termination test of bool_pe.csl:1048-1100 (nf == 0 ends
// the search), the direction of round L + 1, and block 0's record of the
// round.  nf, mf, vd: the next frontier's vertices, their out-degrees and (in
// a pull round) in-degrees summed.  solo_max, solo_edges: the largest frontier
// block 0 takes alone.  heavy_work: kHeavyWork or the search's own.  Thread 0 of a
// block calls; returns the payload.
__device__ __forceinline__ unsigned close_round(const BfsParams &p, int L, int dir,
                                                unsigned long long nf, unsigned long long mf,
                                                unsigned long long vd, unsigned solo_max,
                                                unsigned solo_edges, unsigned long long heavy_work,
                                                SearchState &ss) {
  BfsCtl *ctl = p.ctl;
  ss.pull_rounds += dir == kPull ? 1 : 0;
  ss.visited += nf;
  bool done = nf == 0;
  bool capped = false;
  if (!done && L + 1 >= p.level_cap) {
    capped = true;
    done = true;
  }
  const int next = next_direction(p, dir, nf, ss.prev_nf, mf, ss.explored);
  ss.explored += vd;
  ss.prev_nf = nf;
  ss.switches += (!done && next != dir) ? 1 : 0;
  if (blockIdx.x == 0) {
    cg_stats *st = p.stats;
    const long long now = global_ns();
    if (L < CG_HISTORY) {
      st->nf_history[L] = (int64_t)nf;
      st->direction_history[L] = dir;
      st->round_ns[L] = now - ss.t_mark;
    }
    ss.t_mark = now;
    if (capped) atomicCAS(&ctl->status, 0, (int)CG_ERR_LEVEL_CAP);
    if (done) {
      const int rounds = L + 1;
      const int stat = *(volatile int *)&ctl->status;
      st->status = stat != 0 ? stat : (capped ? (int)CG_ERR_LEVEL_CAP : 0);
      st->rounds = rounds;
      st->visited = (int64_t)ss.visited;
      st->pull_rounds = ss.pull_rounds;
      st->switches = ss.switches;
      st->history_len = rounds < CG_HISTORY ? rounds : CG_HISTORY;
      st->finish_ns = 0;
      st->device_ms = 0.f;
    }
  }
  // a pull round's work is the unvisited vertices with in-edges, a push
  // round's (from the bitmap) its frontier
  const unsigned long long work =
      next == kPull ? (p.live > (int64_t)ss.visited ? (unsigned long long)p.live - ss.visited : 0ull)
                    : nf;
  const bool heavy = work >= heavy_work * (unsigned long long)((gridDim.x * blockDim.x) >> 5);
  // (after a pull round of a directed graph the edges are not known: vd stands
  // for them)
  const bool solo = !done && next == kPush && nf <= solo_max &&
                    (dir == kPull ? vd : mf) <= solo_edges;
  return (done ? kDone : 0u) | (next == kPull ? kNextPull : 0u) | (heavy ? kHeavy : 0u) |
         (solo ? kSolo : 0u);
}

// End of round L in warp 0 of every block, after the round's barrier.  Lanes
// 0-23 each load one sharded counter of the round record (one L2 round trip),
// lane 0 takes the decision (close_round), the same in every block.  All 32
// lanes call; lane 0's return value is the payload.
template <bool kTeamed, bool kWide>
__device__ unsigned round_decision(const BfsParams &p, int L, int dir, SearchState &ss) {
  BfsCtl *ctl = p.ctl;
  const RoundRec *Rn = &ctl->rec[(L + 1) % kRing];
  const int lane = lane_id();
  const int g = lane >> 3, sh = lane & (kCounterShards - 1);
  static_assert(kCounterShards == 8, "three groups of eight lanes");
  unsigned long long x = 0, q = 0;
  if (g == 0) x = __ldcg(&Rn->nf[sh]);
  else if (g == 1) x = __ldcg(&Rn->mf[sh]);
  else if (g == 2) x = __ldcg(&Rn->visdeg[sh]);
  // F_{L+1}'s queue sizes, for the next push round (same round trip)
  if (lane == 24) q = __ldcg(&Rn->big);
  else if (lane == 25) q = __ldcg(&Rn->nlight);
  const unsigned long long qbig = __shfl_sync(kFull, q, 24);
  const unsigned long long qlight = __shfl_sync(kFull, q, 25);
#pragma unroll
  for (int o = 1; o < kCounterShards; o <<= 1) x += __shfl_xor_sync(kFull, x, o);
  const unsigned long long nf = __shfl_sync(kFull, x, 0);
  const unsigned long long mf = __shfl_sync(kFull, x, 8);
  const unsigned long long vd = __shfl_sync(kFull, x, 16);
  if (lane != 0) return 0u;
  ss.next_light = (unsigned)qlight;
  if constexpr (kWide) {
    const unsigned long long edges = qbig & BigWord<true>::kEdges;
    ss.next_big = ((qbig >> BigWord<true>::kShift) << 32) | (uint32_t)edges;
    return close_round(p, L, dir, nf, mf, vd, 0u, 0u, kHeavyWork, ss) |
           (edges >= kEdges32 ? kUnqueued : 0u);
  }
  ss.next_big = qbig;
  // one block takes over well below what it can hold, so that a frontier near
  // the line does not go back and forth
  if constexpr (kTeamed) {
    // a team takes over where the frontier changes slowly (elsewhere it would be
    // handed out for a round or two)
    const bool steady = 4 * nf >= 3 * ss.prev_nf && 4 * nf <= 5 * ss.prev_nf;
    if (dir == kPush && steady && (nf > (unsigned)kSoloMax / 2 || mf > kSoloEnter) &&
        team_size()) {
      const unsigned x = close_round(p, L, dir, nf, mf, vd, kTeam * kSoloMax / 4, kTeamEdges / 2,
                                     kHeavyWork, ss);
      return (x & kSolo) ? x | kHandOver : x;
    }
  }
  return close_round(p, L, dir, nf, mf, vd, kSoloMax / 2, kSoloEnter,
                     kTeamed ? kHeavyWork : p.heavy_work, ss);
}

// ---- small rounds on one block -------------------------------------------------
// A grid-wide round costs 8 to 9 us however small its frontier is: the barrier
// and its decision, the bitmap sweep, and each step's trips through the L2.
// A frontier of a few hundred vertices is therefore expanded by block 0 alone,
// round after round, while the other blocks wait at one barrier: the frontier
// stays in shared memory, each edge takes one compare-and-swap on the target's
// level, which tells unvisited (-1), claimed this round (L + 1) and visited
// apart, and a round ends with a __syncthreads.  Measured per round: 2.5 us for
// 100 edges, 4 us for 1,000, 5.5 us for 2,000, 8.4 us for 4,000 (one SM makes
// about 1.4 scattered accesses a ns; gathering the targets in a shared hash
// table instead was no faster), against 8.5 to 9.5 us for a grid-wide round.
//
// Bitmaps: on entry the other blocks fold F_L into vis and clear all three
// frontier bitmaps; block 0 sets its claims in vis, and on exit, once every
// block has arrived (so the clearing is over), F_L in the current bitmap and
// the queue.  A run is cut into sessions of a quarter of the wait's time limit
// (SoloExit::still), so a deep graph does not run into it.
constexpr int kSoloSession = 256;  // rounds of a session, at most

__device__ __forceinline__ void solo_load(const BfsParams &p, SoloShared &S, unsigned i,
                                          int32_t v) {
  const int64_t o = __ldg(p.out_off + v);
  S.v[0][i] = v;
  S.s[0][i] = (uint32_t)o;
  S.d[0][i] = (uint32_t)(__ldg(p.out_off + v + 1) - o);
}

// S.x = the exclusive prefix of S.d[c][0 .. cnt); returns the total.  All
// threads call, synchronised; ends synchronised.
__device__ __forceinline__ uint32_t solo_scan(SoloShared &S, int c, unsigned cnt) {
  const int lane = lane_id(), wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t base = 0;
  for (unsigned i0 = 0; i0 < cnt; i0 += blockDim.x) {
    const unsigned i = i0 + threadIdx.x;
    const uint32_t d = i < cnt ? S.d[c][i] : 0u;
    uint32_t incl = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) S.warp_total[wib] = incl;
    __syncthreads();
    // every warp sums the totals of those before it
    const uint32_t w = lane < nw ? S.warp_total[lane] : 0u;
    const uint32_t before = __reduce_add_sync(kFull, lane < wib ? w : 0u);
    const uint32_t all = __reduce_add_sync(kFull, w);
    if (i < cnt) S.x[i] = base + before + incl - d;
    base += all;
    __syncthreads();
  }
  return base;
}

// Expands F_L (S.*[c], cnt vertices of E edges) into F_{L+1} (S.*[c ^ 1]; past
// kSoloMax vertices the rest goes to `spill`).  A thread's U edges go through
// every stage together: the searches' shared loads, the list entries, the
// claims and the claimed targets' list bounds are in flight at once.
template <bool kListed>
__device__ __forceinline__ void solo_expand(const BfsParams &p, SoloShared &S, int c, unsigned cnt,
                                            uint32_t E, int L, int32_t *spill) {
  constexpr int U = 4;  // edges a thread has in flight
  const int lane = lane_id();
  unsigned top = 1;     // search steps: top, top / 2, .. 1 cover cnt - 1
  while (2 * top < cnt) top *= 2;
  for (uint32_t base = 0; base < E; base += blockDim.x * U) {
    const uint32_t t0 = base + threadIdx.x;
    unsigned lo[U];
#pragma unroll
    for (int k = 0; k < U; ++k) lo[k] = 0;
    for (unsigned step = top; step > 0; step >>= 1) {  // the last entry whose prefix is <= t
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const unsigned m = lo[k] + step;
        if (m < cnt && S.x[m] <= t0 + k * blockDim.x) lo[k] = m;
      }
    }
    int32_t v[U], old[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint32_t t = t0 + k * blockDim.x;
      v[k] = t < E ? __ldg(p.out_idx + (S.s[c][lo[k]] + (t - S.x[lo[k]]))) : -1;
    }
#pragma unroll
    for (int k = 0; k < U; ++k)
      old[k] = v[k] >= 0 ? atomicCAS(p.levels + orig_id(p, v[k]), -1, L + 1) : 0;
    unsigned mine = 0;  // claims of this thread
    uint32_t s[U], d[U], edges = 0;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      s[k] = d[k] = 0;
      const bool claimed = old[k] == -1;
      if (claimed) {
        const int64_t o = __ldg(p.out_off + v[k]);
        d[k] = (uint32_t)(__ldg(p.out_off + v[k] + 1) - o);
        s[k] = (uint32_t)o;
        atomicOr(p.vis + ((uint32_t)v[k] >> 5), 1u << (v[k] & 31));
        ++mine;
      }
      if (claimed || old[k] == L + 1)
        atomicMin(reinterpret_cast<unsigned *>(p.parents) + orig_id(p, v[k]),
                  (unsigned)orig_id(p, S.v[c][lo[k]]));
    }
    // places in the next frontier: one shared atomic a warp
    unsigned before = 0, total = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const unsigned m = __ballot_sync(kFull, (mine >> b) & 1u);
      before += (unsigned)__popc(m & ((1u << lane) - 1u)) << b;
      total += (unsigned)__popc(m) << b;
    }
    static_assert(U < 8, "three bits of claims per thread");
    if (!total) continue;
#pragma unroll
    for (int k = 0; k < U; ++k) edges += d[k];
    edges = __reduce_add_sync(kFull, edges);
    unsigned at = 0;
    if (lane == 0) {
      at = atomicAdd(&S.n, total);
      atomicAdd(&S.mf, edges);
    }
    at = __shfl_sync(kFull, at, 0) + before;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (old[k] != -1) continue;
      if (at < (unsigned)kSoloMax) {
        S.v[c ^ 1][at] = v[k];
        S.s[c ^ 1][at] = s[k];
        S.d[c ^ 1][at] = d[k];
      } else {
        spill[kListed ? atomicAdd(&p.ctl->team.listed, 1u) : at] = v[k];
      }
      ++at;
    }
  }
}

// ---- small rounds on a team of blocks -----------------------------------------
// One SM makes about 1.5 requests a ns past its L1, so that a grid graph's
// round of 2,400 edges takes the lead block 7 us, 2.5 of it latency.  Sixteen
// blocks share such rounds: each keeps the vertices it claims in its own shared
// memory (the compare-and-swap on the level is the same), and a round ends with
// one wait on a sum that carries the frontier's totals, about 2.5 us.  The
// lead hands its frontier out as a list in memory and gets one back, at least
// every kTeamSession rounds, which also evens out the shares.  A search of a
// 1000^2 grid 9.9 -> 6.8 ms, of a 4000^2 grid 51.4 -> 42.7 ms; three handles
// taking turns on a 1000^2 grid 5.5 -> 3.3 ms a search (with 4 blocks 4.7, 8 3.95,
// 12 3.7, 16 3.55, 24 3.5, all with 512 threads a block).
// This block's place in the team (the lead's is 0), kTeam or more outside it.
// Members are spread over the grid: neighbours may share an SM.
__device__ __forceinline__ unsigned team_rank() {
  const unsigned stride = gridDim.x / kTeam;
  return team_size() && blockIdx.x % stride == 0 ? blockIdx.x / stride : kTeam;
}
__device__ __forceinline__ bool in_team() { return team_rank() < kTeam; }

// F_L's list while the team runs: the queue that F_L is not put in.
__device__ __forceinline__ int32_t *team_list(const BfsParams &p, int L) {
  return (L & 1) ? p.queue0 : p.queue1;
}

// Bounded wait of thread 0 until *at satisfies `ready`; its value, or ~0 after
// the time limit (or another block's error).
template <class Ready>
__device__ __forceinline__ unsigned long long team_wait(const unsigned long long *at, int *status,
                                                        long long timeout_ns, Ready ready) {
  long long t0 = 0;
  unsigned spins = 0;
  unsigned long long x;
  while (true) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(at) : "memory");
    if (ready(x)) break;
    if ((++spins & 255u) == 0) {
      if (t0 == 0) t0 = global_ns();
      if (*(volatile int *)status != 0 || global_ns() - t0 > timeout_ns) {
        atomicCAS(status, 0, (int)CG_ERR_TIMEOUT);
        return ~0ull;
      }
    }
  }
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  return x;
}

// The team's rounds from L on, its frontier the first cnt entries of
// team_list(L).  Every block of the team calls with the same ss, and all take
// the same decisions from the sums of TeamRound; ends with the frontier of the
// round to run next listed again.  Returns its payload (all threads), with the
// frontier's edges (saturated) and L in S.warp_total[1] and [2].
__device__ __noinline__ unsigned team_rounds(const BfsParams &p, SearchState &ss, unsigned cnt,
                                             int L) {
  SoloShared &S = s_round.solo;
  TeamCtl *T = &p.ctl->team;
  const unsigned team = team_size(), rank = team_rank();
  const bool leader = threadIdx.x == 0;
  // sum: 8 bits of arrivals, the lead's word that the session's time is over, 7
  // bits of blocks that overflowed, 8 of blocks with too
  // many out-degrees for their 20 bits, 23 of out-degrees, 17 of vertices
  constexpr unsigned kMfBits = 23, kNfBits = 17;
  static_assert(kTeamEdges < (1u << kNfBits), "a round's claims fit");
  static_assert(kMfBits + kNfBits <= 40, "flags above");
  const unsigned lo = (unsigned)((unsigned long long)cnt * rank / team);
  unsigned mine = (unsigned)((unsigned long long)cnt * (rank + 1) / team) - lo;
  {
    const int32_t *list = team_list(p, L) + lo;
    for (unsigned i = threadIdx.x; i < mine; i += blockDim.x) solo_load(p, S, i, __ldcg(list + i));
  }
  __syncthreads();
  int c = 0;
  unsigned payload;
  for (int ran = 1;; ++ran) {
    const uint32_t E = solo_scan(S, c, mine);
    if (leader) S.n = S.mf = 0;
    __syncthreads();
    solo_expand<true>(p, S, c, mine, E, L, team_list(p, L + 1));
    __syncthreads();
    if (leader) {
      const unsigned nf = S.n, mf = S.mf;
      const bool over = nf > (unsigned)kSoloMax, many = mf >= (1u << kMfBits) / kTeam;
      TeamRound *R = &T->round[L & 3];
      if (rank == 0) {  // its readers were done before the last round's arrivals
        TeamRound *Z = &T->round[(L + 2) & 3];
        Z->sum = Z->mf = 0;
      }
      if (many) atomicAdd(&R->mf, (unsigned long long)mf);
      const bool late = rank == 0 && ss.t_mark - ss.t_session > p.timeout_ns / 4;
      const unsigned long long add = (1ull << 56) | ((unsigned long long)late << 55) |
                                     ((unsigned long long)over << 48) |
                                     ((unsigned long long)many << 40) |
                                     ((unsigned long long)(many ? 0u : mf) << kNfBits) | nf;
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&R->sum), "l"(add) : "memory");
      const unsigned long long x =
          team_wait(&R->sum, &p.ctl->status, p.timeout_ns,
                    [&](unsigned long long s) { return (unsigned)(s >> 56) >= team; });
      unsigned pay = kWaitFailed;
      if (x != ~0ull) {
        const unsigned long long nfs = x & ((1ull << kNfBits) - 1);
        unsigned long long mfs = (x >> kNfBits) & ((1ull << kMfBits) - 1);
        if ((x >> 40) & 0xffu) mfs += __ldcg(&R->mf);
        const bool lists_fit = ((x >> 48) & 0x7fu) == 0;
        pay = close_round(p, L, kPush, nfs, mfs, mfs, lists_fit ? kTeam * kSoloMax / 2 : 0u,
                          kTeamEdges, kHeavyWork, ss);
        S.d[c][0] = (uint32_t)min(mfs, 0xffffffffull);  // F_L's degrees are done with
        // hand back what one block runs faster, and before the waits' time limit
        S.x[0] = (mfs < kTeamLeave && nfs <= (unsigned)kSoloMax / 2) || ((x >> 55) & 1u);
      }
      S.payload = pay;
    }
    __syncthreads();
    payload = S.payload;
    const uint32_t mf = S.d[c][0];
    const bool back = S.x[0] != 0;
    mine = min(S.n, (unsigned)kSoloMax);
    c ^= 1;
    ++L;
    __syncthreads();  // S is read
    if (payload == kWaitFailed || !(payload & kSolo) || back || ran >= kTeamSession) {
      if (leader) {
        S.warp_total[1] = mf;
        S.warp_total[2] = (uint32_t)L;
      }
      break;
    }
  }
  if (payload == kWaitFailed) return payload;
  // list what this block claimed (past kSoloMax it is listed already)
  if (leader) S.n = atomicAdd(&T->listed, mine);
  __syncthreads();
  int32_t *list = team_list(p, L) + S.n;
  for (unsigned i = threadIdx.x; i < mine; i += blockDim.x) list[i] = S.v[c][i];
  __syncthreads();
  return payload;
}

// The lead's side of one hand-over: F_L (cnt vertices) is in team_list(L).
// Returns the payload, with the next frontier's vertices, edges and round in
// S.warp_total[0 .. 2].
__device__ __noinline__ unsigned team_lead(const BfsParams &p, SearchState &ss, unsigned cnt, int L) {
  SoloShared &S = s_round.solo;
  BfsCtl *ctl = p.ctl;
  TeamCtl *T = &ctl->team;
  if (threadIdx.x == 0) {
    SoloExit *x = &ctl->solo;
    x->visited = ss.visited;
    x->prev_nf = ss.prev_nf;
    x->explored = ss.explored;
    x->pull_rounds = ss.pull_rounds;
    x->switches = ss.switches;
    T->L = L;
    T->cnt = cnt;
    T->listed = T->back = 0;
    // the first round's record; the second's is cleared by the first, and so on
    for (int k = 0; k < 2; ++k) T->round[(L + k) & 3].sum = T->round[(L + k) & 3].mf = 0;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&T->command) : "memory");
  }
  __syncthreads();
  const unsigned payload = team_rounds(p, ss, cnt, L);
  if (payload == kWaitFailed || (payload & kDone)) return payload;
  if (threadIdx.x == 0) {
    // every member's part of the list is written
    const unsigned others = team_size() - 1;
    const unsigned long long x = team_wait(
        reinterpret_cast<const unsigned long long *>(&T->listed), &ctl->status, p.timeout_ns,
        [&](unsigned long long w) { return (unsigned)(w >> 32) >= others; });
    S.warp_total[0] = (unsigned)x;
    S.payload = x == ~0ull ? kWaitFailed : payload;
  }
  __syncthreads();
  return S.payload;
}

// A member's side of the lead block's run of small rounds: arrives at the
// run's grid-wide waits, and serves the lead's commands while it waits.
// False after a time limit (all threads).
__device__ __noinline__ bool team_member(const BfsParams &p, SearchState &ss,
                                         unsigned long long &target, unsigned &commands) {
  SoloShared &S = s_round.solo;
  BfsCtl *ctl = p.ctl;
  TeamCtl *T = &ctl->team;
  enum : unsigned { kPassed, kCommand, kFailed };
  bool arrive = true;
  while (true) {
    if (threadIdx.x == 0) {
      if (arrive) {
        target += gridDim.x;
        flat_arrive(&ctl->arrive);
      }
      const unsigned long long goal = target;
      const unsigned seen = commands;
      unsigned got = kFailed, spins = 0;
      long long t0 = 0;
      while (true) {
        unsigned long long a;
        unsigned w;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(&ctl->arrive) : "memory");
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w) : "l"(&T->command) : "memory");
        if (w != seen) { got = kCommand; break; }
        if (a >= goal) { got = kPassed; break; }
        __nanosleep(50);
        if ((++spins & 255u) == 0) {
          if (t0 == 0) t0 = global_ns();
          if (*(volatile int *)&ctl->status != 0 || global_ns() - t0 > p.timeout_ns) {
            atomicCAS(&ctl->status, 0, (int)CG_ERR_TIMEOUT);
            break;
          }
        }
      }
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      if (got == kCommand) {
        const SoloExit *x = &ctl->solo;
        commands = seen + 1;
        ss.visited = __ldcg(&x->visited);
        ss.prev_nf = __ldcg(&x->prev_nf);
        ss.explored = __ldcg(&x->explored);
        ss.pull_rounds = __ldcg(&x->pull_rounds);
        ss.switches = __ldcg(&x->switches);
        S.n = __ldcg(&T->cnt);
        S.mf = (unsigned)__ldcg(&T->L);
      }
      // a wait of a run that goes on: the next one
      S.payload = got == kPassed && __ldcg(&ctl->solo.still) != 0 ? ~0u : got;
    }
    __syncthreads();
    const unsigned got = S.payload, cnt = S.n;
    const int L = (int)S.mf;
    __syncthreads();
    arrive = got == ~0u;
    if (arrive) continue;
    if (got != kCommand) return got == kPassed;
    if (team_rounds(p, ss, cnt, L) == kWaitFailed) return false;
    if (threadIdx.x == 0)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&T->back) : "memory");
  }
}

// Block 0's run of small rounds from round L on, its frontier in S.*[0] (cnt
// vertices, loaded and synchronised).  Ends with SoloExit written and the
// barrier arrived at; returns the payload of the round to run next (every
// thread), L being that round.
template <bool kTeamed>
__device__ __forceinline__ unsigned solo_rounds(const BfsParams &p, SoloShared &S, SearchState &ss,
                                                unsigned long long &target, unsigned cnt, int &L,
                                                uint32_t *cur, unsigned payload) {
  BfsCtl *ctl = p.ctl;
  const bool leader = threadIdx.x == 0;
  const long long session_ns = p.timeout_ns / 4;
  long long t0 = leader ? global_ns() : 0;
  int c = 0, ran = 0;
  [[maybe_unused]] int large = 0;  // rounds in a row of more than kTeamEnter edges
  // F_L is in team_list(L), not in S
  [[maybe_unused]] bool listed = kTeamed && (payload & kHandOver);
  uint32_t E = 0;
  bool stay = false;
  if (!listed) {
    payload = 0;
    E = solo_scan(S, c, cnt);
    // a first frontier whose edges were not known may hold too many
    stay = E <= kSoloEdges;
  }
  while (true) {
    while (stay) {
      if (leader) S.n = S.mf = 0;
      __syncthreads();
      // what does not fit goes to the queue F_{L+1} is not put in
      solo_expand<false>(p, S, c, cnt, E, L, (L & 1) ? p.queue1 : p.queue0);
      __syncthreads();
      if (leader) {
        const unsigned nf = S.n, mf = S.mf;
        // a frontier that more than doubled is left to the grid: the next one
        // would be too large anyway, and the lists of new parts of the graph are
        // cold (directed ER, 3,363 claims from 3,320 edges: 17 us here, 11 there)
        const unsigned room = min(kSoloEdges, max(kSoloEdges / 4, 2 * E));
        unsigned x = close_round(p, L, kPush, nf, mf, mf, kSoloMax, room,
                                 kTeamed ? kHeavyWork : p.heavy_work, ss);
        if ((x & kSolo) && (++ran >= kSoloSession || ss.t_mark - t0 > session_ns)) {
          // the waiting blocks' time limit: let them through to the next wait
          ctl->solo.still = 1;
          target += gridDim.x;
          flat_arrive(&ctl->arrive);
          ran = 0;
          t0 = ss.t_mark;
        }
        if constexpr (kTeamed) {
          large = mf > kTeamEnter ? large + 1 : 0;
          if ((x & kSolo) && large >= kTeamAfter && team_size()) {
            x |= kHandOver;
            large = 0;
          }
        }
        S.payload = x;
      }
      __syncthreads();
      payload = S.payload;
      cnt = S.n;
      c ^= 1;
      ++L;
      stay = (payload & (kSolo | kHandOver)) == kSolo;
      if (stay) E = solo_scan(S, c, cnt);
    }
    if constexpr (!kTeamed) {
      break;
    } else {
      if (!(payload & kHandOver)) break;
      if (!listed) {
        int32_t *list = team_list(p, L);
        for (unsigned i = threadIdx.x; i < cnt; i += blockDim.x) list[i] = S.v[c][i];
        listed = true;
      }
      do {
        if (leader) ss.t_session = t0;
        __syncthreads();
        payload = team_lead(p, ss, cnt, L);
        if (payload == kWaitFailed) return kWaitFailed;
        cnt = S.warp_total[0];
        E = S.warp_total[1];
        L = (int)S.warp_total[2];
        if (leader && (payload & kSolo) && ss.t_mark - t0 > session_ns) {
          ctl->solo.still = 1;
          target += gridDim.x;
          flat_arrive(&ctl->arrive);
          ran = 0;
          t0 = ss.t_mark;
        }
      } while ((payload & kSolo) && !(E < kTeamLeave && cnt <= (unsigned)kSoloMax / 2));
      if (!(payload & kSolo)) break;
      // small again: back to this block alone
      const int32_t *list = team_list(p, L);
      c = 0;
      for (unsigned i = threadIdx.x; i < cnt; i += blockDim.x) solo_load(p, S, i, __ldcg(list + i));
      __syncthreads();
      E = solo_scan(S, c, cnt);
      listed = false;
      stay = true;
    }
  }
  payload &= ~(kSolo | kHandOver);
  // every other block has arrived: the bitmaps are clear, the records unread
  if (leader)
    S.payload = flat_wait(&ctl->arrive, target + gridDim.x - 1, &ctl->status, p.timeout_ns)
                    ? payload
                    : kWaitFailed;
  __syncthreads();
  if (S.payload == kWaitFailed) return kWaitFailed;
  if (!(payload & kDone)) {
    unsigned long long *z = reinterpret_cast<unsigned long long *>(ctl->rec);
    for (int i = threadIdx.x; i < (int)(sizeof(RoundRec) * kRing / 8); i += blockDim.x) z[i] = 0ull;
    __syncthreads();
    RoundRec *R = &ctl->rec[L % kRing];
    const int32_t *spill = (L & 1) ? p.queue0 : p.queue1;
    Acc unused;
    for (unsigned i0 = 0; i0 < cnt; i0 += blockDim.x) {
      const unsigned i = i0 + threadIdx.x;
      const bool has = i < cnt;
      int32_t v = 0;
      int64_t d = 0;
      if (has) {
        if constexpr (kTeamed)
          v = !listed && i < (unsigned)kSoloMax ? S.v[c][i] : __ldcg(spill + i);
        else
          v = i < (unsigned)kSoloMax ? S.v[c][i] : spill[i];
        d = __ldg(p.out_off + v + 1) - __ldg(p.out_off + v);
        atomicOr(cur + ((uint32_t)v >> 5), 1u << (v & 31));
      }
      enqueue_claims(p, has, v, d, L & 1, R, unused);
    }
    __syncthreads();
    if (leader) {
      ss.next_big = __ldcg(&R->big);
      ss.next_light = __ldcg(&R->nlight);
    }
  }
  if (leader) {
    SoloExit *x = &ctl->solo;
    x->visited = ss.visited;
    x->prev_nf = ss.prev_nf;
    x->explored = ss.explored;
    x->next_big = ss.next_big;
    x->next_light = ss.next_light;
    x->pull_rounds = ss.pull_rounds;
    x->switches = ss.switches;
    x->L = L;
    x->payload = payload;
    x->listed = 0;
    x->still = 0;
    target += gridDim.x;
    flat_arrive(&ctl->arrive);
  }
  return payload;
}

// Folds F_L (bitmap cur) into vis and clears cur and old (F_{L-1}), blocks
// b0 .. of the grid sharing the words.  `list`: also append F_L's vertices to
// it (SoloExit::listed counts them).
__device__ __forceinline__ void solo_fold(const BfsParams &p, uint32_t *cur, uint32_t *old,
                                          unsigned b0, int32_t *list) {
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  const int64_t nthreads = (int64_t)(gridDim.x - b0) * blockDim.x;
  for (int64_t i = (int64_t)(blockIdx.x - b0) * blockDim.x + threadIdx.x;
       i < p.tiles * (kTileWords / 4); i += nthreads) {
    const uint4 c = ld4(cur + 4 * i);
    st4(old + 4 * i, zero4);
    if (!any4(c)) continue;
    st4(cur + 4 * i, zero4);
    const uint32_t w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!w[k]) continue;
      atomicOr(p.vis + 4 * i + k, w[k]);  // block 0 may be adding claims to it
      if (!list) continue;
      unsigned at = atomicAdd(&p.ctl->solo.listed, (unsigned)__popc(w[k]));
      for (uint32_t m = w[k]; m; m &= m - 1)
        list[at++] = (int32_t)((4 * i + k) * 32 + __ffs(m) - 1);
    }
  }
}

// A host caller's outputs, copied by every block into the page-locked
// buffers (16 bytes a thread when n allows).  Kept out of line so the search
// loop's registers are not shared with it.
__device__ __noinline__ void copy_to_host(const BfsParams &p) {
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int a = 0; a < 2; ++a) {
    const int32_t *src = a ? p.parents : p.levels;
    int32_t *dst = a ? p.host_parents : p.host_levels;
    if (!dst) continue;
    if ((p.n & 3) == 0) {
      const int4 *s4 = reinterpret_cast<const int4 *>(src);
      int4 *d4 = reinterpret_cast<int4 *>(dst);
      for (int64_t i = t0; i < (p.n >> 2); i += step) d4[i] = s4[i];
    } else {
      for (int64_t i = t0; i < p.n; i += step) dst[i] = src[i];
    }
  }
}

template <bool kTeamed, bool kWide>
__device__ __forceinline__ void search(const BfsParams &p) {
  __shared__ unsigned s_payload;
  __shared__ int s_L;
  BfsCtl *ctl = p.ctl;
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  // the root in original ids (output positions) and as a resident vertex
  const int32_t root_out = (int32_t)p.root;
  const int32_t root = p.perm ? __ldg(p.perm + p.root) : root_out;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;

  // ---- phase 0: start_spmv -- reset outputs and bitmaps, seed the root ----
  __shared__ SearchState ss;  // thread 0's copy of the search-wide bookkeeping
  if (leader) ss.t_mark = global_ns();
  for (int64_t i = gtid; i < p.n; i += nthreads) {
    p.levels[i] = (i == root_out) ? 0 : -1;
    p.parents[i] = (i == root_out) ? root_out : -1;
  }
  // whole tiles (the padding past `words` too: a bitmap-wide round reads it)
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  const int64_t root_word = root >> 5;
  // a root of few edges starts on block 0 alone: it is in vis then, and the
  // frontier bitmaps are clear
  const int64_t root_deg = __ldg(p.out_off + root + 1) - __ldg(p.out_off + root);
  bool solo = !kWide && root_deg <= (int64_t)kSoloEnter;
  for (int64_t i = gtid; i < p.tiles * (kTileWords / 4); i += nthreads) {
    uint4 f0 = zero4;
    if (i == (root_word >> 2)) {  // F_0 = {root}, seeded by the thread that clears its word
      const uint32_t bit = 1u << (root & 31);
      const int c = (int)(root_word & 3);
      f0 = make_uint4(c == 0 ? bit : 0u, c == 1 ? bit : 0u, c == 2 ? bit : 0u, c == 3 ? bit : 0u);
    }
    st4(p.vis + 4 * i, solo ? f0 : zero4);
    st4(p.fr0 + 4 * i, solo ? zero4 : f0);
    st4(p.fr1 + 4 * i, zero4);
    st4(p.fr2 + 4 * i, zero4);
  }
  if (leader) {
    const int64_t deg = p.out_off[root + 1] - p.out_off[root];
    RoundRec *R0 = &ctl->rec[0];
    R0->nf[0] = 1;
    R0->mf[0] = deg;
    R0->visdeg[0] = deg;
    if (deg <= kLightMax) {
      p.queue0[0] = root;
      R0->nlight = 1;
    } else {
      p.queue0[p.n - 1] = root;
      p.bigoff0[0] = 0;
      R0->big = BigWord<kWide>::pack(1, (unsigned)deg);
    }
  }
  // barrier b of this launch completes at (b + 1) * gridDim.x arrivals
  __shared__ unsigned long long s_target;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long target = gridDim.x;
    s_target = target;
    if constexpr (kTeamed) s_commands = 0;
    // the test hook expects one arrival more than the grid has: it must time out
    const bool ok0 = flat_barrier(&ctl->arrive, target + (p.unmatched_wait ? 1u : 0u),
                                  &ctl->status, p.timeout_ns);
    ss.visited = 1;
    ss.prev_nf = 1;
    ss.explored = (unsigned long long)(__ldg(p.out_off + root + 1) - __ldg(p.out_off + root));
    ss.pull_rounds = 0;
    ss.switches = 0;
    // F_0 = {root}: queued light or big by its degree (phase 0 above)
    ss.next_big = ss.explored > (unsigned long long)kLightMax ? ((1ull << 32) | ss.explored) : 0ull;
    ss.next_light = ss.explored > (unsigned long long)kLightMax ? 0u : 1u;
    if (blockIdx.x == 0 && ok0) {
      const long long now = global_ns();
      p.stats->setup_ns = now - ss.t_mark;
      ss.t_mark = now;
    }
    s_payload = ok0 ? 0u : kWaitFailed;
  }
  __syncthreads();
  bool ok = s_payload != kWaitFailed;

  uint32_t *fr0 = p.fr0, *fr1 = p.fr1, *fr2 = p.fr2;
  int dir = kPush;
  bool heavy = false;
  [[maybe_unused]] bool hand = false;  // a small round for the team
  bool queued = true;  // F_L is in a queue (a pull round leaves it in the bitmap only)
  int L = 0;
  Acc acc;
  while (ok) {
    if (!kWide && solo) {
      // L = 0: the root alone, in vis already (phase 0)
      const bool fold = L > 0, from_queue = L > 0 && queued;
      if (fold && !queued) {
        // the frontier is in the bitmap only: all blocks list it first
        solo_fold(p, fr0, fr2, 0, p.queue0);
        __syncthreads();
        if (threadIdx.x == 0) {
          const unsigned long long target = s_target + gridDim.x;
          s_target = target;
          s_payload = flat_barrier(&ctl->arrive, target, &ctl->status, p.timeout_ns)
                          ? 0u : kWaitFailed;
        }
        __syncthreads();
        if (s_payload == kWaitFailed) break;
      } else if (fold && (blockIdx.x > 0 || gridDim.x == 1)) {
        solo_fold(p, fr0, fr2, gridDim.x == 1 ? 0 : 1, nullptr);
      }
      __syncthreads();
      if (blockIdx.x == 0) {
        SoloShared &S = s_round.solo;
        unsigned cnt = 1;
        if (from_queue) {
          const int32_t *q = (L & 1) ? p.queue1 : p.queue0;
          const unsigned nl = ss.next_light, nb = (unsigned)(ss.next_big >> 32);
          cnt = nl + nb;  // at most kSoloMax / 2 (kTeam * kSoloMax / 4 handed over)
          int32_t *list = team_list(p, L);
          for (unsigned i = threadIdx.x; i < cnt; i += blockDim.x) {
            const int32_t v = i < nl ? q[i] : q[p.n - 1 - (int64_t)(i - nl)];
            if (kTeamed && hand)
              list[i] = v;
            else
              solo_load(p, S, i, v);
          }
        } else if (fold) {
          cnt = __ldcg(&ctl->solo.listed);
          for (unsigned i = threadIdx.x; i < cnt; i += blockDim.x)
            solo_load(p, S, i, p.queue0[i]);
        } else if (threadIdx.x == 0) {
          solo_load(p, S, 0, root);
        }
        __syncthreads();
        const unsigned payload = solo_rounds<kTeamed>(p, S, ss, s_target, cnt, L, fr0, hand ? kHandOver : 0u);
        if (threadIdx.x == 0) s_payload = payload;
        __syncthreads();
      } else {
        if (kTeamed && in_team()) {
          // (ends with the last wait of the run still to make)
          const bool served = team_member(p, ss, s_target, s_commands);
          __syncthreads();
          if (!served) {
            if (threadIdx.x == 0) s_payload = kWaitFailed;
            __syncthreads();
            break;
          }
        }
        if (threadIdx.x == 0) {
          const SoloExit *x = &ctl->solo;
          bool arrived = true;
          if (!(kTeamed && in_team())) do {
            const unsigned long long target = s_target + gridDim.x;
            s_target = target;
            flat_arrive(&ctl->arrive);
            arrived = flat_wait(&ctl->arrive, target, &ctl->status, p.timeout_ns, 100);
          } while (arrived && __ldcg(&x->still) != 0);
          unsigned payload = kWaitFailed;
          if (arrived) {
            ss.visited = __ldcg(&x->visited);
            ss.prev_nf = __ldcg(&x->prev_nf);
            ss.explored = __ldcg(&x->explored);
            ss.next_big = __ldcg(&x->next_big);
            ss.next_light = __ldcg(&x->next_light);
            ss.pull_rounds = __ldcg(&x->pull_rounds);
            ss.switches = __ldcg(&x->switches);
            s_L = __ldcg(&x->L);
            payload = __ldcg(&x->payload);
          }
          s_payload = payload;
        }
        __syncthreads();
        L = s_L;
      }
      const unsigned payload = s_payload;
      if (payload == kWaitFailed || (payload & kDone)) break;
      queued = true;
      dir = (payload & kNextPull) ? kPull : kPush;
      heavy = (payload & kHeavy) != 0;
      solo = false;
      __syncthreads();
      // all three bitmaps were cleared; fr0 holds F_L
    }
    RoundRec *Rc = &ctl->rec[L % kRing];
    RoundRec *Rn = &ctl->rec[(L + 1) % kRing];
    const uint32_t *cur = fr0;  // F_L
    uint32_t *nxt = fr1;        // F_{L+1}
    uint32_t *old = fr2;        // F_{L-1}
    if (dir == kPush) {
      if (queued)
        push_round_queue<kWide>(p, cur, nxt, L, Rc, Rn, ss.next_big, ss.next_light, acc);
      else
        push_round_bitmap<kWide>(p, cur, nxt, L, Rc, Rn, heavy, acc);
      // vis |= F_L (readers test vis | F_L, so this races with nothing) and
      // clear F_{L-1}, which becomes the next round's output bitmap; a pull
      // round does both in its own tile pass
      for (int64_t i = gtid; i < p.tiles * (kTileWords / 4); i += nthreads) {
        const uint4 c = ld4(cur + 4 * i), vv = ld4(p.vis + 4 * i);
        if (any4(c))
          st4(p.vis + 4 * i, make_uint4(vv.x | c.x, vv.y | c.y, vv.z | c.z, vv.w | c.w));
        st4(old + 4 * i, zero4);
      }
    } else {
      pull_round(p, cur, nxt, old, L, Rc, heavy, acc);
    }
    unsigned long long a, b, c;
    block_totals(acc, a, b, c);
    if (threadIdx.x < 32) {
      bool arrived = false;
      if (threadIdx.x == 0) {
        const int sh = blockIdx.x % kCounterShards;
        if (a) atomicAdd(&Rn->nf[sh], a);
        if (b) atomicAdd(&Rn->mf[sh], b);
        if (c) atomicAdd(&Rn->visdeg[sh], c);
        if (blockIdx.x == 0) {
          // the record round L + 1 accumulates into next: its last readers were
          // done before the barrier of round L - 2 (ordered by this arrival)
          RoundRec *Rz = &ctl->rec[(L + 2) % kRing];
          for (int i = 0; i < kCounterShards; ++i) Rz->nf[i] = Rz->mf[i] = Rz->visdeg[i] = 0;
          Rz->big = 0;
          Rz->nlight = Rz->work = 0;
        }
        const unsigned long long target = s_target + gridDim.x;
        s_target = target;
        arrived = flat_barrier(&ctl->arrive, target, &ctl->status, p.timeout_ns);
      }
      // lane 0's acquire fence, then this warp barrier, order the other lanes'
      // counter loads after every block's arrival
      arrived = __shfl_sync(kFull, arrived, 0);
      const unsigned payload = arrived ? round_decision<kTeamed, kWide>(p, L, dir, ss) : kWaitFailed;
      if (threadIdx.x == 0) s_payload = payload;
    }
    __syncthreads();
    const unsigned payload = s_payload;
    if (payload == kWaitFailed || (payload & kDone)) break;
    queued = dir == kPush;  // a push round queued F_{L+1}; a pull round did not
    if constexpr (kWide) queued = queued && !(payload & kUnqueued);
    dir = (payload & kNextPull) ? kPull : kPush;
    heavy = (payload & kHeavy) != 0;
    solo = (payload & kSolo) != 0;
    if constexpr (kTeamed) hand = (payload & kHandOver) != 0;
    uint32_t *t = fr2;  // rotate: F_{L+1} becomes the frontier
    fr2 = fr0;
    fr0 = fr1;
    fr1 = t;
    ++L;
  }
  if (leader && s_payload == kWaitFailed) p.stats->status = *(volatile int *)&ctl->status;
  // after the last wait every output is final
  if (s_payload != kWaitFailed && (p.host_levels || p.host_parents)) copy_to_host(p);
}

__global__ void __launch_bounds__(kBfsBlock, 3) bfs_persistent(BfsParams p) {
  search<false, false>(p);
}

// The same search without small rounds on one block, its list positions in 64
// bits: graphs of kEdges32 entries and more.
__global__ void __launch_bounds__(kBfsBlock, 3) bfs_persistent_wide(BfsParams p) {
  search<false, true>(p);
}

// The same search with rounds that a team runs.  A kernel of its own, so that
// the other keeps its registers (with the team in it R-MAT and random graphs took
// 2 to 3% longer), and of fewer threads, so that it has 56 (one is spilled)
// and three handles' blocks still fit an SM: 512 threads and 64 registers are as fast
// for one handle, 4.6 ms a search for three taking turns where this takes 3.3.
__global__ void __launch_bounds__(kTeamBlock, 3) bfs_persistent_team(BfsParams p) {
  search<true, false>(p);
}

// A vertex's share of Graph500's m (bfs_timing.py:379-398): its entries c <= v
// (row v of a symmetric A is ascending: a binary search), or its out-degree.
__device__ __forceinline__ unsigned edge_weight(int64_t v, int symmetric,
                                                const int64_t *__restrict__ in_off,
                                                const int32_t *__restrict__ in_idx,
                                                const int64_t *__restrict__ out_off) {
  if (!symmetric) return (unsigned)(out_off[v + 1] - out_off[v]);
  const int64_t first = in_off[v];
  int64_t lo = first, hi = in_off[v + 1];
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (in_idx[mid] <= v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return (unsigned)(lo - first);
}

__global__ void edge_weight_kernel(int64_t n, int symmetric, const int64_t *__restrict__ in_off,
                                   const int32_t *__restrict__ in_idx,
                                   const int64_t *__restrict__ out_off, uint32_t *w) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) w[v] = edge_weight(v, symmetric, in_off, in_idx, out_off);
}

// m per search: the reached vertices' weights, kCountGroup searches
// (blockIdx.y) at a time.  The weights are the graph's, the same in every
// search, and kept with it (`w`; null when there was no memory for them: then
// they are found here).  A sum of weights stays below nnz < 2^32.  The rest is
// one read of the levels.  R-MAT scale 20, 16 searches: 158 us with a
// search per vertex and search, 64 us with kept weights, 21 us now.
constexpr int kCountGroup = 16;
__global__ void __launch_bounds__(256) count_edges_kernel(
    int64_t n, int k, int symmetric, const int64_t *__restrict__ in_off,
    const int32_t *__restrict__ in_idx, const int64_t *__restrict__ out_off,
    const uint32_t *__restrict__ w, const int32_t *__restrict__ levels,
    unsigned long long *m_out) {
  const int s0 = (int)blockIdx.y * kCountGroup;
  const int ks = min(kCountGroup, k - s0);
  levels += (int64_t)s0 * n;
  unsigned local[kCountGroup];
#pragma unroll
  for (int s = 0; s < kCountGroup; ++s) local[s] = 0;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (int64_t)gridDim.x * blockDim.x) {
    int32_t lv[kCountGroup];
#pragma unroll
    for (int s = 0; s < kCountGroup; ++s)
      lv[s] = s < ks ? __ldg(levels + (int64_t)s * n + v) : -1;
    const unsigned x = w ? __ldg(w + v) : edge_weight(v, symmetric, in_off, in_idx, out_off);
#pragma unroll
    for (int s = 0; s < kCountGroup; ++s)
      if (lv[s] >= 0) local[s] += x;
  }
  // (32 bits hold the sums: a search's m is at most nnz.)  One atomic a block and
  // search, a block's in one request: the totals share a line, and one from each
  // warp, about 1 ns apart, took 43 of the 64 us
  __shared__ unsigned part[8][kCountGroup];
#pragma unroll
  for (int s = 0; s < kCountGroup; ++s) {
    const unsigned x = __reduce_add_sync(kFull, local[s]);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][s] = x;
  }
  __syncthreads();
  if (threadIdx.x < (unsigned)ks) {
    unsigned x = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) x += part[i][threadIdx.x];
    if (x) atomicAdd(m_out + s0 + threadIdx.x, (unsigned long long)x);
  }
}

int64_t bfs_big_capacity(int64_t n, int64_t nnz) {
  const int64_t c = nnz / (kLightMax + 1) + 1;
  return c < n ? c : n;
}

// Bit v of dead[v / 32]: vertex v has no in-edges, so no round reaches it
// (bits past n are set too, through the tile padding: `words` = stride).  A
// warp takes 32 words, a coalesced load of 33 offsets each.  *live: vertices
// with in-edges.
// hub_edges: entries of vertices of in-degree > kLightMax.
__global__ void dead_map_kernel(int64_t n, int64_t words, const int64_t *__restrict__ in_off,
                                uint32_t *dead, unsigned long long *live,
                                unsigned long long *hub_edges, unsigned long long *wide_edges) {
  const int lane = lane_id();
  unsigned long long alive = 0, hubs = 0, wide = 0;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w0 = (int64_t)warp_id_global() * 32; w0 < words; w0 += warps * 32) {
    uint32_t mine = 0;
    for (int j = 0; j < 32 && w0 + j < words; ++j) {
      const int64_t v = (w0 + j) * 32 + lane;
      const int64_t d = v < n ? __ldg(in_off + v + 1) - __ldg(in_off + v) : 0;
      if (d > kLightMax) hubs += (unsigned long long)d;
      if (d > kTeamDegree) wide += (unsigned long long)d;
      const uint32_t m = __ballot_sync(kFull, d == 0);
      if (lane == j) mine = m;
    }
    if (w0 + lane < words) dead[w0 + lane] = mine;
    if (w0 + lane < words) alive += (unsigned)__popc(~mine);
  }
  alive = warp_sum(alive);
  hubs = warp_sum(hubs);
  wide = warp_sum(wide);
  if (lane == 0 && alive) atomicAdd(live, alive);
  if (lane == 0 && hubs) atomicAdd(hub_edges, hubs);
  if (lane == 0 && wide) atomicAdd(wide_edges, wide);
}

// Each vertex's first in-neighbour and in-degree (of one without, zeros).
__global__ void head_kernel(int64_t n, const int64_t *__restrict__ in_off,
                            const int32_t *__restrict__ in_idx, uint2 *__restrict__ head) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const int64_t s = __ldg(in_off + v), e = __ldg(in_off + v + 1);
  head[v] = s < e ? make_uint2((unsigned)__ldg(in_idx + s), (unsigned)(e - s)) : make_uint2(0u, 0u);
}

int refuse_setup_in_capture(cg_graph *g) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CG_CUDA(cudaStreamIsCapturing(g->stream, &cs));
  if (cs == cudaStreamCaptureStatusNone) return CG_OK;
  set_error_text("a handle's first batched search sets up state: run it outside a capture");
  return CG_ERR_NOT_SUPPORTED;
}

// The per-root search state of a new handle: one allocation, set up on the
// handle's stream behind the upload of its arrays (the caller waits).
int bfs_prepare(cg_graph *g) {
  int dev_coop = 0;
  CG_CUDA(cudaDeviceGetAttribute(&dev_coop, cudaDevAttrCooperativeLaunch, g->device));
  if (!dev_coop) return CG_ERR_NOT_SUPPORTED;
  const int64_t stride = bitmap_stride(g->n);
  const int64_t bcap = bfs_big_capacity(g->n, g->nnz);
  size_t bytes = 0;
  auto piece = [&](size_t size) {
    const size_t at = bytes;
    bytes = (bytes + size + 255) & ~(size_t)255;
    return at;
  };
  const size_t at_ctl = piece(sizeof(BfsCtl));
  const size_t at_stats = piece(sizeof(cg_stats));
  const size_t at_live = piece(3 * sizeof(unsigned long long));  // and entries by in-degree
  const size_t zeroed = bytes;
  const size_t at_bitmaps = piece(sizeof(uint32_t) * 4 * (size_t)stride);
  const size_t at_dead = piece(sizeof(uint32_t) * (size_t)stride);
  const size_t at_queue = piece(sizeof(int32_t) * 2 * (size_t)g->n);
  const size_t at_bigoff = piece(sizeof(uint32_t) * 2 * (size_t)bcap);
  unsigned char *base = nullptr;
  if (cudaMalloc(&base, bytes) != cudaSuccess) {
    cudaGetLastError();
    return CG_ERR_OUT_OF_MEMORY;
  }
  g->state = base;
  g->device_bytes += (int64_t)bytes;
  g->words = (g->n + 31) / 32;
  g->bcap = bcap;
  g->ctl = reinterpret_cast<BfsCtl *>(base + at_ctl);
  g->d_stats = reinterpret_cast<cg_stats *>(base + at_stats);
  g->bitmaps = reinterpret_cast<uint32_t *>(base + at_bitmaps);
  g->dead = reinterpret_cast<uint32_t *>(base + at_dead);
  g->queue = reinterpret_cast<int32_t *>(base + at_queue);
  g->bigoff = reinterpret_cast<uint32_t *>(base + at_bigoff);
  unsigned long long *d_live = reinterpret_cast<unsigned long long *>(base + at_live);
  unsigned long long live[3] = {0, 0, 0};
  CG_CUDA(cudaMemsetAsync(base, 0, zeroed, g->stream));
  const int64_t blocks = (stride + 255) / 256;  // 8 warps of 32 words
  dead_map_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, g->stream>>>(
      g->n, stride, g->in_off, g->dead, d_live, d_live + 1, d_live + 2);
  CG_CUDA(cudaGetLastError());
  CG_CUDA(cudaMemcpyAsync(live, d_live, sizeof(live), cudaMemcpyDeviceToHost, g->stream));
  CG_CUDA(cudaStreamSynchronize(g->stream));
  // Heads for graphs whose hubs hold half of the entries (R-MAT): the first
  // entry of a list is then a hub, the one most vertices resolve at.  Without
  // hubs the first entry is like any other, mostly a miss (directed ER of degree
  // 8: its first pull round of 119 us took 127 with them).
  if (2 * live[1] >= (unsigned long long)g->nnz && g->nnz > 0) {
    if (cudaMalloc(&g->head, sizeof(uint2) * (size_t)g->n) == cudaSuccess) {
      g->device_bytes += (int64_t)sizeof(uint2) * g->n;
      head_kernel<<<(unsigned)((g->n + 255) / 256), 256, 0, g->stream>>>(g->n, g->in_off, g->in_idx,
                                                                        g->head);
      CG_CUDA(cudaGetLastError());
    } else {
      cudaGetLastError();  // searches do without
      g->head = nullptr;
    }
  }
  // Meshes, grids and road networks, which take hundreds of rounds of slowly
  // changing frontiers: bounded degrees, and enough vertices for a frontier of
  // kTeamEnter edges that is as deep as it is wide.  Below, one block runs every
  // round; at the line the team's kernel pays only for several handles in turn
  // (256^2 grid: one handle 1,684 us without and 1,786 with it, three in turn 850 and
  // 704; 500^2: 4,496 and 3,749, 2,424 and 1,488).  The degrees alone do not tell a
  // mesh from a random graph of few edges, which it makes slower (1 M vertices,
  // three random in- and out-edges each 181 -> 193 us, a binary tree of 256 K 250 ->
  // 302; 292 and 441 before there were small rounds); what does, how fast a frontier
  // grows, is known only to a search.
  g->team = g->n >= kTeamVertices && g->nnz > 0 &&
            1024 * live[2] <= (unsigned long long)g->nnz;
  g->live = (int64_t)live[0];
  return CG_OK;
}

// The search pulls from its first rounds on.
static bool pulls_early(const cg_graph *g) {
  return g->opt.direction == CG_DIR_BOTTOMUP ||
         (g->opt.direction == CG_DIR_TAU && g->opt.tau_switch_count < g->n / 256);
}

// Blocks per SM of a search whose options leave it open, at most what fits (3).
// Fewer blocks make every round's barrier cheaper, and with one the searches of
// three handles run side by side (R-MAT n = 4 K, three handles in turn: 55 -> 19
// us a search); more keep more list reads in flight.  Measured, all rounds of
// one search with 3 / 2 / 1 blocks, us: direction-optimizing R-MAT n = 4 K 47 / 46
// / 45, 64 K 57 / 51 / 48, 256 K 67 / 63 / 61, 1 M 85 / 82 / 84, 2 M 127 / 122 /
// 128, 4 M 177 / 183 / 230; directed ER 300 K 100 / 93 / 90, 1 M 139 / 136 / 147, 3
// M 292 / 305 / 374; a 1000^2 grid is the same with all.  Top-down, which pushes
// every edge: R-MAT 16 K (0.4 M entries) 56 / 56 / 57, 64 K (1.8 M) 76 / 77 / 92,
// 256 K 136 / 159 / 204; ER 100 K (0.8 M) 94 / 90 / 94.  Searches that pull from the
// start scan whole lists, a hub's by one warp together with its neighbours' (the
// more warps, the fewer of them): bottom-up R-MAT 64 K of degree 16 93 / 84 / 79, 128
// K of degree 128 789 / 769 / 746, 256 K of 32 122 / 116 / 124, 1 M of 4 876 / 1,076 /
// 1,618, 2 M of 16 5,560 / 7,446 / 12,211; ER 250 K of 64 203 / 172 / 239.  A one-way
// switch at 15% of the vertices pushes most edges first: R-MAT 128 K of degree 128
// 158 / 168 / 220, 1 M of 32 149 / 203 / 247, but 256 K of 32 (14 M entries) 76 / 72 / 71.
static int blocks_for(const cg_graph *g) {
  if (g->opt.direction == CG_DIR_TOPDOWN)
    return g->nnz < (1 << 19) ? 1 : (g->nnz < (1 << 20) ? 2 : 3);
  if (pulls_early(g)) return g->n <= (1 << 17) ? 1 : (g->n <= (1 << 18) ? 2 : 3);
  if (g->opt.direction == CG_DIR_TAU && g->nnz >= (1 << 24)) return 3;
  if (g->n <= 300000 || g->nnz < (1 << 22)) return 1;
  return g->n <= (1 << 21) ? 2 : 3;
}

// The team's kernel has 1,152 threads an SM where the common one has 1,536: rounds
// that only pull want those from 4 M vertices on (bottom-up, us with the team's / the
// common kernel: a ring of 4 M with few long edges 31,300 / 28,200, a 3000^2 grid
// 327,800 / 291,600, directed ER of 4 M vertices and degree 1.2 79 / 73; but a 2000^2
// grid 100,200 / 101,200 and the ring of 1 M 11,000 / 12,100).
using BfsKernel = void (*)(BfsParams);
static BfsKernel kernel_for(const cg_graph *g) {
  return g->team && !(pulls_early(g) && g->n >= (1 << 22)) ? bfs_persistent_team : bfs_persistent;
}

static int bfs_grid(cg_graph *g) {
  const BfsKernel kernel = kernel_for(g);
  int block = g->opt.block_size > 0 ? g->opt.block_size : kBfsBlock;
  if (block > kBfsBlock) block = kBfsBlock;
  if (kernel == bfs_persistent_team && block > kTeamBlock) block = kTeamBlock;
  block = (block / 32) * 32;
  if (block < 64) block = 64;
  int per_sm = 0;
  CG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0));
  if (per_sm <= 0) return CG_ERR_NOT_SUPPORTED;
  const int want = g->opt.blocks_per_sm > 0 ? g->opt.blocks_per_sm : blocks_for(g);
  if (want < per_sm) per_sm = want;
  g->bfs_grid = per_sm * g->num_sms;
  g->bfs_block = block;
  return CG_OK;
}

int bfs_launch(cg_graph *g, int64_t root, int32_t *d_levels, int32_t *d_parents,
               int32_t *host_levels, int32_t *host_parents) {
  const int rc = bfs_grid(g);
  if (rc) return rc;
  BfsParams p;
  p.n = g->n;
  p.nnz = g->nnz;
  p.words = g->words;
  const int64_t stride = bitmap_stride(g->n);
  p.tiles = stride / kTileWords;
  p.in_off = g->in_off;
  p.in_idx = g->in_idx;
  p.out_off = g->out_off;
  p.out_idx = g->out_idx;
  p.vis = g->bitmaps;
  p.fr0 = g->bitmaps + stride;
  p.fr1 = g->bitmaps + 2 * stride;
  p.fr2 = g->bitmaps + 3 * stride;
  p.dead = g->dead;
  p.live = g->live;
  p.head = g->head;
  p.orig = g->orig;
  p.perm = g->perm;
  p.queue0 = g->queue;
  p.queue1 = g->queue + g->n;
  p.bigoff0 = g->bigoff;
  p.bigoff1 = g->bigoff + g->bcap;
  p.levels = d_levels;
  p.parents = d_parents;
  p.host_levels = host_levels;
  p.host_parents = host_parents;
  p.ctl = g->ctl;
  p.stats = g->d_stats;
  p.root = root;
  p.direction = g->opt.direction;
  p.alpha = g->opt.alpha > 0 ? g->opt.alpha : 15.f;
  p.beta = g->opt.beta > 0 ? g->opt.beta : 18.f;
  p.tau = g->opt.tau_switch_count;
  p.level_cap = g->opt.level_cap > 0 ? g->opt.level_cap
                                     : (int)((g->n + 1) < 0x7fffffff ? g->n + 1 : 0x7fffffff);
  p.timeout_ns = (long long)(g->opt.wait_timeout_ms > 0 ? g->opt.wait_timeout_ms : 1000) * 1000000ll;
  p.unmatched_wait = g->opt.test_unmatched_wait;
  p.heavy_work = g->head && pulls_early(g) ? kHeavyWorkEarly : kHeavyWork;
  // every launch starts from a clean control block (round records, wait counter)
  CG_CUDA(cudaMemsetAsync(g->ctl, 0, sizeof(BfsCtl), g->stream));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g->bfs_grid);
  cfg.blockDim = dim3(g->bfs_block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = g->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // all blocks co-resident (grid waits)
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CG_CUDA(cudaLaunchKernelEx(&cfg, kernel_for(g), p));
  return CG_OK;
}

int count_edges_launch(cg_graph *g, const int32_t *d_levels, int32_t k,
                       unsigned long long *d_m) {
  const int sym = g->symmetric ? 1 : 0;
  if (!g->edge_w) {
    uint32_t *w = nullptr;
    if (cudaMalloc(&w, sizeof(uint32_t) * (size_t)g->n) == cudaSuccess) {
      edge_weight_kernel<<<(unsigned)((g->n + 255) / 256), 256, 0, g->stream>>>(
          g->n, sym, g->in_off, g->in_idx, g->out_off, w);
      g->edge_w = w;
      g->device_bytes += (int64_t)sizeof(uint32_t) * g->n;
    } else {
      cudaGetLastError();
    }
  }
  CG_CUDA(cudaMemsetAsync(d_m, 0, sizeof(unsigned long long) * (size_t)k, g->stream));
  const int64_t blocks = (g->n + 255) / 256, cap = (int64_t)g->num_sms * 8;
  count_edges_kernel<<<dim3((unsigned)(blocks < cap ? blocks : cap),
                            (k + kCountGroup - 1) / kCountGroup),
                       256, 0, g->stream>>>(g->n, k, sym, g->in_off, g->in_idx, g->out_off,
                                            g->edge_w, d_levels, d_m);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

}  // namespace cg
