// Multi-source BFS with the outputs written after the search ("ledger"
// mode).  The rounds advance the W-word lane masks -- vis, and the frontier
// F_L of every round, kept as a history F_0 .. F_D in HBM -- and write no
// per-(lane, vertex) output.  After the last round a scan pass resolves the
// parents the rounds left open and one output pass writes every (lane, vertex)
// output exactly once:
//   level(l, v)  = the round L whose F_L[v] holds bit l      (-1 if none)
//   parent(l, v) = v at level 0, roots[l] at level 1, else the lowest
//                  in-neighbour u of v with bit l in F_{level - 1}[u]
// which is the lowest-index rule of the per-root search and of the direct
// batched kernel (bfs/README.md:208-224), so the outputs are identical.
//
// Why: written during the rounds, every discovery is a 4-byte store into one
// of 64 rows -- 32 scattered stores per warp instruction, each a separate L1
// wavefront and L2 transaction, and sectors completed across rounds (partial
// sector writes).  Here the output pass writes, lane by lane, the 32 values of
// a warp's 32 consecutive vertices as one 128-byte row.
//
// Parents: vertices of in-degree > kPullLight have a slot of 64 W parent
// candidates.  A push round relaxing u -> v takes atomicMin(slot[l], u) for
// each new lane l (ms_relax); a pull round scans such a vertex's ascending
// in-list with one warp (or its chunks, for hubs, with several) and records
// each lane's first hit (or_warp_first).  Vertices of smaller in-degree keep the
// position of each lane's parent in their in-list, as kPosBits bit slices: a
// pull round's thread scan knows it for the lanes it finds (the first entry
// holding a lane is its lowest-index parent, the in-list being ascending), the
// scan pass finds it for the lanes that pushes gave them.  The size is fixed
// and no later pass has to sort overlaps out: (source, lanes) records, up to 8
// of them, ran out on a directed graph of in-degree 8 and left 0.79 ms of
// fix-ups and 0.59 ms of rescans of a 2.4 ms batch (n = 1 M, 100 lanes).
//
// Rounds: a pull round ORs the frontier masks of a vertex's in-neighbours
// until every wanted lane is found; a push round ORs frontier masks into
// out-neighbours' next masks with atomicOr.  Hubs' in-lists are split into
// chunks across warps as in the direct kernel.  The frontier set of round L is
// a claim bitmap T_L (one bit per vertex, set by whoever first gives the
// vertex a lane): push rounds find their light frontier vertices there and
// only big ones (out-degree > kLightMax) go through a queue, so no per-vertex
// atomic on a shared queue counter.  vis is merged lazily: round L folds F_L
// into vis for its frontier vertices and tests "visited" as vis | F_L, so a
// push round needs no second phase.
//
// A search that needs more rounds than the history holds sets a flag and
// stops; the output pass then only clears the control block, and the direct
// kernel, launched after it gated on the flag, runs the batch from scratch.
#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_ms.cuh"

namespace cg {
namespace {

constexpr int kOutBlock = 128;                 // output pass: 4 warps a block
constexpr int kOutWarps = kOutBlock / 32;
constexpr size_t kSmemOfSm = 228 * 1024;       // shared memory of an SM at most, and what
constexpr size_t kSmemReserved = 1024;         // the system takes of it for a block
constexpr int kOutLevels = 4;                  // levels resolved per in-list scan
// A warp's shared tile: one parent table of kTab words per thread.  A vertex
// with a candidate slot has its 64 parents there, lane l at column (l - 8 t) mod
// 64 for thread t (the 32 threads reading the same lane hit 32 different banks,
// kTab - 8 being odd); a light vertex the in-list entries that positions point
// at, from column 0; -1 (unreached) is at kTabNone.  A lane's parent is one
// table read at a byte index.
constexpr int kTabNone = 64;
constexpr int kTab = kTabNone + 1;
// Behind the table, the bytes of 32 lanes' levels and table indices: word t of
// row g has those of lanes g, g + 8, g + 16, g + 24 for thread t's vertex (rows
// of 33 words: eight threads each on four rows read different banks).
constexpr int kStageRow = 33;
constexpr int kStage = 8 * kStageRow;
constexpr int kOutWarpBytes = (32 * kTab + 2 * kStage) * 4;
static_assert((kTab - 8) % 2 == 1, "same lane, different banks");
static_assert((1 << kPosBits) == kPullLight, "a position in a light in-list");
constexpr int kSlices = 7;                     // bit slices of a level (levels 0..64)

// Four bytes from global to shared memory, asynchronously; the wait covers all
// copies of the calling thread.
__device__ __forceinline__ void copy_async4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int W>
__device__ __forceinline__ uint64_t *plane(const MsParams &p, int L) {
  return p.hist + (int64_t)L * p.n * W;
}

// Adds lanes to slice b of light vertex v's positions; `used` is its pos_used.
template <int W>
__device__ __forceinline__ void add_slice(const MsParams &p, int64_t v, int b, const Mask<W> &a,
                                          unsigned &used) {
  if (!a.any()) return;
  const int64_t at = (int64_t)b * p.n + v;
  st_mask<W>(p.pos, at, (used >> b) & 1u ? a | ld_mask<W>(p.pos, at) : a);
  used |= 1u << b;
}

// The scan of light vertex v's in-list in a pull round: ORs its in-neighbours'
// frontier masks for the lanes of `want` until all are found (returned), and
// keeps the position of each lane's first entry, its lowest-index parent.
// `want1`, after a push round: the lanes that push gave v at this round's
// level L, whose parents are the first entries holding them in F_{L-1}
// (`prev`) -- found in the same pass, so the scan pass need not rescan v.
template <int W>
__device__ __forceinline__ Mask<W> or_thread_pos(const MsParams &p, int64_t v, int64_t s,
                                                 int64_t e, const Mask<W> &want,
                                                 const uint64_t *cur, const uint64_t *prev,
                                                 const Mask<W> &want1) {
  constexpr int G = 4;
  Mask<W> got = Mask<W>::zero(), got1 = Mask<W>::zero();
  // the lanes at positions with bit 0 .. 4 set; with 128 lanes the last three
  // would spill and go to memory as they are found
  constexpr int kKept = W == 1 ? kPosBits : 2;
  Mask<W> A[kKept];
#pragma unroll
  for (int b = 0; b < kKept; ++b) A[b] = Mask<W>::zero();
  const unsigned used0 = p.pos_used[v];
  unsigned used = used0;
  const bool two = want1.any();
  for (int64_t i0 = s; i0 < e; i0 += G) {
    int32_t u[G];
    Mask<W> m[G], m1[G];
#pragma unroll
    for (int k = 0; k < G; ++k) u[k] = i0 + k < e ? __ldg(p.in_idx + i0 + k) : -1;
#pragma unroll
    for (int k = 0; k < G; ++k) {
      m[k] = u[k] >= 0 ? ld_mask<W>(cur, u[k]) : Mask<W>::zero();
      m1[k] = two && u[k] >= 0 ? ld_mask<W>(prev, u[k]) : Mask<W>::zero();
    }
    // entry i0 + k is at position i0 - s + k: its low two bits are k's
    Mask<W> four = Mask<W>::zero();
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const Mask<W> nb = (m[k] & want).andnot(got);
      const Mask<W> nb1 = (m1[k] & want1).andnot(got1);
      const Mask<W> r = nb | nb1;  // disjoint: want1 lanes are visited, want lanes are not
      if (k & 1) A[0] = A[0] | r;
      if (k & 2) A[1] = A[1] | r;
      four = four | r;
      got = got | nb;
      got1 = got1 | nb1;
    }
    const int hi = (int)(i0 - s) >> 2;
#pragma unroll
    for (int b = 2; b < kPosBits; ++b) {
      if (!((hi >> (b - 2)) & 1)) continue;
      if (b < kKept)
        A[b < kKept ? b : 0] = A[b < kKept ? b : 0] | four;
      else
        add_slice<W>(p, v, b, four, used);
    }
    if (got == want && got1 == want1) break;
  }
#pragma unroll
  for (int b = 0; b < kKept; ++b) add_slice<W>(p, v, b, A[b], used);
  if (used != used0) p.pos_used[v] = (uint8_t)used;
  return got;
}

// 32 x 32 bit-matrix transpose across the warp: lane r holds row r (bit c =
// entry (r, c)); afterwards lane t holds column t (bit r = entry (r, t)).
// Five butterfly steps, each swapping off-diagonal blocks with the partner
// lane t ^ j.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x) {
  const int lane = lane_id();
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t m = j == 16 ? 0x0000ffffu
                     : j == 8  ? 0x00ff00ffu
                     : j == 4  ? 0x0f0f0f0fu
                     : j == 2  ? 0x33333333u
                               : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(kMsFull, x, j);
    x = (lane & j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
  }
  return x;
}

// OR of the frontier masks of in-list entries [s, e) restricted to `want`, by the
// whole warp, recording per lane of `want` the first in-list entry
// holding it -- the lowest-index parent -- into row[lane] (plain stores when
// the warp scans the whole in-list, atomicMin when other warps scan other
// chunks of it).  The hits of 32 entries form a 32 x 64 W bit matrix that is
// transposed a word at a time, so warp lane t resolves lanes t and t + 32 of
// each word at once.
template <int W>
__device__ __forceinline__ Mask<W> or_warp_first(const MsParams &p, int64_t s, int64_t e,
                                                 const Mask<W> &want, const uint64_t *cur,
                                                 uint32_t *row, bool atomic) {
  constexpr int G = 4;
  const int lane = lane_id();
  Mask<W> got = Mask<W>::zero();
  for (int64_t base = s; base < e; base += 32 * G) {
    int32_t u[G];
    Mask<W> f[G];
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int64_t i = base + 32 * k + lane;
      u[k] = i < e ? __ldg(p.in_idx + i) : -1;
    }
#pragma unroll
    for (int k = 0; k < G; ++k) f[k] = u[k] >= 0 ? ld_mask<W>(cur, u[k]) : Mask<W>::zero();
    {
      // nothing new among these 4 x 32 entries (the common case late in a
      // list that some lanes only reach in a later round): one reduction
      Mask<W> any = Mask<W>::zero();
#pragma unroll
      for (int k = 0; k < G; ++k) any = any | f[k];
      if (!warp_or<W>(any & want).andnot(got).any()) continue;
    }
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const Mask<W> fk = (f[k] & want).andnot(got);
      const Mask<W> F = warp_or<W>(fk);
      if (!F.any()) continue;
#pragma unroll
      for (int j = 0; j < W; ++j) {
        if (!F.w[j]) continue;
        uint32_t *r = row + 64 * j;
        if (__popcll(F.w[j]) <= 6) {
          // few lanes: one ballot each
          uint64_t bits = F.w[j];
          while (bits) {
            const int b = __ffsll((long long)bits) - 1;
            bits &= bits - 1;
            const unsigned who = __ballot_sync(kMsFull, (fk.w[j] >> b) & 1ull);
            if (lane == __ffs(who) - 1) {
              if (atomic)
                atomicMin(r + b, (unsigned)u[k]);
              else
                r[b] = (uint32_t)u[k];
            }
          }
          continue;
        }
        const uint32_t lo = warp_transpose32((uint32_t)fk.w[j]);
        const uint32_t hi = warp_transpose32((uint32_t)(fk.w[j] >> 32));
        const int32_t plo = __shfl_sync(kMsFull, u[k], lo ? __ffs(lo) - 1 : 0);
        const int32_t phi = __shfl_sync(kMsFull, u[k], hi ? __ffs(hi) - 1 : 0);
        if (atomic) {
          if (lo) atomicMin(r + lane, (unsigned)plo);
          if (hi) atomicMin(r + lane + 32, (unsigned)phi);
        } else {
          if (lo) r[lane] = (uint32_t)plo;
          if (hi) r[lane + 32] = (uint32_t)phi;
        }
      }
      got = got | F;
      if (got == want) return got;
    }
  }
  return got;
}

// Claimed vertices of out-degree > kLightMax on their way to the next queue
// (light ones are found in the claim bitmap): a warp keeps them in shared
// memory and queues 32 with one atomic, instead of one returning atomic on the
// queue's counter per step with any -- the round's warps queue up there.
struct HeavyQueue {
  int32_t v[64];
  uint32_t deg[64];
};
__shared__ HeavyQueue s_heavy[kMsBlock / 32];
struct HeavyOut {
  MsRound *Rn;                // the record of the next frontier
  int parity;                 // its queue
  unsigned count = 0;         // entries waiting, the same in every lane
};

// Queues entries [from, from + n), n <= 32.  All 32 lanes call.
__device__ __forceinline__ void heavy_flush(const MsParams &p, HeavyOut &H, unsigned from,
                                            unsigned n) {
  const int lane = lane_id();
  HeavyQueue &S = s_heavy[threadIdx.x >> 5];
  const bool has = (unsigned)lane < n;
  const uint32_t d = has ? S.deg[from + lane] : 0u;
  uint32_t incl = d;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kMsFull, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t total = __shfl_sync(kMsFull, incl, 31);
  unsigned long long old = 0;
  if (lane == 0) old = atomicAdd(&H.Rn->big, ((unsigned long long)n << 32) | total);
  old = __shfl_sync(kMsFull, old, 0);
  if (has) {
    const unsigned idx = (unsigned)(old >> 32) + (unsigned)lane;
    (H.parity ? p.queue1 : p.queue0)[p.n - 1 - (int64_t)idx] = S.v[from + lane];
    (H.parity ? p.bigoff1 : p.bigoff0)[idx] = (uint32_t)old + incl - d;
  }
  __syncwarp();
}

// Counts the claims of one warp-wide step and keeps the heavy ones.  All 32
// lanes call.
__device__ __forceinline__ void claim_step(const MsParams &p, bool claimed, int32_t v, int64_t deg,
                                           HeavyOut &H, MsAcc &acc) {
  if (claimed) {
    acc.nf += 1;
    acc.mf += (unsigned long long)deg;
  }
  const bool heavy = claimed && deg > kLightMax;
  const unsigned m = __ballot_sync(kMsFull, heavy);
  if (!m) return;
  HeavyQueue &S = s_heavy[threadIdx.x >> 5];
  if (heavy) {
    const unsigned at = H.count + __popc(m & ((1u << lane_id()) - 1u));
    S.v[at] = v;
    S.deg[at] = (uint32_t)deg;
  }
  H.count += __popc(m);
  __syncwarp();
  if (H.count >= 32) {
    H.count -= 32;
    heavy_flush(p, H, H.count, 32);
  }
}

__device__ __forceinline__ void heavy_rest(const MsParams &p, HeavyOut &H) {
  if (H.count) heavy_flush(p, H, 0, H.count);
  H.count = 0;
}

// Claim bitmap T_L: one bit per vertex with a nonzero frontier mask F_L --
// round L's frontier set.  Round L reads T_L (push rounds enumerate light
// frontier vertices from it), sets T_{L+1}, and clears T_{L+2}; three rotate.
__device__ __forceinline__ uint32_t *claims(const MsParams &p, int L) {
  const int r = L % 3;
  return r == 0 ? p.touched0 : (r == 1 ? p.touched1 : p.touched2);
}

// vis is merged lazily: a vertex's frontier lanes F_L[v] join vis[v] during
// round L (pull rounds for every vertex, push rounds for every frontier
// vertex), so round L tests "visited" as vis | F_L.

// Pull round: light vertices one thread each, medium vertices one warp each,
// hub in-lists by chunks (ORed into hub_found, merged after the wait).
template <int W>
__device__ void lg_pull(const MsParams &p, int L, const uint64_t *cur, uint64_t *nxt,
                        const Mask<W> &active, bool after_push, MsRound *Rc, MsRound *Rn,
                        MsAcc &acc) {
  // after a push round, light vertices also resolve the parents of the lanes
  // that push gave them (F_L) against F_{L-1} (64 lanes; with 128 the registers
  // would spill, and the scan pass does it)
  after_push = after_push && W == 1;
  const uint64_t *prev = after_push ? plane<W>(p, L - 1) : cur;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  HeavyOut H{Rn, (L + 1) & 1};
  uint32_t *tnext = claims(p, L + 1);
  const int lane = lane_id();
  // a symmetric graph stores one list per vertex: out-degree = in-degree
  const bool sym = p.out_off == p.in_off;
  // light vertices by groups of p.light_grab bitmap words, then medium vertices
  // by p.med_grab, then hub chunks by p.hub_grab (pull_grabs), handed out
  // dynamically -- one item per warp, then a counter -- so that the round's
  // last warps are not the ones with the longest lists
  const unsigned nwarps = (unsigned)(nthreads >> 5);
  unsigned item = (unsigned)warp_id_global();
  while (item < p.light_items + p.med_items + p.hub_items) {
    // the next item is claimed before this one is worked, hiding the atomic
    unsigned nextitem = 0;
    if (lane == 0) nextitem = nwarps + atomicAdd(&Rc->work, 1u);
    if (item < p.light_items) {
      // the light vertices of a group's words not yet finished, compacted 32
      // at a time (vertices without in-edges are not light: none can reach
      // them).  Lane j holds word j; the t-th vertex is the
      // (t - prefix)-th set bit of the first word whose inclusive count
      // exceeds t.  Only this warp touches these words of fin this round.
      const int64_t w0 = (int64_t)item * p.light_grab;
      uint32_t finw = 0, mine = 0;
      if ((unsigned)lane < p.light_grab && w0 + lane < p.words) {
        finw = p.fin[w0 + lane];
        mine = __ldg(p.light + w0 + lane) & ~finw;
      }
      const uint32_t fin0 = finw;
      const int cnt = __popc(mine);
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kMsFull, incl, o);
        if (lane >= o) incl += t;
      }
      const int total = __shfl_sync(kMsFull, incl, 31);
      for (int b0 = 0; b0 < total; b0 += 32) {
        const int t = b0 + lane;
        int wsel = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (__shfl_sync(kMsFull, incl, wsel + step - 1) <= t) wsel += step;
        const uint32_t wbits = __shfl_sync(kMsFull, mine, wsel);
        const int before = __shfl_sync(kMsFull, incl - cnt, wsel);
        const bool has = t < total;
        int64_t v = 0;
        Mask<W> want = Mask<W>::zero(), want1 = Mask<W>::zero();
        int64_t s = 0, e = 0;
        if (has) {
          v = (w0 + wsel) * 32 + (__fns(wbits, 0, t - before + 1) & 31);
          const Mask<W> fv = ld_mask<W>(cur, v);
          const Mask<W> seen = ld_mask<W>(p.vis, v) | fv;
          if (fv.any()) st_mask<W>(p.vis, v, seen);
          want = active.andnot(seen);
          if (after_push) want1 = fv;
          if (want.any() || want1.any()) {
            s = __ldg(p.in_off + v);
            e = __ldg(p.in_off + v + 1);
          }
        }
        // every running lane visited: no lane can reach v again (finished
        // lanes never run again), so later rounds skip it
        const bool done = has && !want.any();
        bool claimed = false;
        int64_t deg = 0;
        const bool scan = want.any() || want1.any();
        if (__ballot_sync(kMsFull, scan)) {
          Mask<W> got = Mask<W>::zero();
          if (scan) got = or_thread_pos<W>(p, v, s, e, want, cur, prev, want1);
          claimed = got.any();
          if (claimed) {
            st_mask<W>(nxt, v, got);
            acc_lanes<W>(acc, got);
            deg = sym ? e - s : __ldg(p.out_off + v + 1) - __ldg(p.out_off + v);
          }
        }
        // per word of the batch: claim bits (T_{L+1}), finished bits
        const unsigned mybit = 1u << (unsigned)(v & 31);
        const int wlo = __shfl_sync(kMsFull, wsel, 0);
        const int whi = __shfl_sync(kMsFull, wsel, min(31, total - 1 - b0));
        for (int j = wlo; j <= whi; ++j) {  // uniform: the whole warp
          const bool inj = has && wsel == j;
          const unsigned cb = __reduce_or_sync(kMsFull, inj && claimed ? mybit : 0u);
          const unsigned db = __reduce_or_sync(kMsFull, inj && done ? mybit : 0u);
          if (lane == j) {
            finw |= db;
            if (cb) atomicOr(tnext + w0 + j, cb);
          }
        }
        claim_step(p, claimed, (int32_t)v, deg, H, acc);
      }
      if (finw != fin0) p.fin[w0 + lane] = finw;
    } else if (item < p.light_items + p.med_items) {
      const unsigned mi = item - p.light_items;
      const int64_t j0 = (int64_t)mi * p.med_grab;
      const int64_t j1 = min(j0 + (int64_t)p.med_grab, p.nmed);
      // 64 lanes: the first lanes look at the group's vertices at once
      // (the lanes each still wants and its in-list) and the warp then scans
      // those wanting any; 128 lanes (more registers): one vertex at a time
      int32_t vq = 0;
      Mask<W> wq = Mask<W>::zero();
      int64_t sq = 0, eq = 0;
      bool cq = false;  // 64 lanes: lane t's vertex was claimed (queued once, at the end)
      if (W == 1 && lane < j1 - j0) {
        vq = p.med_vtx[j0 + lane];
        // F_L joins vis here for medium vertices (the light loop does it
        // for light ones, the hub merge for hubs)
        const Mask<W> fq = ld_mask<W>(cur, vq);
        const Mask<W> sq0 = ld_mask<W>(p.vis, vq) | fq;
        if (fq.any()) st_mask<W>(p.vis, vq, sq0);
        wq = active.andnot(sq0);
        sq = __ldg(p.in_off + vq);
        eq = __ldg(p.in_off + vq + 1);
      }
      unsigned pend = W == 1 ? __ballot_sync(kMsFull, wq.any())
                             : kMsFull >> (32u - (unsigned)(j1 - j0));
      while (pend) {
        const int t = __ffs(pend) - 1;
        pend &= pend - 1;
        const int64_t j = j0 + t;
        int32_t v;
        Mask<W> want;
        int64_t s, e;
        if (W == 1) {
          v = __shfl_sync(kMsFull, vq, t);
#pragma unroll
          for (int w = 0; w < W; ++w) want.w[w] = __shfl_sync(kMsFull, wq.w[w], t);
          s = __shfl_sync(kMsFull, sq, t);
          e = __shfl_sync(kMsFull, eq, t);
        } else {
          v = p.med_vtx[j];
          const Mask<W> fvm = ld_mask<W>(cur, v);
          const Mask<W> svm = ld_mask<W>(p.vis, v) | fvm;
          __syncwarp();
          if (lane == 0 && fvm.any()) st_mask<W>(p.vis, v, svm);
          want = active.andnot(svm);
          if (!want.any()) continue;
          s = __ldg(p.in_off + v);
          e = __ldg(p.in_off + v + 1);
        }
        // medium vertex j has candidate slot j: its parents of this round go there
        const Mask<W> got = or_warp_first<W>(p, s, e, want, cur, p.cand + j * (64 * W), false);
        const bool claimed = lane == 0 && got.any();
        int64_t deg = 0;
        if (claimed) {
          st_mask<W>(nxt, v, got);
          atomicOr(tnext + (v >> 5), 1u << (v & 31));
          acc_lanes<W>(acc, got);
          if (W != 1) deg = __ldg(p.out_off + v + 1) - __ldg(p.out_off + v);
        }
        if (W == 1) {
          if (lane == t && got.any()) cq = true;
        } else {
          claim_step(p, claimed, v, deg, H, acc);
        }
      }
      // the group's claimed vertices together
      if (W == 1) {
        const int64_t dq =
            !cq ? 0 : (sym ? eq - sq : __ldg(p.out_off + vq + 1) - __ldg(p.out_off + vq));
        claim_step(p, cq, vq, dq, H, acc);
      }
    } else {
      const unsigned hi_item = item - p.light_items - p.med_items;
      const unsigned c1 = min((hi_item + 1) * p.hub_grab, p.hub_chunks);
      // a hub whose chunk c' < c found every wanted lane: chunk c holds only
      // higher-index entries, which could not be parents (known to this item
      // at once, to others through hub_done, tagged with the round)
      const unsigned tag = (unsigned)(L + 1) << 24;
      int done_h = -1;
      for (unsigned ci = hi_item * p.hub_grab; ci < c1; ++ci) {
        const unsigned c = p.hub_chunk_order[ci];  // by rank within the hub, then hub
        const int h = (int)p.hub_of_chunk[c];
        if (h == done_h) continue;
        const unsigned d = *(volatile unsigned *)(p.hub_done + h);
        if ((d & 0xFF000000u) == tag && 0xFFFFFFu - (d & 0xFFFFFFu) < c) continue;
        const int32_t v = p.hub_vtx[h];
        const Mask<W> want = active.andnot(ld_mask<W>(p.vis, v) | ld_mask<W>(cur, v));
        if (!want.any()) continue;
        const int64_t s = __ldg(p.in_off + v) + (int64_t)(c - p.hub_choff[h]) * kHubChunk;
        const int64_t e = min(s + (int64_t)kHubChunk, __ldg(p.in_off + v + 1));
        // hub h has candidate slot nmed + h; several warps scan its chunks
        const Mask<W> got = or_warp_first<W>(p, s, e, want, cur,
                                             p.cand + (p.nmed + h) * (64 * W), true);
        if (got == want) {
          done_h = h;
          if (lane == 0) atomicMax(p.hub_done + h, tag | (0xFFFFFFu - c));
        }
        if (lane == 0) {
#pragma unroll
          for (int w = 0; w < W; ++w)
            if (got.w[w])
              atomicOr(reinterpret_cast<unsigned long long *>(p.hub_found + (int64_t)h * W + w),
                       (unsigned long long)got.w[w]);
        }
      }
    }
    item = __shfl_sync(kMsFull, nextitem, 0);
  }
  heavy_rest(p, H);
}

// After the wait that ends a pull round's scans: hubs found this round get
// their next mask and claim bit, and are queued if big.
template <int W>
__device__ void lg_hub_merge(const MsParams &p, int L, const uint64_t *cur, uint64_t *nxt,
                             MsRound *Rn, MsAcc &acc) {
  const int lane = lane_id();
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  HeavyOut H{Rn, (L + 1) & 1};
  uint32_t *tnext = claims(p, L + 1);
  for (int64_t h0 = (int64_t)warp_id_global() * 32; h0 < p.nhub; h0 += (int64_t)nwarps * 32) {
    const int64_t h = h0 + lane;
    bool claimed = false;
    int32_t v = 0;
    int64_t deg = 0;
    if (h < p.nhub) {
      // F_L joins vis for the hubs (their chunk scans have ended)
      const int32_t vh = p.hub_vtx[h];
      const Mask<W> fh = ld_mask<W>(cur, vh);
      if (fh.any()) st_mask<W>(p.vis, vh, ld_mask<W>(p.vis, vh) | fh);
      const Mask<W> found = ld_mask<W>(p.hub_found, h);
      if (found.any()) {
        v = vh;
        st_mask<W>(nxt, v, found);
        st_mask<W>(p.hub_found, h, Mask<W>::zero());
        atomicOr(tnext + (v >> 5), 1u << (v & 31));
        acc_lanes<W>(acc, found);
        deg = __ldg(p.out_off + v + 1) - __ldg(p.out_off + v);
        claimed = true;
      }
    }
    claim_step(p, claimed, v, deg, H, acc);
  }
  heavy_rest(p, H);
}

// Edge u -> v of a push round: the lanes of u's frontier that v has neither
// visited nor in its own frontier of this round are ORed into v's next mask
// (after a read, so hot targets see few atomics); a vertex with a candidate
// slot also takes u as a parent candidate per lane (atomicMin).  The loads
// that depend only on v go out together; with a sparse frontier (`tfront`,
// its claim bitmap) v's own frontier mask is read only if v is in it.
// Returns whether this thread claimed v (set its bit in the next claim
// bitmap first).
template <int W>
struct Target {
  int32_t v = -1;             // -1: no edge
  int32_t slot = -1;
  uint32_t tw = 0;
  Mask<W> f, add;             // new lanes, and those v's next mask lacks
};

template <int W>
__device__ __forceinline__ void lg_load(const MsParams &p, Target<W> &t, const Mask<W> &fu,
                                        const uint64_t *cur, const uint64_t *nxt,
                                        const uint32_t *tnext, const uint32_t *tfront) {
  t.f = t.add = Mask<W>::zero();
  if (t.v < 0) return;
  const Mask<W> seen = ld_mask<W>(p.vis, t.v);
  Mask<W> have;
#pragma unroll
  for (int i = 0; i < W; ++i) have.w[i] = __ldcg(nxt + (int64_t)t.v * W + i);
  t.slot = p.cand_slot[t.v];
  t.tw = __ldcg(tnext + (t.v >> 5));
  Mask<W> now = Mask<W>::zero();
  if (!tfront || ((tfront[t.v >> 5] >> (t.v & 31)) & 1u)) now = ld_mask<W>(cur, t.v);
  t.f = fu.andnot(seen | now);
  t.add = t.f.andnot(have);
}

template <int W>
__device__ __forceinline__ bool lg_relax(const MsParams &p, int32_t u, const Target<W> &t,
                                         uint64_t *nxt, uint32_t *tnext, MsAcc &acc) {
  if (!t.f.any()) return false;
  acc_lanes<W>(acc, t.f);
  if (t.slot >= 0) {
    // lowest source per new lane: read first (a lower one is often there
    // already), four lanes' reads in flight at a time
    uint32_t *cand = p.cand + (int64_t)t.slot * (64 * W);
#pragma unroll
    for (int j = 0; j < W; ++j) {
      uint64_t bits = t.f.w[j];
      while (bits) {
        int b[4];
        uint32_t c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          b[k] = bits ? __ffsll((long long)bits) - 1 : -1;
          bits &= bits ? bits - 1 : 0ull;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = b[k] >= 0 ? __ldcg(cand + j * 64 + b[k]) : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (b[k] >= 0 && (unsigned)u < c[k]) atomicMin(cand + j * 64 + b[k], (unsigned)u);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < W; ++i)
    if (t.add.w[i])
      atomicOr(reinterpret_cast<unsigned long long *>(nxt + (int64_t)t.v * W + i),
               (unsigned long long)t.add.w[i]);
  const uint32_t tb = 1u << (t.v & 31);
  if (t.tw & tb) return false;
  return (atomicOr(tnext + (t.v >> 5), tb) & tb) == 0;
}

// The claims of one warp-wide step of edges.
template <int W>
__device__ __forceinline__ void lg_apply(const MsParams &p, int32_t u, const Target<W> &t,
                                         uint64_t *nxt, uint32_t *tnext, HeavyOut &H, MsAcc &acc) {
  const bool claimed = lg_relax<W>(p, u, t, nxt, tnext, acc);
  const int64_t deg = claimed ? __ldg(p.out_off + t.v + 1) - __ldg(p.out_off + t.v) : 0;
  claim_step(p, claimed, t.v, deg, H, acc);
}

// Edge positions [x0, x1) of the big-vertex edge space (queue entries
// q[cap-1-j] with prefix offsets boff[j], all of out-degree > kLightMax).  With
// 64 lanes two steps of 32 edges go together: their list entries, then their
// targets' masks, are in flight at once (with 128 the registers would spill).
template <int W>
__device__ void lg_push_chunk(const MsParams &p, const uint64_t *cur, uint64_t *nxt,
                              uint32_t *tnext, const int32_t *bq, const uint32_t *boff,
                              unsigned nbig, unsigned x0, unsigned x1, const uint32_t *tfront,
                              HeavyOut &H, MsAcc &acc) {
  constexpr int U = W == 1 ? 2 : 1;
  const int lane = lane_id();
  const int64_t cap = p.n;
  unsigned lo = 0, hi = nbig - 1;
  while (lo < hi) {
    const unsigned mid = (lo + hi + 1) >> 1;
    if (boff[mid] <= x0)
      lo = mid;
    else
      hi = mid - 1;
  }
  unsigned j = lo;
  int32_t vj = bq[cap - 1 - (int64_t)j];
  int64_t sj = __ldg(p.out_off + vj);
  unsigned oj = boff[j];
  unsigned endj = oj + (unsigned)(__ldg(p.out_off + vj + 1) - sj);
  Mask<W> fj = ld_mask<W>(cur, vj);
  for (unsigned base = x0; base < x1; base += 32 * U) {
    int32_t u[U];
    Mask<W> fu[U];
    Target<W> t[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const unsigned at = base + 32 * k;
      if (at < x1) {  // uniform
        while (at >= endj) {
          ++j;
          vj = bq[cap - 1 - (int64_t)j];
          sj = __ldg(p.out_off + vj);
          oj = boff[j];
          endj = oj + (unsigned)(__ldg(p.out_off + vj + 1) - sj);
          fj = ld_mask<W>(cur, vj);
        }
      }
      const unsigned x = at + lane;
      const bool valid = x < x1 && x >= at;
      u[k] = vj;
      int64_t e = sj + (int64_t)(x - oj);
      fu[k] = fj;
      if (__ballot_sync(kMsFull, valid && x >= endj)) {
        const int32_t vn = bq[cap - 1 - (int64_t)(j + 1)];
        if (valid && x >= endj) {
          u[k] = vn;
          e = __ldg(p.out_off + vn) + (int64_t)(x - endj);
          fu[k] = ld_mask<W>(cur, vn);
        }
      }
      if (valid) t[k].v = __ldg(p.out_idx + e);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) lg_load<W>(p, t[k], fu[k], cur, nxt, tnext, tfront);
#pragma unroll
    for (int k = 0; k < U; ++k) lg_apply<W>(p, u[k], t[k], nxt, tnext, H, acc);
    if (base + 32 * U < base) break;  // x1 within a step of 2^32
  }
}

// Push round.  The big vertices' edges go in chunks (from the queue, as in the
// direct kernel), handed out dynamically; then every warp takes 32 claim words
// at a time, one a lane, a grid apart from each other -- neighbouring words are
// alike, so this spreads them evenly without a counter: the frontier vertices
// there merge their lanes into vis, and the light ones (out-degree <=
// kLightMax) spread their edges over the warp.  A warp's steps follow one
// another: 200,000 frontier vertices among 1 M took 116 us with 32 neighbouring
// words to a warp, 42 us so.
template <int W>
__device__ void lg_push(const MsParams &p, int L, const uint64_t *cur, uint64_t *nxt,
                        bool sparse, MsRound *Rc, MsRound *Rn, MsAcc &acc) {
  __shared__ int32_t s_u[kMsBlock / 32][32];
  __shared__ int64_t s_s[kMsBlock / 32][32];
  __shared__ int64_t s_x[kMsBlock / 32][32];
  const int lane = lane_id();
  const int wib = threadIdx.x >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int parity = L & 1;
  const int32_t *qc = parity ? p.queue1 : p.queue0;
  const uint32_t *bc = parity ? p.bigoff1 : p.bigoff0;
  HeavyOut H{Rn, parity ^ 1};
  const uint32_t *tcur = claims(p, L);
  uint32_t *tnext = claims(p, L + 1);
  // a frontier of under n/1024 vertices (few targets are in it): its claim
  // bitmap (1/64 of a mask plane, cache-resident) is tested before a
  // target's frontier mask is read
  const uint32_t *tfront = sparse ? tcur : nullptr;

  const unsigned long long bigw = *(volatile unsigned long long *)&Rc->big;
  const unsigned nbig = (unsigned)(bigw >> 32), big_edges = (unsigned)bigw;
  unsigned chunk = ((big_edges / (unsigned)nwarps) + 31u) & ~31u;
  chunk = chunk < 32u ? 32u : (chunk > (unsigned)kPushChunk ? (unsigned)kPushChunk : chunk);
  const unsigned nb = (big_edges + chunk - 1) / chunk;
  unsigned item = (unsigned)warp_id_global();
  while (item < nb) {
    // the next item is claimed before this one is worked, hiding the atomic
    unsigned nextitem = 0;
    if (lane == 0) nextitem = (unsigned)nwarps + atomicAdd(&Rc->work, 1u);
    const unsigned x0 = item * chunk;
    lg_push_chunk<W>(p, cur, nxt, tnext, qc, bc, nbig, x0, min(x0 + chunk, big_edges), tfront, H,
                     acc);
    item = __shfl_sync(kMsFull, nextitem, 0);
  }
  for (int64_t w0 = warp_id_global(); w0 < p.words; w0 += 32 * (int64_t)nwarps) {
    // the words' frontier vertices, compacted 32 at a time: lane j holds word
    // w0 + j nwarps; the t-th frontier vertex is the (t - prefix)-th set bit
    // of the word whose prefix count covers t
    const int64_t wi = w0 + (int64_t)lane * nwarps;
    const uint32_t mine = wi < p.words ? tcur[wi] : 0u;
    const int cnt = __popc(mine);
    int incl_c = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kMsFull, incl_c, o);
      if (lane >= o) incl_c += t;
    }
    const int total_v = __shfl_sync(kMsFull, incl_c, 31);
    for (int b0 = 0; b0 < total_v; b0 += 32) {
      const int t = b0 + lane;
      int32_t u = -1;
      int64_t s = 0, d = 0;
      // word holding the t-th vertex: the first lane whose inclusive count
      // exceeds t (the counts never decrease)
      int wsel = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(kMsFull, incl_c, wsel + step - 1) <= t) wsel += step;
      const uint32_t wbits = __shfl_sync(kMsFull, mine, wsel);
      const int before = __shfl_sync(kMsFull, incl_c - cnt, wsel);
      if (t < total_v) {
        const int bit = __fns(wbits, 0, t - before + 1);
        const int64_t v = (w0 + (int64_t)wsel * nwarps) * 32 + bit;
        const Mask<W> fv = ld_mask<W>(cur, v);
        st_mask<W>(p.vis, v, ld_mask<W>(p.vis, v) | fv);
        s = __ldg(p.out_off + v);
        d = __ldg(p.out_off + v + 1) - s;
        if (d > kLightMax)
          d = 0;  // big: its edges are in the chunks above
        else
          u = (int32_t)v;
      }
      int64_t incl = d;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t tt = __shfl_up_sync(kMsFull, incl, o);
        if (lane >= o) incl += tt;
      }
      const int64_t total = __shfl_sync(kMsFull, incl, 31);
      s_u[wib][lane] = u;
      s_s[wib][lane] = s;
      s_x[wib][lane] = incl - d;
      __syncwarp();
      for (int64_t base = 0; base < total; base += 32) {
        const int64_t t2 = base + lane;
        const bool valid = t2 < total;
        int64_t e = 0;
        int32_t uu = 0;
        Mask<W> fu = Mask<W>::zero();
        if (valid) {
          int lo = 0, hi = 31;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_x[wib][mid] <= t2)
              lo = mid;
            else
              hi = mid - 1;
          }
          uu = s_u[wib][lo];
          fu = ld_mask<W>(cur, uu);
          e = s_s[wib][lo] + (t2 - s_x[wib][lo]);
        }
        Target<W> t;
        if (valid) t.v = __ldg(p.out_idx + e);
        lg_load<W>(p, t, fu, cur, nxt, tnext, tfront);
        lg_apply<W>(p, uu, t, nxt, tnext, H, acc);
      }
      __syncwarp();
    }
  }
  heavy_rest(p, H);
}

// End of round L (last block to arrive): termination, the next direction,
// statistics, the history bound -- round L + 1 writes F_{L+2}, which must be
// a plane -- and the reset of the record round L + 1 fills.  Lane discoveries
// per round are counted by the output pass, from the history.
template <int W>
__device__ unsigned lg_decide(const MsParams &p, int L, int dir, int ran) {
  MsCtl *ctl = p.ctl;
  const MsRound *Rn = &ctl->rec[(L + 1) % kRing];
  unsigned long long nf = 0, mf = 0;
#pragma unroll
  for (int i = 0; i < kCounterShards; ++i) {
    nf += *(volatile const unsigned long long *)&Rn->nf[i];
    mf += *(volatile const unsigned long long *)&Rn->mf[i];
  }
  cg_stats *st = p.stats;
  const long long now = global_ns();
  if (ran < CG_HISTORY) {
    st->direction_history[ran] = dir;
    st->round_ns[ran] = now - ctl->t_round;
  }
  ctl->t_round = now;
  if (dir == 1) ctl->pull_rounds += 1;
  bool stop = nf == 0;
  if (!stop && L + 1 >= p.level_cap) {
    atomicCAS(&ctl->status, 0, (int)CG_ERR_LEVEL_CAP);
    stop = true;
  }
  if (!stop && L + 2 >= p.hist_planes) {
    *(volatile int *)p.flag = 1;  // outgrew the history: the direct kernel takes over
    stop = true;
  }
  int next;
  if (p.direction == CG_DIR_TOPDOWN)
    next = 0;
  else if (p.direction == CG_DIR_BOTTOMUP)
    next = 1;
  else
    next = ((double)mf * (double)p.ms_alpha > (double)p.nnz) ? 1 : 0;
  if (next != dir) ctl->switches += 1;
  ctl->L = L + 1;
  ctl->dir = next;
  MsRound *Rz = &ctl->rec[(L + 2) % kRing];  // last used in round L - 2
  for (int i = 0; i < kCounterShards; ++i) Rz->nf[i] = Rz->visits[i] = Rz->mf[i] = 0;
  Rz->big = 0;
  Rz->res_light = Rz->res_big = 0;
  Rz->nlight = Rz->work = 0;
  Rz->lanes[0] = Rz->lanes[1] = 0;
  if (stop) {
    const int rounds = ran + 1;
    st->status = *(volatile int *)&ctl->status;
    st->rounds = rounds;
    st->pull_rounds = ctl->pull_rounds;
    st->switches = ctl->switches;
    st->history_len = rounds < CG_HISTORY ? rounds : CG_HISTORY;
    st->device_ms = 0.f;
  }
  return (stop ? kMsStop : 0u) | (next ? kMsNextPull : 0u) |
         (nf * 1024 < (unsigned long long)p.n ? kMsSparse : 0u);
}

template <int W>
struct LgRoundDecision {
  const MsParams *p;
  int L, dir, ran;
  __device__ unsigned operator()() const { return lg_decide<W>(*p, L, dir, ran); }
};

struct LgSetupDecision {
  MsCtl *ctl;
  cg_stats *st;
  __device__ unsigned operator()() const {
    const long long now = global_ns();
    st->setup_ns = now - ctl->t_start;
    st->finish_ns = 0;
    st->visited = 0;
    for (int i = 0; i < CG_HISTORY; ++i) st->nf_history[i] = 0;
    ctl->t_round = now;
    return 0u;
  }
};

// The rounds of one batch (cooperative, persistent): roots[0..k) seeded in
// F_0 and T_0; round L reads F_L and T_L, writes F_{L+1} and T_{L+1}, clears
// F_{L+2} and T_{L+2}.
template <int W>
__global__ void __launch_bounds__(kMsBlock, 2) msbfs_ledger(MsParams p) {
  __shared__ unsigned s_payload;
  MsCtl *ctl = p.ctl;
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t_start = global_ns();
  uint64_t *f0 = plane<W>(p, 0), *f1 = plane<W>(p, 1);
  for (int64_t i = gtid; i < p.n * W; i += nthreads) {
    p.vis[i] = 0;
    f0[i] = 0;
    f1[i] = 0;
  }
  for (int64_t w = gtid; w < p.words; w += nthreads) {
    p.touched0[w] = 0;
    p.touched1[w] = 0;
    p.touched2[w] = 0;
    p.scanmap[w] = 0;
    p.fin[w] = 0;
  }
  uint32_t *pn = reinterpret_cast<uint32_t *>(p.pos_used);
  for (int64_t w = gtid; w < (p.n + 3) / 4; w += nthreads) pn[w] = 0;
  bool ok = grid_wait(&ctl->wait, &ctl->status, p.timeout_ns);
  if (ok && blockIdx.x == 0 && threadIdx.x < p.k) {
    const int i = threadIdx.x;
    const int32_t r = p.roots[i];
    const unsigned long long bit = 1ull << (i & 63);
    atomicOr(reinterpret_cast<unsigned long long *>(f0 + (int64_t)r * W + (i >> 6)), bit);
    atomicOr(p.touched0 + (r >> 5), 1u << (r & 31));
    bool first = true;
    for (int j = 0; j < i; ++j) first = first && (p.roots[j] != r);
    if (first) {
      const int64_t deg = p.out_off[r + 1] - p.out_off[r];
      MsRound *R0 = &ctl->rec[0];
      if (deg > kLightMax) {
        const unsigned long long old = atomicAdd(&R0->big, (1ull << 32) | (unsigned long long)deg);
        p.queue0[p.n - 1 - (int64_t)(old >> 32)] = r;
        p.bigoff0[old >> 32] = (unsigned)old;
      }
      atomicAdd(&R0->nf[0], 1ull);
      atomicAdd(&R0->mf[0], (unsigned long long)deg);
    }
    if (i == 0) {
      const Mask<W> a0 = lane_mask<W>(p.k);
      ctl->rec[0].lanes[0] = a0.w[0];
      ctl->rec[0].lanes[1] = W == 2 ? a0.w[W - 1] : 0ull;
    }
  }
  if (ok) {
    __syncthreads();
    if (threadIdx.x == 0)
      s_payload = arrive_and_wait(&ctl->wait, &ctl->status, p.timeout_ns, 0u,
                                  LgSetupDecision{ctl, p.stats});
    __syncthreads();
    ok = s_payload != kWaitFailed;
  }
  int L = 0, dir = 0, pdir = 0, ran = 0;
  bool sparse = false;  // this round's frontier has under n/1024 vertices (round 0: not tested)
  MsAcc acc, tot;
  while (ok) {
    const uint64_t *cur = plane<W>(p, L);
    uint64_t *nxt = plane<W>(p, L + 1);
    MsRound *Rc = &ctl->rec[L % kRing];
    MsRound *Rn = &ctl->rec[(L + 1) % kRing];
    if (L + 2 < p.hist_planes) {
      uint64_t *clr = plane<W>(p, L + 2);
      for (int64_t i = gtid; i < p.n * W; i += nthreads) clr[i] = 0;
    }
    uint32_t *tclr = claims(p, L + 2);
    for (int64_t w = gtid; w < p.words; w += nthreads) tclr[w] = 0;
    if (L >= 1 && pdir == 0 && (dir == 0 || W != 1)) {
      // a push round gave these vertices lanes and this round is a push too
      // (or 128 lanes): the scan pass resolves their parents (else this pull
      // round's light scans do, or_thread_pos); open_levels has the same rule
      const uint32_t *tcur = claims(p, L);
      for (int64_t w = gtid; w < p.words; w += nthreads) {
        const uint32_t t = tcur[w];
        if (t) atomicOr(p.scanmap + w, t);
      }
    }
    if (dir == 1) {
      Mask<W> active;
#pragma unroll
      for (int i = 0; i < W; ++i) active.w[i] = *(volatile unsigned long long *)&Rc->lanes[i];
      lg_pull<W>(p, L, cur, nxt, active, L >= 1 && pdir == 0, Rc, Rn, acc);
      if (p.nhub > 0) {
        if (!(ok = grid_wait(&ctl->wait, &ctl->status, p.timeout_ns))) break;
        lg_hub_merge<W>(p, L, cur, nxt, Rn, acc);
      }
    } else {
      lg_push<W>(p, L, cur, nxt, sparse, Rc, Rn, acc);
    }
    ms_block_totals(acc, tot);
    if (threadIdx.x == 0) {
      const int sh = blockIdx.x % kCounterShards;
      if (tot.nf) atomicAdd(&Rn->nf[sh], tot.nf);
      if (tot.mf) atomicAdd(&Rn->mf[sh], tot.mf);
      if (tot.lanes[0]) atomicOr(&Rn->lanes[0], tot.lanes[0]);
      if (tot.lanes[1]) atomicOr(&Rn->lanes[1], tot.lanes[1]);
      s_payload = arrive_and_wait(&ctl->wait, &ctl->status, p.timeout_ns, 0u,
                                  LgRoundDecision<W>{&p, L, dir, ran});
    }
    __syncthreads();
    const unsigned payload = s_payload;
    if (payload == kWaitFailed) {
      ok = false;
      break;
    }
    if (payload & kMsStop) break;
    pdir = dir;
    dir = (payload & kMsNextPull) ? 1 : 0;
    sparse = (payload & kMsSparse) != 0;
    ++L;
    ++ran;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && !ok)
    p.stats->status = *(volatile int *)&ctl->status;
}

// ---- scan pass, output pass ---------------------------------------------------

constexpr int kScanBlock = 256;  // scan pass: threads a block
constexpr int kScanWords = 16;   // scan pass: scanmap words a warp takes at a time, at most
constexpr int kScanG = 2;        // in-list entries loaded together (most lanes resolve at the first)
constexpr int kPre = 8;          // history planes loaded together (the output pass needs 8)

// The planes the rounds filled: F_0 .. F_{rounds - 1} (F_rounds is empty).
__device__ __forceinline__ int history_rounds(const MsParams &p) {
  int rounds = *(volatile int *)&p.ctl->L;
  if (rounds > p.hist_planes) rounds = p.hist_planes;
  if (rounds > CG_HISTORY + 1) rounds = CG_HISTORY + 1;
  return rounds;
}

// Bit L: the parents of level L's light vertices were left open -- round L - 1
// pushed, and round L was no pull round that resolves them.
template <int W>
__device__ __forceinline__ uint64_t open_levels(const MsParams &p, int rounds) {
  uint64_t open = 0;
  for (int L = 1; L < rounds && L < CG_HISTORY; ++L) {
    const bool pushed = p.stats->direction_history[L - 1] == 0;
    const bool resolved = W == 1 && p.stats->direction_history[L] == 1;
    if (pushed && !resolved) open |= 1ull << L;
  }
  return open;
}

// Scan pass, between the rounds and the output pass, over the light vertices
// (in-degree 1 .. kPullLight; heavier ones have candidate slots) that the
// rounds marked in scanmap.  A warp takes `grab` words of the map at a time
// (the first by its index, the next from a counter, claimed before the current
// chunk is worked; at 4 words a time the counter's 65,536 atomics took the whole
// 60 us at R-MAT scale 23, 35 us at 16), compacts their marked vertices in shared memory, and gives
// each thread one, whose in-list it scans for the parents of up to kOutLevels
// open levels at once: the first entry u holding a lane of F_L in F_{L-1} is
// its parent, and its position joins the vertex's slices.
template <int W>
__global__ void __launch_bounds__(kScanBlock) msbfs_scan(MsParams p, int grab) {
  __shared__ int32_t s_list[kScanBlock / 32][kScanWords * 32];
  if (*(volatile int *)p.flag || *(volatile int *)&p.ctl->status != 0) return;
  const uint64_t open = open_levels<W>(p, history_rounds(p));
  if (!open) return;
  const int lane = lane_id();
  int32_t *list = s_list[threadIdx.x >> 5];
  const unsigned nwarps = gridDim.x * (kScanBlock / 32);
  const unsigned nchunks = (unsigned)((p.words + grab - 1) / grab);
  unsigned chunk = (unsigned)warp_id_global();
  while (chunk < nchunks) {
    unsigned next = 0;
    if (lane == 0) next = nwarps + atomicAdd(&p.ctl->scan_work, 1u);
    const int64_t w0 = (int64_t)chunk * grab;
    const int64_t wi = w0 + lane;
    uint32_t bits =
        lane < grab && wi < p.words ? p.scanmap[wi] & __ldg(p.light + wi) : 0u;
    const int c = __popc(bits);
    int incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(kMsFull, incl, d);
      if (lane >= d) incl += y;
    }
    const int total = __shfl_sync(kMsFull, incl, 31);
    for (int at = incl - c; bits; bits &= bits - 1) list[at++] = (int32_t)(wi * 32 + __ffs(bits) - 1);
    __syncwarp();
    for (int i = lane; i < total; i += 32) {
      const int64_t v = list[i];
      const int64_t s = __ldg(p.in_off + v), e = __ldg(p.in_off + v + 1);
      Mask<W> A[kPosBits];
#pragma unroll
      for (int b = 0; b < kPosBits; ++b) A[b] = Mask<W>::zero();
      for (uint64_t left = open; left;) {
        int Ls[kOutLevels];
        Mask<W> Ms[kOutLevels], todo = Mask<W>::zero();
#pragma unroll
        for (int k = 0; k < kOutLevels; ++k) {
          Ls[k] = left ? __ffsll((long long)left) - 1 : 0;
          left &= left ? left - 1 : 0ull;
          Ms[k] = Ls[k] ? ld_mask<W>(plane<W>(p, Ls[k]), v) : Mask<W>::zero();
        }
#pragma unroll
        for (int k = 0; k < kOutLevels; ++k) todo = todo | Ms[k];
        for (int64_t j0 = s; j0 < e && todo.any(); j0 += kScanG) {
          int32_t u[kScanG];
          Mask<W> hit[kScanG];
#pragma unroll
          for (int q = 0; q < kScanG; ++q) {
            u[q] = j0 + q < e ? __ldg(p.in_idx + j0 + q) : -1;
            hit[q] = Mask<W>::zero();
          }
#pragma unroll
          for (int q = 0; q < kScanG; ++q)
#pragma unroll
            for (int k = 0; k < kOutLevels; ++k)
              if (u[q] >= 0 && (Ms[k] & todo).any())
                hit[q] = hit[q] | (Ms[k] & ld_mask<W>(plane<W>(p, Ls[k] - 1), u[q]));
#pragma unroll
          for (int q = 0; q < kScanG; ++q) {
            const Mask<W> r = hit[q] & todo;
            const int pos = (int)(j0 - s) + q;
            if (!r.any()) continue;
            todo = todo.andnot(r);
#pragma unroll
            for (int b = 0; b < kPosBits; ++b)
              if ((pos >> b) & 1) A[b] = A[b] | r;
          }
        }
      }
      const unsigned used0 = p.pos_used[v];
      unsigned used = used0;
#pragma unroll
      for (int b = 0; b < kPosBits; ++b) add_slice<W>(p, v, b, A[b], used);
      if (used != used0) p.pos_used[v] = (uint8_t)used;
    }
    __syncwarp();
    chunk = __shfl_sync(kMsFull, next, 0);
  }
}

// Output pass.  Each warp takes 32 consecutive vertices (one per thread).  Per
// 64-lane half of the batch a thread reads its vertex's history masks once
// and keeps each lane's level as bit slices in registers; the parents of a
// vertex with a slot are its candidates (in-degree > kPullLight), copied by
// the warp into the vertex's row of the shared table, those of a light vertex
// the in-list entries at its lanes' positions, bit slices like the levels.
// The bytes of four lanes (levels, table indices) come out of the slices
// together: lanes g, g + 8, g + 16 and g + 24 lie under the same 0x01010101
// mask, one shift and one logic operation a slice.  They are turned round in
// shared memory, so that a thread has four vertices of a lane and writes 16
// bytes at a time, eight threads a 128-byte row piece.  Where rows do not all
// start on 16 bytes (n no multiple of 4), tiles overlap: a tile has the four
// vertices before its own 28 as well, and a row that starts r elements past 16
// bytes (the four lanes of a word share r) gets the 28 from r vertices earlier,
// so every store is still 16 aligned bytes.  Writing such a tile's ends element
// by element instead took 545 us where this takes 289 (n = 1,000,003, 100
// lanes).  Lanes at level 0 are their own vertex's and are written last.
//
// Integer issue bound it when each thread wrote its vertex's values one by one
// (3,900 instructions per tile of 32 vertices and 64 lanes, 2,000 now).  R-MAT
// scale 23, 64 lanes: 1345 -> 1077 us for 5.3 GB; scale 18: 50 -> 34 us.
template <int W>
__global__ void __launch_bounds__(kOutBlock, 5) msbfs_outputs(MsParams p) {
  extern __shared__ __align__(16) unsigned char s_tile[];
  __shared__ unsigned s_cnt[CG_HISTORY + 1];  // lane discoveries per level
  MsCtl *ctl = p.ctl;
  if (*(volatile int *)p.flag) {
    // the gated direct launch that follows needs a clean control block
    if (blockIdx.x == 0) {
      unsigned long long *c = reinterpret_cast<unsigned long long *>(ctl);
      for (int i = threadIdx.x; i < (int)(sizeof(MsCtl) / 8); i += blockDim.x) c[i] = 0ull;
    }
    return;
  }
  if (*(volatile int *)&ctl->status != 0) return;  // timed out or over the level cap
  const int rounds = history_rounds(p);
  for (int i = threadIdx.x; i <= CG_HISTORY; i += blockDim.x) s_cnt[i] = 0;
  __syncthreads();
  constexpr uint32_t kOne = 0x01010101u;
  const int lane = lane_id();
  const int wib = threadIdx.x >> 5;
  int32_t *tab = reinterpret_cast<int32_t *>(s_tile + wib * kOutWarpBytes);
  int32_t *my_tab = tab + lane * kTab;
  uint32_t *s_level = reinterpret_cast<uint32_t *>(tab) + 32 * kTab, *s_index = s_level + kStage;
  my_tab[kTabNone] = -1;
  unsigned found[kPre];  // lanes of my vertices at levels 0 .. kPre - 1
#pragma unroll
  for (int j = 0; j < kPre; ++j) found[j] = 0;
  int nsl = 1;  // bit slices needed for levels 0 .. rounds - 1
  while (nsl < kSlices && (rounds - 1) >> nsl) ++nsl;
  const int64_t nwarps = (int64_t)gridDim.x * kOutWarps;
  // rows aligned alike in both outputs (else they are written one by one), and
  // whether any is off 16 bytes: then tiles are 28 vertices and the 4 before
  const bool same_align = ((reinterpret_cast<uintptr_t>(p.levels) ^
                            reinterpret_cast<uintptr_t>(p.parents)) & 15u) == 0;
  const int before = (p.n & 3) || (reinterpret_cast<uintptr_t>(p.levels) & 15u) ? 4 : 0;
  const int own_tile = 32 - before;  // vertices of a tile
  const int64_t tiles = (p.n + (before ? 3 : 0) + own_tile - 1) / own_tile;
  // a tile's slots, position flags and list bounds are loaded one tile ahead:
  // the tile's history, candidate and list loads then all go out at its start
  int64_t tile = (int64_t)blockIdx.x * kOutWarps + wib;
  int next_slot = -1;
  unsigned next_used = 0, next_deg = 0;
  int64_t next_s = 0;
  auto look_ahead = [&](int64_t v) {
    next_slot = -1;
    next_used = next_deg = 0;
    if (v >= 0 && v < p.n) {
      next_slot = p.cand_slot[v];
      next_used = p.pos_used[v];
      next_s = __ldg(p.in_off + v);
      next_deg = (unsigned)min(__ldg(p.in_off + v + 1) - next_s, (int64_t)kPullLight);
    }
  };
  look_ahead(tile * own_tile - before + lane);
  for (; tile < tiles; tile += nwarps) {
    const int64_t v = tile * own_tile - before + lane;
    const bool valid = v >= 0 && v < p.n;
    const int slot = next_slot;
    const unsigned used = slot < 0 ? next_used : 0u;
    const int64_t s = next_s;
    // entries that positions can point at: 2^(slices in use), within the list
    const unsigned entries = slot < 0 ? min(next_deg, 1u << (32 - __clz(used))) : 0u;
    const unsigned tile_used = __reduce_or_sync(kMsFull, used);
    look_ahead((tile + nwarps) * own_tile - before + lane);
#pragma unroll 1
    for (int h = 0; h < W && 64 * h < p.k; ++h) {
      // the first kPre history planes: independent of the loads below, so they
      // are issued first and their latency overlaps
      uint64_t pm0[kPre];
#pragma unroll
      for (int j = 0; j < kPre; ++j)
        pm0[j] = valid && j < rounds ? plane<W>(p, j)[v * W + h] : 0ull;
      uint64_t Q[kPosBits];  // bit l of Q[b]: bit b of lane l's position
#pragma unroll
      for (int b = 0; b < kPosBits; ++b)
        Q[b] = (used >> b) & 1u ? p.pos[((int64_t)b * p.n + v) * W + h] : 0ull;
      // a light vertex's list entries, and the 256-byte candidate rows of the
      // tile's slotted vertices (by the warp), go into the table while the
      // slices are made: asynchronous copies, all in flight at once
      if (h == 0)
        for (unsigned q = 0; q < entries; ++q) copy_async4(my_tab + q, p.in_idx + s + q);
      for (unsigned pend = __ballot_sync(kMsFull, slot >= 0); pend; pend &= pend - 1) {
        const int src = __ffs(pend) - 1;
        const uint32_t *row =
            p.cand + (int64_t)__shfl_sync(kMsFull, slot, src) * (64 * W) + 64 * h;
        int32_t *t = tab + src * kTab;
        copy_async4(t + ((lane - 8 * src) & 63), row + lane);
        copy_async4(t + ((lane + 32 - 8 * src) & 63), row + lane + 32);
      }
      // each lane's level as bit slices: bit l of S[b] = bit b of lane l's level
      uint64_t S[kSlices], reached = 0;
#pragma unroll
      for (int b = 0; b < kSlices; ++b) S[b] = 0;
      const uint64_t own = pm0[0];  // lanes whose root is v
      for (int L0 = 0; L0 < rounds; L0 += kPre) {  // uniform: the whole warp
        uint64_t pm[kPre];
#pragma unroll
        for (int j = 0; j < kPre; ++j)
          pm[j] = L0 == 0 ? pm0[j]
                          : (valid && L0 + j < rounds ? plane<W>(p, L0 + j)[v * W + h] : 0ull);
        // L0 is a multiple of kPre = 8: bits 0..2 of level L0 + j are those
        // of j, known at compile time; bits 3.. those of L0, the same for the
        // whole batch
        uint64_t batch = 0;
#pragma unroll
        for (int j = 0; j < kPre; ++j) {
          const uint64_t m = pm[j];
          const unsigned mine = lane >= before ? (unsigned)__popcll(m) : 0u;  // once a vertex
          if (L0 == 0) {
            found[j] += mine;
          } else {
            const unsigned c = __reduce_add_sync(kMsFull, mine);
            if (lane == 0 && c) atomicAdd(&s_cnt[L0 + j], c);
          }
          batch |= m;
#pragma unroll
          for (int b = 0; b < 3; ++b)
            if ((j >> b) & 1) S[b] |= m;
        }
        reached |= batch;
#pragma unroll
        for (int b = 3; b < kSlices; ++b)
          if ((L0 >> b) & 1) S[b] |= batch;
      }
      copy_async_wait();
      __syncwarp();  // the candidate rows copied by the warp are in place
      // rows: lane l of this half, vertices tile*32 .. tile*32 + 31, a 32-lane
      // word of the masks at a time
      const int lanes = min(64, p.k - 64 * h);
      const int64_t n = p.n;
      const uint32_t slotted = slot >= 0 ? ~0u : 0u;
#pragma unroll 1
      for (int hw = 0; hw < 2 && 32 * hw < lanes; ++hw) {
        uint32_t sl[kSlices], qs[kPosBits];
#pragma unroll
        for (int b = 0; b < kSlices; ++b) sl[b] = (uint32_t)(S[b] >> (32 * hw));
#pragma unroll
        for (int b = 0; b < kPosBits; ++b) qs[b] = (uint32_t)(Q[b] >> (32 * hw));
        const uint32_t rw = (uint32_t)(reached >> (32 * hw));
        // table columns of lanes 0, 8, 16, 24 of the word (a slotted vertex):
        // multiples of 8, so lane l + 8 i's is l more, without a wrap
        const uint32_t col =
            ((((uint32_t)(32 * hw - 8 * lane) & 63u) * kOne + 0x18100800u) & 0x3f3f3f3fu) & slotted;
        // bit g + 8 i of x at bit b of byte i
        auto bits_at = [](uint32_t x, int g, int b) {
          return (g >= b ? x >> (g - b) : x << (b - g)) & (kOne << b);
        };
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          // lanes g + 8 i, i = 0..3, in byte i: 0xFF where unreached (um), the
          // level (0xFF unreached sign-extends to -1), the table index
          const uint32_t um = bits_at(~rw, g, 0) * 0xFFu;
          uint32_t word = um, pos = 0;
#pragma unroll
          for (int b = 0; b < 3; ++b) word |= bits_at(sl[b], g, b);
          if (nsl > 3) {
#pragma unroll
            for (int b = 3; b < kSlices; ++b) word |= bits_at(sl[b], g, b);
          }
#pragma unroll
          for (int b = 0; b < 3; ++b) pos |= bits_at(qs[b], g, b);
          if (tile_used >> 3) {
#pragma unroll
            for (int b = 3; b < kPosBits; ++b) pos |= bits_at(qs[b], g, b);
          }
          const uint32_t at = pos | ((col + (uint32_t)g * kOne) & slotted);
          s_level[kStageRow * g + lane] = word;
          s_index[kStageRow * g + lane] = (at & ~um) | (kTabNone * kOne & um);
        }
        __syncwarp();
        // thread (g, j): four vertices of lanes g + 8 i
        const int j = lane & 7;
        const int64_t v0 = tile * own_tile;
        const bool inner = same_align && v0 >= before && v0 + own_tile <= n;
#pragma unroll 1
        for (int g = lane >> 3; g < 8; g += 4) {
          const int64_t at0 = (int64_t)(64 * h + 32 * hw + g) * n;
          // elements past 16 bytes at v0, the same for every i (8 n is a
          // multiple of 4)
          const int r = (int)((reinterpret_cast<uintptr_t>(p.levels + at0 + v0) >> 2) & 3u);
          const int first = 4 * j - r;  // this thread's vertices are v0 + first ..
          uint32_t lws[4], iws[4];
          const int32_t *row[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int t = (before + first + c) & 31;
            lws[c] = s_level[kStageRow * g + t];
            iws[c] = s_index[kStageRow * g + t];
            row[c] = tab + t * kTab;
          }
          const bool mine = 4 * j < own_tile;
          int32_t *pl = p.levels + at0 + v0 + first, *pp = p.parents + at0 + v0 + first;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (32 * hw + 8 * i >= lanes) break;  // uniform: no such lanes
            int32_t lv[4], pv[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              lv[c] = (int32_t)(int8_t)(uint8_t)(lws[c] >> (8 * i));
              pv[c] = row[c][(iws[c] >> (8 * i)) & 0xFFu];
            }
            if (mine && 32 * hw + g + 8 * i < lanes) {
              if (inner) {  // written once, never read here: evict-first
                __stcs(reinterpret_cast<int4 *>(pl), make_int4(lv[0], lv[1], lv[2], lv[3]));
                __stcs(reinterpret_cast<int4 *>(pp), make_int4(pv[0], pv[1], pv[2], pv[3]));
              } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                  const int64_t x = v0 + first + c;
                  if (x >= 0 && x < n) {
                    __stcs(pl + c, lv[c]);
                    __stcs(pp + c, pv[c]);
                  }
                }
              }
            }
            pl += 8 * n;
            pp += 8 * n;
          }
        }
        __syncwarp();  // the staged words are read
      }
      // (after the syncwarp, so after whichever thread wrote these elements; an
      // overlapped vertex is in the tile that wrote the row's element)
      for (uint64_t x = own; x; x &= x - 1) {
        const int64_t at = (int64_t)(64 * h + __ffsll((long long)x) - 1) * n;
        const int r =
            (int)((reinterpret_cast<uintptr_t>(p.levels + at + tile * own_tile) >> 2) & 3u);
        const int t = lane - before + r;
        if (t >= 0 && t < own_tile) p.parents[at + v] = (int32_t)v;
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int j = 0; j < kPre; ++j) {
    const unsigned c = __reduce_add_sync(kMsFull, found[j]);
    if (lane == 0 && c) atomicAdd(&s_cnt[j], c);
  }
  // the statistics: lane discoveries per round (level L came from round
  // L - 1) and in all; the last block out records the time since the last
  // round ended
  __syncthreads();
  for (int i = threadIdx.x; i < rounds; i += blockDim.x) {
    const unsigned long long c = s_cnt[i];  // widened for the global sums
    if (!c) continue;
    atomicAdd(reinterpret_cast<unsigned long long *>(&p.stats->visited), c);
    if (i >= 1)
      atomicAdd(reinterpret_cast<unsigned long long *>(&p.stats->nf_history[i - 1]), c);
  }
  if (threadIdx.x == 0 && atomicAdd(&ctl->exited, 1u) + 1u == gridDim.x)
    p.stats->finish_ns = global_ns() - *(volatile long long *)&ctl->t_round;
}

// What warps take at a time: the largest power of two that still leaves two
// items for every warp.  More items than that only add atomics on
// the round's work counter (one each, about 1 ns apart: the last pull round of 64
// lanes on R-MAT scale 23 spent 220 us on 190,000 items, 171 us on 53,000), fewer
// leave warps idle (scale 18: 4,864 warps shared 1,024 groups of 8 words; rounds
// 125 / 84 us, 80 / 58 us now).
unsigned grab_of(int64_t things, unsigned least, unsigned most, int64_t warps, unsigned *items) {
  unsigned g = least;
  while (g < most && things >= 4 * (int64_t)g * warps) g <<= 1;
  *items = (unsigned)((things + g - 1) / g);
  return g;
}

void pull_grabs(MsParams &p, int64_t warps) {
  p.light_grab = grab_of(p.words, 1, 32, warps, &p.light_items);
  p.med_grab = grab_of(p.nmed, 1, 32, warps, &p.med_items);
  p.hub_grab = grab_of(p.hub_chunks, 1, 4, warps, &p.hub_items);
}

template <int W>
int ledger_pass(cg_graph *g, MsState *s, const int64_t *roots, int k, int32_t *d_levels,
                int32_t *d_parents) {
  MsParams p = ms_params<W>(g, s);
  p.levels = d_levels;
  p.parents = d_parents;
  p.k = k;
  for (int i = 0; i < kMsMaxLanes; ++i) p.roots[i] = i < k ? (int32_t)roots[i] : 0;
  int rc = ms_reset<W>(s, g->stream);
  if (rc) return rc;
  int block = g->opt.block_size > 0 ? g->opt.block_size : kMsBlock;
  if (block > kMsBlock) block = kMsBlock;
  block = (block / 32) * 32;
  if (block < 128) block = 128;  // seeding uses threads 0..k-1 of block 0
  int per_sm = 0;
  CG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, msbfs_ledger<W>, block, 0));
  if (per_sm <= 0) return CG_ERR_NOT_SUPPORTED;
  if (g->opt.blocks_per_sm > 0 && g->opt.blocks_per_sm < per_sm) per_sm = g->opt.blocks_per_sm;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(per_sm * g->num_sms);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = g->stream;
  // The rounds gather through the L1, which is what shared memory leaves of an
  // SM.  Without a stated share the SM keeps the split of the kernel before it
  // where that is large enough, and started right behind another handle's
  // output pass (209 KB of shared memory a block set) every round ran on 20 KB
  // of L1: three handles taking turns, n = 1,000,003, 100 lanes, rounds 829 us
  // for 566; R-MAT scale 23, 64 lanes, 8.1 ms for 3.5.  Whole batches there:
  // 1,223 -> 970 us and 4.5 to 5.4 -> 3.9 ms.
  cudaFuncAttributes fa;
  CG_CUDA(cudaFuncGetAttributes(&fa, msbfs_ledger<W>));
  const size_t shared = (fa.sharedSizeBytes + kSmemReserved) * (size_t)per_sm;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  attr[1].val.sharedMemCarveout = (unsigned)((shared * 100 + kSmemOfSm - 1) / kSmemOfSm);
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  pull_grabs(p, per_sm * g->num_sms * (block / 32));
  CG_CUDA(cudaLaunchKernelEx(&cfg, msbfs_ledger<W>, p));
  int scan_per_sm = 0;
  CG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&scan_per_sm, msbfs_scan<W>, kScanBlock, 0));
  if (scan_per_sm <= 0) return CG_ERR_NOT_SUPPORTED;
  unsigned scan_items = 0;
  const int64_t scan_warps = (int64_t)scan_per_sm * g->num_sms * (kScanBlock / 32);
  const int scan_words = (int)grab_of(p.words, 4, kScanWords, scan_warps, &scan_items);
  int64_t scan_blocks = ((int64_t)scan_items + kScanBlock / 32 - 1) / (kScanBlock / 32);
  if (scan_blocks > (int64_t)scan_per_sm * g->num_sms) scan_blocks = (int64_t)scan_per_sm * g->num_sms;
  msbfs_scan<W><<<(unsigned)scan_blocks, kScanBlock, 0, g->stream>>>(p, scan_words);
  const int smem = kOutWarps * kOutWarpBytes;
  CG_CUDA(cudaFuncSetAttribute(msbfs_outputs<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               smem));
  int out_per_sm = 0;
  CG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&out_per_sm, msbfs_outputs<W>, kOutBlock,
                                                        smem));
  if (out_per_sm <= 0) return CG_ERR_NOT_SUPPORTED;
  const int64_t tiles = (g->n + 3 + 27) / 28;  // of 28 vertices where rows are ragged, else 32
  int64_t blocks = (tiles + kOutWarps - 1) / kOutWarps;
  const int64_t cap = (int64_t)out_per_sm * g->num_sms;
  if (blocks > cap) blocks = cap;
  msbfs_outputs<W><<<(unsigned)blocks, kOutBlock, smem, g->stream>>>(p);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

}  // namespace

int ms_ledger_pass(cg_graph *g, MsState *s, const int64_t *roots, int k, int32_t *d_levels,
                   int32_t *d_parents) {
  return s->lane_words == 2 ? ledger_pass<2>(g, s, roots, k, d_levels, d_parents)
                            : ledger_pass<1>(g, s, roots, k, d_levels, d_parents);
}

}  // namespace cg
