// Kernel-1 construction on the device: synthetic edge generation and the
// edge-list -> CSR/CSC build, so that graphs at scale 23-26 are built in
// seconds instead of the reference's tens of host seconds
// (docs/ERRORS.md:121-136 reports ~20 s for the s17 upload alone).
//
// R-MAT (datasets/gen_rmat.py:15-44) draws one double per edge per level
// from np.random.default_rng(seed) -- a PCG64 stream (128-bit LCG, XSL-RR
// output) consumed level by level, rng.random(m) each.  Each thread here owns
// R consecutive edges: it jumps its generator to the first of them once, draws
// its R doubles of a level, then jumps by m - R to the same edges of the next
// level.  Jump-ahead is Brown's arbitrary-stride LCG method ("Random number
// generation with arbitrary strides", 1994): the affine map s -> a s + c
// applied d times, by square-and-multiply.  A double is (x >> 11) * 2^-53, so
// every quadrant test "r >= t" is done exactly on the 53-bit integer against
// ceil(t * 2^53), computed on the host.
//
// CSR build: CUB radix sorts of as few keys and as few bits as will do.  A
// symmetrised graph sorts each undirected edge once, as (low end, high end);
// that is the upper triangle, and its stable sort by the high end (32-bit keys)
// is the lower one, whose entries precede the upper ones in every row.  A
// directed graph's CSC is the stable sort of its CSR by column.  Keys hold
// 2 * ceil(log2 n) bits, dropped loops the key 0 = (0, 0), which cannot be an
// entry then.  Offsets come from the places where the sorted rows change.
// Bound by the sorts' passes over memory (8 bits a pass).  R-MAT scale 20, 16.8
// M edges: 5 passes of 16.8 M 64-bit keys and 3 of 15.7 M 32-bit pairs where one
// sort of both directions took 7 of 33.5 M; device time 2580 -> 1620 us (with
// one search).
#include <cuda_runtime.h>
#include <stdint.h>

#include <cub/cub.cuh>
#include <new>

#include "cg_internal.cuh"

namespace cg {

typedef unsigned __int128 u128;

__host__ __device__ __forceinline__ u128 mk128(uint64_t hi, uint64_t lo) {
  return ((u128)hi << 64) | (u128)lo;
}

static constexpr uint64_t kPcgMulHi = 0x2360ED051FC65DA4ull;
static constexpr uint64_t kPcgMulLo = 0x4385DF649FCCF645ull;

struct Affine {  // s -> mul * s + add (mod 2^128)
  u128 mul, add;
};

__host__ __device__ inline Affine lcg_jump(u128 inc, uint64_t delta) {
  u128 cur_mul = mk128(kPcgMulHi, kPcgMulLo), cur_add = inc;
  u128 acc_mul = 1, acc_add = 0;
  while (delta) {
    if (delta & 1) {
      acc_mul *= cur_mul;
      acc_add = acc_add * cur_mul + cur_add;
    }
    cur_add = (cur_mul + 1) * cur_add;
    cur_mul *= cur_mul;
    delta >>= 1;
  }
  return Affine{acc_mul, acc_add};
}

__device__ __forceinline__ uint64_t pcg_next(u128 &s, u128 inc) {
  s = s * mk128(kPcgMulHi, kPcgMulLo) + inc;
  const uint64_t x = (uint64_t)(s >> 64) ^ (uint64_t)s;
  const unsigned rot = (unsigned)(s >> 122);
  return (x >> rot) | (x << ((64u - rot) & 63u));
}

struct RmatParams {
  uint64_t st_hi, st_lo, inc_hi, inc_lo;  // generator state after seeding
  uint64_t t_a, t_ab, t_abc;              // ceil(t * 2^53) of A, A+B, A+B+C
  uint64_t skip_mul_hi, skip_mul_lo, skip_add_hi, skip_add_lo;  // jump by m - R
  int64_t m;
  int scale;
};

template <int R>
__global__ void rmat_kernel(RmatParams p, uint32_t *__restrict__ u_out,
                            uint32_t *__restrict__ v_out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t e0 = t * R;
  if (e0 >= p.m) return;
  const u128 inc = mk128(p.inc_hi, p.inc_lo);
  const int64_t cnt = (p.m - e0) < R ? (p.m - e0) : R;
  Affine j0 = lcg_jump(inc, (uint64_t)e0);
  u128 s = j0.mul * mk128(p.st_hi, p.st_lo) + j0.add;
  Affine skip;
  if (cnt == R)
    skip = Affine{mk128(p.skip_mul_hi, p.skip_mul_lo), mk128(p.skip_add_hi, p.skip_add_lo)};
  else
    skip = lcg_jump(inc, (uint64_t)(p.m - cnt));
  uint32_t u[R], v[R];
#pragma unroll
  for (int j = 0; j < R; ++j) u[j] = v[j] = 0;
  for (int level = 0; level < p.scale; ++level) {
    const uint32_t bit = 1u << (p.scale - 1 - level);
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (j < cnt) {
        const uint64_t k = pcg_next(s, inc) >> 11;
        const bool ub = k >= p.t_ab;
        const bool vb = (k >= p.t_a && k < p.t_ab) || k >= p.t_abc;
        u[j] |= ub ? bit : 0u;
        v[j] |= vb ? bit : 0u;
      }
    }
    s = skip.mul * s + skip.add;
  }
#pragma unroll
  for (int j = 0; j < R; ++j)
    if (j < cnt) {
      u_out[e0 + j] = u[j];
      v_out[e0 + j] = v[j];
    }
}

// k-th double of the stream -> floor(r * 2^bits), k = first + e
__global__ void uniform_bits_kernel(uint64_t st_hi, uint64_t st_lo, uint64_t inc_hi,
                                    uint64_t inc_lo, uint64_t first, int64_t count, int bits,
                                    uint32_t *__restrict__ out) {
  constexpr int R = 16;
  const int64_t e0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * R;
  if (e0 >= count) return;
  const u128 inc = mk128(inc_hi, inc_lo);
  Affine j0 = lcg_jump(inc, first + (uint64_t)e0);
  u128 s = j0.mul * mk128(st_hi, st_lo) + j0.add;
  for (int j = 0; j < R && e0 + j < count; ++j)
    out[e0 + j] = (uint32_t)((pcg_next(s, inc) >> 11) >> (53 - bits));
}

// One key per edge: (row = dst) << bits | (col = src), or, symmetrised, the
// smaller end << bits | the larger one.
__global__ void edge_keys_kernel(int64_t m, const uint32_t *__restrict__ src,
                                 const uint32_t *__restrict__ dst, int symmetrize,
                                 int drop_loops, int bits, uint64_t *__restrict__ keys) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m;
       e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t s = src[e], d = dst[e];
    const uint64_t hi = symmetrize ? min(s, d) : d, lo = symmetrize ? max(s, d) : s;
    keys[e] = drop_loops && s == d ? 0ull : (hi << bits) | lo;
  }
}

// Rows without entries between two that have some, too many for one thread.
struct Gap {
  uint32_t first, last, at;  // rows [first, last] start at position `at`
};
constexpr int64_t kGapRows = 64;        // rows a thread fills itself
constexpr int64_t kGapPiece = 1 << 16;  // rows per listed piece of a longer gap
static int64_t gap_capacity(int64_t n) { return n / kGapRows + n / kGapPiece + 2; }

// first[r] = the first position whose row is >= r, for the rows after that of
// position i - 1 up to that of position i (every r <= n over all i <= count);
// long gaps go on a list for fill_gaps_kernel.  Rows past n count as n.
__device__ __forceinline__ void mark_rows(int64_t n, int64_t count, int64_t i, int64_t before,
                                          int64_t row, uint32_t *__restrict__ first,
                                          Gap *__restrict__ gaps, unsigned *ngaps) {
  const int64_t r0 = i > 0 ? min(before, n) + 1 : 0, r1 = i < count ? min(row, n) : n;
  if (r1 - r0 < kGapRows) {
    for (int64_t r = r0; r <= r1; ++r) first[r] = (uint32_t)i;
    return;
  }
  const unsigned pieces = (unsigned)((r1 - r0) / kGapPiece) + 1;
  unsigned at = atomicAdd(ngaps, pieces);
  for (int64_t r = r0; r <= r1; r += kGapPiece)
    gaps[at++] = Gap{(uint32_t)r, (uint32_t)min(r + kGapPiece - 1, r1), (uint32_t)i};
}

__global__ void fill_gaps_kernel(const Gap *__restrict__ gaps, const unsigned *ngaps,
                                 uint32_t *__restrict__ first) {
  const unsigned count = *ngaps;
  for (unsigned g = blockIdx.x; g < count; g += gridDim.x) {
    const Gap x = gaps[g];
    for (uint32_t r = x.first + threadIdx.x; r <= x.last && r >= x.first; r += blockDim.x)
      first[r] = x.at;
  }
}

// Row starts of the sorted keys, and each key's (column, row) for the sort by
// column.  `loop_row`, if not negative: the column given to a loop (a
// symmetrised graph's upper triangle holds it already).
__global__ void split_keys_kernel(int64_t n, int64_t count, const uint64_t *__restrict__ keys,
                                  int bits, int64_t loop_row, uint32_t *__restrict__ first,
                                  uint32_t *__restrict__ cols, uint32_t *__restrict__ rows,
                                  Gap *__restrict__ gaps, unsigned *ngaps) {
  const uint64_t mask = (1ull << bits) - 1ull;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= count;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = i < count ? keys[i] : 0ull;
    const int64_t row = (int64_t)(k >> bits);
    mark_rows(n, count, i, i > 0 ? (int64_t)(keys[i - 1] >> bits) : 0, row, first, gaps, ngaps);
    if (i == count) continue;
    const uint32_t col = (uint32_t)(k & mask);
    cols[i] = loop_row >= 0 && col == row ? (uint32_t)loop_row : col;
    rows[i] = (uint32_t)row;
  }
}

__global__ void row_starts_kernel(int64_t n, int64_t count, const uint32_t *__restrict__ rows,
                                  uint32_t *__restrict__ first, Gap *__restrict__ gaps,
                                  unsigned *ngaps) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= count;
       i += (int64_t)gridDim.x * blockDim.x)
    mark_rows(n, count, i, i > 0 ? rows[i - 1] : 0, i < count ? rows[i] : 0, first, gaps, ngaps);
}

// CSR of the sorted keys (first: its row starts).
__global__ void csr_kernel(int64_t n, int64_t nnz, const uint64_t *__restrict__ keys, int bits,
                           const uint32_t *__restrict__ first, int64_t *__restrict__ off,
                           int32_t *__restrict__ idx) {
  const uint64_t mask = (1ull << bits) - 1ull;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = t0; i < nnz; i += stride) idx[i] = (int32_t)(keys[i] & mask);
  for (int64_t r = t0; r <= n; r += stride) off[r] = first[r];
}

// The same from (row, column) pairs sorted by row.
__global__ void csr_pairs_kernel(int64_t n, int64_t nnz, const uint32_t *__restrict__ cols,
                                 const uint32_t *__restrict__ first, int64_t *__restrict__ off,
                                 int32_t *__restrict__ idx) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = t0; i < nnz; i += stride) idx[i] = (int32_t)cols[i];
  for (int64_t r = t0; r <= n; r += stride) off[r] = first[r];
}

// CSR of a symmetrised graph.  up: row starts of the upper triangle's keys;
// low: row starts of the lower triangle's pairs.  A row's lower entries come
// first, so row r starts at up[r] + low[r]; the upper entry at position i lies
// behind the lower entries of rows 0 .. its own, at i + low[row + 1], the lower
// one at position j behind the upper entries of the rows before, at j + up[row].
__global__ void csr_symmetric_kernel(int64_t n, int64_t nu, int64_t nl,
                                     const uint64_t *__restrict__ keys, int bits,
                                     const uint32_t *__restrict__ up,
                                     const uint32_t *__restrict__ low_rows,
                                     const uint32_t *__restrict__ low_cols,
                                     const uint32_t *__restrict__ low, int64_t *__restrict__ off,
                                     int32_t *__restrict__ idx) {
  const uint64_t mask = (1ull << bits) - 1ull;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = t0; i < nu; i += stride) {
    const uint64_t k = keys[i];
    const int64_t row = min((int64_t)(k >> bits), n - 1);
    idx[i + low[row + 1]] = (int32_t)(k & mask);
  }
  for (int64_t j = t0; j < nl; j += stride)
    idx[j + up[min((int64_t)low_rows[j], n)]] = (int32_t)low_cols[j];
  for (int64_t r = t0; r <= n; r += stride) off[r] = (int64_t)up[r] + low[r];
}

// A == A^T exactly when the CSR and the CSC of the same entries coincide.
__global__ void same_arrays_kernel(int64_t n, int64_t nnz, const int64_t *__restrict__ a_off,
                                   const int32_t *__restrict__ a_idx,
                                   const int64_t *__restrict__ b_off,
                                   const int32_t *__restrict__ b_idx, unsigned *differ) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool d = false;
  for (int64_t i = t0; i < nnz; i += stride) d |= a_idx[i] != b_idx[i];
  for (int64_t r = t0; r <= n; r += stride) d |= a_off[r] != b_off[r];
  if (__any_sync(0xffffffffu, d) && (threadIdx.x & 31) == 0) atomicOr(differ, 1u);
}

static int grid_for(int64_t work, int num_sms) {
  int64_t b = (work + 255) / 256;
  const int64_t cap = (int64_t)num_sms * 32;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

static int value_bits(int64_t n) {  // bits of the values 0 .. n - 1, at least 1
  int b = 1;
  while (b < 62 && (1ll << b) < n) ++b;
  return b;
}

// A build's device scratch: one allocation, cut into 256-byte aligned pieces.
struct Scratch {
  unsigned char *base = nullptr;
  size_t used = 0;
  template <class T>
  T *take(int64_t count) {
    T *p = reinterpret_cast<T *>(base + used);
    used = (used + sizeof(T) * (size_t)count + 255) & ~(size_t)255;
    return p;
  }
};

// The buffers of one build, laid out in `s` (once without memory, for the
// size).  The second sort's pairs take the space of the first's input; its
// other set that of the unique keys when those are done with (a directed
// graph), else space of its own.
struct BuildSpace {
  uint64_t *keys, *tmp;      // [m]
  uint32_t *pairs;           // [2 m], symmetrised graphs only
  uint32_t *first[2];        // [n + 1] row starts of the two sorts
  Gap *gaps;
  int64_t *count;
  unsigned *zeros;           // two gap counts and the symmetry flag
  void *temp;
  BuildSpace(Scratch &s, int64_t n, int64_t m, bool sym, size_t temp_bytes) {
    keys = s.take<uint64_t>(m);
    tmp = s.take<uint64_t>(m);
    pairs = s.take<uint32_t>(sym ? 2 * m : 0);
    for (int i = 0; i < 2; ++i) first[i] = s.take<uint32_t>(n + 1);
    gaps = s.take<Gap>(gap_capacity(n));
    count = s.take<int64_t>(1);
    zeros = s.take<unsigned>(3);
    temp = s.take<unsigned char>((int64_t)temp_bytes);
  }
};

}  // namespace cg

using namespace cg;

extern "C" {

int cg_rmat_edges(int32_t scale, int64_t m, const uint64_t *gen_state,
                  const uint64_t *thresholds, uint32_t *d_u, uint32_t *d_v, void *stream) {
  if (scale < 1 || scale > 31 || m <= 0 || !gen_state || !thresholds || !d_u || !d_v)
    return CG_ERR_INVALID_ARG;
  constexpr int R = 16;
  RmatParams p;
  p.st_hi = gen_state[0];
  p.st_lo = gen_state[1];
  p.inc_hi = gen_state[2];
  p.inc_lo = gen_state[3];
  p.t_a = thresholds[0];
  p.t_ab = thresholds[1];
  p.t_abc = thresholds[2];
  const Affine skip = lcg_jump(mk128(p.inc_hi, p.inc_lo), (uint64_t)(m - R));
  p.skip_mul_hi = (uint64_t)(skip.mul >> 64);
  p.skip_mul_lo = (uint64_t)skip.mul;
  p.skip_add_hi = (uint64_t)(skip.add >> 64);
  p.skip_add_lo = (uint64_t)skip.add;
  p.m = m;
  p.scale = scale;
  const int64_t threads = (m + R - 1) / R;
  const int block = 128;
  rmat_kernel<R><<<(unsigned)((threads + block - 1) / block), block, 0, (cudaStream_t)stream>>>(
      p, d_u, d_v);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

int cg_uniform_bits(const uint64_t *gen_state, uint64_t first, int64_t count, int32_t bits,
                    uint32_t *d_out, void *stream) {
  if (!gen_state || count <= 0 || bits < 1 || bits > 32 || !d_out) return CG_ERR_INVALID_ARG;
  const int64_t threads = (count + 15) / 16;
  uniform_bits_kernel<<<(unsigned)((threads + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
      gen_state[0], gen_state[1], gen_state[2], gen_state[3], first, count, bits, d_out);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

int cg_graph_from_edges(int64_t n, int64_t m, const uint32_t *d_src, const uint32_t *d_dst,
                        int32_t flags, cg_graph **out) {
  if (!out || n <= 0 || n > 0x7fffffffLL || m < 0 || (m > 0 && (!d_src || !d_dst)))
    return CG_ERR_INVALID_ARG;
  *out = nullptr;
  const bool sym = (flags & CG_EDGES_SYMMETRIZE) != 0;
  const bool drop = (flags & CG_EDGES_DROP_LOOPS) != 0;
  const bool detect = (flags & CG_EDGES_DETECT_SYMMETRIC) != 0;
  int dev = 0, sms = 0;
  CG_CUDA(cudaGetDevice(&dev));
  CG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  cudaStream_t st = nullptr;
  CG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  const int bits = value_bits(n);
  // the second sort's rows: a kept loop of a symmetrised graph gets row n there
  const bool loops = sym && !drop;
  const int row_bits = loops ? value_bits(n + 1) : bits;
  Scratch mem;
  int64_t *off[2] = {nullptr, nullptr};
  int32_t *idx[2] = {nullptr, nullptr};
  int64_t nnz = 0;
  bool found_sym = false;
  int rc = CG_OK;
  auto fail = [&](cudaError_t e, const char *what) { rc = cuda_fail(e, what); };
  auto alloc = [&](auto **p, int64_t count) {
    if (cudaMalloc(p, sizeof(**p) * (size_t)(count > 0 ? count : 1)) == cudaSuccess) return true;
    cudaGetLastError();
    rc = CG_ERR_OUT_OF_MEMORY;
    return false;
  };
  do {
    if (m == 0) {
      if (!alloc(&off[0], n + 1) || !alloc(&idx[0], 1)) break;
      const cudaError_t e = cudaMemsetAsync(off[0], 0, sizeof(int64_t) * (size_t)(n + 1), st);
      if (e != cudaSuccess) { fail(e, "empty offsets"); break; }
      break;
    }
    size_t tb_keys = 0, tb_pairs = 0, tb_uniq = 0;
    {
      cub::DoubleBuffer<uint64_t> kb(nullptr, nullptr);
      cub::DoubleBuffer<uint32_t> pk(nullptr, nullptr), pv(nullptr, nullptr);
      cudaError_t e = cub::DeviceRadixSort::SortKeys(nullptr, tb_keys, kb, m, 0, 2 * bits, st);
      if (e == cudaSuccess)
        e = cub::DeviceRadixSort::SortPairs(nullptr, tb_pairs, pk, pv, m, 0, row_bits, st);
      if (e == cudaSuccess)
        e = cub::DeviceSelect::Unique(nullptr, tb_uniq, (uint64_t *)nullptr, (uint64_t *)nullptr,
                                      (int64_t *)nullptr, m, st);
      if (e != cudaSuccess) { fail(e, "sort sizes"); break; }
    }
    size_t tb = tb_keys > tb_pairs ? tb_keys : tb_pairs;
    tb = tb > tb_uniq ? tb : tb_uniq;
    Scratch size;
    BuildSpace(size, n, m, sym, tb);
    if (!alloc(&mem.base, (int64_t)size.used)) break;
    BuildSpace b(mem, n, m, sym, tb);
    cudaError_t e = cudaMemsetAsync(b.zeros, 0, 3 * sizeof(unsigned), st);
    if (e != cudaSuccess) { fail(e, "build counters"); break; }
    edge_keys_kernel<<<grid_for(m, sms), 256, 0, st>>>(m, d_src, d_dst, sym ? 1 : 0, drop ? 1 : 0,
                                                       bits, b.keys);
    e = cudaGetLastError();
    if (e != cudaSuccess) { fail(e, "edge_keys"); break; }
    cub::DoubleBuffer<uint64_t> kb(b.keys, b.tmp);
    e = cub::DeviceRadixSort::SortKeys(b.temp, tb_keys, kb, m, 0, 2 * bits, st);
    if (e != cudaSuccess) { fail(e, "SortKeys"); break; }
    uint64_t *const uniq = kb.Alternate();
    e = cub::DeviceSelect::Unique(b.temp, tb_uniq, kb.Current(), uniq, b.count, m, st);
    if (e != cudaSuccess) { fail(e, "Unique"); break; }
    int64_t nu = 0;
    uint64_t lowest = 1;
    e = cudaMemcpyAsync(&nu, b.count, sizeof(nu), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(&lowest, uniq, sizeof(lowest), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { fail(e, "Unique count"); break; }
    const uint64_t *res = uniq;
    if (drop && lowest == 0) {  // the dropped loops
      ++res;
      --nu;
    }
    if (nu >= (1ll << 32) - (1ll << 16)) { rc = CG_ERR_NOT_SUPPORTED; break; }
    if (sym || nu > 0) {
      uint32_t *pair[2][2];  // [set][key, value]
      pair[0][0] = reinterpret_cast<uint32_t *>(kb.Current());
      pair[1][0] = sym ? b.pairs : reinterpret_cast<uint32_t *>(uniq);
      for (int i = 0; i < 2; ++i) pair[i][1] = pair[i][0] + m;
      split_keys_kernel<<<grid_for(nu + 1, sms), 256, 0, st>>>(
          n, nu, res, bits, loops ? n : -1, b.first[0], pair[0][0], pair[0][1], b.gaps, b.zeros);
      fill_gaps_kernel<<<sms, 256, 0, st>>>(b.gaps, b.zeros, b.first[0]);
      e = cudaGetLastError();
      if (e != cudaSuccess) { fail(e, "split_keys"); break; }
      const int grid = grid_for(nu > n ? nu : n + 1, sms);
      if (!sym) {
        // the CSR before the second sort, which takes the keys' space
        nnz = nu;
        if (!alloc(&off[0], n + 1) || !alloc(&idx[0], nnz) || !alloc(&off[1], n + 1) ||
            !alloc(&idx[1], nnz))
          break;
        csr_kernel<<<grid, 256, 0, st>>>(n, nnz, res, bits, b.first[0], off[0], idx[0]);
      }
      cub::DoubleBuffer<uint32_t> pk(pair[0][0], pair[1][0]), pv(pair[0][1], pair[1][1]);
      if (nu > 0) e = cub::DeviceRadixSort::SortPairs(b.temp, tb_pairs, pk, pv, nu, 0, row_bits, st);
      if (e != cudaSuccess) { fail(e, "SortPairs"); break; }
      row_starts_kernel<<<grid_for(nu + 1, sms), 256, 0, st>>>(n, nu, pk.Current(), b.first[1],
                                                               b.gaps, b.zeros + 1);
      fill_gaps_kernel<<<sms, 256, 0, st>>>(b.gaps, b.zeros + 1, b.first[1]);
      e = cudaGetLastError();
      if (e != cudaSuccess) { fail(e, "row_starts"); break; }
      if (sym) {
        uint32_t nl = (uint32_t)nu;  // lower triangle: all but the loops
        if (loops) {
          e = cudaMemcpyAsync(&nl, b.first[1] + n, sizeof(nl), cudaMemcpyDeviceToHost, st);
          if (e == cudaSuccess) e = cudaStreamSynchronize(st);
          if (e != cudaSuccess) { fail(e, "loop count"); break; }
        }
        nnz = nu + (int64_t)nl;
        if (nnz >= (1ll << 32) - (1ll << 16)) { rc = CG_ERR_NOT_SUPPORTED; break; }
        if (!alloc(&off[0], n + 1) || !alloc(&idx[0], nnz)) break;
        csr_symmetric_kernel<<<grid, 256, 0, st>>>(n, nu, nl, res, bits, b.first[0], pk.Current(),
                                                   pv.Current(), b.first[1], off[0], idx[0]);
      } else {
        csr_pairs_kernel<<<grid, 256, 0, st>>>(n, nnz, pv.Current(), b.first[1], off[1], idx[1]);
      }
      e = cudaGetLastError();
      if (e != cudaSuccess) { fail(e, "csr"); break; }
      if (!sym && detect) {
        same_arrays_kernel<<<grid, 256, 0, st>>>(n, nnz, off[0], idx[0], off[1], idx[1],
                                                 b.zeros + 2);
        e = cudaGetLastError();
        unsigned differ = 1u;
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(&differ, b.zeros + 2, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) { fail(e, "symmetry check"); break; }
        found_sym = differ == 0u;
      }
    } else {
      if (!alloc(&off[0], n + 1) || !alloc(&idx[0], 1)) break;
      e = cudaMemsetAsync(off[0], 0, sizeof(int64_t) * (size_t)(n + 1), st);
      if (e != cudaSuccess) { fail(e, "empty offsets"); break; }
    }
  } while (0);
  if (rc == CG_OK) {
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) fail(e, "cg_graph_from_edges");
  } else {
    cudaStreamSynchronize(st);
  }
  cudaFree(mem.base);
  cudaStreamDestroy(st);
  const bool out_sym = sym || nnz == 0 || found_sym;
  if (rc == CG_OK && out_sym) {
    cudaFree(off[1]);
    cudaFree(idx[1]);
    off[1] = nullptr;
    idx[1] = nullptr;
  }
  if (rc == CG_OK) return graph_adopt(n, nnz, off[0], idx[0], off[1], idx[1], out_sym, out);
  for (int i = 0; i < 2; ++i) {
    cudaFree(off[i]);
    cudaFree(idx[i]);
  }
  return rc;
}

int cg_graph_export(const cg_graph *g, int64_t *in_off, int32_t *in_idx, int64_t *out_off,
                    int32_t *out_idx) {
  if (g) {
    if (int r = refuse_reordered(g, "cg_graph_export")) return r;
  }
  if (!g) return CG_ERR_INVALID_ARG;
  const size_t ob = sizeof(int64_t) * (size_t)(g->n + 1), ib = sizeof(int32_t) * (size_t)g->nnz;
  if (in_off) CG_CUDA(cudaMemcpyAsync(in_off, g->in_off, ob, cudaMemcpyDeviceToHost, g->stream));
  if (in_idx && ib)
    CG_CUDA(cudaMemcpyAsync(in_idx, g->in_idx, ib, cudaMemcpyDeviceToHost, g->stream));
  if (out_off)
    CG_CUDA(cudaMemcpyAsync(out_off, g->out_off, ob, cudaMemcpyDeviceToHost, g->stream));
  if (out_idx && ib)
    CG_CUDA(cudaMemcpyAsync(out_idx, g->out_idx, ib, cudaMemcpyDeviceToHost, g->stream));
  CG_CUDA(cudaStreamSynchronize(g->stream));
  return CG_OK;
}

}  // extern "C"
