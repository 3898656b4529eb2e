// kernels_read.cu -- read-out kernels: probabilities, marginals, sampling,
// amplitude gather, Pauli expectations.  Every reduction is deterministic:
// per-block partial sums in a fixed tree order, then a fixed-order combine,
// all in FP64 whatever the state precision.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "pauli_terms.cuh"
#include "read.h"

namespace ket {

namespace {

template <typename R>
__device__ __forceinline__ double pref(const typename Vec2<R>::T* a, uint64_t i) {
  typename Vec2<R>::T v = a[i];
  return norm2_ref(v.x, v.y);
}

// ------------------------------------------------------------------ sums
template <typename R, int NT>
__global__ void __launch_bounds__(NT) k_norm_partial(const typename Vec2<R>::T* a, uint64_t N, uint64_t chunk,
                                                     double* partial) {
  __shared__ double red[32];
  uint64_t lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  double acc = 0.0;
  for (uint64_t i = lo + threadIdx.x; i < hi; i += NT) acc += pref<R>(a, i);
  double t = block_sum<NT>(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// Fixed-order sum of n partials (one block): thread t sums a strided subset
// sequentially, then a block tree.
template <int NT>
__global__ void __launch_bounds__(NT) k_sum(const double* partial, uint64_t n, double* out) {
  __shared__ double red[32];
  double acc = 0.0;
  for (uint64_t i = threadIdx.x; i < n; i += NT) acc += partial[i];
  double t = block_sum<NT>(acc, red);
  if (threadIdx.x == 0) *out = t;
}

// out[j] = sum over rows b of partial[b*width + j], in a fixed order: 32 threads
// a column, each a strided run of rows (64 of the 2048 partials marginals makes,
// several loads in flight), then their sums in order.  One thread a column took
// 179 us for those 2048 rows, this takes 12.
constexpr int kColRows = 32;
__device__ __forceinline__ void column_combine(double acc, int j, int width, double* out) {
  __shared__ double red[kColRows][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  red[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && j < width) {
    double t = red[0][tx];
    for (int r = 1; r < kColRows; r++) t += red[r][tx];
    out[j] = t;
  }
}
__global__ void __launch_bounds__(32 * kColRows) k_sum_columns(const double* partial, uint64_t rows, int width,
                                                               double* out) {
  const int j = blockIdx.x * 32 + (threadIdx.x & 31);
  double acc = 0.0;
  if (j < width) {
#pragma unroll 8
    for (uint64_t b = threadIdx.x >> 5; b < rows; b += kColRows) acc += partial[b * width + j];
  }
  column_combine(acc, j, width, out);
}

// ------------------------------------------------------------------ state comparison
// Per block: sum of conj(a_i) b_i (re, im) and max |a_i - b_i|, all in FP64.
template <typename RA, typename RB, int NT>
__global__ void __launch_bounds__(NT) k_compare(const typename Vec2<RA>::T* a, const typename Vec2<RB>::T* b,
                                                uint64_t N, uint64_t chunk, double* partial) {
  __shared__ double red[32];
  uint64_t lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  double sr = 0.0, si = 0.0, mx = 0.0;
  for (uint64_t i = lo + threadIdx.x; i < hi; i += NT) {
    const typename Vec2<RA>::T u = a[i];
    const typename Vec2<RB>::T v = b[i];
    const double ur = u.x, ui = u.y, vr = v.x, vi = v.y;
    sr += ur * vr + ui * vi;
    si += ur * vi - ui * vr;
    const double dr = ur - vr, di = ui - vi;
    mx = fmax(mx, sqrt(dr * dr + di * di));
  }
  const double tr = block_sum<NT>(sr, red);
  const double ti = block_sum<NT>(si, red);
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int w = 0; w < NT / 32; w++) m = fmax(m, red[w]);
    partial[3 * blockIdx.x] = tr;
    partial[3 * blockIdx.x + 1] = ti;
    partial[3 * blockIdx.x + 2] = m;
  }
}

// Fixed-order combine of the block partials (one thread).
__global__ void k_compare_combine(const double* partial, uint64_t nb, double* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double r = 0.0, i = 0.0, m = 0.0;
  for (uint64_t b = 0; b < nb; b++) {
    r += partial[3 * b];
    i += partial[3 * b + 1];
    m = fmax(m, partial[3 * b + 2]);
  }
  out[0] = r;
  out[1] = i;
  out[2] = m;
}

// ------------------------------------------------------------------ probabilities
template <typename R>
__global__ void k_probs_dense(const typename Vec2<R>::T* a, uint64_t off, uint64_t cnt, double thr, double* out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt; i += (uint64_t)gridDim.x * blockDim.x) {
    double p = pref<R>(a, off + i);
    out[i] = p > thr ? p : 0.0;
  }
}

template <typename R, int NT>
__global__ void __launch_bounds__(NT) k_count_kept(const typename Vec2<R>::T* a, uint64_t N, uint64_t chunk, double thr,
                                                   uint64_t* counts) {
  __shared__ unsigned long long red;
  if (threadIdx.x == 0) red = 0;
  __syncthreads();
  uint64_t lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  unsigned long long c = 0;
  for (uint64_t i = lo + threadIdx.x; i < hi; i += NT) c += pref<R>(a, i) > thr ? 1 : 0;
  atomicAdd(&red, c);  // integer: order does not matter
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = red;
}

// Compaction preserving ascending index order within each chunk.
template <typename R, int NT>
__global__ void __launch_bounds__(NT) k_compact_kept(const typename Vec2<R>::T* a, uint64_t N, uint64_t chunk, double thr,
                                                     const uint64_t* offsets, uint64_t cap, uint64_t* oidx, double* op) {
  __shared__ uint32_t wsum[NT / 32];
  __shared__ uint64_t running;
  if (threadIdx.x == 0) running = offsets[blockIdx.x];
  __syncthreads();
  uint64_t lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (uint64_t s = lo; s < hi; s += NT) {
    uint64_t i = s + threadIdx.x;
    double p = 0.0;
    bool keep = false;
    if (i < hi) { p = pref<R>(a, i); keep = p > thr; }
    uint32_t bal = __ballot_sync(0xffffffffu, keep);
    uint32_t before = __popc(bal & ((1u << lane) - 1));
    if (lane == 0) wsum[w] = __popc(bal);
    __syncthreads();
    uint64_t wbase = running;
    for (int j = 0; j < w; j++) wbase += wsum[j];
    if (keep) {
      uint64_t pos = wbase + before;
      if (pos < cap) { oidx[pos] = i; op[pos] = p; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t t = 0;
      for (int j = 0; j < NT / 32; j++) t += wsum[j];
      running += t;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ marginals
// P(q = 1) for every qubit: per-block partials [block][n].  A block covers 2^c
// indices; index bits 0-7 are thread bits, 8-11 register bits (16 amplitudes in
// flight a thread), 12..c-1 loop bits, the rest the block's.  The 16
// probabilities are added pairwise, level by level, and each level's odd halves are
// its bit's marginal: about 3 additions an amplitude in place of one for every
// qubit, which made the pass FP64-bound (27 qubits: 2.03 -> 0.36 ms; one read of
// the state is 0.33).
constexpr int kMargLoopBits = KET_MAX_QUBITS - 11 - 12;  // marg_chunk() leaves at most 2^11 blocks

template <typename R>
__global__ void __launch_bounds__(256) k_marginals(const typename Vec2<R>::T* a, int n, int c, double* partial) {
  constexpr int NV = 1 + 4 + 5 + kMargLoopBits;  // total, register bits, lane bits, loop bits
  __shared__ double ws[8][NV];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint64_t N = uint64_t(1) << n, base = (uint64_t)blockIdx.x << c;
  double tot = 0.0, mj[4] = {0.0, 0.0, 0.0, 0.0}, mo[kMargLoopBits];
#pragma unroll
  for (int b = 0; b < kMargLoopBits; b++) mo[b] = 0.0;
  for (uint64_t o = 0; o < uint64_t(1) << (c - 12); o++) {
    double p[16];
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const uint64_t i = base | (o << 12) | (uint64_t)(j << 8) | t;
      p[j] = i < N ? pref<R>(a, i) : 0.0;
    }
#pragma unroll
    for (int b = 0; b < 4; b++) {
      double odd = 0.0;
#pragma unroll
      for (int j = 0; j < (8 >> b); j++) {
        odd += p[2 * j + 1];
        p[j] = p[2 * j] + p[2 * j + 1];
      }
      mj[b] += odd;
    }
    tot += p[0];
#pragma unroll
    for (int b = 0; b < kMargLoopBits; b++)
      if ((o >> b) & 1) mo[b] += p[0];
  }
  auto put = [&](int k, double v) {
    v = warp_sum(v);
    if (lane == 0) ws[w][k] = v;
  };
  put(0, tot);
#pragma unroll
  for (int b = 0; b < 4; b++) put(1 + b, mj[b]);
#pragma unroll
  for (int b = 0; b < 5; b++) put(5 + b, ((lane >> b) & 1) ? tot : 0.0);
#pragma unroll
  for (int b = 0; b < kMargLoopBits; b++)
    if (b < c - 12) put(10 + b, mo[b]);
  __syncthreads();
  if (t < n) {
    const int q = t;
    const int k = q < 5 ? 5 + q : q < 8 ? 0 : q < 12 ? 1 + (q - 8) : q < c ? 10 + (q - 12) : 0;
    double sum = 0.0;
    for (int x = 0; x < 8; x++)
      if (q < 5 || q >= 8 || ((x >> (q - 5)) & 1)) sum += ws[x][k];
    if (q >= c && !((base >> q) & 1)) sum = 0.0;
    partial[blockIdx.x * (uint64_t)n + q] = sum;
  }
}

// Joint distribution of the qubits in `mask`: per-block sums over the in-block
// bins (bin bits in ascending qubit order).  A block covers 2^c indices, split as
// in k_marginals.  Register sums v[j] run over the loop bits outside the mask;
// for each setting of the masked loop bits the register bits, then the lane bits
// outside the mask are folded, and the warps' sums added in shared memory.  Every
// load is of consecutive amplitudes and every block runs 16 of them a thread, where
// a thread a bin over 2^20 indices left most of the chip idle (20 qubits, 10 low
// qubits: one block, 489 -> 16 us, half of them k_marginal_dist_combine's; 27 qubits: 2.86 ->
// 0.31 ms).
template <typename R>
__global__ void __launch_bounds__(256) k_marginal_dist(const typename Vec2<R>::T* a, int n, int c, uint64_t mask,
                                                       double* partial) {
  __shared__ double red[8][16][32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint64_t N = uint64_t(1) << n, base = (uint64_t)blockIdx.x << c, inmask = mask & ((uint64_t(1) << c) - 1);
  const uint32_t tmask = (uint32_t)inmask & 0xffu, jmask = (uint32_t)(inmask >> 8) & 15u;
  const uint64_t omask = inmask >> 12, oother = ((uint64_t(1) << (c - 12)) - 1) & ~omask;
  const uint32_t tj = tmask | jmask << 8, wother = 7u & ~(tmask >> 5);
  const uint32_t nout = 1u << __popc(tj);
  double* dst = partial + ((uint64_t)blockIdx.x << __popcll(inmask));
  uint64_t uo = 0;
  do {
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = 0.0;
    uint64_t x = 0;
    do {
      const uint64_t i0 = base | ((uo | x) << 12) | t;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const uint64_t i = i0 | (uint64_t)(j << 8);
        if (i < N) v[j] += pref<R>(a, i);
      }
      x = (x - oother) & oother;
    } while (x != 0);
#pragma unroll
    for (int b = 0; b < 4; b++)
      if (!((jmask >> b) & 1)) {
#pragma unroll
        for (int j = 0; j < 16; j++)
          if (!((j >> b) & 1)) v[j] += v[j | 1 << b];
      }
#pragma unroll
    for (int j = 0; j < 16; j++) {
      if (j & ~jmask) continue;
#pragma unroll
      for (int b = 0; b < 5; b++)
        if (!((tmask >> b) & 1)) v[j] += __shfl_xor_sync(0xffffffffu, v[j], 1 << b);
    }
    __syncthreads();  // the last round's sums are read
    if (!(lane & ~tmask)) {
#pragma unroll
      for (int j = 0; j < 16; j++)
        if (!(j & ~jmask)) red[w][j][lane] = v[j];
    }
    __syncthreads();
    for (uint32_t e = t; e < nout; e += 256) {
      uint32_t at = 0, m = tj;  // e scattered over the masked thread and register bits
      for (uint32_t y = e; y; y >>= 1, m &= m - 1)
        if (y & 1) at |= m & (0u - m);
      double sum = 0.0;
      uint32_t z = 0;
      do {
        sum += red[((at >> 5) & 7u) | z][at >> 8][at & 31];
        z = (z - wother) & wother;
      } while (z != 0);
      dst[e] = sum;
    }
    dst += nout;
    uo = (uo - omask) & omask;
  } while (uo != 0);
}

// out[bin] = sum of the blocks' sums whose out-of-block bits match the bin, in
// ascending block order within each of 32 strided runs, the runs in order.
__global__ void __launch_bounds__(32 * kColRows) k_marginal_dist_combine(const double* partial, int n, int c,
                                                                         MarginalSpec spec, double* out) {
  const uint32_t bin = blockIdx.x * 32 + (threadIdx.x & 31), width = 1u << spec.m;
  const uint64_t inmask = spec.mask & ((uint64_t(1) << c) - 1);
  const int nin = __popcll(inmask);
  double acc = 0.0;
  if (bin < width) {
    uint64_t at = 0, ob = 0;  // the bin's place in a block, and its block bits
    for (int k = 0; k < spec.m; k++) {
      if (!((bin >> k) & 1)) continue;
      if (spec.q[k] < c) at |= uint64_t(1) << __popcll(inmask & ((uint64_t(1) << spec.q[k]) - 1));
      else ob |= uint64_t(1) << (spec.q[k] - c);
    }
    const uint64_t other = n > c ? ((uint64_t(1) << (n - c)) - 1) & ~(spec.mask >> c) : 0;
    const uint64_t rows = uint64_t(1) << __popcll(other);
    auto scatter = [&](uint64_t r) {
      uint64_t o = 0, m = other;
      for (; r; r >>= 1, m &= m - 1)
        if (r & 1) o |= m & (0ull - m);
      return o;
    };
    const uint64_t r0 = threadIdx.x >> 5;
    if (r0 < rows) {
      uint64_t b = scatter(r0);
      const uint64_t step = rows > kColRows ? scatter(kColRows) : 0;
      for (uint64_t r = r0; r < rows; r += kColRows) {
        acc += partial[((ob | b) << nin) + at];
        b = (b + ~other + step) & other;  // + step, carrying over the bits not in `other`
      }
    }
  }
  column_combine(acc, (int)bin, (int)width, out);
}

// ------------------------------------------------------------------ sampling
// The sampling CDF is the reference's running FP64 sum over kept entries in
// ascending index order, rounded after every addition (circuit.ts:3429-3436),
// reproduced bit for bit at every state size.  It is kept as checkpoints:
// ck[k] = the running sum before entry 32k, ck[nk] = the total.  A draw finds
// its 32-entry sub-chunk by binary search over ck and finishes with the
// reference's own FP64 additions from ck[k].
//
// While the running sum s stays in one binade [2^(e-1), 2^e), every value it
// takes is a multiple of u = 2^(e-53): s = S u with S an integer in
// [2^52, 2^53).  Adding p rounds to the nearest multiple of u, so
// s + p = (S + d) u with d = round(p / u) -- an increment that does not
// depend on s, except when p / u lies exactly halfway (the tie goes to the
// even S + d) or when S + d reaches 2^53 (the sum leaves the binade and rounds
// on the next grid).  A run of entries inside one binade is therefore an
// integer prefix sum of the d's.  Five kernels build the checkpoints:
//   k_cdf_block_sums    per block of 4096 entries, the plain sum of the kept
//                       p's and the first and last kept index;
//   k_cdf_block_prefix  an approximate exclusive prefix of those sums -- it
//                       only guesses the binade each block starts in -- and
//                       the first and last kept index of the state;
//   k_cdf_block_d       per block, in the guessed binade, the d's, their sum D
//                       and their exclusive prefix at every 32-entry
//                       sub-chunk; a block holding a tie or an oversized d, or
//                       with nothing kept before it, is marked unclean;
//   k_cdf_walk          one CTA carries the exact running sum across windows
//                       of blocks.  A block is taken whole when nothing in it
//                       is kept, or when it is clean in the binade the exact
//                       sum is in and S + D stays below 2^53 -- its integer
//                       prefix is then exact.  Any other block runs entry by
//                       entry (cdf_exact_range): integer prefix sums up to the
//                       next tie or crossing, which takes the FP64 addition
//                       itself;
//   k_cdf_fill          the checkpoints of the blocks taken whole, from their
//                       exact start and the sub-chunk prefixes.
// Only blocks holding a binade crossing, a tie or the first kept entry run
// entry by entry: a crossing happens about once per doubling of s.
constexpr int kCdfThreads = 1024;
constexpr int kWalkThreads = 1024;                  // the walker's
constexpr int kCdfPer = 4;                          // entries of a block per walker thread
constexpr int kCdfHead = 128;                       // entries after the first kept one, added one by one
constexpr int kCdfBlock = 4096;                     // entries per block
constexpr int kCdfSub = 32;                         // entries per checkpoint
constexpr int kCdfSubPerBlock = kCdfBlock / kCdfSub;
constexpr int kCdfWalkPer = 4;                      // blocks per walker thread per window
constexpr long long kTwo52 = 4503599627370496ll;
constexpr long long kTwo53 = 9007199254740992ll;
static_assert(kWalkThreads * kCdfPer == kCdfBlock, "a thread's share of a block");

enum : int { kBlkUnclean = 0, kBlkClean = 1, kBlkEmpty = 2, kBlkExact = 3 };

// Inclusive block scan of v over NT threads; `wsum` holds 32 partials.
template <int NT, typename T>
__device__ __forceinline__ T block_scan_incl(T v, T* wsum) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) wsum[w] = v;
  __syncthreads();
  if (w == 0) {
    T x = lane < NT / 32 ? wsum[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T t = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += t;
    }
    wsum[lane] = x;
  }
  __syncthreads();
  const T r = v + (w > 0 ? wsum[w - 1] : T(0));
  __syncthreads();  // wsum is reused by the next scan
  return r;
}

// Block minimum of v over NT threads; every thread gets it.
template <int NT>
__device__ __forceinline__ unsigned long long block_min_u64(unsigned long long v, unsigned long long* wred) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) wred[w] = v;
  __syncthreads();
  if (w == 0) {
    unsigned long long x = lane < NT / 32 ? wred[lane] : ~0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = min(x, __shfl_xor_sync(0xffffffffu, x, o));
    if (lane == 0) wred[32] = x;
  }
  __syncthreads();
  const unsigned long long r = wred[32];
  __syncthreads();
  return r;
}

// The kept probability of entry i: p when p > thr, else +0.0 (adds nothing).
template <typename R>
__device__ __forceinline__ double kept_p(const typename Vec2<R>::T* a, uint64_t i, double thr) {
  const double p = pref<R>(a, i);
  return p > thr ? p : 0.0;
}

template <typename R>
__global__ void __launch_bounds__(256) k_cdf_block_sums(const typename Vec2<R>::T* a, uint64_t N, double thr,
                                                        double* bsum, unsigned long long* bfirst,
                                                        unsigned long long* blast) {
  __shared__ double red[32];
  __shared__ unsigned long long wred[33];
  const uint64_t lo = (uint64_t)blockIdx.x * kCdfBlock;
  double acc = 0.0;
  unsigned long long f = ~0ull, l = ~0ull;  // l holds ~index, so the minimum is the largest index
#pragma unroll 4
  for (int k = 0; k < kCdfBlock / 256; k++) {
    const uint64_t i = lo + (uint64_t)k * 256 + threadIdx.x;
    if (i < N) {
      const double p = pref<R>(a, i);
      if (p > thr) {
        acc += p;
        if (f == ~0ull) f = i;
        l = ~(unsigned long long)i;
      }
    }
  }
  const double t = block_sum<256>(acc, red);
  f = block_min_u64<256>(f, wred);
  l = block_min_u64<256>(l, wred);
  if (threadIdx.x == 0) {
    bsum[blockIdx.x] = t;
    bfirst[blockIdx.x] = f;
    blast[blockIdx.x] = l;
  }
}

// bsum[0..nb) -> its exclusive prefix, bsum[nb] = the total; fl[0] = the
// first kept index, fl[1] = the last (~0: nothing kept).
__global__ void __launch_bounds__(kCdfThreads) k_cdf_block_prefix(double* bsum, const unsigned long long* bfirst,
                                                                  const unsigned long long* blast, uint64_t nb,
                                                                  unsigned long long* fl) {
  __shared__ double wsd[32];
  __shared__ unsigned long long wred[33];
  const uint64_t per = (nb + kCdfThreads - 1) / kCdfThreads;
  const uint64_t lo = min(nb, (uint64_t)threadIdx.x * per), hi = min(nb, lo + per);
  double t = 0.0;
  unsigned long long f = ~0ull, l = ~0ull;
  for (uint64_t b = lo; b < hi; b++) {
    t += bsum[b];
    f = min(f, bfirst[b]);
    l = min(l, blast[b]);
  }
  const double incl = block_scan_incl<kCdfThreads>(t, wsd);
  double x = incl - t;
  for (uint64_t b = lo; b < hi; b++) {
    const double v = bsum[b];
    bsum[b] = x;
    x += v;
  }
  f = block_min_u64<kCdfThreads>(f, wred);
  l = block_min_u64<kCdfThreads>(l, wred);
  if (threadIdx.x == kCdfThreads - 1) bsum[nb] = incl;
  if (threadIdx.x == 0) {
    fl[0] = f;
    fl[1] = l == ~0ull ? ~0ull : ~l;
  }
}

// Warp w handles sub-chunks 16w .. 16w + 15; lane l reads entry 32j + l of
// sub-chunk j, so every load is 32 consecutive amplitudes.
template <typename R>
__global__ void __launch_bounds__(256) k_cdf_block_d(const typename Vec2<R>::T* a, uint64_t N, double thr,
                                                     const double* bstart_approx, long long* ckd, long long* bd,
                                                     int* bst, int* be) {
  static_assert(kCdfSubPerBlock == 8 * 16, "8 warps of 16 sub-chunks");
  __shared__ long long wsum[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t b = blockIdx.x, lo = b * kCdfBlock;
  const double A = bstart_approx[b];
  int e = 0;
  if (A > 0.0) frexp(A, &e);
  const bool guess = A > 0.0;
  const bool tiny = e < -900;  // (1 / u leaves the normal numbers)
  const double inv_u = __longlong_as_double((long long)(1023 + 53 - (tiny ? 0 : e)) << 52);
  bool pos = false, bad = false;
  long long mine = 0;  // lane k < 16: the d-sum of sub-chunk 16w + k
#pragma unroll 4
  for (int k = 0; k < 16; k++) {
    const uint64_t i = lo + (uint64_t)(16 * w + k) * kCdfSub + lane;
    const double p = i < N ? kept_p<R>(a, i, thr) : 0.0;
    pos |= p > 0.0;
    long long d = 0;
    if (guess) {
      const double q = tiny ? ldexp(p, 53 - e) : p * inv_u;  // p / u, exact
      // rounded to an integer (ties to even) by the 2^52 that it is added to
      const double y = q + 4503599627370496.0, r = y - 4503599627370496.0;
      if (q >= 4503599627370496.0) bad = true;   // 2^52: S + d would leave the binade
      else if (fabs(q - r) == 0.5) bad = true;    // a tie: the rounding depends on S
      else d = __double_as_longlong(y) - 0x4330000000000000ll;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (lane == k) mine = d;
  }
  const bool any_pos = __syncthreads_or(pos);
  const bool any_bad = __syncthreads_or(bad);
  // a sub-chunk sum is below 2^57; clamped at 2^53 the block total stays exact
  // below 2^53 and cannot overflow
  const long long v = lane < 16 ? (mine < kTwo53 ? mine : kTwo53) : 0;
  const long long incl = block_scan_incl<256>(v, wsum);
  __shared__ long long total;
  if (threadIdx.x == 255) total = incl;
  __syncthreads();
  const uint64_t j = 16 * w + lane;
  if (lane < 16 && lo + j * kCdfSub < N) ckd[b * kCdfSubPerBlock + j] = incl - v;
  if (threadIdx.x == 0) {
    int st;
    if (!any_pos) st = kBlkEmpty;
    else if (!guess || any_bad || total >= kTwo53) st = kBlkUnclean;
    else st = kBlkClean;
    bst[b] = st;
    be[b] = e;
    bd[b] = total;
  }
}

// p 2^k, exact where the result is a normal number (k as frexp of a sum gives it).
__device__ __forceinline__ double scaled(double p, int k) {
  return k >= -1000 && k <= 1000 ? p * __longlong_as_double((long long)(1023 + k) << 52) : ldexp(p, k);
}

// Exclusive prefix of v and block minimum over the walker's threads, each with one
// barrier: every warp reduces the 32 warps' values for itself.  `buf` holds values
// that no thread reads any more (callers alternate between two).
__device__ __forceinline__ long long walk_scan(long long v, long long* buf) {
  static_assert(kWalkThreads == 1024, "one value a lane");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) buf[w] = x;
  __syncthreads();
  long long z = buf[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, z, o);
    if (lane >= o) z += y;
  }
  const long long before = __shfl_sync(0xffffffffu, z, w > 0 ? w - 1 : 0);
  return (w > 0 ? before : 0) + x - v;
}
__device__ __forceinline__ uint32_t walk_min(uint32_t v, uint32_t* buf) {
  v = __reduce_min_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = v;
  __syncthreads();
  return __reduce_min_sync(0xffffffffu, buf[threadIdx.x & 31]);
}

// What the walker's threads share.  s: the exact running sum before position c.
struct WalkShared {
  long long scan[2][32];
  uint32_t red[2][32];
  double head[kCdfHead];
  double s;
  uint32_t c;
};

// The running sum over a block's entries [lo, hi) in the reference's rounding,
// from the exact sum sh.s before lo.  Writes the checkpoints ck[(i + 1) / 32]
// for entries i with (i + 1) % 32 == 0 and i + 1 < hi, and leaves the sum after
// entry hi - 1 in sh.s.  Called by the whole CTA of kWalkThreads threads.
//
// A thread's entries lo + kCdfPer t + k stay in its registers; a step runs from
// position c to the next tie or crossing, with three barriers (reloading the
// entries of each step and twelve barriers took 5 us a step, a dozen steps a
// block).
template <typename R>
__device__ void cdf_exact_range(const typename Vec2<R>::T* a, uint64_t lo, uint64_t hi, double thr, double* ck,
                                WalkShared& sh, int& turn) {
  const uint32_t tid = threadIdx.x, len = (uint32_t)(hi - lo), NONE = ~0u, i0 = kCdfPer * tid;
  double pv[kCdfPer];
#pragma unroll
  for (int k = 0; k < kCdfPer; k++) pv[k] = i0 + k < len ? kept_p<R>(a, lo + i0 + k, thr) : 0.0;
  auto checkpoint = [&](uint32_t i, double v) {  // the sum after entry i
    if (((lo + i + 1) & (kCdfSub - 1)) == 0 && i + 1 < len) ck[(lo + i + 1) / kCdfSub] = v;
  };
  if (tid == 0) sh.c = 0;
  __syncthreads();
  for (;;) {
    const uint32_t c = sh.c;
    const double s = sh.s;
    if (c >= len) break;
    turn ^= 1;
    if (s == 0.0) {
      // before the first positive kept entry the sum is +0.0; that entry sets
      // it exactly
      uint32_t f = NONE;
#pragma unroll
      for (int k = kCdfPer - 1; k >= 0; k--)
        if (i0 + k >= c && pv[k] > 0.0) f = i0 + k;
      const uint32_t z = min(walk_min(f, sh.red[turn]), len);
#pragma unroll
      for (int k = 0; k < kCdfPer; k++) {
        const uint32_t i = i0 + k;
        if (i >= c && i < z) checkpoint(i, 0.0);
        if (i >= z && i < len && i - z < (uint32_t)kCdfHead) sh.head[i - z] = pv[k];
      }
      __syncthreads();
      // from there the sum doubles every few entries, and a step ends at each
      // doubling: one thread adds the first entries as the reference does
      if (tid == 0) {
        const uint32_t cnt = min(len - z, (uint32_t)kCdfHead);
        double t = 0.0;
        for (uint32_t i = 0; i < cnt; i++) {
          t += sh.head[i];
          checkpoint(z + i, t);
        }
        sh.s = t;
        sh.c = z + cnt;
      }
      __syncthreads();
      continue;
    }
    // s in [2^(e-1), 2^e): u = 2^(e-53), S = s / u
    int e;
    frexp(s, &e);
    const long long S0 = (long long)scaled(s, 53 - e);
    uint32_t stop = NONE;  // this thread's first entry that is a tie or crosses
    long long d[kCdfPer];
    long long tsum = 0;
#pragma unroll
    for (int k = 0; k < kCdfPer; k++) {
      const uint32_t i = i0 + k;
      d[k] = 0;
      if (i < c || i >= len || stop != NONE) continue;
      const double q = scaled(pv[k], 53 - e);  // p / u, exact
      // 2^53: the sum leaves the binade; half: a tie, the rounding depends on S
      if (q >= 9007199254740992.0 || q - floor(q) == 0.5) {
        stop = i;
        continue;
      }
      d[k] = (long long)rint(q);
      tsum += d[k];
    }
    // (past the first such entry of the block the prefix is of no use, but then
    // neither is a crossing found there: the earliest position counts)
    const long long S1 = S0 + walk_scan(tsum, sh.scan[turn]);
    long long Sr = S1;  // S before this thread's first entry
#pragma unroll
    for (int k = 0; k < kCdfPer; k++) {
      const uint32_t i = i0 + k;
      if (i < c || i >= len || i >= stop) continue;
      if (Sr + d[k] >= kTwo53) { stop = i; continue; }
      Sr += d[k];
    }
    stop = min(walk_min(stop, sh.red[turn]), len);
    // the exact sums of the entries before `stop`
    Sr = S1;
#pragma unroll
    for (int k = 0; k < kCdfPer; k++) {
      const uint32_t i = i0 + k;
      if (i < c || i > stop || i >= len) continue;
      if (i == stop) {
        // the special entry, by the reference's own FP64 addition
        const double sp = scaled((double)Sr, e - 53) + pv[k];
        checkpoint(i, sp);
        sh.s = sp;
        continue;
      }
      Sr += d[k];
      const double v = scaled((double)Sr, e - 53);
      checkpoint(i, v);
      if (i + 1 == len) sh.s = v;  // (stop == len)
    }
    if (tid == 0) sh.c = stop < len ? stop + 1 : len;
    __syncthreads();
  }
}

// Windows of kCdfWalkPer blocks a thread: their states are read once, and the walk
// steps through them as cdf_exact_range steps through entries.  27 qubits (32768
// blocks, 27 doublings of the sum): 337 -> 222 us; 16 qubits 139 -> 71.
template <typename R>
__global__ void __launch_bounds__(kWalkThreads) k_cdf_walk(const typename Vec2<R>::T* a, uint64_t N, double thr,
                                                          uint64_t nb, uint64_t nk, double* ck, const long long* bd,
                                                          int* bst, const int* be, double* bstart) {
  __shared__ WalkShared sh;
  __shared__ uint32_t at_sh;           // the next block, in the window
  __shared__ double sum_sh;            // the exact running sum before it
  const uint32_t tid = threadIdx.x, NONE = ~0u, j0 = kCdfWalkPer * tid;
  int turn = 0;
  if (tid == 0) sum_sh = 0.0;
  for (uint64_t win = 0; win < nb; win += kCdfWalkPer * kWalkThreads) {
    const uint32_t len = (uint32_t)(nb - win < kCdfWalkPer * kWalkThreads ? nb - win : kCdfWalkPer * kWalkThreads);
    int st[kCdfWalkPer], eb[kCdfWalkPer];
    long long D[kCdfWalkPer];
#pragma unroll
    for (int k = 0; k < kCdfWalkPer; k++) {
      st[k] = kBlkEmpty;
      eb[k] = 0;
      D[k] = 0;
      if (j0 + k < len) {
        st[k] = bst[win + j0 + k];
        eb[k] = be[win + j0 + k];
        D[k] = bd[win + j0 + k];
      }
    }
    if (tid == 0) at_sh = 0;
    __syncthreads();
    for (;;) {
      const uint32_t c = at_sh;
      const double s = sum_sh;
      if (c >= len) break;
      turn ^= 1;
      int e = 0;
      long long S0 = 0;
      if (s > 0.0) {
        frexp(s, &e);
        S0 = (long long)scaled(s, 53 - e);
      }
      uint32_t stop = NONE;  // this thread's first block that is not taken whole
      long long dv[kCdfWalkPer];
      long long tsum = 0;
#pragma unroll
      for (int k = 0; k < kCdfWalkPer; k++) {
        const uint32_t j = j0 + k;
        dv[k] = 0;
        if (j < c || j >= len || stop != NONE || st[k] == kBlkEmpty) continue;
        if (st[k] == kBlkClean && s > 0.0 && eb[k] == e) dv[k] = D[k];
        else stop = j;
        tsum += dv[k];
      }
      const long long S1 = S0 + walk_scan(tsum, sh.scan[turn]);  // (blocks of one binade: no overflow)
      long long Sr = S1;
#pragma unroll
      for (int k = 0; k < kCdfWalkPer; k++) {
        const uint32_t j = j0 + k;
        if (j < c || j >= len || j >= stop) continue;
        if (Sr + dv[k] >= kTwo53) { stop = j; continue; }  // the sum reaches 2^53 u
        Sr += dv[k];
      }
      stop = min(walk_min(stop, sh.red[turn]), len);
      // blocks before `stop` are taken whole
      Sr = S1;
#pragma unroll
      for (int k = 0; k < kCdfWalkPer; k++) {
        const uint32_t j = j0 + k;
        if (j < c || j > stop || j >= len) continue;
        const double before = s > 0.0 ? scaled((double)Sr, e - 53) : 0.0;
        bstart[win + j] = before;
        if (j == stop) {
          bst[win + j] = kBlkExact;
          ck[(win + j) * kCdfSubPerBlock] = before;
          sh.s = before;
          continue;
        }
        Sr += dv[k];
        if (j + 1 == len) sum_sh = s > 0.0 ? scaled((double)Sr, e - 53) : 0.0;  // (stop == len)
      }
      __syncthreads();
      if (stop < len) {
        // block `stop` entry by entry
        const uint64_t lo = (win + stop) * kCdfBlock;
        cdf_exact_range<R>(a, lo, lo + kCdfBlock < N ? lo + kCdfBlock : N, thr, ck, sh, turn);
        if (tid == 0) {
          sum_sh = sh.s;
          at_sh = stop + 1;
        }
      } else if (tid == 0) {
        at_sh = len;
      }
      __syncthreads();
    }
    __syncthreads();  // (at_sh is reset for the next window)
  }
  if (tid == 0) ck[nk] = sum_sh;
}

// Checkpoints of the blocks taken whole: the exact start plus the sub-chunk's
// d prefix, in the block's binade (ck holds the prefixes as integers until now).
__global__ void k_cdf_fill(double* ck, uint64_t nk, const int* bst, const int* be, const double* bstart) {
  long long* ckd = (long long*)ck;
  for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < nk; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = k / kCdfSubPerBlock;
    const int st = bst[b];
    if (st == kBlkEmpty) {
      ck[k] = bstart[b];
    } else if (st == kBlkClean) {
      const int e = be[b];
      const long long S = (long long)ldexp(bstart[b], 53 - e);
      ck[k] = ldexp((double)(S + ckd[k]), e - 53);
    }
  }
}

// One draw per thread: the first kept entry whose running sum is >= r, the
// last kept entry's sum taken as 1.0 (circuit.ts:3438-3451).  The host checks
// 0 <= r <= 1, so the walk ends inside one sub-chunk.
template <typename R>
__global__ void k_sample_ck(const typename Vec2<R>::T* a, uint64_t N, double thr, const double* ck, uint64_t nk,
                            const double* r, uint64_t shots, const unsigned long long* fl, uint64_t* out) {
  const uint64_t first = fl[0], last = fl[1];
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < shots; s += (uint64_t)gridDim.x * blockDim.x) {
    if (last == ~uint64_t(0)) { out[s] = 0; continue; }
    const double rv = r[s];
    if (ck[nk] < rv) { out[s] = last; continue; }
    uint64_t lo = 0, hi = nk;  // the first checkpoint >= r
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (ck[mid] < rv) lo = mid + 1; else hi = mid;
    }
    const uint64_t k = lo > 0 ? lo - 1 : 0;
    double acc = ck[k];
    uint64_t i = k * kCdfSub;
    if (i < first) i = first;
    uint64_t res = last;
    for (; i < last; i++) {
      const double p = pref<R>(a, i);
      if (p > thr) {
        acc = acc + p;
        if (acc >= rv) { res = i; break; }
      }
    }
    out[s] = res;
  }
}

// ------------------------------------------------------------------ gather, Pauli
template <typename R>
__global__ void k_gather(const typename Vec2<R>::T* a, const uint64_t* idx, uint64_t k, double* out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < k; i += (uint64_t)gridDim.x * blockDim.x) {
    typename Vec2<R>::T v = a[idx[i]];
    out[2 * i] = (double)v.x;
    out[2 * i + 1] = (double)v.y;
  }
}

// <psi|P|psi> partials for a group of Pauli terms sharing the flip mask f:
// sum_y Re( psi_y * conj(psi_{y^f}) * i^nY ) * sum_t coeff_t (-1)^popc(y & zm_t).
template <typename R, int NT>
__global__ void __launch_bounds__(NT) k_pauli_group(const typename Vec2<R>::T* a, uint64_t N, uint64_t chunk,
                                                    PauliGroup grp, double* partial) {
  __shared__ double red[32];
  uint64_t lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  double acc = 0.0;
  for (uint64_t y = lo + threadIdx.x; y < hi; y += NT) {
    typename Vec2<R>::T v = a[y], w = a[y ^ grp.flip];
    double vr = v.x, vi = v.y, wr = w.x, wi = -(double)w.y;  // conj(psi_{y^f})
    double pr = vr * wr - vi * wi, pi = vr * wi + vi * wr;
    double base;
    switch (grp.ny & 3) {
      case 0: base = pr; break;
      case 1: base = -pi; break;   // * i
      case 2: base = -pr; break;
      default: base = pi; break;   // * -i
    }
    double c = 0.0;
    for (int t = 0; t < grp.nterms; t++) c += (__popcll(y & grp.zm[t]) & 1) ? -grp.coeff[t] : grp.coeff[t];
    acc += base * c;
  }
  double t = block_sum<NT>(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// Sums of Pauli terms over tiles of 2^12 amplitudes held in shared memory: every
// term whose flips lie inside the tile is evaluated on one read of the state,
// where k_pauli_group reads it once per flip mask.
//
// Thread t of 512 holds amplitudes t + 512 j, so tile bits 9-11 are register bits
// (8 amplitudes in 64 registers let 32 warps cover each other's loads; 16
// amplitudes in 128 registers were several times slower).  A group's products are
// |psi_y|^2 (8 a thread) or, with flips, Re or Im of conj(psi_x) psi_y, one per
// pair, so 4 a thread: the pairs of a register flip by the member with its top
// flip bit clear, those of a thread flip half by either thread; the other member
// comes from shared memory.  A term's sign is a tile part, folded into its
// coefficient once a tile, a thread part, and a parity of the products' index:
// a group of several terms takes one Walsh transform over that index, after
// which a term costs one addition.
// Bound: HBM for few groups; for many, issue and the latency of the partners'
// shared-memory reads (half a tile a group).  25 qubits, 24 Z Z and 25 X terms:
// 26 passes of 136 us before, 3 passes of 374, 225 and 178 us now (12, 8 and 5
// flips; one read of the state is 82 us).  Below 12 qubits a tile is not full and
// a group a pass costs a launch each.
constexpr int kPauliThreads = 512;

template <typename R>
__global__ void __launch_bounds__(kPauliThreads, 2) k_pauli_tile(const typename Vec2<R>::T* a, PauliTileArgs g,
                                                                 const PauliTileGroup* groups,
                                                                 const PauliTileTerm* terms, double* partial) {
  typedef typename Vec2<R>::T V;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* s = reinterpret_cast<V*>(smraw);
  __shared__ double red[32];
  __shared__ double sc[KET_PAULI_TILE_TERMS];
  __shared__ uint32_t zm[KET_PAULI_TILE_TERMS];
  __shared__ PauliTileGroup gs[KET_PAULI_TILE_TERMS];
  const int t = threadIdx.x;
  static_assert(kPauliThreads == KET_PAULI_TILE_TERMS, "one term and one group a thread");
  if (t < g.ngroups) gs[t] = groups[t];
  double coeff = 0.0;
  uint64_t zctx = 0;
  if (t < g.nterms) {
    coeff = terms[t].coeff;
    zctx = terms[t].zctx;
    zm[t] = terms[t].zm;
  }
  const int lane = t & 31, ctxq = lane < g.nctx ? g.ctxbits[lane] : 63;
  auto coeff_of = [&](int i) { return sc[i]; };
  auto mask_of = [&](int i) { return zm[i]; };
  uint64_t toff = 0;
#pragma unroll
  for (int b = 0; b < 9; b++)
    if ((t >> b) & 1) toff |= uint64_t(1) << g.bits[b];
  double acc = 0.0;
  for (uint64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
    // lane b places tile bit b (at most 28 qubits lie outside the tile)
    const uint64_t mine = ((tile >> lane) & 1) << ctxq;
    const uint64_t ctx = ((uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(mine >> 32)) << 32) |
                         __reduce_or_sync(0xffffffffu, (uint32_t)mine);
    V v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint64_t o = ctx | toff;
#pragma unroll
      for (int b = 0; b < 3; b++)
        if ((j >> b) & 1) o |= uint64_t(1) << g.bits[9 + b];
      v[j] = a[o];
    }
    __syncthreads();  // the last tile's reads of s and sc are done
    if (t < g.nterms) sc[t] = (__popcll(ctx & zctx) & 1) ? -coeff : coeff;
    if (g.flips) {
#pragma unroll
      for (int j = 0; j < 8; j++) s[t + 512 * j] = v[j];
    }
    __syncthreads();
    for (int k = 0; k < g.ngroups; k++) {
      const PauliTileGroup G = gs[k];
      if (G.flip == 0) {
        double b[8];
#pragma unroll
        for (int j = 0; j < 8; j++) b[j] = norm2_ref(v[j].x, v[j].y);
        acc += pauli_terms<8>(b, coeff_of, mask_of, G.first, G.nterms, t);
        continue;
      }
      double b[4];
      // this thread's pairs: register index u with a bit inserted at P, clear for a
      // register flip, the thread's top flip bit (`set`) for a thread flip
      auto products = [&](auto PP, auto ODD, bool set) {
        constexpr int P = decltype(PP)::value;
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int j0 = ((u >> P) << (P + 1)) | (u & ((1 << P) - 1)), j1 = j0 | (1 << P);
          const V w = s[(t + 512 * (set ? j1 : j0)) ^ G.flip];
          const double vr = set ? v[j1].x : v[j0].x, vi = set ? v[j1].y : v[j0].y, wr = w.x, wi = w.y;
          b[u] = decltype(ODD)::value ? vi * wr - vr * wi : vr * wr + vi * wi;
        }
      };
      auto by_top = [&](auto ODD) {
        switch (G.top) {
          case 9: products(std::integral_constant<int, 0>(), ODD, false); break;
          case 10: products(std::integral_constant<int, 1>(), ODD, false); break;
          case 11: products(std::integral_constant<int, 2>(), ODD, false); break;
          default: products(std::integral_constant<int, 2>(), ODD, (t >> G.top) & 1); break;
        }
      };
      if (G.odd) by_top(std::true_type());
      else by_top(std::false_type());
      acc += pauli_terms<4>(b, coeff_of, mask_of, G.first, G.nterms, t);
    }
  }
  const double sum = block_sum<kPauliThreads>(acc, red);
  if (t == 0) partial[blockIdx.x] = sum;
}

// lambda = H psi by the same tiles (c128): a pass adds the terms it holds to
// lambda, every amplitude's partner coming from shared memory; the last pass sums
// Re <psi|lambda>.  A group's coefficients over the register bits are one number
// (a term without Z or Y there), or the Walsh transform of its terms'.
// Bound: shared memory (the tile once a group) and, for few groups, HBM.  24
// qubits, 23 Z Z and 24 X terms: 3 passes of 167 us,
// where one kernel over all terms took 1340 (and 43 for a serial sum).
__global__ void __launch_bounds__(kPauliThreads, 2) k_hpsi_tile(const double2* psi, double2* lam, PauliTileArgs g,
                                                                const PauliTileGroup* groups,
                                                                const PauliTileTerm* terms, double ident, int first,
                                                                int last, double* partial) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* s = reinterpret_cast<double2*>(smraw);
  __shared__ double red[32];
  __shared__ double sc[KET_PAULI_TILE_TERMS];
  __shared__ uint32_t zm[KET_PAULI_TILE_TERMS];
  __shared__ PauliTileGroup gs[KET_PAULI_TILE_TERMS];
  const int t = threadIdx.x, lane = t & 31, ctxq = lane < g.nctx ? g.ctxbits[lane] : 63;
  if (t < g.ngroups) gs[t] = groups[t];
  double coeff = 0.0;
  uint64_t zctx = 0;
  if (t < g.nterms) {
    coeff = terms[t].coeff;
    zctx = terms[t].zctx;
    zm[t] = terms[t].zm;
  }
  uint64_t toff = 0;
#pragma unroll
  for (int b = 0; b < 9; b++)
    if ((t >> b) & 1) toff |= uint64_t(1) << g.bits[b];
  auto signed_coeff = [&](int i, uint32_t z) { return flip_sign(sc[i], __popc(t & z & 0xffffu) & 1); };
  double e = 0.0;
  for (uint64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
    const uint64_t mine = ((tile >> lane) & 1) << ctxq;
    const uint64_t ctx = ((uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(mine >> 32)) << 32) |
                         __reduce_or_sync(0xffffffffu, (uint32_t)mine);
    auto at = [&](int j) {
      uint64_t o = ctx | toff;
#pragma unroll
      for (int b = 0; b < 3; b++)
        if ((j >> b) & 1) o |= uint64_t(1) << g.bits[9 + b];
      return o;
    };
    __syncthreads();  // the last tile's reads of s and sc are done
    if (t < g.nterms) sc[t] = (__popcll(ctx & zctx) & 1) ? -coeff : coeff;
    double2 l[8];
#pragma unroll
    for (int j = 0; j < 8; j++) s[t + 512 * j] = psi[at(j)];
    if (first) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const double2 v = s[t + 512 * j];
        l[j] = make_double2(ident * v.x, ident * v.y);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) l[j] = lam[at(j)];
    }
    __syncthreads();
    for (int k = 0; k < g.ngroups; k++) {
      const PauliTileGroup G = gs[k];
      const uint32_t z0 = zm[G.first];
      double c[8];
      if (G.nterms == 1) {
        const double c0 = signed_coeff(G.first, z0);
#pragma unroll
        for (int j = 0; j < 8; j++) c[j] = ((0x96u >> (j & (z0 >> 16))) & 1u) ? -c0 : c0;
      } else {
        int i = G.first;
#pragma unroll
        for (int w = 0; w < 8; w++) {
          c[w] = 0.0;
          for (; i < G.first + G.nterms; i++) {
            const uint32_t z = zm[i];
            if ((z >> 16) != w) break;
            c[w] += signed_coeff(i, z);
          }
        }
#pragma unroll
        for (int st = 1; st < 8; st <<= 1)
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (!(j & st)) {
              const double x = c[j], y = c[j | st];
              c[j] = x + y;
              c[j | st] = x - y;
            }
      }
      if (G.odd) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const double2 w = s[(t + 512 * j) ^ G.flip];
          l[j].x = fma(-c[j], w.y, l[j].x);
          l[j].y = fma(c[j], w.x, l[j].y);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const double2 w = s[(t + 512 * j) ^ G.flip];
          l[j].x = fma(c[j], w.x, l[j].x);
          l[j].y = fma(c[j], w.y, l[j].y);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) lam[at(j)] = l[j];
    if (last) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const double2 v = s[t + 512 * j];
        e += v.x * l[j].x + v.y * l[j].y;
      }
    }
  }
  if (last) {
    const double sum = block_sum<kPauliThreads>(e, red);
    if (t == 0) partial[blockIdx.x] = sum;
  }
}

inline unsigned gridn(uint64_t work, int nt, int cap_per_sm = 16) {
  uint64_t b = (work + nt - 1) / nt;
  uint64_t cap = (uint64_t)num_sms() * cap_per_sm;
  return (unsigned)std::max<uint64_t>(1, std::min(b, cap));
}

}  // namespace

// ------------------------------------------------------------------ launchers
template <typename R>
static cudaError_t norm2_t(const void* amp, int n, double* scratch, double* out, cudaStream_t s) {
  const uint64_t N = uint64_t(1) << n;
  const uint64_t chunk = std::max<uint64_t>(N / 4096, 4096);
  const uint64_t nb = (N + chunk - 1) / chunk;
  k_norm_partial<R, 256><<<(unsigned)nb, 256, 0, s>>>((const typename Vec2<R>::T*)amp, N, chunk, scratch);
  k_sum<256><<<1, 256, 0, s>>>(scratch, nb, out);
  return cudaGetLastError();
}

cudaError_t launch_norm2(const void* amp, int n, int prec, double* scratch, double* out, cudaStream_t s) {
  return prec == KET_C64 ? norm2_t<float>(amp, n, scratch, out, s) : norm2_t<double>(amp, n, scratch, out, s);
}
size_t norm2_scratch(int n) { return 8 * 4096 + 64; }

template <typename R>
static cudaError_t probs_dense_t(const void* amp, uint64_t off, uint64_t cnt, double thr, double* out, cudaStream_t s) {
  k_probs_dense<R><<<gridn(cnt, 256), 256, 0, s>>>((const typename Vec2<R>::T*)amp, off, cnt, thr, out);
  return cudaGetLastError();
}
cudaError_t launch_probs_dense(const void* amp, int prec, uint64_t off, uint64_t cnt, double thr, double* out,
                               cudaStream_t s) {
  return prec == KET_C64 ? probs_dense_t<float>(amp, off, cnt, thr, out, s)
                         : probs_dense_t<double>(amp, off, cnt, thr, out, s);
}

uint64_t kept_chunk(int n) {
  uint64_t N = uint64_t(1) << n;
  return std::max<uint64_t>(N / 8192, 1024);
}
template <typename R>
static cudaError_t count_kept_t(const void* amp, int n, double thr, uint64_t* counts, cudaStream_t s) {
  uint64_t N = uint64_t(1) << n, chunk = kept_chunk(n), nb = (N + chunk - 1) / chunk;
  k_count_kept<R, 256><<<(unsigned)nb, 256, 0, s>>>((const typename Vec2<R>::T*)amp, N, chunk, thr, counts);
  return cudaGetLastError();
}
cudaError_t launch_count_kept(const void* amp, int n, int prec, double thr, uint64_t* counts, cudaStream_t s) {
  return prec == KET_C64 ? count_kept_t<float>(amp, n, thr, counts, s) : count_kept_t<double>(amp, n, thr, counts, s);
}
template <typename R>
static cudaError_t compact_t(const void* amp, int n, double thr, const uint64_t* offs, uint64_t cap, uint64_t* oi,
                             double* op, cudaStream_t s) {
  uint64_t N = uint64_t(1) << n, chunk = kept_chunk(n), nb = (N + chunk - 1) / chunk;
  k_compact_kept<R, 256><<<(unsigned)nb, 256, 0, s>>>((const typename Vec2<R>::T*)amp, N, chunk, thr, offs, cap, oi, op);
  return cudaGetLastError();
}
cudaError_t launch_compact_kept(const void* amp, int n, int prec, double thr, const uint64_t* offs, uint64_t cap,
                                uint64_t* oidx, double* op, cudaStream_t s) {
  return prec == KET_C64 ? compact_t<float>(amp, n, thr, offs, cap, oidx, op, s)
                         : compact_t<double>(amp, n, thr, offs, cap, oidx, op, s);
}

// At most 2048 blocks, of at least 2^12 indices (16 a thread).
static int marg_chunk_bits(int n) { return std::max(12, n - 11); }
uint64_t marg_chunk(int n) { return uint64_t(1) << marg_chunk_bits(n); }
template <typename R>
static cudaError_t marginals_t(const void* amp, int n, double* partial, double* out, cudaStream_t s) {
  const int c = marg_chunk_bits(n);
  const uint64_t nb = n > c ? uint64_t(1) << (n - c) : 1;
  k_marginals<R><<<(unsigned)nb, 256, 0, s>>>((const typename Vec2<R>::T*)amp, n, c, partial);
  k_sum_columns<<<(n + 31) / 32, 32 * kColRows, 0, s>>>(partial, nb, n, out);
  return cudaGetLastError();
}
cudaError_t launch_marginals(const void* amp, int n, int prec, double* partial, double* out, cudaStream_t s) {
  return prec == KET_C64 ? marginals_t<float>(amp, n, partial, out, s) : marginals_t<double>(amp, n, partial, out, s);
}

// At most 1024 blocks of at least 2^12 indices: the blocks' sums (2^12 bins at
// most) stay below a thirtieth of a large state's bytes.
static int mdist_chunk_bits(int n) { return std::max(12, n - 10); }
size_t mdist_partials(int n, uint64_t mask) {
  const int c = mdist_chunk_bits(n);
  return (size_t)(n > c ? uint64_t(1) << (n - c) : 1) << __builtin_popcountll(mask & ((uint64_t(1) << c) - 1));
}
template <typename R>
static cudaError_t mdist_t(const void* amp, int n, const MarginalSpec& spec, double* partial, double* out,
                           cudaStream_t s) {
  const int c = mdist_chunk_bits(n);
  const uint64_t nb = n > c ? uint64_t(1) << (n - c) : 1;
  k_marginal_dist<R><<<(unsigned)nb, 256, 0, s>>>((const typename Vec2<R>::T*)amp, n, c, spec.mask, partial);
  k_marginal_dist_combine<<<((1u << spec.m) + 31) / 32, 32 * kColRows, 0, s>>>(partial, n, c, spec, out);
  return cudaGetLastError();
}
cudaError_t launch_marginal_dist(const void* amp, int n, int prec, const MarginalSpec& spec, double* partial,
                                 double* out, cudaStream_t s) {
  return prec == KET_C64 ? mdist_t<float>(amp, n, spec, partial, out, s) : mdist_t<double>(amp, n, spec, partial, out, s);
}

// Scratch layout of the sampler: nk + 1 checkpoints, then per block the
// approximate prefix (nb + 1), the first and last kept index, D, the exact
// start, the state and the binade; the state's first and last kept index.
struct CdfScratch {
  double* ck;
  double* bsum;
  unsigned long long* bfirst;
  unsigned long long* blast;
  long long* bd;
  double* bstart;
  int* bst;
  int* be;
  unsigned long long* fl;
  size_t bytes;
};
static CdfScratch cdf_scratch(int n, void* base) {
  const uint64_t N = uint64_t(1) << n;
  const uint64_t nk = (N + kCdfSub - 1) / kCdfSub, nb = (N + kCdfBlock - 1) / kCdfBlock;
  CdfScratch c;
  char* p = (char*)base;
  auto take = [&](size_t bytes) {
    char* r = p;
    p += (bytes + 255) & ~size_t(255);
    return (void*)r;
  };
  c.ck = (double*)take(8 * (nk + 1));
  c.bsum = (double*)take(8 * (nb + 1));
  c.bfirst = (unsigned long long*)take(8 * nb);
  c.blast = (unsigned long long*)take(8 * nb);
  c.bd = (long long*)take(8 * nb);
  c.bstart = (double*)take(8 * nb);
  c.bst = (int*)take(4 * nb);
  c.be = (int*)take(4 * nb);
  c.fl = (unsigned long long*)take(16);
  c.bytes = (size_t)(p - (char*)base);
  return c;
}

template <typename R>
static cudaError_t sample_t(const void* amp, int n, double thr, const double* r, uint64_t shots, void* scratch,
                            uint64_t* out, cudaStream_t s) {
  const typename Vec2<R>::T* a = (const typename Vec2<R>::T*)amp;
  const uint64_t N = uint64_t(1) << n;
  const uint64_t nk = (N + kCdfSub - 1) / kCdfSub, nb = (N + kCdfBlock - 1) / kCdfBlock;
  const CdfScratch c = cdf_scratch(n, scratch);
  k_cdf_block_sums<R><<<(unsigned)nb, 256, 0, s>>>(a, N, thr, c.bsum, c.bfirst, c.blast);
  k_cdf_block_prefix<<<1, kCdfThreads, 0, s>>>(c.bsum, c.bfirst, c.blast, nb, c.fl);
  k_cdf_block_d<R><<<(unsigned)nb, 256, 0, s>>>(a, N, thr, c.bsum, (long long*)c.ck, c.bd, c.bst, c.be);
  k_cdf_walk<R><<<1, kWalkThreads, 0, s>>>(a, N, thr, nb, nk, c.ck, c.bd, c.bst, c.be, c.bstart);
  k_cdf_fill<<<gridn(nk, 256), 256, 0, s>>>(c.ck, nk, c.bst, c.be, c.bstart);
  k_sample_ck<R><<<gridn(shots, 128), 128, 0, s>>>(a, N, thr, c.ck, nk, r, shots, c.fl, out);
  return cudaGetLastError();
}
size_t sample_scratch(int n) { return cdf_scratch(n, nullptr).bytes; }
int sample_launches() { return 6; }
cudaError_t launch_sample(const void* amp, int n, int prec, double thr, const double* r, uint64_t shots, void* scratch,
                          uint64_t* out, cudaStream_t s) {
  return prec == KET_C64 ? sample_t<float>(amp, n, thr, r, shots, scratch, out, s)
                         : sample_t<double>(amp, n, thr, r, shots, scratch, out, s);
}

cudaError_t launch_gather(const void* amp, int prec, const uint64_t* idx, uint64_t k, double* out, cudaStream_t s) {
  if (prec == KET_C64) k_gather<float><<<gridn(k, 256), 256, 0, s>>>((const float2*)amp, idx, k, out);
  else k_gather<double><<<gridn(k, 256), 256, 0, s>>>((const double2*)amp, idx, k, out);
  return cudaGetLastError();
}

template <typename R>
static cudaError_t pauli_t(const void* amp, int n, const PauliGroup& g, double* partial, double* out, cudaStream_t s) {
  const uint64_t N = uint64_t(1) << n;
  const uint64_t chunk = std::max<uint64_t>(N / 4096, 2048);
  const uint64_t nb = (N + chunk - 1) / chunk;
  k_pauli_group<R, 256><<<(unsigned)nb, 256, 0, s>>>((const typename Vec2<R>::T*)amp, N, chunk, g, partial);
  k_sum<256><<<1, 256, 0, s>>>(partial, nb, out);
  return cudaGetLastError();
}
cudaError_t launch_pauli_group(const void* amp, int n, int prec, const PauliGroup& g, double* partial, double* out,
                               cudaStream_t s) {
  return prec == KET_C64 ? pauli_t<float>(amp, n, g, partial, out, s) : pauli_t<double>(amp, n, g, partial, out, s);
}
size_t pauli_scratch(int n) { return 8 * 4096 + 64; }

unsigned pauli_tile_grid(int n) {
  return (unsigned)std::min<uint64_t>(uint64_t(1) << (n - KET_PAULI_TILE_BITS), (uint64_t)num_sms() * 2);
}
template <typename R>
static cudaError_t pauli_tile_t(const void* amp, const PauliTileArgs& g, const PauliTileGroup* groups,
                                const PauliTileTerm* terms, double* partial, unsigned grid, cudaStream_t s) {
  const int smem = (int)(sizeof(typename Vec2<R>::T) << KET_PAULI_TILE_BITS);
  cudaError_t e = cudaFuncSetAttribute(k_pauli_tile<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  k_pauli_tile<R><<<grid, kPauliThreads, smem, s>>>((const typename Vec2<R>::T*)amp, g, groups, terms, partial);
  return cudaGetLastError();
}
cudaError_t launch_pauli_tile(const void* amp, int n, int prec, const PauliTileArgs& g, const PauliTileGroup* groups,
                              const PauliTileTerm* terms, double* partial, cudaStream_t s) {
  return prec == KET_C64 ? pauli_tile_t<float>(amp, g, groups, terms, partial, pauli_tile_grid(n), s)
                         : pauli_tile_t<double>(amp, g, groups, terms, partial, pauli_tile_grid(n), s);
}
cudaError_t launch_hpsi_tile(const void* psi, void* lam, int n, const PauliTileArgs& g, const PauliTileGroup* groups,
                             const PauliTileTerm* terms, double ident, bool first, bool last, double* partial,
                             cudaStream_t s) {
  const int smem = (int)(sizeof(double2) << KET_PAULI_TILE_BITS);
  cudaError_t e = cudaFuncSetAttribute(k_hpsi_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  k_hpsi_tile<<<pauli_tile_grid(n), kPauliThreads, smem, s>>>((const double2*)psi, (double2*)lam, g, groups, terms, ident,
                                                              first, last, partial);
  return cudaGetLastError();
}
cudaError_t launch_sum(const double* partial, uint64_t count, double* out, cudaStream_t s) {
  k_sum<256><<<1, 256, 0, s>>>(partial, count, out);
  return cudaGetLastError();
}

template <typename RA, typename RB>
static cudaError_t compare_t(const void* a, const void* b, int n, double* scratch, double* out, cudaStream_t s) {
  const uint64_t N = uint64_t(1) << n;
  const uint64_t chunk = std::max<uint64_t>(N / 4096, 4096);
  const uint64_t nb = (N + chunk - 1) / chunk;
  k_compare<RA, RB, 256><<<(unsigned)nb, 256, 0, s>>>((const typename Vec2<RA>::T*)a,
                                                      (const typename Vec2<RB>::T*)b, N, chunk, scratch);
  k_compare_combine<<<1, 32, 0, s>>>(scratch, nb, out);
  return cudaGetLastError();
}
cudaError_t launch_compare(const void* a, int pa, const void* b, int pb, int n, double* scratch, double* out,
                           cudaStream_t s) {
  if (pa == KET_C64 && pb == KET_C64) return compare_t<float, float>(a, b, n, scratch, out, s);
  if (pa == KET_C64) return compare_t<float, double>(a, b, n, scratch, out, s);
  if (pb == KET_C64) return compare_t<double, float>(a, b, n, scratch, out, s);
  return compare_t<double, double>(a, b, n, scratch, out, s);
}
size_t compare_scratch(int) { return 3 * 8 * 4096 + 64; }

}  // namespace ket
