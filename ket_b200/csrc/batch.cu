// batch.cu -- thousands of QAOA MaxCut circuits of uneven width in one
// persistent launch (ket_batch_qaoa).
//
// Each instance: H on all n qubits, then per layer exp(-i gamma Z_u Z_v) on
// every edge and Rx(2 beta) on every qubit; output <C> = sum_e (1 - <Z_u Z_v>)/2.
// The reference builds the same circuit as qaoa(n, E, -2 gamma, beta)
// (algorithms.ts:260-276: cnot . rz . cnot per edge) and measures it with
// vqe(., maxCutHamiltonian(n, E)) (algorithms.ts:231-241, 301-336).
//
// Work items are pulled from global queues by persistent grids:
//   * an instance of n <= TILE qubits is one item of k_qaoa_chip, its whole state in
//     shared memory (all layers and the <C> reduction);
//   * a wider instance is split into p + 1 passes of tiles of 2^TILE amplitudes
//     (k_batch_qaoa).
//     A tile holds either the low TILE qubits (even passes) or the qubits above
//     them with the lowest qubits (odd passes).  Rx gates commute and the cost
//     phase is diagonal, so pass k finishes layer k - 1 on its qubits, applies
//     layer k's phase (every other qubit's Rx of layer k - 1 was done in pass k - 1)
//     and starts layer k on its qubits: one read and write of the state a layer.
//     A tile of pass k waits (bounded spin, error flag on timeout) until every tile
//     of pass k-1 of its instance has been written back; the queue hands items
//     out in an order where everything a tile waits on was handed out earlier, so
//     the fully resident grid cannot deadlock.
// A tile of a wide instance lives in registers, 2^K consecutive values of K of its bits a thread; Rx on
// those bits needs no exchange, and the other bits come round through shared memory.
// Rx(2 beta) = cos(beta) (1 - i tan(beta) X) is applied without its scalar, so an
// amplitude takes two FMAs a gate; <C> is divided by the norm that is left.  Where
// |tan(beta)| > 1, beta - pi/2 stands in for beta: the two differ by X on every
// qubit, which commutes with the circuit and leaves every cut as it is.
// The cost phase exp(-i gamma (|E| - 2 cut(x))) comes from a table of |E|+1 phases
// a layer; a thread counts cut(x) once and follows its register bits from there.
// Partials of <C> and of the norm are written per (instance, tile) and reduced
// in a fixed order.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "launch.h"
#include "rounds.h"

namespace ket {

namespace {

#define KQ_MAX_EDGES 64
#define KQ_MAX_P 16

struct QInst {
  int n, ne, p, ntiles;     // ntiles = 2^(n - tile) for split instances, 0 on the chip
  int multi, pad;           // an edge occurs twice: cut(x) is counted for every amplitude
  int64_t state;            // offset (amplitudes) of the instance's state in the workspace (split only)
  int64_t edge_off;         // first edge in the edge array
  int64_t part_off;         // first <C> partial of the instance
  int64_t tab_off;          // first phase of layer 0; a layer has ne + 1
};

// The queue's items in order: run r holds items [first, the next run's first), the
// tiles of one pass (0..p) of a wide instance.
struct QRun {
  int first, inst, pass, pad;
};

struct QArgs {
  const QInst* inst;
  const QRun* runs;         // and an end mark
  const int* chip;          // the instances that fit the chip, widest first
  const uint32_t* emask;    // edge masks (1<<u | 1<<v)
  const double* gamma;      // [inst * p + l]
  const double* beta;
  double* tan;              // [inst * p + l]: tan(beta), beta taken to [-pi/4, pi/4]
  double2* tab;             // phases by instance, layer and cut
  double2* work;            // split-instance states
  double2* part;            // (<C>, norm) partials
  double* out;              // <C> by instance
  unsigned int* next;       // queue heads: tiles of wide instances, chip instances
  unsigned int* done;       // per instance: tiles finished (pass-major)
  int* status;
  uint32_t spin_limit;      // polls before a wait gives up (status KET_ERR_TIMEOUT)
  int nitems;
  int nchip, chip_bits;     // instances on the chip, qubits of the widest
  int drop;                 // test hook: an item that is left out (-1: none)
};

// Layer angles to phase tables and tangents, once a call: a CTA a (instance, layer).
__global__ void k_qaoa_tables(QArgs a, int p) {
  const int i = blockIdx.x / p, l = blockIdx.x % p;
  const QInst I = a.inst[i];
  if (I.ntiles == 0) return;
  const double gamma = a.gamma[blockIdx.x];
  for (int c = threadIdx.x; c <= I.ne; c += blockDim.x) {
    double s, co;
    sincos(-gamma * (double)(I.ne - 2 * c), &s, &co);
    a.tab[I.tab_off + (int64_t)l * (I.ne + 1) + c] = make_double2(co, s);
  }
  if (threadIdx.x == 0) {
    double sb, cb;
    sincos(a.beta[blockIdx.x], &sb, &cb);
    a.tan[blockIdx.x] = fabs(cb) < fabs(sb) ? -cb / sb : sb / cb;
  }
}

// What a CTA keeps of an instance in shared memory beside the tile.
struct QShared {
  double2 tab[KQ_MAX_EDGES + 1];
  uint32_t em[KQ_MAX_EDGES];
  uint32_t nbr[32];          // neighbours of each qubit
  double red[32];
  int item[2], failed;
  QRun run;
  QInst inst;
};

__device__ __forceinline__ int cut_of(uint32_t x, const uint32_t* em, int ne) {
  int c = 0;
  for (int e = 0; e < ne; e++) c += __popc(x & em[e]) & 1;
  return c;
}

// The layouts of a tile of T bits on NT threads: in layout g the thread's 2^K
// amplitudes run over the tile bits reg(g, 0..K-1), and thread bit b is tile bit
// thr(g, b).  Every tile bit is turned in one layout.  The last layout's lanes are
// the lowest tile bits, so loads and stores are of runs.
//
// In general layout g holds the bits from K g (the last reaches back when K does not
// divide T).  A tile of 12 bits on 256 threads orders them so that layouts 1 and 2
// keep the same warp bits (9-11): that move stays inside a warp, and a pass meets
// two CTA barriers instead of four (19.3 -> 18.7 ms on 512 instances).  The lowest
// three lanes of each layout fall on three different bank bits.
template <int NT, int T>
struct QLay {
  static constexpr int LT = NT == 128 ? 7 : NT == 256 ? 8 : 9;
  static constexpr int K = T - LT, NS = 1 << K, NG = (T + K - 1) / K;
  // CTAs an SM holds: by registers (4 an amplitude and as many again), by shared memory
  static constexpr int CTAS = T == 11 ? (NT == 512 ? 2 : 4) : 2;
  static constexpr bool WARP = T == 12 && NT == 256;
  static constexpr int s(int g) { return K * g < T - K ? K * g : T - K; }
  __host__ __device__ static constexpr int reg(int g, int b) {
    if (!WARP) return s(g) + b;
    return g == 0 ? (b == 0 ? 0 : 8 + b) : g == 1 ? 1 + b : 5 + b;
  }
  __host__ __device__ static constexpr int thr(int g, int b) {
    if (!WARP) return b < s(g) ? b : b + K;
    constexpr int one[8] = {0, 5, 7, 6, 8, 9, 10, 11};
    return g == 0 ? 1 + b : g == 1 ? one[b] : b < 5 ? b : 4 + b;
  }
  // whether layout g turns its register bit b (the last layout reaches back)
  __host__ __device__ static constexpr bool turns(int g, int b) { return WARP || s(g) + b >= K * g; }
  __host__ __device__ static constexpr bool in_warp(int g, int h) { return WARP && g + h == 3; }  // 1 <-> 2
};

// Tile qubits to global qubits: pass A tiles hold qubits 0..T-1; pass B tiles the
// low lowB qubits and qubits T..n-1.
struct QMap {
  uint32_t base;   // global index of tile element 0
  int lowB, T;     // lowB = T: pass A
  __device__ __forceinline__ int qubit(int b) const { return b < lowB ? b : T + b - lowB; }
  __device__ __forceinline__ uint32_t index(uint32_t i) const {  // of tile element i, but for base
    return (i & ((1u << lowB) - 1)) | (i >> lowB) << T;
  }
};

template <int NT, int T, int G>
__device__ __forceinline__ uint32_t tile_index(int t) {  // of the thread's register index 0
  uint32_t i = 0;
#pragma unroll
  for (int b = 0; b < QLay<NT, T>::LT; b++) i |= (((uint32_t)t >> b) & 1u) << QLay<NT, T>::thr(G, b);
  return i;
}
template <int NT, int T, int G>
__host__ __device__ constexpr uint32_t reg_index(int j) {  // tile bits of register index j
  uint32_t i = 0;
  for (int b = 0; b < QLay<NT, T>::K; b++)
    if ((j >> b) & 1) i |= 1u << QLay<NT, T>::reg(G, b);
  return i;
}

// Rx on the layout's own bits in `rotate` (tile bits).  The others turn by zero,
// which leaves them as they are: with a branch a bit, half of the new values moved
// back to their old registers, as many moves as FMAs (17.5 -> 16.0 ms on 512
// instances).
template <int NT, int T, int G>
__device__ __forceinline__ void rotate_regs(double2* v, uint32_t rotate, double tan) {
  constexpr int K = QLay<NT, T>::K, NS = QLay<NT, T>::NS;
#pragma unroll
  for (int b = 0; b < K; b++) {
    if (!QLay<NT, T>::turns(G, b)) continue;
    const double r = (rotate >> QLay<NT, T>::reg(G, b)) & 1 ? tan : 0.0;
#pragma unroll
    for (int j = 0; j < NS; j++) {
      if (j & (1 << b)) continue;
      // x' = x - i r y, y' = y - i r x
      const double2 x = v[j], y = v[j | 1 << b];
      v[j] = make_double2(fma(r, y.y, x.x), fma(-r, y.x, x.y));
      v[j | 1 << b] = make_double2(fma(r, x.y, y.x), fma(-r, x.x, y.y));
    }
  }
}

// cut(x) of the thread's 2^K amplitudes: counted at register index 0, then
// followed bit by bit -- setting a bit whose qubit has d neighbours, c of them
// set, changes the cut by d - 2 c.
template <int NT, int T, int G>
__device__ __forceinline__ void cuts(int (&c)[QLay<NT, T>::NS], const QMap& m, int t, const QShared& sh, const QInst& I) {
  typedef QLay<NT, T> L;
  constexpr int K = L::K, NS = L::NS;
  const uint32_t x0 = m.base | m.index(tile_index<NT, T, G>(t));
  c[0] = cut_of(x0, sh.em, I.ne);
  if (I.multi) {
#pragma unroll
    for (int j = 1; j < NS; j++) {
      uint32_t x = x0;
#pragma unroll
      for (int b = 0; b < K; b++)
        if ((j >> b) & 1) x |= 1u << m.qubit(L::reg(G, b));
      c[j] = cut_of(x, sh.em, I.ne);
    }
    return;
  }
#pragma unroll
  for (int b = K - 1; b >= 0; b--) {
    const uint32_t nb = sh.nbr[m.qubit(L::reg(G, b))];
    uint32_t adj = 0;  // the register bits above b that neighbour it
#pragma unroll
    for (int u = b + 1; u < K; u++) adj |= ((nb >> m.qubit(L::reg(G, u))) & 1u) << u;
    const int d = __popc(nb) - 2 * __popc(x0 & nb);
#pragma unroll
    for (int j = 0; j < NS; j++)
      if (((j >> b) & 1) && !(j & ((1 << b) - 1))) c[j] = c[j ^ (1 << b)] + d - 2 * __popc(j & adj);
  }
}

template <int NT, int T, int G>
__device__ __forceinline__ void phase_regs(double2* v, const QMap& m, int t, const QShared& sh, const QInst& I) {
  constexpr int NS = QLay<NT, T>::NS;
  int c[NS];
  cuts<NT, T, G>(c, m, t, sh, I);
#pragma unroll
  for (int j = 0; j < NS; j++) {
    const double2 ph = sh.tab[c[j]], x = v[j];
    v[j] = make_double2(fma(ph.x, x.x, -ph.y * x.y), fma(ph.x, x.y, ph.y * x.x));
  }
}

// From layout G to layout H through shared memory.  A thread writes the slots it
// read last, which no other thread reads until the barrier: one barrier a move (of
// the warp where it moves only between its own threads).
template <int NT, int T, int G, int H>
__device__ __forceinline__ void relayout(double2* v, double2* s, int t) {
  constexpr int NS = QLay<NT, T>::NS;
  const uint32_t g0 = round_slot(tile_index<NT, T, G>(t)), h0 = round_slot(tile_index<NT, T, H>(t));
#pragma unroll
  for (int j = 0; j < NS; j++) s[g0 ^ round_slot(reg_index<NT, T, G>(j))] = v[j];
  if constexpr (QLay<NT, T>::in_warp(G, H)) __syncwarp();
  else __syncthreads();
#pragma unroll
  for (int j = 0; j < NS; j++) v[j] = s[h0 ^ round_slot(reg_index<NT, T, H>(j))];
}

// Rx on every bit in `rotate`, from layout G up to the top layout / down to layout 0.
template <int NT, int T, int G>
__device__ __forceinline__ void rx_up(double2* v, double2* s, int t, uint32_t rotate, double r) {
  rotate_regs<NT, T, G>(v, rotate, r);
  if constexpr (G + 1 < QLay<NT, T>::NG) {
    relayout<NT, T, G, G + 1>(v, s, t);
    rx_up<NT, T, G + 1>(v, s, t, rotate, r);
  }
}
template <int NT, int T, int G>
__device__ __forceinline__ void rx_down(double2* v, double2* s, int t, uint32_t rotate, double r) {
  rotate_regs<NT, T, G>(v, rotate, r);
  if constexpr (G > 0) {
    relayout<NT, T, G, G - 1>(v, s, t);
    rx_down<NT, T, G - 1>(v, s, t, rotate, r);
  }
}

// Sums of |a|^2 cut(x) and |a|^2 over the tile, in layout G.
template <int NT, int T, int G>
__device__ __forceinline__ void tile_cut(const double2* v, const QMap& m, int t, QShared& sh, const QInst& I, double2* out) {
  constexpr int NS = QLay<NT, T>::NS;
  int c[NS];
  cuts<NT, T, G>(c, m, t, sh, I);
  double acc = 0.0, nrm = 0.0;
#pragma unroll
  for (int j = 0; j < NS; j++) {
    const double q = v[j].x * v[j].x + v[j].y * v[j].y;
    nrm += q;
    acc = fma(q, (double)c[j], acc);
  }
  acc = block_sum<NT>(acc, sh.red);
  __syncthreads();
  nrm = block_sum<NT>(nrm, sh.red);
  if (t == 0) *out = make_double2(acc, nrm);
}

// Bound: for wide instances the state's traffic (2 p reads and writes) and shared
// memory's (a tile moves through it four times a pass), then the FP64 pipe (two
// FMAs an amplitude and Rx).  512 instances of 10 to 22 qubits, p = 4:
// 35.9 ms as 2 p passes of three-bit rounds, 15.3 now (96 of 13 to 20 qubits: FP64 pipe 27%
// busy, HBM 20%; two CTAs of 8 warps wait for barriers and loads).
template <int NT, int T>
__global__ void __launch_bounds__(NT, QLay<NT, T>::CTAS) k_batch_qaoa(QArgs a) {
  typedef QLay<NT, T> L;
  constexpr int NS = L::NS, TOP = L::NG - 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* s = reinterpret_cast<double2*>(smraw);
  QShared& sh = *reinterpret_cast<QShared*>(smraw + (sizeof(double2) << T));
  const int t = threadIdx.x;
  if (t == 0) sh.item[0] = (int)atomicAdd(a.next, 1u);
  __syncthreads();
  // A CTA's items ascend, so its place in the runs only moves on; what a run's tiles
  // share is read once, and its wait is over once it has been.
  int run = 0, have = -1, end = a.runs[1].first;
  bool ready = false;
  const QRun& w = sh.run;
  const QInst& I = sh.inst;
  for (int turn = 0;; turn ^= 1) {
    const int it = sh.item[turn];
    if (it >= a.nitems) break;
    if (t == 0) sh.item[turn ^ 1] = (int)atomicAdd(a.next, 1u);  // the next item, while this one runs
    while (it >= end) end = a.runs[++run + 1].first;
    const bool fresh = run != have;
    if (fresh) {
      have = run;
      if (t == 0) {
        sh.run = a.runs[run];
        sh.inst = a.inst[sh.run.inst];
      }
      if (t < 32) sh.nbr[t] = 0;
      __syncthreads();
      ready = w.pass == 0;
      for (int e = t; e < I.ne; e += NT) sh.em[e] = a.emask[I.edge_off + e];
      __syncthreads();
      for (int e = t; e < I.ne; e += NT) {
        const uint32_t m = sh.em[e], u = __ffs(m) - 1, q = 31 - __clz(m);
        atomicOr(&sh.nbr[u], 1u << q);
        atomicOr(&sh.nbr[q], 1u << u);
      }
    }
    const int tile = it - w.first;
    if (it == a.drop) {
      __syncthreads();
      continue;
    }
    const int n = I.n;
    auto load_table = [&](int l) {
      for (int c = t; c <= I.ne; c += NT) sh.tab[c] = a.tab[I.tab_off + (int64_t)l * (I.ne + 1) + c];
    };
    double2 v[NS];
    if (fresh && w.pass < I.p) load_table(w.pass);
    if (!ready) {
      // wait until every tile of the previous pass has been written back; a
      // wait that ran out anywhere (status set) ends every later wait at once
      const unsigned int need = (unsigned int)w.pass * (unsigned int)I.ntiles;
      if (t == 0) {
        volatile unsigned int* d = a.done + w.inst;
        volatile int* st = a.status;
        uint32_t spins = 0;
        while (*d < need) {
          if (*st != 0) break;
          if (++spins > a.spin_limit) { atomicExch(a.status, (int)KET_ERR_TIMEOUT); break; }
          __nanosleep(100);
        }
        __threadfence();
        sh.failed = *st;
      }
      __syncthreads();  // (masks and table are in, too)
      if (sh.failed != 0) {
        // the call reports the timeout; drain the queue without the tile's work
        __syncthreads();
        if (t == 0) atomicAdd(a.done + w.inst, 1u);
        continue;
      }
      ready = true;
    } else if (fresh) {
      __syncthreads();
    }
    const bool passA = (w.pass & 1) == 0;
    const int nhigh = n - T;                          // qubits >= T
    const QMap m = passA ? QMap{(uint32_t)tile << T, T, T}
                         : QMap{(uint32_t)tile << (T - nhigh), T - nhigh, T};
    const uint32_t rotate = passA ? (1u << T) - 1u : ((1u << T) - 1u) & ~((1u << m.lowB) - 1u);
    double2* g = a.work + I.state + m.base + m.index(tile_index<NT, T, TOP>(t));
    auto off = [&](int j) {
      uint32_t o = 0;
#pragma unroll
      for (int b = 0; b < L::K; b++)
        if ((j >> b) & 1) o |= 1u << m.qubit(L::reg(TOP, b));
      return o;
    };
    if (w.pass == 0) {
      const double amp0 = 1.0 / sqrt((double)(1u << n));
#pragma unroll
      for (int j = 0; j < NS; j++) v[j] = make_double2(amp0, 0.0);
    } else {
#pragma unroll
      for (int j = 0; j < NS; j++) v[j] = __ldcg(g + off(j));
      rx_down<NT, T, TOP>(v, s, t, rotate, a.tan[(int64_t)w.inst * I.p + w.pass - 1]);
    }
    if (w.pass == I.p) {
      tile_cut<NT, T, 0>(v, m, t, sh, I, a.part + I.part_off + tile);
    } else {
      phase_regs<NT, T, 0>(v, m, t, sh, I);
      rx_up<NT, T, 0>(v, s, t, rotate, a.tan[(int64_t)w.inst * I.p + w.pass]);
#pragma unroll
      for (int j = 0; j < NS; j++) g[off(j)] = v[j];
    }
    __syncthreads();
    if (t == 0) {
      __threadfence();
      atomicAdd(a.done + w.inst, 1u);
    }
  }
}

// <C> of a wide instance: its partials added by a warp (strided runs, then a tree).
__global__ void k_qaoa_reduce(const QInst* inst, int ninst, const double2* part, double* out) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= ninst) return;
  const QInst I = inst[i];
  if (I.ntiles == 0) return;
  double acc = 0.0, nrm = 0.0;
  for (int t = lane; t < I.ntiles; t += 32) {
    const double2 p = part[I.part_off + t];
    acc += p.x;
    nrm += p.y;
  }
  acc = warp_sum(acc);
  nrm = warp_sum(nrm);
  if (lane == 0) out[i] = acc / nrm;
}

// ---------------------------------------------------------------- instances on the chip
// Shared-memory position of amplitude i: the three low index bits are XORed with
// bits 3-5.  For every group of rotated bits below, the eight threads of a quarter
// warp then touch eight distinct 16-byte slots of a 128-byte row (conflict-free),
// whichever bits the group holds.
__device__ __forceinline__ uint32_t sw(uint32_t i) { return i ^ ((i >> 3) & 7u); }

// Rx(2 beta) = [[c, -i s], [-i s, c]] on one pair, in registers.
__device__ __forceinline__ void rx_pair(double2& a, double2& b, double cb, double sb) {
  const double2 x = a, y = b;
  a = make_double2(fma(cb, x.x, sb * y.y), fma(cb, x.y, -sb * y.x));
  b = make_double2(fma(cb, y.x, sb * x.y), fma(cb, y.y, -sb * x.x));
}

// Rx(2 beta) on the K bits g[0] < ... < g[K-1] of a block of 2^m amplitudes: each
// thread loads the 2^K amplitudes of a subcube into registers, rotates every bit of
// the group there (lowest first), and stores them back -- one shared-memory round
// trip per group instead of one per bit.
template <int NT, int K>
__device__ void rx_group(double2* s, int m, uint32_t gp, double cb, double sb) {
  int g[K];  // the group's bits, packed one per byte of gp (kept in registers)
#pragma unroll
  for (int q = 0; q < K; q++) g[q] = (int)((gp >> (8 * q)) & 0xffu);
  const uint32_t nsub = 1u << (m - K);
  for (uint32_t u = threadIdx.x; u < nsub; u += NT) {
    uint32_t b = u;
#pragma unroll
    for (int q = 0; q < K; q++) b = insert0_32(b, g[q]);
    double2 v[1 << K];
#pragma unroll
    for (int j = 0; j < (1 << K); j++) {
      uint32_t o = b;
#pragma unroll
      for (int q = 0; q < K; q++)
        if ((j >> q) & 1) o |= 1u << g[q];
      v[j] = s[sw(o)];
    }
#pragma unroll
    for (int q = 0; q < K; q++)
#pragma unroll
      for (int j = 0; j < (1 << K); j++)
        if (!((j >> q) & 1)) rx_pair(v[j], v[j | (1 << q)], cb, sb);
#pragma unroll
    for (int j = 0; j < (1 << K); j++) {
      uint32_t o = b;
#pragma unroll
      for (int q = 0; q < K; q++)
        if ((j >> q) & 1) o |= 1u << g[q];
      s[sw(o)] = v[j];
    }
  }
}

// Bits per group: three at 256 threads per CTA, so that the registers of three
// resident CTAs (what 12 qubits of shared memory allow) hold a group's 8 amplitudes
// without spills; four at 128 and 512 threads.
template <int NT>
constexpr int rx_group_bits() { return NT == 256 ? 3 : 4; }
template <int NT>
constexpr int chip_min_blocks() { return NT == 512 ? 1 : 3; }

// Rx(2 beta) on all m bits, in ascending order, a group of bits per shared-memory
// round trip.
template <int NT>
__device__ void rx_bits(double2* s, int m, double cb, double sb) {
  constexpr int KM = rx_group_bits<NT>();
  for (int b = 0; b < m; b += KM) {
    const uint32_t gp = 0x03020100u + 0x01010101u * (uint32_t)b;
    const int k = min(KM, m - b);
    __syncthreads();
    if constexpr (KM == 4) {
      if (k == 4) { rx_group<NT, 4>(s, m, gp, cb, sb); continue; }
    }
    switch (k) {
      case 3: rx_group<NT, 3>(s, m, gp, cb, sb); break;
      case 2: rx_group<NT, 2>(s, m, gp, cb, sb); break;
      default: rx_group<NT, 1>(s, m, gp, cb, sb); break;
    }
  }
}

// Shared memory of a CTA: state, phase table, edge masks, sums, cut(x) per amplitude.
constexpr size_t kChipFixed = 16 * (KQ_MAX_EDGES + 1) + 4 * KQ_MAX_EDGES + 8 * 32;
static_assert(kChipFixed % 16 == 0, "cut bytes 16-byte aligned");
size_t chip_smem(int bits) { return kChipFixed + (size_t(17) << bits) + 16; }

// One instance a CTA at a time, 2^n amplitudes in shared memory.  Bound: latency -- a
// layer is n / 3 round trips and as many barriers.  The wide kernel's tiles take every
// layout move of 12 bits and a launch for their tables, whatever the instance's
// width: 2000 instances of 2 qubits and 6 layers 365 us on them, 48 here; 500 of 12
// qubits and 3 layers, which fill a tile, 93 and 69.
template <int NT>
__global__ void __launch_bounds__(NT, chip_min_blocks<NT>()) k_qaoa_chip(QArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* s = reinterpret_cast<double2*>(smraw);
  double2* tab = s + (1u << a.chip_bits);
  uint32_t* em = reinterpret_cast<uint32_t*>(tab + KQ_MAX_EDGES + 1);
  double* red = reinterpret_cast<double*>(em + KQ_MAX_EDGES);
  uint8_t* cutb = reinterpret_cast<uint8_t*>(red + 32);
  __shared__ int item_sh;
  for (;;) {
    if (threadIdx.x == 0) item_sh = (int)atomicAdd(a.next + 1, 1u);
    __syncthreads();
    const int it = item_sh;
    __syncthreads();
    if (it >= a.nchip) break;
    const int i = a.chip[it];
    const QInst I = a.inst[i];
    if (I.p == 0) {  // <C> of the uniform state, whatever n
      if (threadIdx.x == 0) a.out[i] = 0.5 * I.ne;
      continue;
    }
    for (int e = threadIdx.x; e < I.ne; e += NT) em[e] = a.emask[I.edge_off + e];
    const int n = I.n;
    const uint32_t N = 1u << n;
    const double amp0 = 1.0 / sqrt((double)N);
    __syncthreads();  // edge masks in
    // cut(x) depends on x only: computed once, read by every layer and <C>
    for (uint32_t x = threadIdx.x; x < N; x += NT) {
      s[sw(x)] = make_double2(amp0, 0.0);
      cutb[x] = (uint8_t)cut_of(x, em, I.ne);
    }
    for (int l = 0; l < I.p; l++) {
      const double gamma = a.gamma[(int64_t)i * I.p + l];
      __syncthreads();
      for (int c = threadIdx.x; c <= I.ne; c += NT) {
        double sn, co;
        sincos(-gamma * (double)(I.ne - 2 * c), &sn, &co);
        tab[c] = make_double2(co, sn);
      }
      __syncthreads();
      for (uint32_t x = threadIdx.x; x < N; x += NT) {
        const double2 ph = tab[cutb[x]];
        const double2 v = s[sw(x)];
        s[sw(x)] = make_double2(fma(ph.x, v.x, -ph.y * v.y), fma(ph.x, v.y, ph.y * v.x));
      }
      double sb, cb;
      sincos(a.beta[(int64_t)i * I.p + l], &sb, &cb);
      rx_bits<NT>(s, n, cb, sb);
    }
    __syncthreads();
    // over the norm: n p rotations with one rounded cosine and sine let it drift (9
    // qubits, 4 layers: <C> off by 1.9e-14, over the norm by 1.6e-15)
    double acc = 0.0, nrm = 0.0;
    for (uint32_t x = threadIdx.x; x < N; x += NT) {
      const double2 v = s[sw(x)];
      const double q = v.x * v.x + v.y * v.y;
      nrm += q;
      acc = fma(q, (double)cutb[x], acc);
    }
    acc = block_sum<NT>(acc, red);
    __syncthreads();
    nrm = block_sum<NT>(nrm, red);
    if (threadIdx.x == 0) a.out[i] = acc / nrm;
    __syncthreads();
  }
}

// Test hook (ket_debug_batch_hook): leave one work item out and
// shorten the waits, so that the tiles depending on it time out.
int g_drop_item = -1;
uint32_t g_spin_limit = 1u << 24;

}  // namespace
}  // namespace ket

using namespace ket;

// Launch the wide instances' tables, their persistent kernel (NT threads per CTA, every
// CTA resident at once) and its fixed-order reduction, then the instances that fit
// the chip, captured in a CUDA graph when use_graph is set.
template <int NT, int T>
static cudaError_t run_batch(ket_ctx* c, const QArgs& a, int p, int ninst, int use_graph) {
  const size_t smem = (sizeof(double2) << T) + sizeof(QShared), smem_chip = chip_smem(a.chip_bits);
  // the shared-memory limit is a per-device attribute of the kernels
  static std::atomic<uint64_t> attr_set{0};
  const uint64_t bit = uint64_t(1) << (c->device & 63);
  if (!(attr_set.load() & bit)) {
    cudaError_t e = cudaFuncSetAttribute(k_batch_qaoa<NT, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_qaoa_chip<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chip_smem(12));
    if (e != cudaSuccess) return e;
    attr_set.fetch_or(bit);
  }
  int per_sm = 0, grid = 0, grid_chip = 0;
  if (a.nitems) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_qaoa<NT, T>, NT, smem);
    grid = num_sms() * std::max(1, per_sm);
  }
  if (a.nchip) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_qaoa_chip<NT>, NT, smem_chip);
    grid_chip = std::min(a.nchip, num_sms() * std::max(1, per_sm));
  }
  auto record = [&]() -> cudaError_t {
    cudaMemsetAsync(a.next, 0, 4 * (a.nitems ? (size_t)ninst + 2 : 2), c->stream);
    if (a.nitems) {
      k_qaoa_tables<<<(unsigned)ninst * p, 64, 0, c->stream>>>(a, p);
      k_batch_qaoa<NT, T><<<grid, NT, smem, c->stream>>>(a);
      k_qaoa_reduce<<<(ninst + 3) / 4, 128, 0, c->stream>>>(a.inst, ninst, a.part, a.out);
    }
    if (a.nchip) k_qaoa_chip<NT><<<grid_chip, NT, smem_chip, c->stream>>>(a);
    return cudaGetLastError();
  };
  if (!use_graph) return record();
  // A batch of the same shape reuses the executable graph: its inputs were
  // re-uploaded to the same addresses, so only a changed launch (sizes,
  // buffers, shape) is captured and instantiated again.
  uint64_t key = 1469598103934665603ull;
  auto mix = [&](const void* p, size_t nb) {
    for (size_t i = 0; i < nb; i++) key = (key ^ ((const unsigned char*)p)[i]) * 1099511628211ull;
  };
  const int nt = NT, tile = T;
  mix(&a, sizeof(a));
  mix(&tile, sizeof(tile));
  mix(&p, sizeof(p));
  mix(&ninst, sizeof(ninst));
  mix(&nt, sizeof(nt));
  mix(&grid, sizeof(grid));
  mix(&grid_chip, sizeof(grid_chip));
  if (c->graph_exec && c->graph_key == key) return cudaGraphLaunch(c->graph_exec, c->stream);
  cudaGraph_t graph;
  cudaError_t e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  e = record();
  cudaError_t e2 = cudaStreamEndCapture(c->stream, &graph);
  if (e != cudaSuccess) return e;
  if (e2 != cudaSuccess) return e2;
  if (c->graph_exec) { cudaGraphExecDestroy(c->graph_exec); c->graph_exec = nullptr; }
  c->graph_key = 0;
  e = cudaGraphInstantiate(&c->graph_exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) return e;
  c->graph_key = key;
  return cudaGraphLaunch(c->graph_exec, c->stream);
}

extern "C" int ket_batch_config(ket_ctx* c, int block_threads, int tile_bits) {
  if (!c) return fail(KET_ERR_TYPE, "null context");
  if (block_threads == 0) block_threads = 256;
  if (tile_bits == 0) tile_bits = 12;
  if (block_threads != 128 && block_threads != 256 && block_threads != 512)
    return fail(KET_ERR_TYPE, "block_threads must be 128, 256 or 512");
  if (tile_bits != 11 && tile_bits != 12) return fail(KET_ERR_TYPE, "tile_bits must be 11 or 12");
  c->batch_threads = block_threads;
  c->batch_tile = tile_bits;
  return KET_OK;
}

extern "C" int ket_debug_batch_hook(int drop_item, uint32_t spin_limit) {
  g_drop_item = drop_item;
  g_spin_limit = spin_limit ? spin_limit : (1u << 24);
  return KET_OK;
}

extern "C" int ket_batch_qaoa(ket_ctx* c, int ninst, const int* n, const int* ne, const int64_t* eoff,
                              const int* edges, int p, const double* gamma, const double* beta, int use_graph,
                              double* out) {
  if (!c || (ninst > 0 && (!n || !ne || !eoff || !edges || !gamma || !beta || !out)))
    return fail(KET_ERR_TYPE, "null argument");
  if (ninst < 0 || p < 0 || p > KQ_MAX_P) return fail(KET_ERR_TYPE, "bad instance count or layer count");
  if (ninst == 0) return KET_OK;
  cudaSetDevice(c->device);
  const int T = c->batch_tile;
  std::vector<QInst> inst(ninst, QInst{});
  std::vector<uint32_t> masks;
  int64_t work = 0, parts = 0, phases = 0;
  int chip_bits = 0;
  for (int i = 0; i < ninst; i++) {
    if (n[i] < 1 || n[i] > 30) return fail(KET_ERR_RANGE, "instance qubit count out of range (1..30)");
    if (ne[i] < 0 || ne[i] > KQ_MAX_EDGES) return fail(KET_ERR_TYPE, "instance edge count out of range (0..64)");
    if (n[i] > T && n[i] - T > T)
      return fail(KET_ERR_UNSUPPORTED, "instance wider than twice the tile width (" + std::to_string(2 * T) + " qubits)");
    QInst& I = inst[i];
    I.n = n[i];
    I.ne = ne[i];
    I.p = p;
    I.edge_off = (int64_t)masks.size();
    for (int e = 0; e < ne[i]; e++) {
      int u = edges[2 * (eoff[i] + e)], v = edges[2 * (eoff[i] + e) + 1];
      if (u < 0 || v < 0 || u >= n[i] || v >= n[i]) return fail(KET_ERR_RANGE, "edge endpoint out of range");
      if (u == v) return fail(KET_ERR_TYPE, "self-loop edge");
      masks.push_back((uint32_t(1) << u) | (uint32_t(1) << v));
    }
    if (I.n <= T || p == 0) {
      chip_bits = std::max(chip_bits, p > 0 ? I.n : 0);
      continue;
    }
    std::vector<uint32_t> em(masks.begin() + I.edge_off, masks.end());
    std::sort(em.begin(), em.end());
    I.multi = std::adjacent_find(em.begin(), em.end()) != em.end();
    I.tab_off = phases;
    phases += (int64_t)p * (ne[i] + 1);
    I.ntiles = 1 << (I.n - T);
    I.state = work;
    work += int64_t(1) << I.n;
    I.part_off = parts;
    parts += I.ntiles;
  }
  // Work order: wide instances (largest first), then those that fit the chip.
  std::vector<int> order(ninst);
  for (int i = 0; i < ninst; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return inst[x].n > inst[y].n; });
  std::vector<QRun> runs;
  int64_t nitems = 0;
  auto add = [&](int i, int pass) {
    runs.push_back(QRun{(int)nitems, i, pass, 0});
    nitems += inst[i].ntiles;
  };
  // Wide instances go in sets whose states share the 126 MB L2, all passes of a set
  // before the next, the set's instances in turn so that a tile rarely waits (512
  // instances of up to 64 MB: 15.9 ms in one set, 15.3 in sets of 80 MB, 15.5 and
  // 15.7 of 70 and 112 MB).
  constexpr int64_t kSetBytes = int64_t(80) << 20;
  std::vector<int> wide, chip;
  for (int i : order) (inst[i].ntiles ? wide : chip).push_back(i);
  while (!wide.empty()) {
    std::vector<int> set, rest;
    int64_t bytes = 0;
    for (int i : wide) {
      const int64_t b = int64_t(16) << inst[i].n;
      if (set.empty() || bytes + b <= kSetBytes) { set.push_back(i); bytes += b; }
      else rest.push_back(i);
    }
    for (int k = 0; k <= p; k++)
      for (int i : set) add(i, k);
    wide.swap(rest);
  }
  if (nitems > INT32_MAX / 2) return fail(KET_ERR_UNSUPPORTED, "too many tiles in a batch");
  runs.push_back(QRun{INT32_MAX, 0, 0, 0});  // end marks
  runs.push_back(QRun{INT32_MAX, 0, 0, 0});
  // device buffers in the second scratch pool
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  size_t off_inst = 0, off_runs = al(sizeof(QInst) * ninst), off_mask = off_runs + al(sizeof(QRun) * runs.size());
  size_t off_chip = off_mask + al(4 * std::max<size_t>(masks.size(), 1));
  size_t off_g = off_chip + al(4 * chip.size());
  size_t off_b = off_g + al(8 * (size_t)ninst * p + 8);
  size_t off_tan = off_b + al(8 * (size_t)ninst * p + 8);
  size_t off_tab = off_tan + al(8 * std::max<size_t>((size_t)ninst * p, 1));
  size_t off_part = off_tab + al(16 * std::max<size_t>((size_t)phases, 1));
  size_t off_out = off_part + al(16 * std::max<size_t>((size_t)parts, 1));
  size_t off_cnt = off_out + al(8 * (size_t)ninst);
  size_t off_work = off_cnt + al(4 * ((size_t)ninst + 2));
  size_t total = off_work + al(16 * (size_t)work) + 256;
  if (c->scratch2_bytes < total) {
    int rc = ctx_wait(c);
    if (rc) return rc;
    if (c->graph_exec) { cudaGraphExecDestroy(c->graph_exec); c->graph_exec = nullptr; }
    c->graph_key = 0;
    if (c->scratch2) cudaFree(c->scratch2);
    c->scratch2 = nullptr;
    c->scratch2_bytes = 0;
    rc = dev_alloc(&c->scratch2, total);
    if (rc) return rc;
    c->scratch2_bytes = total;
  }
  char* base = (char*)c->scratch2;
  std::vector<double> gv(gamma, gamma + (size_t)ninst * p), bv(beta, beta + (size_t)ninst * p);
  cudaMemcpyAsync(base + off_inst, inst.data(), sizeof(QInst) * ninst, cudaMemcpyHostToDevice, c->stream);
  if (nitems)
    cudaMemcpyAsync(base + off_runs, runs.data(), sizeof(QRun) * runs.size(), cudaMemcpyHostToDevice, c->stream);
  if (!chip.empty())
    cudaMemcpyAsync(base + off_chip, chip.data(), 4 * chip.size(), cudaMemcpyHostToDevice, c->stream);
  if (!masks.empty()) cudaMemcpyAsync(base + off_mask, masks.data(), 4 * masks.size(), cudaMemcpyHostToDevice, c->stream);
  if (p > 0) {
    cudaMemcpyAsync(base + off_g, gv.data(), 8 * gv.size(), cudaMemcpyHostToDevice, c->stream);
    cudaMemcpyAsync(base + off_b, bv.data(), 8 * bv.size(), cudaMemcpyHostToDevice, c->stream);
  }
  c->h2d_bytes += sizeof(QInst) * ninst + (nitems ? sizeof(QRun) * runs.size() : 0) + 4 * chip.size() + 4 * masks.size() +
                  16 * gv.size();
  QArgs a;
  memset(&a, 0, sizeof(a));  // its bytes are the graph's key
  a.inst = (const QInst*)(base + off_inst);
  a.runs = (const QRun*)(base + off_runs);
  a.chip = (const int*)(base + off_chip);
  a.emask = (const uint32_t*)(base + off_mask);
  a.gamma = (const double*)(base + off_g);
  a.beta = (const double*)(base + off_b);
  a.tan = (double*)(base + off_tan);
  a.tab = (double2*)(base + off_tab);
  a.part = (double2*)(base + off_part);
  a.out = (double*)(base + off_out);
  a.next = (unsigned int*)(base + off_cnt);
  a.done = a.next + 2;
  a.status = c->d_status;
  a.spin_limit = g_spin_limit;
  a.work = (double2*)(base + off_work);
  a.nitems = (int)nitems;
  a.nchip = (int)chip.size();
  a.chip_bits = chip_bits;
  a.drop = g_drop_item;
  prof_begin(c);
  cudaError_t e;
  switch (c->batch_threads + T) {
    case 128 + 11: e = run_batch<128, 11>(c, a, p, ninst, use_graph); break;
    case 256 + 11: e = run_batch<256, 11>(c, a, p, ninst, use_graph); break;
    case 512 + 11: e = run_batch<512, 11>(c, a, p, ninst, use_graph); break;
    case 128 + 12: e = run_batch<128, 12>(c, a, p, ninst, use_graph); break;
    case 512 + 12: e = run_batch<512, 12>(c, a, p, ninst, use_graph); break;
    default: e = run_batch<256, 12>(c, a, p, ninst, use_graph); break;
  }
  prof_end(c, PK_BATCH);
  c->launches += (nitems ? 3 : 0) + (chip.empty() ? 0 : 1) - 1;  // (prof_end counted one)
  if (e != cudaSuccess) return cuda_fail(e, "batch launch");
  e = cudaMemcpyAsync(out, a.out, 8 * (size_t)ninst, cudaMemcpyDeviceToHost, c->stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(out)");
  c->d2h_bytes += 8 * (size_t)ninst;
  return ctx_finish(c);
}
