// small.cu -- circuits on complex128 states of up to 20 qubits in one launch
// (ket_apply_ops' automatic path there).  complex64 states keep the tiled passes:
// another order of the FP32 roundings would show in what is read from them.
//
// A pass of the register-tiled kernels costs a launch, and their planning (tile
// choice, layouts) a millisecond of host time for a few hundred gates, whatever the
// state's size; a 16-qubit state then runs on 16 of 148 SMs, one gate at a time.
// Here the whole circuit is one cooperative launch over a state that stays in
// the L2:
//   * CNOTs, swaps and X gates are relabellings over GF(2) of the whole state
//     (rounds.h) and move nothing; the last pass stores the amplitudes in order;
//   * a pass takes the next gates, in program order, while their pair masks span at
//     most 10 to 12 dimensions with the two lowest index bits (so that memory is read in
//     runs of four).  A CTA holds one coset of the span in shared memory and runs
//     the pass's gates there in rounds of up to 16 on amplitudes in registers;
//     diagonals take no dimension, and phases of one target under controls that a
//     thread's amplitudes share (a Fourier transform's) are gathered into one;
//   * between passes the grid meets at a barrier (a bounded wait).
// States of up to 12 qubits are one CTA, which needs no barrier.  Gates keep their
// order, so pruning after each (accumulate(), statevector.ts:19-27) is the
// reference's.  The order of the FMAs differs from the tiled passes', so the two
// agree to rounding.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "fused_ops.cuh"
#include "launch.h"
#include "rounds.h"

namespace ket {
namespace {

constexpr int kTileBits = 12;
constexpr int kMaxRounds = 64, kMaxGates = 64, kMaxSlots = 128;  // of one pass, in shared memory
constexpr uint32_t kSpinLimit = 1u << 22;  // polls of the barrier: seconds

// Test hook (ket_debug_rounds_hook): the co-resident CTAs a launch may count on (0:
// what the device holds) and the barrier's polls.
int g_max_ctas = 0;
uint32_t g_spin_limit = kSpinLimit;

enum : uint8_t { FM_GEN = 0, FM_REAL = 1, FM_RX = 2, FM_DIAG = 3, FM_DIAG2 = 4, FM_X = 5, FM_PHASE = 6 };
enum : uint8_t { GF_PRUNE = 1, GF_CHAIN = 2 };  // CHAIN: the next gate is a phase of the same target, too

// FM_PHASE: diag(1, p) whose controls are the same for a thread's 16 amplitudes.
struct __align__(16) RGate {
  uint8_t form, bit, nc, flags;
  uint16_t r, slot;          // target functional (tile bits); matrix, in 64-byte slots of the pass
  uint32_t flip;             // bit 0 target, 1 and 2 controls, 3 second target: the coset base's parity
  uint16_t rc[2];
  // (the loop over a round's gates reads the 16 bytes above first)
  uint16_t r2;
  uint8_t cj[2], rj[2];
  uint16_t cflip;            // constant part of flip (X gates so far)
  uint32_t g, gc[2], g2;     // the functionals on the whole index
  uint32_t pad;
};
static_assert(sizeof(RGate) == 48, "three 16-byte reads");

struct __align__(16) RRound {
  uint16_t slot[16];
  uint16_t rd[4];
  uint8_t piv[4];
  uint8_t k, dense;
  uint16_t ngates;
  int32_t gate0, pad[3];
};
static_assert(sizeof(RRound) == 64, "copied as words");

struct __align__(16) RPass {
  int32_t round0, nrounds, gate0, ngates, slot0, nslots;
  uint32_t basis[kTileBits];   // index mask of each tile bit
  uint8_t free[12];            // index bits of the tile number
  int32_t pad;
};
static_assert(sizeof(RPass) == 96, "copied as words");

// A pass's records in shared memory.
struct __align__(16) Records {
  double2 mats[4 * kMaxSlots];
  RRound rounds[kMaxRounds];
  RGate gates[kMaxGates];
  RPass pass;
};

struct RArgs {
  double2* amp;
  const RPass* passes;
  const RRound* rounds;
  const RGate* gates;
  const double2* mats;         // by 64-byte slots
  unsigned int* arrived;       // barrier
  int* status;
  int npasses, n, d;           // d: tile bits
  int permute;                 // the relabelling is not the identity
  uint32_t spin_limit;
  uint32_t beta;               // physical index of logical index l: A l ^ beta
  uint32_t acol[20];
  // (in memory: a launch carries what each of its blocks reads)
  const uint32_t* inverse;     // logical index of physical index p: B p ^ lbeta; lbeta, then B's columns
};

__device__ __forceinline__ uint32_t par(uint32_t x) { return (uint32_t)__popc(x) & 1u; }

__device__ __forceinline__ uint32_t pattern(uint32_t j4) {  // bit j = parity(j & j4), j < 16
  return (j4 & 1 ? 0xaaaau : 0u) ^ (j4 & 2 ? 0xccccu : 0u) ^ (j4 & 4 ? 0xf0f0u : 0u) ^ (j4 & 8 ? 0xff00u : 0u);
}
__device__ __forceinline__ uint32_t controls_ok(const RGate& g, uint32_t base) {
  uint32_t ok = 0xffffu;
  for (int c = 0; c < g.nc; c++)
    ok &= pattern(g.cj[c]) ^ ((par(base & g.rc[c]) ^ (g.flip >> (1 + c))) & 1u ? 0xffffu : 0u);
  return ok;
}

template <int K, int I, int FORM>
__device__ __forceinline__ void pair_gate(cpx<double>* v, const double2* M, bool role, bool prune, bool ctl, uint32_t ok) {
  constexpr int NS = 1 << K;
  double m[8];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const double2 t = M[role ? e ^ 3 : e];
    m[2 * e] = t.x;
    m[2 * e + 1] = t.y;
  }
  if (!ctl) mat1_reg<double, I, FORM, NS>(v, m, full_mask<NS>());
  else mat1_reg<double, I, FORM, NS>(v, m, ok & full_mask<NS>());
  if (prune) prune_slots<double, NS>(v, 1e-14, 1e-7);
}
template <int K, int I>
__device__ __forceinline__ void pair_x(cpx<double>* v, uint32_t ok) {
#pragma unroll
  for (int j = 0; j < (1 << K); j++)
    if (!(j & (1 << I)) && ((ok >> j) & 1)) swap_c(v[j], v[j | 1 << I]);
}

template <int K>
__device__ __forceinline__ void run_round(double2* s, const RRound& Q, const RGate* gates,
                                          const double2* mats, int d) {
  constexpr int NS = 1 << K;
  const uint32_t u = threadIdx.x;
  if (u >= 1u << (d - K)) return;
  uint32_t base = u;
#pragma unroll
  for (int i = 0; i < K; i++) base = insert0_32(base, Q.piv[i]);
  const uint32_t sb = round_slot(base);
  cpx<double> v[NS];
  RoundSlots slots;
  slots.read(Q.slot);
#pragma unroll
  for (int j = 0; j < NS; j++) v[j] = ld_amp<double>(s + (sb ^ slots(j)));
  // cosets of zeros stay zeros (most of a state in its first gates)
  if (!__any_sync(__activemask(), !all_zero<double, NS>(v))) return;
  uint4 next = *reinterpret_cast<const uint4*>(gates);
  double fr = 1.0, fi = 0.0;  // phases of one target, gathered
  for (int k = 0; k < Q.ngates; k++) {
    const uint4 q = next;
    const RGate& g = gates[k];
    if (k + 1 < Q.ngates) next = *reinterpret_cast<const uint4*>(gates + k + 1);
    const int form = q.x & 0xff, bit = (q.x >> 8) & 0xff, nc = (q.x >> 16) & 0xff;
    const uint32_t flags = q.x >> 24;
    const double2* M = mats + 4 * (q.y >> 16);
    const uint32_t role = (par(base & q.y & 0xffffu) ^ q.z) & 1u;
    if (form == FM_PHASE) {
      uint32_t on = nc > 0 ? par(base & q.w & 0xffffu) ^ (q.z >> 1) : 1u;
      if (nc > 1) on &= par(base & (q.w >> 16)) ^ (q.z >> 2);
      if (on & 1u) {
        const double2 e = M[3];
        const double x = fr;
        fr = fma(e.x, x, -e.y * fi);
        fi = fma(e.x, fi, e.y * x);
      }
      if (!(flags & GF_CHAIN)) {
        const uint32_t p0 = pattern(g.rj[0]) ^ (role ? 0xffffu : 0u);
#pragma unroll
        for (int j = 0; j < NS; j++)
          if ((p0 >> j) & 1) cmul_in<double>(v[j], fr, fi);
        fr = 1.0;
        fi = 0.0;
      }
      continue;
    }
    const bool ctl = nc != 0;
    const uint32_t ok = ctl ? controls_ok(g, base) : 0xffffu;
    if (form == FM_DIAG || form == FM_DIAG2) {
      // entry by each amplitude's target bits, read from shared memory
      const uint32_t p0 = pattern(g.rj[0]) ^ (role ? 0xffffu : 0u);
      const uint32_t p1 = form == FM_DIAG2 ? pattern(g.rj[1]) ^ ((par(base & g.r2) ^ (q.z >> 3)) & 1u ? 0xffffu : 0u) : p0;
#pragma unroll
      for (int j = 0; j < NS; j++) {
        const double2 e = M[2 * ((p0 >> j) & 1) + ((p1 >> j) & 1)];
        if ((ok >> j) & 1) cmul_in<double>(v[j], e.x, e.y);
      }
      continue;
    }
    const bool pr = flags & GF_PRUNE;
    switch (4 * form + bit) {
#define KET_BIT(F, I) \
  case 4 * F + I: if constexpr (I < K) pair_gate<K, I, F>(v, M, role, pr, ctl, ok); break;
#define KET_FORM(F) KET_BIT(F, 0) KET_BIT(F, 1) KET_BIT(F, 2) KET_BIT(F, 3)
      KET_FORM(0) KET_FORM(1) KET_FORM(2)
#undef KET_FORM
#undef KET_BIT
#define KET_BIT(I) \
  case 4 * FM_X + I: if constexpr (I < K) pair_x<K, I>(v, ok); break;
      KET_BIT(0) KET_BIT(1) KET_BIT(2) KET_BIT(3)
#undef KET_BIT
    }
  }
  slots.read(Q.slot);
#pragma unroll
  for (int j = 0; j < NS; j++) st_amp<double>(s + (sb ^ slots(j)), v[j]);
}

// A dense 2^K x 2^K on the K masks of its round, the products of a row added in
// ascending column order in FP64.
template <int K>
__device__ __forceinline__ void run_dense(double2* s, const RRound& Q, const RGate& g, const double2* mats,
                                          int d) {
  constexpr int D = 1 << K;
  const double2* M = mats + 4 * g.slot;
  for (uint32_t u = threadIdx.x; u < 1u << (d - K); u += blockDim.x) {
    uint32_t base = u;
#pragma unroll
    for (int i = 0; i < K; i++) base = insert0_32(base, Q.piv[i]);
    if (g.nc && !(controls_ok(g, base) & 1)) continue;
    uint32_t l0 = 0;  // local index of the coset's base
#pragma unroll
    for (int i = 0; i < K; i++) l0 |= par(base & Q.rd[i]) << i;
    l0 ^= g.cj[1];    // (a dense gate keeps the base's parities here)
    const uint32_t sb = round_slot(base);
    double xr[D], xi[D];
#pragma unroll
    for (int c = 0; c < D; c++) {
      const cpx<double> x = ld_amp<double>(s + (sb ^ Q.slot[c ^ l0]));
      xr[c] = x.re;
      xi[c] = x.im;
    }
    for (int r = 0; r < D; r++) {
      double sr = 0.0, si = 0.0;
#pragma unroll
      for (int c = 0; c < D; c++) {
        const double2 m = M[r * D + c];
        sr = fma(m.x, xr[c], fma(-m.y, xi[c], sr));
        si = fma(m.x, xi[c], fma(m.y, xr[c], si));
      }
      cpx<double> y = {sr, si};
      if (g.flags & GF_PRUNE) prune_amp(y, 1e-14, 1e-7);
      st_amp<double>(s + (sb ^ Q.slot[r ^ l0]), y);
    }
  }
}

__device__ __forceinline__ void copy_words(void* dst, const void* src, int bytes) {
  for (int i = threadIdx.x; i < bytes / 16; i += blockDim.x)
    static_cast<uint4*>(dst)[i] = __ldg(static_cast<const uint4*>(src) + i);
}

// The grid's barrier in two halves: a CTA's loads and stores before arrive() are done
// for every CTA after wait().  (The grid is co-resident.)
__device__ __forceinline__ void arrive(const RArgs& a) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(a.arrived, 1u);
  }
}
// False: the wait ran out (status set).
__device__ __forceinline__ bool wait(const RArgs& a, unsigned int target, int* failed) {
  if (threadIdx.x == 0) {
    volatile unsigned int* p = a.arrived;
    uint32_t spins = 0;
    int bad = 0;
    while (*p < target) {
      if (++spins > a.spin_limit) {
        atomicExch(a.status, (int)KET_ERR_TIMEOUT);
        bad = 1;
        break;
      }
    }
    __threadfence();
    *failed = bad;
  }
  __syncthreads();
  return *failed == 0;
}

// 2^K amplitudes a thread: 8, or 16 at 20 qubits, where 256 CTAs of 2^12 amplitudes
// have to be resident two an SM.  (16 at 16 qubits: 290 us against 221; a gate's
// straight-line code is half as long and twice the warps hide its latency.)
// Bound: latency -- of a gate (about 0.4 us of dependent reads, FP64 chain and
// pruning screen) and of a pass (about 3 us of barrier, loads and stores); issue slots
// are 13 to 24% taken.  20 brickwork layers of 16 qubits: 487 us in 20 launches and 770 of
// planning before, 210 and 90 now; QFT of 20 qubits 142 and 220, 127 and 75 now.
// ALONE: one CTA, without the grid's code (10 qubits 48.3 -> 46.6 us).
template <int K, bool ALONE>
__global__ void __launch_bounds__(K == 4 ? 256 : 512, K == 4 ? 2 : 1) k_rounds(const __grid_constant__ RArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* s = reinterpret_cast<double2*>(smraw);
  Records* rec = reinterpret_cast<Records*>(smraw + (sizeof(double2) << a.d));
  __shared__ int failed;
  double2* amp = a.amp;
  const uint32_t t = threadIdx.x, T = 1u << a.d, nt = blockDim.x, lnt = 31 - __clz(nt);
  const uint64_t N = uint64_t(1) << a.n;
  unsigned int met = 0;
  // the records of a pass, two passes' at a time: read before the barrier the pass
  // waits at
  auto fetch = [&](int pass) {
    const RPass& P = a.passes[pass];
    Records& r = rec[pass & 1];
    copy_words(r.rounds, a.rounds + P.round0, P.nrounds * sizeof(RRound));
    copy_words(r.gates, a.gates + P.gate0, P.ngates * sizeof(RGate));
    copy_words(r.mats, a.mats + 4 * P.slot0, P.nslots * 64);
    copy_words(&r.pass, &P, sizeof(RPass));
  };
  fetch(0);
  __syncthreads();
  for (int pass = 0; pass < a.npasses; pass++) {
    const Records& W = rec[pass & 1];
    const RPass& P = W.pass;
    uint32_t cbase = 0, tl = 0;
    for (int b = 0; b < a.n - a.d; b++) cbase |= ((blockIdx.x >> b) & 1u) << P.free[b];
    for (uint32_t b = 0; b < lnt; b++)
      if ((t >> b) & 1) tl ^= P.basis[b];
    uint32_t hi[K];  // masks of register bits
#pragma unroll
    for (int b = 0; b < K; b++) hi[b] = lnt + b < (uint32_t)a.d ? P.basis[lnt + b] : 0u;
    auto index = [&](int j) {  // of tile element t + nt j
      uint32_t p = cbase ^ tl;
#pragma unroll
      for (int b = 0; b < K; b++)
        if ((j >> b) & 1) p ^= hi[b];
      return p;
    };
    double2 v[1 << K];
#pragma unroll
    for (int j = 0; j < (1 << K); j++) {
      const uint32_t p = index(j);
      v[j] = make_double2(0.0, 0.0);
      if (t + nt * j < T && p < N) v[j] = __ldcg(amp + p);
    }
    for (int k = t; k < P.ngates; k += nt) {
      RGate& g = rec[pass & 1].gates[k];
      g.flip = (par(cbase & g.g) | par(cbase & g.gc[0]) << 1 | par(cbase & g.gc[1]) << 2 | par(cbase & g.g2) << 3) ^ g.cflip;
      if (g.form == FM_GEN && g.bit >= 4) {
        // dense: g, gc[1], g2 and pad are the functionals of local bits 0..3, and
        // cj[1] keeps their parities
        g.cj[1] = (uint8_t)((par(cbase & g.g) | par(cbase & g.gc[1]) << 1 | par(cbase & g.g2) << 2 | par(cbase & g.pad) << 3) ^
                            (g.cflip >> 8));
        g.flip = (par(cbase & g.gc[0]) << 1) ^ (g.cflip & 2u);
      }
    }
#pragma unroll
    for (int j = 0; j < (1 << K); j++)
      if (t + nt * j < T) s[round_slot(t + nt * j)] = v[j];
    const bool last = pass + 1 == a.npasses, scatter = !ALONE && last && a.permute;
    if (scatter) arrive(a);  // (this CTA's tile is read)
    for (int r = 0; r < P.nrounds; r++) {
      __syncthreads();
      const RRound& Q = W.rounds[r];
      const RGate* G = W.gates + Q.gate0;
      if (!Q.dense) {
        run_round<K>(s, Q, G, W.mats, a.d);
      } else {
        switch (Q.k) {
          case 2: run_dense<2>(s, Q, *G, W.mats, a.d); break;
          case 3: run_dense<3>(s, Q, *G, W.mats, a.d); break;
          default: run_dense<4>(s, Q, *G, W.mats, a.d); break;
        }
      }
    }
    __syncthreads();
    if (ALONE && last) {
      // one tile, whose index is the physical index: written in logical order
      for (uint32_t l = t; l < N; l += nt) {
        uint32_t p = a.beta;
        for (int b = 0; b < a.n; b++)
          if ((l >> b) & 1) p ^= a.acol[b];
        amp[l] = s[round_slot(p)];
      }
      return;
    }
    if (scatter) {
      // in logical order, over other CTAs' tiles: once every CTA has read its own
      met += gridDim.x;
      if (!wait(a, met, &failed)) return;
      auto logical = [&](uint32_t p) {
        uint32_t l = 0;
        for (int b = 0; b < a.n; b++)
          if ((p >> b) & 1) l ^= __ldg(a.inverse + 1 + b);
        return l;
      };
      const uint32_t l0 = logical(cbase ^ tl) ^ __ldg(a.inverse);
      uint32_t lhi[K];
#pragma unroll
      for (int b = 0; b < K; b++) lhi[b] = logical(hi[b]);
#pragma unroll
      for (int j = 0; j < (1 << K); j++) {
        uint32_t l = l0;
#pragma unroll
        for (int b = 0; b < K; b++)
          if ((j >> b) & 1) l ^= lhi[b];
        if (t + nt * j < T) amp[l] = s[round_slot(t + nt * j)];
      }
      return;
    }
#pragma unroll
    for (int j = 0; j < (1 << K); j++) {
      const uint32_t p = index(j);
      if (t + nt * j < T && p < N) amp[p] = s[round_slot(t + nt * j)];
    }
    if (last) return;
    if constexpr (ALONE) {
      fetch(pass + 1);
      __syncthreads();
      continue;
    }
    arrive(a);
    fetch(pass + 1);
    met += gridDim.x;
    if (!wait(a, met, &failed)) return;
  }
}

// ---------------------------------------------------------------- planning

// A gate on the relabelled index.
struct SGate {
  uint8_t form = 0, nc = 0, k = 0;
  bool prune = false;
  uint32_t m[4] = {}, r[4] = {};   // pair masks and functionals (a dense gate's by local bit)
  uint32_t rc[2] = {};
  uint32_t flip = 0;               // constant parities, as RGate::cflip
  const cd* mat = nullptr;         // its matrix: 2 or 4 diagonal entries, else 2^k x 2^k
};

struct SPlan {
  int n, ne, d;
  int rb_;                     // dimension of the rounds: 2^rb_ amplitudes a thread
  std::vector<RPass> passes;
  std::vector<RRound> rounds;
  std::vector<RGate> gates;
  std::vector<double> mats;
  uint32_t col[20], row[20], beta = 0;  // logical index = B (p ^ beta)

  explicit SPlan(int n_) : n(n_), ne(std::max(n_, kRoundBits)), d(tile_bits(ne)), rb_(n_ < 20 ? 3 : 4) {
    for (int q = 0; q < 20; q++) col[q] = row[q] = 1u << q;
    reset_span();
  }

  // Tiles: one CTA up to 12 qubits; above, 8 to 256 CTAs, all resident.  Measured on
  // 20 brickwork layers (us of kernel, tiles of 2^9 / 2^10 / 2^11): 13 qubits 175 / 155 /
  // 163, 16 qubits 232 / 210 / 221, 18 qubits 290 / 262 / 260.  Smaller tiles share
  // the FP64 work among more SMs, larger ones meet the grid barrier less often.
  static int tile_bits(int n) { return n <= kTileBits ? n : n <= 17 ? 10 : n <= 19 ? 11 : kTileBits; }

  // Every op that the relabelling does not absorb, in order.
  bool lower(const std::vector<Gate>& gs, bool prune) {
    for (const Gate& g : gs) {
      int cs[2], nc = 0;
      for (int q = 0; q < n; q++)
        if ((g.cmask >> q) & 1) {
          if (nc == 2) return false;
          cs[nc++] = q;
        }
      switch (g.type) {
        case G_X1:
          if (nc == 0) beta ^= col[g.t0];
          else if (nc == 1) cnot(cs[0], g.t0);
          else pair(g.t0, cs, nc, FM_X, nullptr, false);
          break;
        case G_SWAP:
          if (nc == 0) {
            std::swap(col[g.t0], col[g.t1]);
            std::swap(row[g.t0], row[g.t1]);
          } else if (nc == 1) {  // cswap(c, a, b) = cnot(b, a) toffoli(c, a, b) cnot(b, a)
            const int both[2] = {cs[0], g.t0};
            cnot(g.t1, g.t0);
            pair(g.t1, both, 2, FM_X, nullptr, false);
            cnot(g.t1, g.t0);
          } else {
            return false;
          }
          break;
        case G_MAT1: pair(g.t0, cs, nc, form_of(g.m), g.m, prune && g.prune); break;
        case G_DIAG1: case G_DIAG2: {
          SGate o;
          o.form = g.type == G_DIAG1 ? FM_DIAG : FM_DIAG2;
          o.r[0] = row[g.t0];
          o.flip = odd(beta & row[g.t0]);
          if (g.type == G_DIAG2) {
            o.r[1] = row[g.t1];
            o.flip |= odd(beta & row[g.t1]) << 3;
          }
          o.mat = g.m;
          put(o, cs, nc);
          break;
        }
        case G_MAT2: {
          const int q[2] = {g.t0, g.t1};
          if (nc > 1) return false;
          dense(q, 2, cs, nc, g.m, prune && g.prune);
          break;
        }
        case G_MATK:
          if (g.tk.size() > 4 || nc) return false;
          dense(g.tk.data(), (int)g.tk.size(), cs, 0, g.mk.data(), prune && g.prune);
          break;
        default: return false;
      }
    }
    close();
    if (passes.empty()) close(true);  // relabelling only
    return true;
  }

 private:
  std::vector<SGate> cur_;
  std::vector<uint32_t> span_;  // echelon form, pivots at the lowest bits
  int slots_ = 0;

  static uint32_t odd(uint32_t x) { return (uint32_t)__builtin_popcount(x) & 1u; }
  void cnot(int c, int t) { row[t] ^= row[c]; col[c] ^= col[t]; }
  static uint8_t form_of(const cd* m) {
    if (m[0].im == 0 && m[1].im == 0 && m[2].im == 0 && m[3].im == 0) return FM_REAL;
    if (m[0].im == 0 && m[3].im == 0 && m[1].re == 0 && m[2].re == 0) return FM_RX;
    return FM_GEN;
  }
  void pair(int q, const int* cs, int nc, uint8_t form, const cd* m, bool prune) {
    SGate o;
    o.form = form;
    o.k = 1;
    o.prune = prune;
    o.m[0] = col[q];
    o.r[0] = row[q];
    o.flip = odd(beta & row[q]);
    o.mat = m;
    put(o, cs, nc);
  }
  void dense(const int* q, int k, const int* cs, int nc, const cd* m, bool prune) {
    SGate o;
    o.form = FM_GEN;
    o.k = (uint8_t)k;
    o.prune = prune;
    for (int i = 0; i < k; i++) {
      o.m[i] = col[q[k - 1 - i]];
      o.r[i] = row[q[k - 1 - i]];
      o.flip |= odd(beta & o.r[i]) << (8 + i);
    }
    o.mat = m;
    put(o, cs, nc);
  }
  static int slots_of(const SGate& g) { return g.form == FM_X ? 0 : g.k <= 1 ? 1 : 1 << (2 * g.k - 2); }
  uint32_t reduce(uint32_t m) const {
    for (uint32_t e : span_)
      if (m & (e & (0u - e))) m ^= e;
    return m;
  }
  bool extend(uint32_t m) {  // add to the span if it has room
    m = reduce(m);
    if (!m) return true;
    if ((int)span_.size() == d) return false;
    const uint32_t low = m & (0u - m);
    for (uint32_t& e : span_)
      if (e & low) e ^= m;
    span_.push_back(m);
    return true;
  }
  void reset_span() {
    span_.clear();
    for (int b = 0; b < (ne > d ? 2 : d); b++) extend(1u << b);  // one tile: the whole index
  }
  void put(SGate& o, const int* cs, int nc) {
    o.nc = (uint8_t)nc;
    for (int c = 0; c < nc; c++) {
      o.rc[c] = row[cs[c]];
      o.flip |= odd(beta & o.rc[c]) << (1 + c);
    }
    // (rounds and gates: a round may end for every gate)
    bool fits = (int)cur_.size() < kMaxRounds && slots_ + slots_of(o) <= kMaxSlots;
    if (fits) {
      const std::vector<uint32_t> keep = span_;
      for (int i = 0; fits && i < o.k; i++) fits = extend(o.m[i]);
      if (!fits) span_ = keep;
    }
    if (!fits) {
      close();
      for (int i = 0; i < o.k; i++) extend(o.m[i]);
    }
    slots_ += slots_of(o);
    cur_.push_back(o);
  }
  void close(bool empty = false) {
    if (cur_.empty() && !empty) return;
    for (int b = 0; b < ne && (int)span_.size() < d; b++) extend(1u << b);
    std::sort(span_.begin(), span_.end(), [](uint32_t x, uint32_t y) { return (x & (0u - x)) < (y & (0u - y)); });
    RPass P = {};
    uint32_t pivots = 0;
    for (int k = 0; k < d; k++) {
      P.basis[k] = span_[k];
      pivots |= span_[k] & (0u - span_[k]);
    }
    for (int b = 0, f = 0; b < ne; b++)
      if (!((pivots >> b) & 1)) P.free[f++] = (uint8_t)b;
    // a mask's tile bits are its bits at the pivots; a functional's, its values on the basis
    auto tile_mask = [&](uint32_t m) {
      uint32_t x = 0;
      for (int k = 0; k < d; k++)
        if (m & span_[k] & (0u - span_[k])) x |= 1u << k;
      return (uint16_t)x;
    };
    auto tile_row = [&](uint32_t r) {
      uint32_t x = 0;
      for (int k = 0; k < d; k++) x |= odd(r & span_[k]) << k;
      return (uint16_t)x;
    };
    RoundBuilder rb(d, rb_);
    for (size_t i = 0; i < cur_.size(); i++) {
      const SGate& o = cur_[i];
      uint16_t rc[2];
      for (int c = 0; c < o.nc; c++) rc[c] = tile_row(o.rc[c]);
      if (o.form == FM_DIAG || o.form == FM_DIAG2) {
        rb.add_diag(tile_row(o.r[0]), tile_row(o.r[1]), o.form == FM_DIAG2, rc, o.nc, (int)i);
      } else if (o.k == 1) {
        rb.add(tile_mask(o.m[0]), tile_row(o.r[0]), rc, o.nc, o.form == FM_X, (int)i);
      } else {
        uint16_t ms[4], rs[4];
        for (int b = 0; b < o.k; b++) { ms[b] = tile_mask(o.m[b]); rs[b] = tile_row(o.r[b]); }
        rb.add_dense(ms, rs, o.k, rc, o.nc, (int)i);
      }
    }
    rb.close();
    P.round0 = (int)rounds.size();
    P.nrounds = (int)rb.rounds.size();
    P.gate0 = (int)gates.size();
    P.ngates = (int)rb.gates.size();
    P.slot0 = (int)(mats.size() / 8);
    for (const Round& r : rb.rounds) {
      RRound Q = {};
      std::copy(r.slot, r.slot + 16, Q.slot);
      std::copy(r.rd, r.rd + 4, Q.rd);
      std::copy(r.piv, r.piv + 4, Q.piv);
      Q.k = r.k;
      Q.dense = r.dense;
      Q.ngates = (uint16_t)r.ngates;
      Q.gate0 = r.gate0;
      rounds.push_back(Q);
    }
    std::vector<char> at_round_end(rb.gates.size(), 0);
    for (const Round& r : rb.rounds) at_round_end[r.gate0 + r.ngates - 1] = 1;
    int last_phase = -1;
    for (size_t gi = 0; gi < rb.gates.size(); gi++) {
      const RoundGate& r = rb.gates[gi];
      const SGate& o = cur_[r.op];
      RGate g = {};
      g.form = o.form;
      g.bit = o.k > 1 ? 4 : r.bit;
      g.nc = o.nc;
      g.flags = o.prune ? GF_PRUNE : 0;
      g.r = r.r;
      g.r2 = r.r2;
      std::copy(r.rc, r.rc + 2, g.rc);
      std::copy(r.cj, r.cj + 2, g.cj);
      std::copy(r.rj, r.rj + 2, g.rj);
      g.cflip = (uint16_t)o.flip;
      g.g = o.r[0];
      g.gc[0] = o.rc[0];
      g.gc[1] = o.rc[1];
      g.g2 = o.form == FM_DIAG2 ? o.r[1] : 0;
      if (o.k > 1) { g.gc[1] = o.r[1]; g.g2 = o.r[2]; g.pad = o.r[3]; }
      g.slot = (uint16_t)((mats.size() / 8) - P.slot0);
      if (o.form != FM_X) {
        const size_t at = mats.size();
        mats.resize(at + 8 * (size_t)slots_of(o), 0.0);
        auto entry = [&](int e, const cd& z) { mats[at + 2 * e] = z.re; mats[at + 2 * e + 1] = z.im; };
        if (o.form == FM_DIAG && o.mat[0].re == 1 && o.mat[0].im == 0 && (o.nc < 1 || r.cj[0] == 0) && (o.nc < 2 || r.cj[1] == 0)) {
          g.form = FM_PHASE;
          // the round's gate before it, when that is a phase of the same target
          if (last_phase >= 0 && gates[last_phase].r == g.r && gates[last_phase].g == g.g && !((gates[last_phase].cflip ^ g.cflip) & 1))
            gates[last_phase].flags |= GF_CHAIN;
        }
        if (o.form == FM_DIAG) {  // read at 2 b + b
          entry(0, o.mat[0]);
          entry(3, o.mat[1]);
        } else if (o.form == FM_DIAG2) {
          for (int e = 0; e < 4; e++) entry(e, o.mat[e]);
        } else {
          for (int e = 0; e < 1 << (2 * o.k); e++) entry(e, o.mat[e]);
        }
      }
      gates.push_back(g);
      last_phase = g.form == FM_PHASE && at_round_end[gi] == 0 ? (int)gates.size() - 1 : -1;
    }
    P.nslots = (int)(mats.size() / 8) - P.slot0;
    passes.push_back(P);
    cur_.clear();
    slots_ = 0;
    reset_span();
  }
};

// Dynamic shared memory and threads of a launch on tiles of 2^d amplitudes.
size_t rounds_smem(int d) { return (sizeof(double2) << d) + 2 * sizeof(Records); }
template <int K>
unsigned rounds_threads(int d) { return std::max(32u, 1u << (d - K)); }
// A launch of one CTA has four warps from 8 qubits on: those beyond a round's cosets share
// the loads and the ordered store (an H on 8 qubits by one warp: 39.5 us a call, 32.8 by
// four; on 10 qubits sixteen in place of four make every round's barrier dearer,
// 112 us a circuit and 118).
template <int K>
unsigned rounds_threads_alone(int d) { return std::max(d >= 8 ? 128u : 32u, 1u << (d - K)); }

// CTAs that are resident together.
template <int K>
cudaError_t rounds_resident(int device, int d, int* ctas) {
  const int smem = (int)rounds_smem(d);
  int per_sm = 0, sms = 0;
  cudaError_t e = cudaFuncSetAttribute(k_rounds<K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rounds<K, false>, rounds_threads<K>(d), smem);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  *ctas = per_sm * sms;
  return e;
}

template <int K>
cudaError_t launch_rounds(const RArgs& a, unsigned grid, cudaStream_t s) {
  const size_t smem = rounds_smem(a.d);
  if constexpr (K == 3) {  // (tiles of fewer than 2^10 amplitudes are never part of a grid)
    if (grid == 1) {
      const cudaError_t e =
          cudaFuncSetAttribute(k_rounds<K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      k_rounds<K, true><<<1, rounds_threads_alone<K>(a.d), smem, s>>>(a);
      return cudaGetLastError();
    }
  }
  const cudaError_t e = cudaFuncSetAttribute(k_rounds<K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<RArgs*>(&a)};
  return cudaLaunchCooperativeKernel((const void*)k_rounds<K, false>, dim3(grid), dim3(rounds_threads<K>(a.d)), args, smem, s);
}

}  // namespace

// The circuit in one launch (not waited for); *ran = false when it holds something
// this path does not take (unitaries of more than four qubits), or the device has no
// room for all its CTAs at once (a share of a GPU): the passes run it then.
int run_small(ket_state* s, const std::vector<Gate>& gates, bool prune, bool* ran) {
  *ran = false;
  SPlan P(s->n);
  ket_ctx* c = s->ctx;
  cudaSetDevice(c->device);
  const unsigned grid = s->n > P.d ? 1u << (s->n - P.d) : 1u;
  if (grid > 1) {
    int& fit = c->rounds_ctas[P.d - 10];  // (tiles of a grid are of 2^10 to 2^12)
    if (fit == 0) {
      const cudaError_t e =
          P.rb_ == 4 ? rounds_resident<4>(c->device, P.d, &fit) : rounds_resident<3>(c->device, P.d, &fit);
      if (e != cudaSuccess) return cuda_fail(e, "rounds occupancy");
    }
    if (grid > (unsigned)(g_max_ctas > 0 ? g_max_ctas : fit)) return KET_OK;
  }
  if (!P.lower(gates, prune)) return KET_OK;
  constexpr size_t kInverse = 128;
  size_t total = 256;  // the barrier's counter, then the relabelling's inverse
  auto place = [&](size_t bytes) {
    const size_t at = total;
    total += (bytes + 255) & ~size_t(255);
    return at;
  };
  const size_t o_pass = place(sizeof(RPass) * P.passes.size()), o_round = place(sizeof(RRound) * P.rounds.size()),
               o_gate = place(sizeof(RGate) * P.gates.size()), o_mat = place(8 * P.mats.size());
  void* dev = nullptr;
  int rc = ctx_scratch(c, total, &dev);
  if (rc) return rc;
  std::vector<unsigned char> img(total, 0);
  memcpy(img.data() + o_pass, P.passes.data(), sizeof(RPass) * P.passes.size());
  if (!P.rounds.empty()) memcpy(img.data() + o_round, P.rounds.data(), sizeof(RRound) * P.rounds.size());
  if (!P.gates.empty()) memcpy(img.data() + o_gate, P.gates.data(), sizeof(RGate) * P.gates.size());
  if (!P.mats.empty()) memcpy(img.data() + o_mat, P.mats.data(), 8 * P.mats.size());
  const bool permute = [&] {
    for (int q = 0; q < s->n; q++)
      if (P.col[q] != 1u << q) return true;
    return P.beta != 0;
  }();
  if (permute && grid > 1) {
    uint32_t inv[21] = {};
    for (int q = 0; q < s->n; q++) {
      for (uint32_t r = P.row[q]; r; r &= r - 1) inv[1 + __builtin_ctz(r)] |= 1u << q;
      inv[0] |= ((uint32_t)__builtin_popcount(P.beta & P.row[q]) & 1u) << q;
    }
    static_assert(kInverse + sizeof(inv) <= 256, "before the passes");
    memcpy(img.data() + kInverse, inv, sizeof(inv));
  }
  c->h2d_bytes += total;
  rc = ctx_upload(c, dev, img.data(), total);
  if (rc) return rc;
  char* base = (char*)dev;
  RArgs a;
  memset(&a, 0, sizeof(a));
  a.amp = (double2*)s->amp;
  a.passes = (const RPass*)(base + o_pass);
  a.rounds = (const RRound*)(base + o_round);
  a.gates = (const RGate*)(base + o_gate);
  a.mats = (const double2*)(base + o_mat);
  a.arrived = (unsigned int*)base;
  a.status = c->d_status;
  a.npasses = (int)P.passes.size();
  a.n = s->n;
  a.d = P.d;
  a.spin_limit = g_spin_limit;
  a.beta = P.beta;
  a.permute = permute;
  a.inverse = (const uint32_t*)(base + kInverse);
  std::copy(P.col, P.col + 20, a.acol);
  prof_begin(c);
  const cudaError_t e = P.rb_ == 4 ? launch_rounds<4>(a, grid, c->stream) : launch_rounds<3>(a, grid, c->stream);
  prof_end(c, PK_FUSED1);
  if (e != cudaSuccess) return cuda_fail(e, "rounds launch");
  *ran = true;
  return KET_OK;
}

}  // namespace ket

extern "C" int ket_debug_rounds_hook(int max_ctas, uint32_t spin_limit) {
  if (max_ctas < 0) return ket::fail(KET_ERR_TYPE, "negative CTA count");
  ket::g_max_ctas = max_ctas;
  ket::g_spin_limit = spin_limit ? spin_limit : ket::kSpinLimit;
  return KET_OK;
}
