// shots.cu -- run()'s per-shot path: mid-circuit measure / reset / if and
// stochastic Pauli noise (circuit.ts:55-83, :169-207, :289-304, :3455-3481).
//
// One device trajectory per shot.  The host walks the op list the way
// applyOps does and draws the reference's xorshift32 stream in the
// reference's order; every operation on the state runs on the device:
//   * runs of gates go through the fused engine (ket_apply_ops, with the
//     reference's per-gate pruning), with the Paulis that the noise draws
//     select spliced in right after their gate -- the draws never depend on
//     the state, so a run of noisy gates is still one engine call;
//   * measure and reset reduce P(q=1) on the device (k_prob_one, fixed-order
//     partial sums), the host compares it with its draw, and k_collapse
//     zeroes the other half and rescales the kept half in place by
//     1/sqrt(p) as collapseQubit does;
//   * the final readout is the sampling kernel with no probability
//     threshold: sampleSV walks every entry of its Map, and the engine's
//     pruned state holds exactly those entries as its nonzero amplitudes.
//     The sampler's running sum is sampleSV's, ascending index order and
//     rounding included; the in-shared-memory trajectories below walk chunk
//     sums and then one chunk, which differs from it only in rounding.
// The device state is the caller's ket_state, reset to |init> per shot.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "engine.h"
#include "fused_ops.cuh"
#include "launch.h"
#include "rounds.h"

using namespace ket;

namespace {

constexpr int KNT = 256;

// partial[b] = sum of |a_i|^2 over i with bit q set, for the b-th slice of
// the N/2 such indices (j -> i inserts a 1 at bit q).
template <typename R>
__global__ void __launch_bounds__(KNT) k_prob_one(const typename Vec2<R>::T* a, uint64_t half, int q, uint64_t chunk,
                                                  double* partial) {
  __shared__ double sh[KNT];
  const uint64_t lo = (uint64_t)blockIdx.x * chunk;
  const uint64_t hi = lo + chunk < half ? lo + chunk : half;
  const uint64_t low = (uint64_t(1) << q) - 1;
  double acc = 0.0;
  for (uint64_t j = lo + threadIdx.x; j < hi; j += KNT) {
    const uint64_t i = ((j & ~low) << 1) | (uint64_t(1) << q) | (j & low);
    const typename Vec2<R>::T v = a[i];
    const double re = (double)v.x, im = (double)v.y;
    acc += re * re + im * im;
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int w = KNT / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// out = the partials summed in index order (one thread: nb <= 4096).
__global__ void k_sum_in_order(const double* partial, int nb, double* out) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double s = 0.0;
  for (int b = 0; b < nb; b++) s += partial[b];
  *out = s;
}

// collapseQubit's projection: keep the amplitudes whose bit q equals the
// outcome, scaled by inv; zero the others.
template <typename R>
__global__ void k_collapse(typename Vec2<R>::T* a, uint64_t N, int q, int outcome, double inv) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    typename Vec2<R>::T v = a[i];
    if ((int)((i >> q) & 1) == outcome) {
      v.x = (R)((double)v.x * inv);
      v.y = (R)((double)v.y * inv);
    } else {
      v.x = (R)0;
      v.y = (R)0;
    }
    a[i] = v;
  }
}

#define TRY(x) do { int _rc = (x); if (_rc) return _rc; } while (0)

// ---------------------------------------------------------------- batched trajectories
// Small states (2^n amplitudes fit in shared memory) run one shot per CTA,
// many shots at a time.  Gate arithmetic rounds exactly as the reference's
// complex.ts does (products and sums each rounded, no fused multiply-add; the
// products of zero matrix entries, which add nothing, are left out), pruning as
// accumulate() does.
//
// The op list is planned once for all shots (plan_shots): one-qubit gates run in
// rounds on cosets of 16 amplitudes held in registers, and CNOTs and swaps outside
// if-bodies are relabellings of the shared-memory state (rounds.h).  What differs
// from shot to shot is carried beside the plan:
//   * the Paulis the noise draws select are a frame: an X on a qubit moves the
//     physical indices by a mask (beta), a Z signs them by a functional (zeta), and
//     a gate reads both as of its place in the program -- the swapped rows and
//     columns, or negated off-diagonal entries, a Pauli before it amounts to.
//     (A Y is both, up to a phase that no probability sees.)
//   * draw d of the shot's xorshift32 stream is the start state under a GF(2) power
//     of the step, so the threads make the draws of a segment in parallel.

enum { T_NOISE1 = 20, T_NOISE2 = 21 };

struct TOp {
  int32_t kind;  // ket_op_kind, or T_NOISE1 / T_NOISE2 (a dep1 / dep2 draw after the gate before it)
  int32_t q[4];  // gate qubits; MEASURE {q, cbit}; RESET {q}; IF {first bit, size, value, body length}
  int32_t mat;   // complex offset of the matrix in the matrix table (-1: none)
  int32_t k;     // UNITARY: qubit count
  int32_t pad;
};

struct cd { double re, im; };
__device__ __forceinline__ cd cmul_rn(cd a, cd b) {  // complex.ts mul
  return {__dsub_rn(__dmul_rn(a.re, b.re), __dmul_rn(a.im, b.im)),
          __dadd_rn(__dmul_rn(a.re, b.im), __dmul_rn(a.im, b.re))};
}
__device__ __forceinline__ cd cadd_rn(cd a, cd b) { return {__dadd_rn(a.re, b.re), __dadd_rn(a.im, b.im)}; }
__device__ __forceinline__ double norm2_rn(cd a) { return __dadd_rn(__dmul_rn(a.re, a.re), __dmul_rn(a.im, a.im)); }
__device__ __forceinline__ cd pruned(cd a) {
  // (the high words rule out all but components of about 1e-7 and below)
  if (fmaxf(hiabs(a.re), hiabs(a.im)) < tiny_screen(0.0) && norm2_rn(a) < 1e-14) return cd{0.0, 0.0};
  return a;
}

template <typename V>
__device__ __forceinline__ cd ldc(const V* st, uint32_t i) { const V v = st[i]; return {(double)v.x, (double)v.y}; }
template <typename V>
__device__ __forceinline__ void stc(V* st, uint32_t i, cd a) {
  V v;
  v.x = (decltype(v.x))a.re;
  v.y = (decltype(v.y))a.im;
  st[i] = v;
}

constexpr int kShotBits = kRoundBits;
constexpr int kShotMinQubits = 4;  // narrower states get idle qubits, so that a coset of 16 exists

struct __align__(16) SRound {
  uint16_t slot[16], m[4], rd[4];
  uint8_t piv[4];
  uint8_t k, dense;
  uint16_t ngates;
  int32_t gate0;      // in the segment
  int32_t pad;
};
enum : uint8_t { SF_GEN = 0, SF_REAL = 1, SF_RX = 2, SF_DIAG = 3, SF_X = 4 };
struct __align__(16) SGate {
  uint8_t form, bit, nc, pad;
  uint16_t r, m;      // the target's functional and mask
  int32_t slot;       // matrix, in 64-byte slots of the segment
  uint32_t frame;     // beta | zeta << 16 as of this gate (shared memory only)
  uint16_t rc[2];     // controls
  uint8_t cj[2];
  uint16_t pad2;
  int32_t dpos;       // noise draws of the segment before this gate
  int32_t pad3;
};
static_assert(sizeof(SGate) == 32, "two 16-byte reads");
// A noise draw: the masks and functionals of its qubits at its place in the program.
struct SNoise {
  uint16_t ma, ra, mb, rb;
  int32_t two;
};
// Gates between measurements, resets and ifs, as many as shared memory holds: round0,
// gate0 and slot0 are places in the segment's chunk.
struct SSeg {
  int32_t chunk, round0, nrounds, gate0, ngates, slot0;
  int32_t noise0, ndraws, per, jump0;  // draws, draws a thread, first jump row
};
// Segments whose records are in shared memory together (a program that fits is read
// once a CTA; one that measures after every gate is not read again for each: with draws
// stepped from the draw before, 200 measurements of 4 qubits, 100 shots, 1260 us before
// and 990 now, 100 of 10 qubits, 1000 shots, 1400 and 1270, 50 of 12, 2000, 3440 and 3120).
struct SChunk {
  int32_t round0, nrounds, gate0, ngates, slot0, nslots;
};
enum { ST_SEG = 0, ST_MEASURE = 1, ST_RESET = 2, ST_IF = 3 };
struct SStep {
  int32_t kind;
  // SEG: index; MEASURE: cbit, jump row, steps from the draw of the one before (0: jump);
  // RESET: -, jump row, steps; IF: first, size, value, steps to skip
  int32_t a, b, c, d;
  uint16_t r, m;       // MEASURE, RESET: the qubit's functional and mask (r = 0: a qubit outside the state)
};

struct SArgs {
  const SStep* steps;
  const SSeg* segs;
  const SChunk* chunks;
  const SRound* rounds;
  const SGate* gates;
  const double2* mats;   // by 64-byte slots
  const SNoise* noise;
  const uint32_t* jump;  // rows of 32 columns: the step's power that makes the row's draw
  const uint32_t* start;
  uint64_t* out_idx;
  uint8_t* out_bits;
  uint64_t shots, init;
  ket_noise nz;
  int nsteps, n, ne, ncbits;  // ne: qubits with idle ones
  int last_row, last_gap;     // jump row of the sampling draw, or its steps
  // shared-memory layout (bytes)
  int off_mats, off_rounds, off_gates, off_events, off_red, off_bits;
  uint16_t acol[kRoundQubits];  // the final relabelling: physical mask of each logical bit
};

struct SEvent {
  int32_t d;
  uint32_t bz;  // beta | zeta << 16
};

__device__ __forceinline__ uint32_t xs_step(uint32_t s) {  // xorshift32 (circuit.ts:813-819)
  s ^= s << 13;
  s ^= s >> 17;
  return s ^ (s << 5);
}
__device__ __forceinline__ double xs_value(uint32_t s) { return (double)s / 4294967296.0; }
__device__ __forceinline__ uint32_t xs_jump(const uint32_t* row, uint32_t s) {
  uint32_t o = 0;
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const uint4 c = __ldg(reinterpret_cast<const uint4*>(row + k));
    o ^= ((s >> k) & 1 ? c.x : 0u) ^ ((s >> (k + 1)) & 1 ? c.y : 0u) ^ ((s >> (k + 2)) & 1 ? c.z : 0u) ^
         ((s >> (k + 3)) & 1 ? c.w : 0u);
  }
  return o;
}

__device__ __forceinline__ double neg_if(double v, uint32_t odd) {
  return __hiloint2double(__double2hiint(v) ^ (int)(odd << 31), __double2loint(v));
}
__device__ __forceinline__ uint32_t par(uint32_t x) { return (uint32_t)__popc(x) & 1u; }

// The amplitudes j of a coset whose controls all hold (p: the base, moved by beta).
__device__ __forceinline__ uint32_t shot_controls(const SGate& g, uint32_t p) {
  uint32_t ok = 0xffffu;
  for (int c = 0; c < g.nc; c++) {
    const uint32_t cj = g.cj[c];
    uint32_t x = par(p & g.rc[c]) ? 0xffffu : 0u;
    x ^= (cj & 1 ? 0xaaaau : 0u) ^ (cj & 2 ? 0xccccu : 0u) ^ (cj & 4 ? 0xf0f0u : 0u) ^ (cj & 8 ? 0xff00u : 0u);
    ok &= x;
  }
  return ok;
}

// A 2x2 on register bit I.  role: the amplitude with the bit clear holds logical 1
// (entry e becomes e ^ 3); neg: the off-diagonal entries change sign.
// The pair's new values, in place: inline PTX with tied operands (the cross products
// first), so that every amplitude keeps its registers across the forms the gate loop
// switches between.  Written as expressions, the loop re-homed the thread's 64
// registers of amplitudes at every gate.  Each product and sum is rounded.
template <int FORM>
__device__ __forceinline__ void shot_pair(cd& a, cd& b, const cd* g) {
  if (FORM == SF_REAL) {
    asm("{\n .reg .f64 x, y, u, w;\n"
        " mul.rn.f64 x, %5, %2;\n mul.rn.f64 y, %5, %3;\n mul.rn.f64 u, %6, %0;\n mul.rn.f64 w, %6, %1;\n"
        " mul.rn.f64 %0, %4, %0;\n add.rn.f64 %0, %0, x;\n mul.rn.f64 %1, %4, %1;\n add.rn.f64 %1, %1, y;\n"
        " mul.rn.f64 %2, %7, %2;\n add.rn.f64 %2, u, %2;\n mul.rn.f64 %3, %7, %3;\n add.rn.f64 %3, w, %3;\n}"
        : "+d"(a.re), "+d"(a.im), "+d"(b.re), "+d"(b.im)
        : "d"(g[0].re), "d"(g[1].re), "d"(g[2].re), "d"(g[3].re));
  } else if (FORM == SF_RX) {
    asm("{\n .reg .f64 x, y, u, w;\n"
        " mul.rn.f64 x, %5, %3;\n mul.rn.f64 y, %5, %2;\n mul.rn.f64 u, %6, %1;\n mul.rn.f64 w, %6, %0;\n"
        " mul.rn.f64 %0, %4, %0;\n sub.rn.f64 %0, %0, x;\n mul.rn.f64 %1, %4, %1;\n add.rn.f64 %1, %1, y;\n"
        " mul.rn.f64 %2, %7, %2;\n sub.rn.f64 %2, %2, u;\n mul.rn.f64 %3, %7, %3;\n add.rn.f64 %3, w, %3;\n}"
        : "+d"(a.re), "+d"(a.im), "+d"(b.re), "+d"(b.im)
        : "d"(g[0].re), "d"(g[1].im), "d"(g[2].im), "d"(g[3].re));
  } else if (FORM == SF_DIAG) {
    asm("{\n .reg .f64 x, y;\n"
        " mul.rn.f64 x, %5, %1;\n mul.rn.f64 y, %5, %0;\n mul.rn.f64 %0, %4, %0;\n sub.rn.f64 %0, %0, x;\n"
        " mul.rn.f64 %1, %4, %1;\n add.rn.f64 %1, %1, y;\n"
        " mul.rn.f64 x, %7, %3;\n mul.rn.f64 y, %7, %2;\n mul.rn.f64 %2, %6, %2;\n sub.rn.f64 %2, %2, x;\n"
        " mul.rn.f64 %3, %6, %3;\n add.rn.f64 %3, %3, y;\n}"
        : "+d"(a.re), "+d"(a.im), "+d"(b.re), "+d"(b.im)
        : "d"(g[0].re), "d"(g[0].im), "d"(g[3].re), "d"(g[3].im));
  } else {
    asm("{\n .reg .f64 x, y, u, w, t, s;\n"
        // x + i y = g1 b, u + i w = g2 a
        " mul.rn.f64 x, %6, %2;\n mul.rn.f64 t, %7, %3;\n sub.rn.f64 x, x, t;\n"
        " mul.rn.f64 y, %6, %3;\n mul.rn.f64 t, %7, %2;\n add.rn.f64 y, y, t;\n"
        " mul.rn.f64 u, %8, %0;\n mul.rn.f64 t, %9, %1;\n sub.rn.f64 u, u, t;\n"
        " mul.rn.f64 w, %8, %1;\n mul.rn.f64 t, %9, %0;\n add.rn.f64 w, w, t;\n"
        // a = g0 a + (x + i y), b = (u + i w) + g3 b
        " mul.rn.f64 t, %5, %1;\n mul.rn.f64 s, %5, %0;\n"
        " mul.rn.f64 %0, %4, %0;\n sub.rn.f64 %0, %0, t;\n add.rn.f64 %0, %0, x;\n"
        " mul.rn.f64 %1, %4, %1;\n add.rn.f64 %1, %1, s;\n add.rn.f64 %1, %1, y;\n"
        " mul.rn.f64 t, %11, %3;\n mul.rn.f64 s, %11, %2;\n"
        " mul.rn.f64 %2, %10, %2;\n sub.rn.f64 %2, %2, t;\n add.rn.f64 %2, u, %2;\n"
        " mul.rn.f64 %3, %10, %3;\n add.rn.f64 %3, %3, s;\n add.rn.f64 %3, w, %3;\n}"
        : "+d"(a.re), "+d"(a.im), "+d"(b.re), "+d"(b.im)
        : "d"(g[0].re), "d"(g[0].im), "d"(g[1].re), "d"(g[1].im), "d"(g[2].re), "d"(g[2].im), "d"(g[3].re), "d"(g[3].im));
  }
}

template <typename R, int K, int I, int FORM>
__device__ __forceinline__ void shot_gate(cpx<R>* v, const double2* M, bool role, uint32_t neg, bool ctl, uint32_t ok) {
  constexpr int NS = 1 << K;
  cd g[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const double2 t = M[role ? e ^ 3 : e];
    g[e] = (e == 1 || e == 2) ? cd{neg_if(t.x, neg), neg_if(t.y, neg)} : cd{t.x, t.y};
  }
#pragma unroll
  for (int j = 0; j < NS; j++) {
    if (j & (1 << I)) continue;
    const int j1 = j | 1 << I;
    if (ctl && !((ok >> j) & 1)) continue;
    cd a = {(double)v[j].re, (double)v[j].im}, b = {(double)v[j1].re, (double)v[j1].im};
    shot_pair<FORM>(a, b, g);
    if constexpr (sizeof(R) == 4) {  // the pruning reads the value before its rounding to FP32
      a = pruned(a);
      b = pruned(b);
    }
    v[j] = cpx<R>{(R)a.re, (R)a.im};
    v[j1] = cpx<R>{(R)b.re, (R)b.im};
  }
  if constexpr (sizeof(R) == 8) {  // one screen over the thread's amplitudes
    // (an exact zero, of which a state has many in its first gates, need not be
    // flushed: less one, its word is the largest)
    uint32_t tiny = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < NS; j++)
      tiny = min(tiny, __float_as_uint(fmaxf(hiabs(v[j].re), hiabs(v[j].im))) - 1u);
    if (tiny < __float_as_uint(tiny_screen(0.0)) - 1u) {
#pragma unroll
      for (int j = 0; j < NS; j++) {
        const cd y = pruned(cd{v[j].re, v[j].im});
        v[j] = cpx<R>{(R)y.re, (R)y.im};
      }
    }
  }
}
// X under controls: the two trade places, with the sign the frame puts between them.
template <typename R, int K, int I>
__device__ __forceinline__ void shot_x(cpx<R>* v, uint32_t neg, uint32_t ok) {
#pragma unroll
  for (int j = 0; j < (1 << K); j++) {
    if ((j & (1 << I)) || !((ok >> j) & 1)) continue;
    const cpx<R> a = v[j], b = v[j | 1 << I];
    v[j] = cpx<R>{neg ? -b.re : b.re, neg ? -b.im : b.im};
    v[j | 1 << I] = cpx<R>{neg ? -a.re : a.re, neg ? -a.im : a.im};
  }
}

#define KET_BITS KET_BIT(0) KET_BIT(1) KET_BIT(2) KET_BIT(3)
static_assert(kShotBits == 4, "one KET_BIT a register bit");

template <typename R, int NT>
__device__ __forceinline__ void shot_round(typename Vec2<R>::T* st, const SRound& Q, const SGate* gates,
                                           const double2* mats, int n) {
  constexpr int K = kShotBits;
  const uint32_t nsub = 1u << (n - K);
  for (uint32_t u = threadIdx.x; u < nsub; u += NT) {
    uint32_t base = u;
#pragma unroll
    for (int i = 0; i < K; i++) base = insert0_32(base, Q.piv[i]);
    const uint32_t sb = round_slot(base);
    cpx<R> v[1 << K];
    RoundSlots slots;
    slots.read(Q.slot);
#pragma unroll
    for (int j = 0; j < (1 << K); j++) v[j] = ld_amp<R>(st + (sb ^ slots(j)));
    // cosets of zeros stay zeros (most of a state in its first gates)
    if (!__any_sync(__activemask(), !all_zero<R, 1 << K>(v))) continue;
    for (int k = 0; k < Q.ngates; k++) {
      // form, bit, controls | functional, mask | matrix | frame
      const uint4 g = *reinterpret_cast<const uint4*>(gates + k);
      const uint32_t p = base ^ (g.w & 0xffffu), neg = par((g.y >> 16) & (g.w >> 16));
      const bool role = par(p & g.y & 0xffffu);
      const double2* M = mats + 4 * g.z;
      const int form = g.x & 0xff, bit = (g.x >> 8) & 0xff;
      if (g.x >> 16) {
        const uint32_t ok = shot_controls(gates[k], p);
        switch (2 * bit + (form == SF_X)) {
#define KET_BIT(I)                                                                    \
  case 2 * I: shot_gate<R, K, I, SF_GEN>(v, M, role, neg, true, ok); break;           \
  case 2 * I + 1: shot_x<R, K, I>(v, neg, ok); break;
          KET_BITS
#undef KET_BIT
        }
        continue;
      }
      switch (4 * bit + form) {
#define KET_BIT(I)                                                                      \
  case 4 * I + SF_GEN: shot_gate<R, K, I, SF_GEN>(v, M, role, neg, false, 0); break;    \
  case 4 * I + SF_REAL: shot_gate<R, K, I, SF_REAL>(v, M, role, neg, false, 0); break;  \
  case 4 * I + SF_RX: shot_gate<R, K, I, SF_RX>(v, M, role, neg, false, 0); break;      \
  case 4 * I + SF_DIAG: shot_gate<R, K, I, SF_DIAG>(v, M, role, neg, false, 0); break;
        KET_BITS
#undef KET_BIT
      }
    }
    slots.read(Q.slot);
#pragma unroll
    for (int j = 0; j < (1 << K); j++) st_amp<R>(st + (sb ^ slots(j)), v[j]);
  }
}

// A dense 2^K x 2^K (two-qubit gates, csrswap, unitaries of up to 4 qubits):
// applyTwo and applyUnitary add a row's products in ascending column order.
template <typename R, int NT, int K>
__device__ void shot_dense(typename Vec2<R>::T* st, const SRound& Q, const SGate& g, const double2* mats,
                           int n) {
  constexpr int D = 1 << K;
  const uint32_t f = g.frame;
  const uint32_t nsub = 1u << (n - K);
  const double2* M = mats + 4 * g.slot;
  uint32_t z = 0;  // the frame's sign of mask i
#pragma unroll
  for (int i = 0; i < K; i++) z |= par(Q.m[i] & (f >> 16)) << i;
  for (uint32_t u = threadIdx.x; u < nsub; u += NT) {
    uint32_t base = u;
#pragma unroll
    for (int i = 0; i < K; i++) base = insert0_32(base, Q.piv[i]);
    const uint32_t p = base ^ (f & 0xffffu), sb = round_slot(base);
    if (g.nc && !(shot_controls(g, p) & 1)) continue;
    uint32_t l0 = 0;  // local index of the coset's base
#pragma unroll
    for (int i = 0; i < K; i++) l0 |= par(p & Q.rd[i]) << i;
    cd x[D];
#pragma unroll
    for (int c = 0; c < D; c++) {
      const cd t = ldc(st, sb ^ Q.slot[c ^ l0]);
      const uint32_t odd = par((c ^ l0) & z);
      x[c] = cd{neg_if(t.re, odd), neg_if(t.im, odd)};
    }
    for (int r = 0; r < D; r++) {
      cd out = {0.0, 0.0};
#pragma unroll
      for (int c = 0; c < D; c++) {
        const double2 m = M[r * D + c];
        out = cadd_rn(out, cmul_rn(cd{m.x, m.y}, x[c]));
      }
      out = pruned(out);
      const uint32_t odd = par((r ^ l0) & z);
      stc(st, sb ^ Q.slot[r ^ l0], cd{neg_if(out.re, odd), neg_if(out.im, odd)});
    }
  }
}

// block sum of v in a fixed order (warps, then their sums in order)
template <int NT>
__device__ double shot_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = red[0];
#pragma unroll
  for (int w = 1; w < NT / 32; w++) s = __dadd_rn(s, red[w]);
  return s;
}

// collapseQubit (circuit.ts:55-72) on the shared-memory state
template <typename R, int NT>
__device__ int shot_collapse(typename Vec2<R>::T* st, int n, uint32_t r, uint32_t beta, double rand, double* red) {
  if (r == 0) return 0;  // a qubit outside the state reads 0; the state is unchanged
  const uint32_t N = 1u << n;
  double acc = 0.0;
  for (uint32_t i = threadIdx.x; i < N; i += NT)
    if (par((i ^ beta) & r)) acc = __dadd_rn(acc, norm2_rn(ldc(st, round_slot(i))));
  const double p1 = shot_sum<NT>(acc, red);
  const int outcome = rand < p1 ? 1 : 0;
  const double inv = 1 / sqrt(outcome == 1 ? p1 : 1 - p1);
  for (uint32_t i = threadIdx.x; i < N; i += NT) {
    cd a = ldc(st, round_slot(i));
    if ((int)par((i ^ beta) & r) == outcome) a = {__dmul_rn(a.re, inv), __dmul_rn(a.im, inv)};
    else a = {0.0, 0.0};
    stc(st, round_slot(i), a);
  }
  __syncthreads();
  return outcome;
}

__device__ __forceinline__ void copy_words(void* dst, const void* src, int bytes, int nt) {
  for (int i = threadIdx.x; i < bytes / 4; i += nt)
    static_cast<uint32_t*>(dst)[i] = __ldg(static_cast<const uint32_t*>(src) + i);
}

// Bound: the FP64 pipe (unfused products and sums).  In place of one pass over
// shared memory and one barrier per op, every gate as a general complex one:
// 16384 shots of 12 qubits, 120 one-qubit gates and 55 CNOTs with noise, 22.6 ->
// 8.4 ms (FP64 pipe 28% busy, issue slots 52%: register moves between the gate
// forms take a fifth of the instructions).  Cosets of 16 at 16 warps an SM beat
// cosets of 8 at 32 warps (9.9 ms), which pass over shared memory more often.
template <typename R, int NT>
__global__ void __launch_bounds__(NT, NT <= 64 ? 8 : 512 / NT) k_shots(const __grid_constant__ SArgs a) {
  typedef typename Vec2<R>::T V;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* st = reinterpret_cast<V*>(smraw);
  double2* mats = reinterpret_cast<double2*>(smraw + a.off_mats);
  SRound* rounds = reinterpret_cast<SRound*>(smraw + a.off_rounds);
  SGate* gates = reinterpret_cast<SGate*>(smraw + a.off_gates);
  SEvent* events = reinterpret_cast<SEvent*>(smraw + a.off_events);
  double* red = reinterpret_cast<double*>(smraw + a.off_red);
  uint8_t* bits = smraw + a.off_bits;
  __shared__ int nev;
  __shared__ uint32_t pick, last;
  const int t = threadIdx.x, n = a.ne;
  int loaded = -1;
  for (uint64_t shot = blockIdx.x; shot < a.shots; shot += gridDim.x) {
    const uint32_t s0 = a.start[shot];
    uint32_t beta = 0, zeta = 0;
    uint32_t xd = s0;  // the stream at the last measurement's or reset's draw
    auto draw = [&](int gap, int row) {
      if (gap > 0) {
        for (int k = 0; k < gap; k++) xd = xs_step(xd);
      } else {
        xd = xs_jump(a.jump + 32 * row, s0);
      }
      return xd;
    };
    for (uint32_t i = t; i < 1u << n; i += NT) stc(st, round_slot(i), cd{i == a.init ? 1.0 : 0.0, 0.0});
    for (int b = t; b < a.ncbits; b += NT) bits[b] = 0;
    __syncthreads();
    for (int pc = 0; pc < a.nsteps; pc++) {
      const SStep& o = a.steps[pc];
      const int kind = o.kind;
      if (kind == ST_SEG) {
        const SSeg S = a.segs[o.a];
        if (loaded != S.chunk) {
          const SChunk C = a.chunks[S.chunk];
          copy_words(rounds, a.rounds + C.round0, C.nrounds * sizeof(SRound), NT);
          copy_words(gates, a.gates + C.gate0, C.ngates * sizeof(SGate), NT);
          copy_words(mats, a.mats + 4 * C.slot0, C.nslots * 64, NT);
          loaded = S.chunk;
        }
        SGate* sgates = gates + S.gate0;
        const double2* smats = mats + 4 * S.slot0;
        if (t == 0) nev = 0;
        __syncthreads();
        const int d0 = t * S.per, d1 = min(d0 + S.per, S.ndraws);
        if (d0 < d1) {
          uint32_t x = xs_jump(a.jump + 32 * (S.jump0 + t), s0);
          for (int d = d0; d < d1; d++) {
            const SNoise q = a.noise[S.noise0 + d];
            const double r = xs_value(x), p = q.two ? a.nz.p2 : a.nz.p1;
            x = xs_step(x);
            if (!(r < p)) continue;
            int pa, pb = 0;  // 0 none, 1 X, 2 Y, 3 Z
            const double u = r / p;
            if (q.two) {  // dep2 (circuit.ts:298-304), TWO_PAULI order
              int k = (int)floor(u * 15);
              if (k > 14) k = 14;
              pa = (k + 1) >> 2;  // k + 1 = 4 * pa + pb over {I, X, Y, Z}^2 \ {II}
              pb = (k + 1) & 3;
            } else {  // dep1 (circuit.ts:289-295)
              pa = u < 1.0 / 3 ? 1 : u < 2.0 / 3 ? 2 : 3;
            }
            const uint32_t be = (pa == 1 || pa == 2 ? q.ma : 0u) ^ (pb == 1 || pb == 2 ? q.mb : 0u);
            const uint32_t ze = (pa >= 2 ? q.ra : 0u) ^ (pb >= 2 ? q.rb : 0u);
            events[atomicAdd(&nev, 1)] = SEvent{d, be | ze << 16};  // (their order does not matter: XORs)
          }
        }
        __syncthreads();
        const int ne = nev;
        for (int g = t; g < S.ngates; g += NT) {
          uint32_t f = beta | zeta << 16;
          for (int e = 0; e < ne; e++)
            if (events[e].d < sgates[g].dpos) f ^= events[e].bz;
          sgates[g].frame = f;
        }
        for (int e = 0; e < ne; e++) {
          beta ^= events[e].bz & 0xffffu;
          zeta ^= events[e].bz >> 16;
        }
        for (int q = 0; q < S.nrounds; q++) {
          __syncthreads();
          const SRound& Q = rounds[S.round0 + q];
          const SGate* G = sgates + Q.gate0;
          if (Q.dense) {
            switch (Q.k) {
              case 2: shot_dense<R, NT, 2>(st, Q, *G, smats, n); break;
              case 3: shot_dense<R, NT, 3>(st, Q, *G, smats, n); break;
              default: shot_dense<R, NT, 4>(st, Q, *G, smats, n); break;
            }
          } else {
            shot_round<R, NT>(st, Q, G, smats, n);
          }
        }
      } else if (kind == ST_MEASURE || kind == ST_RESET) {
        uint32_t x = draw(o.c, o.b);
        const int outcome = shot_collapse<R, NT>(st, n, o.r, beta, xs_value(x), red);
        if (kind == ST_RESET) {
          if (outcome == 1) beta ^= o.m;
        } else {
          x = xs_step(x);
          const int reported = (a.nz.pmeas != 0 && xs_value(x) < a.nz.pmeas) ? 1 - outcome : outcome;
          if (t == 0 && o.a >= 0) bits[o.a] = (uint8_t)reported;
        }
      } else {
        int v = 0;
        for (int kk = 0; kk < o.b; kk++)
          if (bits[o.a + kk]) v |= 1 << kk;
        if (v != o.c) pc += o.d;
      }
      __syncthreads();
    }
    // sampleSV (circuit.ts:75-83): the first logical index whose running sum of
    // |a|^2 reaches the draw, else the last nonzero entry.  Thread t holds logical
    // indices 16 t .. 16 t + 15; a scan gives it the sum before them.
    uint32_t x = draw(a.last_gap, a.last_row);
    const double r = xs_value(x);
    if (t == 0) { pick = 0xffffffffu; last = 0; }
    const uint32_t N = 1u << a.n;
    constexpr int NW = NT / 32;
    double carry = 0.0;  // sums of the tiles of 16 NT indices before this one
    for (uint32_t l0 = 0; l0 < N; l0 += 16 * NT) {
      const uint32_t l = l0 + 16 * t;
      uint32_t phys = beta;
      for (int b = 4; b < n; b++)
        if ((l >> b) & 1) phys ^= a.acol[b];
      double pv[16], csum = 0.0;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const uint32_t pj = phys ^ (j & 1 ? a.acol[0] : 0) ^ (j & 2 ? a.acol[1] : 0) ^ (j & 4 ? a.acol[2] : 0) ^
                            (j & 8 ? a.acol[3] : 0);
        pv[j] = l + j < N ? norm2_rn(ldc(st, round_slot(pj))) : 0.0;
        if (pv[j] > 0) csum = __dadd_rn(csum, pv[j]);
      }
      double incl = csum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((t & 31) >= o) incl = __dadd_rn(incl, y);
      }
      __syncthreads();
      if ((t & 31) == 31) red[t >> 5] = incl;
      __syncthreads();
      double before = carry;
      for (int w = 0; w < (t >> 5); w++) before = __dadd_rn(before, red[w]);
      for (int w = 0; w < NW; w++) carry = __dadd_rn(carry, red[w]);
      // the sum before the thread's own entries
      const double y = __shfl_up_sync(0xffffffffu, incl, 1);
      if (t & 31) before = __dadd_rn(before, y);
      double w = before;
      uint32_t hit = 0xffffffffu, end = 0;
#pragma unroll
      for (int j = 15; j >= 0; j--)
        if (pv[j] > 0 && end == 0) end = l + j + 1;
      for (int j = 0; j < 16; j++) {
        if (!(pv[j] > 0)) continue;
        w = __dadd_rn(w, pv[j]);
        if (hit == 0xffffffffu && r <= w) hit = l + j;
      }
      if (hit != 0xffffffffu) atomicMin(&pick, hit);
      if (end) atomicMax(&last, end);
    }
    __syncthreads();
    uint64_t idx = pick != 0xffffffffu ? pick : last ? last - 1 : 0;
    if (a.nz.pmeas != 0)
      for (int q = 0; q < a.n; q++) {
        x = xs_step(x);
        if (xs_value(x) < a.nz.pmeas) idx ^= uint64_t(1) << q;
      }
    if (t == 0) a.out_idx[shot] = idx;
    for (int b = t; b < a.ncbits; b += NT) a.out_bits[shot * (uint64_t)a.ncbits + b] = bits[b];
    __syncthreads();
  }
}

// xorshift32 as a linear map over GF(2)^32: col[k] = image of bit k
struct Jump {
  uint32_t col[32];
  static uint32_t step(uint32_t s) {
    s ^= s << 13;
    s ^= s >> 17;
    return s ^ (s << 5);
  }
  uint32_t apply(uint32_t v) const {
    uint32_t o = 0;
    for (int k = 0; k < 32; k++)
      if ((v >> k) & 1) o ^= col[k];
    return o;
  }
};
Jump jump_power(uint64_t d) {
  Jump step, acc;
  for (int k = 0; k < 32; k++) {
    step.col[k] = Jump::step(1u << k);
    acc.col[k] = 1u << k;
  }
  if (d <= 64) {  // (few steps are cheaper than their squares)
    for (; d; d--)
      for (int k = 0; k < 32; k++) acc.col[k] = Jump::step(acc.col[k]);
    return acc;
  }
  while (d) {
    if (d & 1) {
      Jump t;
      for (int k = 0; k < 32; k++) t.col[k] = step.apply(acc.col[k]);
      acc = t;
    }
    Jump sq;
    for (int k = 0; k < 32; k++) sq.col[k] = step.apply(step.col[k]);
    step = sq;
    d >>= 1;
  }
  return acc;
}

// Draws that ops[b, e) make per shot when that number does not depend on
// outcomes (no draw inside an if body), else -1.  Also lowers the ops to the
// device form.
int64_t lower_shots(const ket_op* ops, size_t b, size_t e, const ket_noise& nz, bool in_if, std::vector<TOp>& out) {
  int64_t draws = 0;
  for (size_t i = b; i < e; i++) {
    const ket_op& o = ops[i];
    TOp t;
    memset(&t, 0, sizeof(t));
    t.kind = o.kind;
    for (int j = 0; j < 4 && j < o.nq; j++) t.q[j] = o.q[j];
    t.mat = (int32_t)o.mat;
    t.k = o.nq;
    int64_t d = 0;
    bool noisy = false;
    switch (o.kind) {
      case KET_OP_SINGLE: noisy = nz.p1 != 0; break;
      case KET_OP_CNOT: case KET_OP_CONTROLLED: case KET_OP_SWAP: case KET_OP_TWO: noisy = nz.p2 != 0; break;
      case KET_OP_UNITARY: if (o.nq > 4) return -1; break;
      case KET_OP_MEASURE: d = 1 + (nz.pmeas != 0 ? 1 : 0); break;
      case KET_OP_RESET: d = 1; break;
      case KET_OP_IF: {
        out.push_back(t);
        const size_t at = out.size() - 1;
        const int64_t inner = lower_shots(ops, i + 1, i + 1 + o.q[3], nz, true, out);
        if (inner != 0) return -1;  // a body that draws makes the draw count depend on outcomes
        out[at].q[3] = (int32_t)(out.size() - at - 1);
        i += o.q[3];
        continue;
      }
      default: break;
    }
    out.push_back(t);
    if (noisy) {
      TOp z;
      memset(&z, 0, sizeof(z));
      z.kind = o.kind == KET_OP_SINGLE ? T_NOISE1 : T_NOISE2;
      z.q[0] = o.q[0];
      z.q[1] = o.q[1];
      out.push_back(z);
      d = 1;
    }
    if (in_if && d) return -1;
    draws += d;
  }
  return draws;
}

// What a segment may hold of shared memory beside the state.
struct SCaps {
  int rounds, gates, slots, draws;
};
SCaps shot_caps(int nt) { return nt <= 64 ? SCaps{32, 64, 64, 128} : SCaps{64, 192, 192, 1024}; }

// Threads of a CTA: 16 amplitudes each.
int shot_threads(int ne) { return std::max(32, 1 << (ne - kShotBits)); }

// The plan all shots of a call share.
struct ShotPlan {
  int ne = 0, nt = 0;
  std::vector<SStep> steps;
  std::vector<SSeg> segs;
  std::vector<SChunk> chunks;
  std::vector<SRound> rounds;
  std::vector<SGate> gates;
  std::vector<double> mats;    // 8 doubles a slot
  std::vector<SNoise> noise;
  std::vector<int64_t> rows;   // draw index (0-based) of each jump row
  SCaps used = {0, 0, 0, 0};
  int last_gap = 0;
  uint16_t acol[kRoundQubits];
};

class ShotPlanner {
 public:
  ShotPlanner(ShotPlan& p, int n, const std::vector<TOp>& ops, const std::vector<double>& mats)
      : P(p), n_(n), ops_(ops), mats_(mats), caps_(shot_caps(p.nt)), rp_(p.ne) {}

  void run(size_t b, size_t e, bool in_if) {
    for (size_t i = b; i < e; i++) {
      const TOp& o = ops_[i];
      const int* q = o.q;
      switch (o.kind) {
        case KET_OP_SINGLE: gate(q[0], nullptr, 0, false, (int)i); break;
        case KET_OP_CONTROLLED: gate(q[1], q, 1, false, (int)i); break;
        case KET_OP_CNOT:
          if (in_if) gate(q[1], q, 1, true, (int)i);
          else rp_.cnot(q[0], q[1]);
          break;
        case KET_OP_TOFFOLI: gate(q[2], q, 2, true, (int)i); break;
        case KET_OP_SWAP:
          if (!in_if) { rp_.swap(q[0], q[1]); break; }
          x1(q[0], q[1], (int)i);  // an if-body runs in some shots only: its swaps move data
          x1(q[1], q[0], (int)i);
          x1(q[0], q[1], (int)i);
          break;
        case KET_OP_CSWAP: {  // cswap(c, a, b) = cnot(b, a) toffoli(c, a, b) cnot(b, a)
          const int cs[2] = {q[0], q[1]};
          if (in_if) x1(q[2], q[1], (int)i); else rp_.cnot(q[2], q[1]);
          gate(q[2], cs, 2, true, (int)i);
          if (in_if) x1(q[2], q[1], (int)i); else rp_.cnot(q[2], q[1]);
          break;
        }
        case KET_OP_TWO: dense(q, 2, nullptr, 0, (int)i); break;
        case KET_OP_CSRSWAP: dense(q + 1, 2, q, 1, (int)i); break;
        case KET_OP_UNITARY:
          if (o.k == 1) gate(q[0], nullptr, 0, false, (int)i);
          else dense(q, o.k, nullptr, 0, (int)i);
          break;
        case T_NOISE1: case T_NOISE2: {
          if (ndraws_ == caps_.draws) end_segment();
          SNoise z = {rp_.col[q[0]], rp_.row[q[0]], 0, 0, o.kind == T_NOISE2};
          if (z.two) { z.mb = rp_.col[q[1]]; z.rb = rp_.row[q[1]]; }
          noise_.push_back(z);
          ndraws_++;
          break;
        }
        case KET_OP_MEASURE: case KET_OP_RESET: {
          end_segment();
          SStep s = {};
          s.kind = o.kind == KET_OP_MEASURE ? ST_MEASURE : ST_RESET;
          s.a = o.kind == KET_OP_MEASURE ? q[1] : -1;
          s.c = gap();
          s.b = (int)P.rows.size();
          if (!s.c) P.rows.push_back(draw_);
          draw_ += o.kind == KET_OP_MEASURE && flips_ ? 2 : 1;
          if (q[0] >= 0 && q[0] < n_) { s.r = rp_.row[q[0]]; s.m = rp_.col[q[0]]; }
          P.steps.push_back(s);
          break;
        }
        case KET_OP_IF: {
          end_segment();
          const size_t at = P.steps.size();
          P.steps.push_back(SStep{ST_IF, q[0], q[1], q[2], 0, 0, 0});
          run(i + 1, i + 1 + q[3], true);
          end_segment();
          P.steps[at].d = (int)(P.steps.size() - at - 1);
          i += q[3];
          break;
        }
        default: break;  // barrier
      }
    }
  }
  void finish() {
    end_segment();
    std::copy(rp_.col, rp_.col + kRoundQubits, P.acol);
    P.last_gap = gap();
    if (!P.last_gap) P.rows.push_back(draw_);
  }
  void set_flips(bool f) { flips_ = f; }

 private:
  ShotPlan& P;
  int n_;
  const std::vector<TOp>& ops_;
  const std::vector<double>& mats_;
  SCaps caps_;
  RoundPlan rp_;
  std::vector<SNoise> noise_;          // of the segment under construction
  std::vector<int> dpos_;              // per gate of it, in program order
  int ndraws_ = 0;
  int64_t draw_ = 0;                   // first draw of the segment
  int64_t last_draw_ = -1;             // of the last measurement or reset
  bool flips_ = false;

  // Steps from there to the next draw, which becomes the last; 0 where a jump is the
  // shorter way (a row from memory, 32 columns: as long as some 30 steps).
  int gap() {
    const int64_t g = draw_ - last_draw_;
    last_draw_ = draw_;
    return g <= 24 ? (int)g : 0;
  }
  void x1(int c, int t, int op) { gate(t, &c, 1, true, op); }
  static int slots_of(int k) { return k <= 1 ? 1 : 1 << (2 * k - 2); }
  void room(int slots) {
    // (a round under construction may hold kRoundGates gates that are not in rp_.gates yet)
    if ((int)dpos_.size() + 1 > caps_.gates - 1 || (int)rp_.rounds.size() + 2 > caps_.rounds || slots_ + slots > caps_.slots)
      end_segment();
    slots_ += slots;
  }
  int slots_ = 0;
  void gate(int q, const int* cs, int nc, bool x, int op) {
    room(x ? 0 : 1);
    rp_.gate(q, cs, nc, x, op);
    dpos_.push_back(ndraws_);
  }
  void dense(const int* qs, int k, const int* cs, int nc, int op) {
    room(slots_of(k));
    rp_.dense(qs, k, cs, nc, op);
    dpos_.push_back(ndraws_);
  }
  void end_segment() {
    rp_.close();
    if (rp_.rounds.empty() && ndraws_ == 0) return;
    SSeg S = {};
    const int slot0 = (int)(P.mats.size() / 8);
    S.nrounds = (int)rp_.rounds.size();
    S.ngates = (int)rp_.gates.size();
    int nslots = 0;
    for (const Round& r : rp_.rounds)
      for (int g = r.gate0; g < r.gate0 + r.ngates; g++) nslots += rp_.gates[g].x ? 0 : r.dense ? slots_of(r.k) : 1;
    if (P.chunks.empty() || P.chunks.back().nrounds + S.nrounds > caps_.rounds ||
        P.chunks.back().ngates + S.ngates > caps_.gates || P.chunks.back().nslots + nslots > caps_.slots)
      P.chunks.push_back(SChunk{(int)P.rounds.size(), 0, (int)P.gates.size(), 0, slot0, 0});
    SChunk& C = P.chunks.back();
    S.chunk = (int)P.chunks.size() - 1;
    S.round0 = C.nrounds;
    S.gate0 = C.ngates;
    S.slot0 = C.nslots;
    C.nrounds += S.nrounds;
    C.ngates += S.ngates;
    C.nslots += nslots;
    int slot = 0;
    for (const Round& r : rp_.rounds) {
      SRound Q = {};
      std::copy(r.slot, r.slot + 16, Q.slot);
      std::copy(r.m, r.m + 4, Q.m);
      std::copy(r.rd, r.rd + 4, Q.rd);
      std::copy(r.piv, r.piv + 4, Q.piv);
      Q.k = r.k;
      Q.dense = r.dense;
      Q.ngates = (uint16_t)r.ngates;
      Q.gate0 = r.gate0;
      P.rounds.push_back(Q);
      for (int g = r.gate0; g < r.gate0 + r.ngates; g++) {
        const RoundGate& o = rp_.gates[g];
        SGate G = {};
        G.bit = o.bit;
        G.nc = o.nc;
        G.r = o.r;
        G.m = o.m;
        std::copy(o.cj, o.cj + 2, G.cj);
        std::copy(o.rc, o.rc + 2, G.rc);
        G.slot = slot;
        G.dpos = dpos_[g];
        if (o.x) {
          G.form = SF_X;
        } else {
          const int ns = r.dense ? slots_of(r.k) : 1;
          std::vector<double> m(8 * (size_t)ns, 0.0);
          matrix(ops_[o.op], r.dense ? r.k : 1, m.data());
          G.form = r.dense ? SF_GEN : form_of(m.data());
          P.mats.insert(P.mats.end(), m.begin(), m.end());
          slot += ns;
        }
        P.gates.push_back(G);
      }
    }
    S.noise0 = (int)P.noise.size();
    S.ndraws = ndraws_;
    P.noise.insert(P.noise.end(), noise_.begin(), noise_.end());
    S.per = (ndraws_ + P.nt - 1) / P.nt;
    S.jump0 = (int)P.rows.size();
    for (int d = 0; d < ndraws_; d += std::max(S.per, 1)) P.rows.push_back(draw_ + d);
    draw_ += ndraws_;
    P.used.rounds = std::max(P.used.rounds, C.nrounds);
    P.used.gates = std::max(P.used.gates, C.ngates);
    P.used.slots = std::max(P.used.slots, C.nslots);
    P.used.draws = std::max(P.used.draws, S.ndraws);
    SStep st = {};
    st.kind = ST_SEG;
    st.a = (int)P.segs.size();
    P.segs.push_back(S);
    P.steps.push_back(st);
    rp_.rounds.clear();
    rp_.gates.clear();
    noise_.clear();
    dpos_.clear();
    ndraws_ = slots_ = 0;
  }
  void matrix(const TOp& o, int k, double* m) const {
    if (o.kind == KET_OP_CSRSWAP) {  // applyCsrSwap (statevector.ts:177-207): sqrt(iSWAP)
      const double sq2 = 1.0 / 1.4142135623730951;  // 1 / Math.sqrt(2)
      m[0] = m[30] = 1.0;
      m[2 * 5] = m[2 * 10] = sq2;
      m[2 * 6 + 1] = m[2 * 9 + 1] = sq2;
      return;
    }
    std::copy(mats_.begin() + 2 * (size_t)o.mat, mats_.begin() + 2 * ((size_t)o.mat + (size_t(1) << (2 * k))), m);
  }
  static uint8_t form_of(const double* m) {
    if (m[2] == 0 && m[3] == 0 && m[4] == 0 && m[5] == 0) return SF_DIAG;
    if (m[1] == 0 && m[3] == 0 && m[5] == 0 && m[7] == 0) return SF_REAL;
    if (m[1] == 0 && m[2] == 0 && m[4] == 0 && m[7] == 0) return SF_RX;
    return SF_GEN;
  }
};

template <typename R, int NT>
cudaError_t launch_shots_t(const SArgs& a, size_t smem, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(k_shots<R, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  uint64_t grid = a.shots;
  if (grid > (uint64_t)num_sms()) {
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_shots<R, NT>, NT, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    grid = std::min<uint64_t>(grid, (uint64_t)per_sm * num_sms());
  }
  k_shots<R, NT><<<(unsigned)grid, NT, smem, s>>>(a);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_shots(const SArgs& a, int nt, size_t smem, cudaStream_t s) {
  switch (nt) {
    case 32: return launch_shots_t<R, 32>(a, smem, s);
    case 64: return launch_shots_t<R, 64>(a, smem, s);
    case 128: return launch_shots_t<R, 128>(a, smem, s);
    case 256: return launch_shots_t<R, 256>(a, smem, s);
    default: return launch_shots_t<R, 512>(a, smem, s);
  }
}

// Largest state the batched kernel holds in shared memory.
int batched_max_qubits(int precision) { return precision == KET_C64 ? 13 : 12; }

int g_pershot_path = 0;  // ket_debug_pershot_path: 0 automatic, 1 host-driven only, 2 batched only

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// All shots in one launch: shot i starts from the stream state after i * D
// draws (D = draws per shot), found by the GF(2) jump of xorshift32.
int run_batched(ket_state* st, const std::vector<TOp>& tops, int64_t draws, const std::vector<double>& mats,
                uint64_t init, const ket_noise& nz, size_t shots, uint32_t* prng, int ncbits, uint64_t* out_idx,
                uint8_t* out_bits) {
  ket_ctx* c = st->ctx;
  ShotPlan P;
  P.ne = std::max(st->n, kShotMinQubits);
  P.nt = shot_threads(P.ne);
  ShotPlanner planner(P, st->n, tops, mats);
  planner.set_flips(nz.pmeas != 0);
  planner.run(0, tops.size(), false);
  planner.finish();
  // jump rows: the step's power that leads from a shot's start to the row's draw
  std::vector<uint32_t> jump(32 * P.rows.size());
  {
    Jump J = jump_power(0);
    int64_t at = 0;
    std::vector<size_t> by(P.rows.size());
    for (size_t i = 0; i < by.size(); i++) by[i] = i;
    std::stable_sort(by.begin(), by.end(), [&](size_t x, size_t y) { return P.rows[x] < P.rows[y]; });
    for (size_t i : by) {
      for (; at < P.rows[i] + 1; at++)
        for (int k = 0; k < 32; k++) J.col[k] = Jump::step(J.col[k]);
      std::copy(J.col, J.col + 32, jump.begin() + 32 * i);
    }
  }
  // the shots' start states, a byte of the state at a time (an entry is the XOR of two
  // filled before it: a jump an entry took 30 us, more than a small call's kernel)
  const Jump J = jump_power((uint64_t)draws);
  uint32_t byte_img[4][256];
  for (int b = 0; b < 4; b++) {
    byte_img[b][0] = 0;
    for (int v = 1; v < 256; v++) byte_img[b][v] = byte_img[b][v & (v - 1)] ^ J.col[8 * b + __builtin_ctz(v)];
  }
  std::vector<uint32_t> start(shots);
  uint32_t s = *prng ? *prng : 1u;
  for (size_t i = 0; i < shots; i++) {
    start[i] = s;
    s = byte_img[0][s & 255] ^ byte_img[1][(s >> 8) & 255] ^ byte_img[2][(s >> 16) & 255] ^ byte_img[3][s >> 24];
  }
  size_t total = 0;
  struct Part { const void* src; size_t bytes, at; };
  std::vector<Part> parts;
  auto place = [&](size_t bytes) {
    const size_t at = total;
    total += align256(std::max<size_t>(bytes, 1));
    return at;
  };
  auto part = [&](const auto& v) {
    parts.push_back(Part{v.data(), v.size() * sizeof(v[0]), place(v.size() * sizeof(v[0]))});
    return parts.back().at;
  };
  const size_t o_steps = part(P.steps), o_segs = part(P.segs), o_chunks = part(P.chunks), o_rounds = part(P.rounds), o_gates = part(P.gates),
               o_mats = part(P.mats), o_noise = part(P.noise), o_jump = part(jump), o_start = part(start);
  const size_t image = total, o_idx = place(8 * shots), o_bits = place(shots * ncbits);
  void* scr;
  TRY(ctx_scratch(c, total, &scr));
  char* base = (char*)scr;
  std::vector<unsigned char> img(image, 0);
  for (const Part& p : parts)
    if (p.bytes) memcpy(img.data() + p.at, p.src, p.bytes);
  cudaError_t e = cudaMemcpyAsync(base, img.data(), image, cudaMemcpyHostToDevice, c->stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(trajectory inputs)");
  c->h2d_bytes += image;
  SArgs a;
  memset(&a, 0, sizeof(a));
  a.steps = (const SStep*)(base + o_steps);
  a.segs = (const SSeg*)(base + o_segs);
  a.chunks = (const SChunk*)(base + o_chunks);
  a.rounds = (const SRound*)(base + o_rounds);
  a.gates = (const SGate*)(base + o_gates);
  a.mats = (const double2*)(base + o_mats);
  a.noise = (const SNoise*)(base + o_noise);
  a.jump = (const uint32_t*)(base + o_jump);
  a.start = (const uint32_t*)(base + o_start);
  a.out_idx = (uint64_t*)(base + o_idx);
  a.out_bits = (uint8_t*)(base + o_bits);
  a.shots = shots;
  a.init = init;
  a.nz = nz;
  a.nsteps = (int)P.steps.size();
  a.n = st->n;
  a.ne = P.ne;
  a.ncbits = ncbits;
  a.last_row = (int)P.rows.size() - 1;
  a.last_gap = P.last_gap;
  std::copy(P.acol, P.acol + kRoundQubits, a.acol);
  size_t smem = (st->precision == KET_C64 ? sizeof(float2) : sizeof(double2)) << P.ne;
  auto area = [&](size_t bytes) {
    const size_t at = smem;
    smem += (bytes + 15) & ~size_t(15);
    return (int)at;
  };
  a.off_mats = area(64 * (size_t)P.used.slots);
  a.off_rounds = area(sizeof(SRound) * P.used.rounds);
  a.off_gates = area(sizeof(SGate) * P.used.gates);
  a.off_events = area(sizeof(SEvent) * P.used.draws);
  a.off_red = area(8 * 32);
  a.off_bits = area(ncbits);
  prof_begin(c);
  e = st->precision == KET_C64 ? launch_shots<float>(a, P.nt, smem, c->stream)
                               : launch_shots<double>(a, P.nt, smem, c->stream);
  prof_end(c, PK_BATCH);
  if (e != cudaSuccess) return cuda_fail(e, "trajectory launch");
  e = cudaMemcpyAsync(out_idx, a.out_idx, 8 * shots, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess && ncbits)
    e = cudaMemcpyAsync(out_bits, a.out_bits, shots * (size_t)ncbits, cudaMemcpyDeviceToHost, c->stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(trajectory outputs)");
  c->d2h_bytes += 8 * shots + shots * (size_t)ncbits;
  TRY(ctx_wait(c));
  *prng = s;
  return KET_OK;
}

// The op list's structure: every if-body lies inside its parent range;
// classical operands are in range.  Gates are collected for lower_ops.
int check_range(const ket_op* ops, size_t b, size_t e, int n, int ncbits, std::vector<ket_op>& gates) {
  for (size_t i = b; i < e; i++) {
    const ket_op& o = ops[i];
    switch (o.kind) {
      case KET_OP_MEASURE:
        if (o.nq != 2) return fail(KET_ERR_TYPE, "measure: nq must be 2 (qubit, classical bit)");
        if (o.q[1] < -1 || o.q[1] >= ncbits) return fail(KET_ERR_RANGE, "measure: classical bit out of range");
        break;
      case KET_OP_RESET:
        if (o.nq != 1) return fail(KET_ERR_TYPE, "reset: nq must be 1");
        if (o.q[0] < 0 || o.q[0] >= n)
          return fail(KET_ERR_RANGE, "qubit index " + std::to_string(o.q[0]) + " is out of range for a " +
                                         std::to_string(n) + "-qubit circuit");
        break;
      case KET_OP_IF: {
        if (o.nq != 4) return fail(KET_ERR_TYPE, "if: nq must be 4 (first bit, size, value, body length)");
        const int first = o.q[0], size = o.q[1], len = o.q[3];
        if (size < 0 || size > 31) return fail(KET_ERR_UNSUPPORTED, "if: registers of more than 31 bits");
        if (size > 0 && (first < 0 || first + size > ncbits)) return fail(KET_ERR_RANGE, "if: register out of range");
        if (len < 0 || i + 1 + (size_t)len > e) return fail(KET_ERR_TYPE, "if: body runs past its enclosing list");
        TRY(check_range(ops, i + 1, i + 1 + len, n, ncbits, gates));
        i += len;
        break;
      }
      default:
        gates.push_back(o);
        break;
    }
  }
  return KET_OK;
}

struct Runner {
  ket_state* st = nullptr;
  const ket_op* ops = nullptr;
  std::vector<double> mats;  // the caller's matrices, then X, Y, Z (gates.ts:15-17)
  size_t nmat = 0;
  int64_t pauli[4] = {0, 0, 0, 0};
  ket_noise nz{};
  uint32_t s = 1;
  std::vector<uint8_t> bits;
  std::vector<ket_op> seg;
  ket_exec_opts opts{};

  // makePrng's generator (circuit.ts:813-819)
  double draw() {
    s ^= s << 13;
    s ^= s >> 17;
    s ^= s << 5;
    return (double)s / 4294967296.0;
  }
  int flush() {
    if (seg.empty()) return KET_OK;
    const int rc = ket_apply_ops(st, seg.data(), seg.size(), mats.data(), nmat, &opts);
    seg.clear();
    return rc;
  }
  void push_pauli(int which, int q) {
    ket_op o;
    memset(&o, 0, sizeof(o));
    o.kind = KET_OP_SINGLE;
    o.nq = 1;
    o.q[0] = q;
    o.mat = pauli[which];
    seg.push_back(o);
  }
  // dep1 / dep2 (circuit.ts:289-304): which Paulis a draw selects
  void dep1(int q) {
    const double r = draw();
    if (r >= nz.p1) return;
    const double u = r / nz.p1;
    push_pauli(u < 1.0 / 3 ? 1 : u < 2.0 / 3 ? 2 : 3, q);
  }
  void dep2(int a, int b) {
    static const int pairs[15][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 0}, {1, 1}, {1, 2}, {1, 3}, {2, 0},
                                     {2, 1}, {2, 2}, {2, 3}, {3, 0}, {3, 1}, {3, 2}, {3, 3}};
    const double r = draw();
    if (r >= nz.p2) return;
    int k = (int)std::floor(r / nz.p2 * 15);
    if (k > 14) k = 14;
    if (pairs[k][0]) push_pauli(pairs[k][0], a);
    if (pairs[k][1]) push_pauli(pairs[k][1], b);
  }
  // collapseQubit (circuit.ts:55-72); a qubit outside the state reads 0, as
  // the reference's mask then matches no index
  int collapse(int q, int& outcome) {
    TRY(flush());
    const double r = draw();
    double p1 = 0.0;
    const int n = st->n;
    const bool inside = q >= 0 && q < n;
    ket_ctx* c = st->ctx;
    if (inside) {
      const uint64_t half = uint64_t(1) << (n - 1);
      const uint64_t chunk = half > 4096 * 1024 ? (half + 4095) / 4096 : 1024;
      const int nb = (int)((half + chunk - 1) / chunk);
      void* scr;
      TRY(ctx_scratch(c, 8 * (size_t)nb + 64, &scr));
      double* part = (double*)scr;
      double* sum = part + nb;
      prof_begin(c);
      if (st->precision == KET_C64)
        k_prob_one<float><<<nb, KNT, 0, c->stream>>>((const float2*)st->amp, half, q, chunk, part);
      else
        k_prob_one<double><<<nb, KNT, 0, c->stream>>>((const double2*)st->amp, half, q, chunk, part);
      k_sum_in_order<<<1, 32, 0, c->stream>>>(part, nb, sum);
      prof_end(c, PK_READ);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "collapse reduction launch");
      c->d2h_bytes += 8;
      e = cudaMemcpyAsync(&p1, sum, 8, cudaMemcpyDeviceToHost, c->stream);
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(P(q=1))");
      TRY(ctx_wait(c));
    }
    outcome = r < p1 ? 1 : 0;
    const double inv = 1 / std::sqrt(outcome == 1 ? p1 : 1 - p1);
    if (inside) {
      const uint64_t N = uint64_t(1) << n;
      const unsigned grid = (unsigned)std::min<uint64_t>((N + 255) / 256, 148 * 16);
      prof_begin(c);
      if (st->precision == KET_C64)
        k_collapse<float><<<grid, 256, 0, c->stream>>>((float2*)st->amp, N, q, outcome, inv);
      else
        k_collapse<double><<<grid, 256, 0, c->stream>>>((double2*)st->amp, N, q, outcome, inv);
      prof_end(c, PK_GATE);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "collapse launch");
    }
    return KET_OK;
  }
  // applyOps (circuit.ts:169-207) over ops[b, e)
  int run(size_t b, size_t e) {
    for (size_t i = b; i < e; i++) {
      const ket_op& o = ops[i];
      switch (o.kind) {
        case KET_OP_SINGLE:
          seg.push_back(o);
          if (nz.p1 != 0) dep1(o.q[0]);
          break;
        case KET_OP_CNOT: case KET_OP_CONTROLLED: case KET_OP_SWAP: case KET_OP_TWO:
          seg.push_back(o);
          if (nz.p2 != 0) dep2(o.q[0], o.q[1]);
          break;
        case KET_OP_BARRIER: break;
        case KET_OP_MEASURE: {
          int outcome;
          TRY(collapse(o.q[0], outcome));
          const int reported = (nz.pmeas != 0 && draw() < nz.pmeas) ? 1 - outcome : outcome;
          if (o.q[1] >= 0) bits[o.q[1]] = (uint8_t)reported;
          break;
        }
        case KET_OP_RESET: {
          int outcome;
          TRY(collapse(o.q[0], outcome));
          if (outcome == 1) push_pauli(1, o.q[0]);
          break;
        }
        case KET_OP_IF: {
          // cregValue (circuit.ts:164-166): the register as a little-endian integer
          int v = 0;
          for (int k = 0; k < o.q[1]; k++)
            if (bits[o.q[0] + k]) v |= 1 << k;
          if (v == o.q[2]) TRY(run(i + 1, i + 1 + o.q[3]));
          i += o.q[3];
          break;
        }
        default:  // toffoli, cswap, csrswap, unitary: no noise (circuit.ts:178-183)
          seg.push_back(o);
          break;
      }
    }
    return KET_OK;
  }
};

}  // namespace

extern "C" {

int ket_debug_pershot_path(int mode) {
  if (mode < 0 || mode > 2) return fail(KET_ERR_TYPE, "mode must be 0, 1 or 2");
  g_pershot_path = mode;
  return KET_OK;
}

int ket_run_shots(ket_state* st, const ket_op* ops, size_t nops, const double* mats, size_t nmat,
                  const ket_noise* noise, uint64_t init, size_t shots, uint32_t* prng_state, int ncbits,
                  uint64_t* out_idx, uint8_t* out_bits) {
  if (!st) return fail(KET_ERR_TYPE, "null state");
  if (nops && !ops) return fail(KET_ERR_TYPE, "null op list");
  if (!prng_state) return fail(KET_ERR_TYPE, "null prng state");
  if (ncbits < 0) return fail(KET_ERR_TYPE, "negative classical bit count");
  if (shots && !out_idx) return fail(KET_ERR_TYPE, "null output");
  if (shots && ncbits && !out_bits) return fail(KET_ERR_TYPE, "null classical-bit output");
  if (nmat && !mats) return fail(KET_ERR_TYPE, "null matrix buffer");
  if (init >> st->n) return fail(KET_ERR_RANGE, "initial index out of range");
  cudaSetDevice(st->ctx->device);
  // validate everything before touching the state
  std::vector<ket_op> gates;
  TRY(check_range(ops, 0, nops, st->n, ncbits, gates));
  {
    std::vector<Gate> lowered;
    std::string err;
    const int rc = lower_ops(st->n, gates.data(), gates.size(), mats, nmat, true, lowered, err);
    if (rc) return fail(rc, err);
  }
  const ket_noise nz0 = noise ? *noise : ket_noise{0.0, 0.0, 0.0};
  if (g_pershot_path != 1 && shots > 0 && st->n <= batched_max_qubits(st->precision) && ncbits <= 4096) {
    std::vector<TOp> tops;
    const int64_t op_draws = lower_shots(ops, 0, nops, nz0, false, tops);
    // per shot: the ops' draws, sampleSV's draw and the readout flips' draws
    const int64_t draws = op_draws < 0 ? -1 : op_draws + 1 + (nz0.pmeas != 0 ? st->n : 0);
    bool fits = draws > 0;
    for (const TOp& t : tops) fits = fits && t.mat >= -1;
    if (fits) {
      const std::vector<double> tm(mats, mats + 2 * nmat);
      return run_batched(st, tops, draws, tm, init, nz0, shots, prng_state, ncbits, out_idx, out_bits);
    }
  }
  if (g_pershot_path == 2) return fail(KET_ERR_UNSUPPORTED, "trajectories not batchable (state size or draws inside if)");
  Runner R;
  R.st = st;
  R.ops = ops;
  R.mats.assign(mats, mats + 2 * nmat);
  static const double P[3][8] = {{0, 0, 1, 0, 1, 0, 0, 0},     // X
                                 {0, 0, 0, -1, 0, 1, 0, 0},    // Y
                                 {1, 0, 0, 0, 0, 0, -1, 0}};   // Z
  for (int k = 0; k < 3; k++) {
    R.pauli[k + 1] = (int64_t)(R.mats.size() / 2);
    R.mats.insert(R.mats.end(), P[k], P[k] + 8);
  }
  R.nmat = R.mats.size() / 2;
  if (noise) R.nz = *noise;
  R.s = *prng_state ? *prng_state : 1u;
  R.bits.assign((size_t)ncbits, 0);
  ket_exec_opts_default(&R.opts);
  R.opts.prune = 1;
  for (size_t shot = 0; shot < shots; shot++) {
    TRY(ket_state_set_basis(st, init));
    std::fill(R.bits.begin(), R.bits.end(), 0);
    TRY(R.run(0, nops));
    TRY(R.flush());
    // sampleSV (circuit.ts:75-83) then the readout flips (:3466-3470)
    const double r = R.draw();
    uint64_t idx = 0;
    TRY(sample_indices(st, &r, 1, 0.0, &idx));
    if (R.nz.pmeas != 0)
      for (int q = 0; q < st->n; q++)
        if (R.draw() < R.nz.pmeas) idx ^= uint64_t(1) << q;
    out_idx[shot] = idx;
    if (ncbits) memcpy(out_bits + shot * (size_t)ncbits, R.bits.data(), (size_t)ncbits);
  }
  *prng_state = R.s;
  return KET_OK;
}

}  // extern "C"
