// batch_vqe.cu -- vqe() energies of many parameterised circuits of uneven
// width in one persistent launch (ket_batch_vqe).
//
// The reference evaluates each energy on its own: vqe() (algorithms.ts:301-336)
// re-simulates the circuit per Pauli term, and a parameter sweep calls it once
// per parameter vector.  Here a batch names circuit templates (an op list whose
// parametric ops are bound to parameters, the same bindings as the adjoint
// gradient) and instances (a template and a parameter vector).  A persistent
// grid pulls work from a queue, largest first; one CTA, of 128 to 512 threads by the
// amplitudes it holds, runs one instance with its whole state in shared memory (up to 13
// qubits, 128 KB), or, where not all would run at once, a pack of up to 32 instances of
// one template of fewer qubits:
//   * |0...0>, then the ops in order, with the reference's per-gate pruning
//     (accumulate(), statevector.ts:19-27) after each matrix op.  CNOTs and
//     swaps are relabellings, and one-qubit gates run in rounds of up to 16 on
//     amplitudes held in registers (rounds.h).  Parametric matrices are formed on
//     the device from the instance's parameters with the formulas of gates.ts (Rx,
//     Ry, Rz, U1, Gpi, Gpi2, their controlled forms, Xx, Yy, Zz, Xy);
//   * E = ident + sum_t Re <psi| c_t P_t |psi> over the template's Pauli terms, in
//     physical masks, summed in a fixed order, so results repeat bit for bit.
// The launch (queue reset, kernel) is captured in a CUDA graph that is kept
// and replayed while the batch's shape and buffers stay the same; parameters
// are uploaded to the same addresses before each replay.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "fused_ops.cuh"
#include "launch.h"
#include "pauli_terms.cuh"
#include "read.h"
#include "rounds.h"

namespace ket {
namespace {

constexpr int kVqeMaxQubits = 13;
constexpr int kVqeMinQubits = 4;    // narrower templates get idle qubits: a coset of a round lies in one instance
constexpr int kVqeMaxThreads = 512;
// Threads of a CTA that holds 2^tile amplitudes: 16 amplitudes each, and at least 128 to
// form the matrices.  At 128 registers a thread an SM then has one CTA of 2^13
// amplitudes, two of 2^12 or up to four narrower ones; with 512 threads whatever the tile, an
// SM had one, and 150 instances of 8 qubits ran in two turns (34 us; 24 now).
constexpr int vqe_threads(int tile) { return tile <= 11 ? 128 : 1 << (tile - 4); }
static_assert(vqe_threads(kVqeMaxQubits) == kVqeMaxThreads, "the widest tile");
constexpr int kVqePackBits = 5;     // instances in a pack, at most 32
// What shared memory holds of a template at a time (a chunk): 2x2 matrices (a 4x4
// takes 4), rounds and their gates.
constexpr int kVqeSlots = 512, kVqeRounds = 64, kVqeGates = 256;

// One op of a template after lowering; its matrix is G_fam(scale * theta[param] +
// shift) when fam >= 0, else mats[moff ..].
struct BFactor {
  int16_t fam;
  int16_t two;     // a 4x4
  int32_t param;
  int64_t moff;
  double scale, shift;
};

// One matrix of a template: the product of factors [f0, f0 + nf), the first applied
// first.
struct BMat {
  int32_t f0;
  int16_t nf, two;
  int32_t slot;    // in the template's numbering
};

// Rounds whose matrices are in shared memory together.
struct BChunk {
  int32_t round0, nrounds, gate0, ngates, mat0, nmats, slot0, nslots;
};

struct BRoundGate {
  uint8_t form, bit, nc, pad;  // form: 0 a general 2x2, 1 a real one, 2 X
  uint8_t cj[4];
  uint16_t r, rc[3];
  int32_t slot;
};

struct __align__(16) BRound {
  uint16_t slot[16];
  uint8_t piv[4];
  uint8_t k, two;
  uint16_t r2[2];
  uint16_t ngates;
  int32_t gate0;
};

struct BTmpl {
  int n, lgpack;            // qubits (at least kVqeMinQubits), log2 of the instances in a pack
  int nchunks, ngroups;
  int64_t chunk_first, group_first;
  double ident;
};

struct BItem {
  int tmpl, first, count;   // instances order[first .. first + count)
};

struct BTerm {
  double coeff;             // with the sign of i^ny, and 2 for a pair
  uint32_t zm;              // thread mask | mask over the products' index << 16
  uint32_t pad;
};

struct BArgs {
  const BTmpl* tmpl;
  const BChunk* chunks;
  const BRound* rounds;
  const BRoundGate* gates;
  const BMat* matv;
  const BFactor* factors;
  const double2* mats;
  const PauliTileGroup* groups;
  const BTerm* terms;
  const BItem* items;
  const int* order;
  const double* theta;
  double* energy;
  unsigned int* next;
  int nitems, nparams, tile;  // tile: log2 of the amplitudes a CTA holds
  int slots, rounds_max;      // matrix slots and rounds of the largest chunk
};

// G_fam(a) into m (row-major, 2x2 or 4x4), the formulas of gates.ts.
__device__ void param_matrix(int fam, double a, double2* m) {
  double s, c;
  sincos(0.5 * a, &s, &c);
  const double sq2 = 0.70710678118654752440;
  switch (fam) {
    case KET_PG_RX: case KET_PG_CRX:
      m[0] = make_double2(c, 0); m[1] = make_double2(0, -s); m[2] = make_double2(0, -s); m[3] = make_double2(c, 0);
      return;
    case KET_PG_RY: case KET_PG_CRY:
      m[0] = make_double2(c, 0); m[1] = make_double2(-s, 0); m[2] = make_double2(s, 0); m[3] = make_double2(c, 0);
      return;
    case KET_PG_RZ: case KET_PG_CRZ:
      m[0] = make_double2(c, -s); m[1] = make_double2(0, 0); m[2] = make_double2(0, 0); m[3] = make_double2(c, s);
      return;
    case KET_PG_U1: case KET_PG_CU1: {
      double si, co;
      sincos(a, &si, &co);
      m[0] = make_double2(1, 0); m[1] = make_double2(0, 0); m[2] = make_double2(0, 0); m[3] = make_double2(co, si);
      return;
    }
    case KET_PG_GPI: {
      double si, co;
      sincos(a, &si, &co);
      m[0] = make_double2(0, 0); m[1] = make_double2(co, -si); m[2] = make_double2(co, si); m[3] = make_double2(0, 0);
      return;
    }
    case KET_PG_GPI2: {
      double si, co;
      sincos(a, &si, &co);
      m[0] = make_double2(sq2, 0); m[1] = make_double2(-sq2 * si, -sq2 * co);
      m[2] = make_double2(sq2 * si, -sq2 * co); m[3] = make_double2(sq2, 0);
      return;
    }
    default:
      break;
  }
  for (int k = 0; k < 16; k++) m[k] = make_double2(0, 0);
  if (fam == KET_PG_XX || fam == KET_PG_YY) {
    const double2 ni = make_double2(0, -s);
    const double2 corner = fam == KET_PG_XX ? ni : make_double2(0, s);
    m[0] = m[5] = m[10] = m[15] = make_double2(c, 0);
    m[3] = m[12] = corner;
    m[6] = m[9] = ni;
  } else if (fam == KET_PG_ZZ) {
    m[0] = m[15] = make_double2(c, -s);
    m[5] = m[10] = make_double2(c, s);
  } else {  // XY
    m[0] = m[15] = make_double2(1, 0);
    m[5] = m[10] = make_double2(c, 0);
    m[6] = m[9] = make_double2(0, s);
  }
}

__device__ __forceinline__ double2 cmac(double2 acc, double2 m, double2 x) {
  return make_double2(fma(m.x, x.x, fma(-m.y, x.y, acc.x)), fma(m.x, x.y, fma(m.y, x.x, acc.y)));
}

// accumulate()'s flush: |a|^2 < 1e-14 becomes an exact zero.
__device__ __forceinline__ double2 prune2(double2 v) {
  return norm2_ref(v.x, v.y) < 1e-14 ? make_double2(0.0, 0.0) : v;
}

__device__ __forceinline__ void factor_matrix(const BArgs& a, const BFactor& f, const double* th, double2* m) {
  if (f.fam >= 0) {
    param_matrix(f.fam, f.scale * th[f.param] + f.shift, m);
  } else {
    const int ne = f.two ? 16 : 4;
    for (int e = 0; e < ne; e++) m[e] = a.mats[f.moff + e];
  }
}

__device__ __forceinline__ void copy_words(void* dst, const void* src, int bytes) {
  for (int i = threadIdx.x; i < bytes / 4; i += blockDim.x)
    static_cast<uint32_t*>(dst)[i] = static_cast<const uint32_t*>(src)[i];
}

// The amplitudes j of a thread's coset whose controls all hold.
__device__ __forceinline__ uint32_t controls_ok(const BRoundGate& g, uint32_t base) {
  uint32_t ok = 0xffffu;
  for (int c = 0; c < g.nc; c++) {
    const uint32_t cj = g.cj[c];
    uint32_t p = (__popc(base & g.rc[c]) & 1) ? 0xffffu : 0u;
    p ^= (cj & 1 ? 0xaaaau : 0u) ^ (cj & 2 ? 0xccccu : 0u) ^ (cj & 4 ? 0xf0f0u : 0u) ^ (cj & 8 ? 0xff00u : 0u);
    ok &= p;
  }
  return ok;
}

// A 2x2 on register bit I, then the reference's pruning (by one screen over the
// thread's amplitudes, fused_ops.cuh).  role: the amplitude with the bit clear
// holds logical 1 (rows and columns then trade places: matrix entry e becomes e ^ 3).
template <int K, int I, int FORM>
__device__ __forceinline__ void reg_gate(cpx<double>* v, const double2* M, int role, bool ctl, uint32_t ok) {
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
  prune_slots<double, NS>(v, 1e-14, 1e-7);
}
template <int K, int I>
__device__ __forceinline__ void reg_x(cpx<double>* v, uint32_t ok) {
#pragma unroll
  for (int j = 0; j < (1 << K); j++)
    if (!(j & (1 << I)) && ((ok >> j) & 1)) swap_c(v[j], v[j | 1 << I]);
}

__device__ __forceinline__ void run_round(double2* s, const BRound& R, const BRoundGate* gates, const double2* mats,
                                          int n, int lgpack) {
  constexpr int K = kRoundBits;
  const uint32_t nsub = 1u << (n + lgpack - K);
  for (uint32_t u = threadIdx.x; u < nsub; u += blockDim.x) {
    uint32_t base = u;
#pragma unroll
    for (int i = 0; i < K; i++) base = insert0_32(base, R.piv[i]);
    const uint32_t sb = round_slot(base), inst = base >> n;
    cpx<double> v[1 << K];
    RoundSlots slots;
    slots.read(R.slot);
#pragma unroll
    for (int j = 0; j < (1 << K); j++) {
      const double2 t = s[sb ^ slots(j)];
      v[j] = cpx<double>{t.x, t.y};
    }
    // cosets of zeros stay zeros (most of a state in its first gates)
    if (!__any_sync(__activemask(), !all_zero<double, 1 << K>(v))) continue;
    for (int k = 0; k < R.ngates; k++) {
      const BRoundGate& g = gates[k];
      const uint32_t ok = g.nc ? controls_ok(g, base) : 0xffffu;
      const int role = __popc(base & g.r) & 1;
      const double2* M = mats + 4 * ((g.slot << lgpack) + inst);
      const bool ctl = g.nc != 0;
      switch (g.bit + 4 * g.form) {
#define KET_BIT(I)                                             \
  case I: reg_gate<K, I, 0>(v, M, role, ctl, ok); break;       \
  case 4 + I: reg_gate<K, I, 1>(v, M, role, ctl, ok); break;   \
  case 8 + I: reg_x<K, I>(v, ok); break;
        KET_BIT(0) KET_BIT(1) KET_BIT(2) KET_BIT(3)
#undef KET_BIT
      }
    }
    slots.read(R.slot);
#pragma unroll
    for (int j = 0; j < (1 << K); j++) s[sb ^ slots(j)] = make_double2(v[j].re, v[j].im);
  }
}

// A 4x4 on the two masks of its round.
__device__ __forceinline__ void run_two(double2* s, const BRound& R, const BRoundGate& g, const double2* mats, int n,
                                        int lgpack) {
  const uint32_t nsub = 1u << (n + lgpack - 2);
  for (uint32_t u = threadIdx.x; u < nsub; u += blockDim.x) {
    const uint32_t base = insert0_32(insert0_32(u, R.piv[0]), R.piv[1]);
    if (g.nc && !(controls_ok(g, base) & 1)) continue;
    const uint32_t sb = round_slot(base), l0 = 2 * (__popc(base & R.r2[1]) & 1) + (__popc(base & R.r2[0]) & 1);
    const double2* M = mats + 4 * (g.slot << lgpack) + 16 * (base >> n);
    double2 x[4];
#pragma unroll
    for (int c = 0; c < 4; c++) x[c] = s[sb ^ R.slot[c ^ l0]];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      double2 y = make_double2(0, 0);
#pragma unroll
      for (int c = 0; c < 4; c++) y = cmac(y, M[4 * r + c], x[c]);
      s[sb ^ R.slot[r ^ l0]] = prune2(y);
    }
  }
}

// sum_t Re <psi| c_t P_t |psi> over the 16 amplitudes of thread t, and over the
// pairs it carries (physical masks; amplitude index 16 t + j), of every step-th group
// from `first` on.
__device__ __forceinline__ double thread_energy(const BArgs& a, const double2* s, const BTmpl& T, int t, int first,
                                                int step) {
  double2 v[16];
#pragma unroll
  for (int j = 0; j < 16; j++) v[j] = s[round_slot(16 * t + j)];
  auto coeff = [&](int i) { return a.terms[i].coeff; };
  auto mask = [&](int i) { return a.terms[i].zm; };
  double acc = 0.0;
  PauliTileGroup next = {};
  if (first < T.ngroups) next = a.groups[T.group_first + first];
  for (int k = first; k < T.ngroups; k += step) {
    const PauliTileGroup G = next;
    if (k + step < T.ngroups) next = a.groups[T.group_first + k + step];  // (while this one is worked on)
    if (G.flip == 0) {
      double b[16];
#pragma unroll
      for (int j = 0; j < 16; j++) b[j] = norm2_ref(v[j].x, v[j].y);
      acc += pauli_terms<16>(b, coeff, mask, G.first, G.nterms, t);
      continue;
    }
    // 8 pairs: register index with bit P clear or, of a thread flip, half the pairs
    // by either thread: those with bit 3 clear in the thread whose top bit is clear
    double b[8];
    auto products = [&](auto PP, bool set) {
      constexpr int P = decltype(PP)::value;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int j0 = ((u >> P) << (P + 1)) | (u & ((1 << P) - 1)), j1 = j0 | (1 << P);
        const double2 w = s[round_slot((16 * t + (set ? j1 : j0)) ^ G.flip)];
        const double vr = set ? v[j1].x : v[j0].x, vi = set ? v[j1].y : v[j0].y;
        b[u] = G.odd ? vi * w.x - vr * w.y : vr * w.x + vi * w.y;
      }
    };
    switch (G.top) {
      case 0: products(std::integral_constant<int, 0>(), false); break;
      case 1: products(std::integral_constant<int, 1>(), false); break;
      case 2: products(std::integral_constant<int, 2>(), false); break;
      case 3: products(std::integral_constant<int, 3>(), false); break;
      default: products(std::integral_constant<int, 3>(), ((t >> (G.top - 4)) & 1) && !(G.flip & 8)); break;
    }
    acc += pauli_terms<8>(b, coeff, mask, G.first, G.nterms, t);
  }
  return acc;
}

// Bound: the FP64 pipe (8 FMAs an amplitude and gate).  In place of one pass over
// shared memory and one barrier per op, with one CTA of 8 warps an SM whatever the
// instance's width: 2048 instances of 8 to 13 qubits and 4 layers 2.16 -> 0.41 ms
// (FP64 pipe 31% busy, issue slots 41%; the rest is latency at 16 warps an SM, which
// 128 KB of state allow).
__global__ void __launch_bounds__(kVqeMaxThreads) k_batch_vqe(BArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* s = reinterpret_cast<double2*>(smraw);
  double2* mats = s + (1u << a.tile);
  BRound* rounds = reinterpret_cast<BRound*>(mats + 4 * a.slots);
  BRoundGate* gates = reinterpret_cast<BRoundGate*>(rounds + a.rounds_max);
  __shared__ double red[kVqeMaxThreads / 32], part[kVqeMaxThreads];
  __shared__ int item_sh;
  const int tid = threadIdx.x;
  for (;;) {
    if (tid == 0) item_sh = (int)atomicAdd(a.next, 1u);
    __syncthreads();
    const int it = item_sh;
    if (it >= a.nitems) break;
    const BItem item = a.items[it];
    const BTmpl T = a.tmpl[item.tmpl];
    const int n = T.n, pack = 1 << T.lgpack;
    // a short pack repeats its last instance
    auto instance = [&](int i) { return a.order[item.first + min(i, item.count - 1)]; };
    for (uint32_t i = tid; i < 1u << (n + T.lgpack); i += blockDim.x)
      s[round_slot(i)] = make_double2((i & ((1u << n) - 1)) == 0 ? 1.0 : 0.0, 0.0);
    for (int c = 0; c < T.nchunks; c++) {
      const BChunk C = a.chunks[T.chunk_first + c];
      static_assert(sizeof(BRound) % 4 == 0 && sizeof(BRoundGate) % 4 == 0, "copied as words");
      copy_words(rounds, a.rounds + C.round0, C.nrounds * sizeof(BRound));
      copy_words(gates, a.gates + C.gate0, C.ngates * sizeof(BRoundGate));
      for (int e = tid; e < C.nmats << T.lgpack; e += blockDim.x) {
        const BMat B = a.matv[C.mat0 + (e >> T.lgpack)];
        const int i = e & (pack - 1);
        const double* th = a.theta + (size_t)instance(i) * a.nparams;
        double2 m[16];
        factor_matrix(a, a.factors[B.f0], th, m);
        for (int f = 1; f < B.nf; f++) {
          double2 g[4], p[4];
          factor_matrix(a, a.factors[B.f0 + f], th, g);
#pragma unroll
          for (int r = 0; r < 2; r++)
#pragma unroll
            for (int k = 0; k < 2; k++)
              p[2 * r + k] = cmac(cmac(make_double2(0, 0), g[2 * r], m[k]), g[2 * r + 1], m[2 + k]);
          for (int k = 0; k < 4; k++) m[k] = p[k];
        }
        const int ne = B.two ? 16 : 4;
        double2* dst = mats + 4 * ((B.slot - C.slot0) << T.lgpack) + ne * i;  // (the chunk's gates count from slot0)
        for (int k = 0; k < ne; k++) dst[k] = m[k];
      }
      for (int r = 0; r < C.nrounds; r++) {
        __syncthreads();
        const BRound& R = rounds[r];
        const BRoundGate* G = gates + R.gate0;
        if (R.two) {
          run_two(s, R, *G, mats, n, T.lgpack);
        } else {
          run_round(s, R, G, mats, n, T.lgpack);
        }
      }
      __syncthreads();
    }
    __syncthreads();
    // energies: 2^(n-4) threads an instance, and the CTA's other threads take a share of
    // the flip groups (100 instances of 6 qubits, 400 random strings: a call 571 us
    // by the first threads alone, 390 to 460 so; of 10 qubits 786 and 530)
    const int lgt = n - 4, lgw = n + T.lgpack - 4, slices = (int)blockDim.x >> lgw;
    double e = tid < slices << lgw ? thread_energy(a, s, T, tid & ((1 << lgw) - 1), tid >> lgw, slices) : 0.0;
    if (slices > 1) {  // (a power of two, as 2^lgw is)
      part[tid] = e;
      for (int h = slices >> 1; h > 0; h >>= 1) {
        __syncthreads();
        if (tid < h << lgw) part[tid] += part[tid + (h << lgw)];
      }
      __syncthreads();
      e = tid < 1 << lgw ? part[tid] : 0.0;
    }
    for (int o = 1; o < 32 && o < 1 << lgt; o <<= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lgt <= 5) {
      const int i = tid >> lgt;
      if ((tid & ((1 << lgt) - 1)) == 0 && i < item.count) a.energy[instance(i)] = e + T.ident;
    } else {
      if ((tid & 31) == 0) red[tid >> 5] = e;
      __syncthreads();
      if (tid < item.count) {
        const int nw = 1 << (lgt - 5);
        double sum = 0.0;
        for (int w = 0; w < nw; w++) sum += red[tid * nw + w];
        a.energy[instance(tid)] = sum + T.ident;
      }
    }
    __syncthreads();  // red, item_sh and the state are reused
  }
}

// One op of a template on the host.
struct HOp {
  enum Kind { M1, M2, X, SWAP } kind = M1;
  int q0 = 0, q1 = 0, nc = 0;
  int cs[2] = {0, 0};
  bool diag = false, real = false, dead = false;
  std::vector<BFactor> factors;
};

// Merge an uncontrolled one-qubit gate into the one before it on its qubit where
// no op in between touches the qubit and at most one of the two changes magnitudes
// (the reference prunes between two that do).  The merged gate stands where the
// magnitude-changing one stood.
void fold_ops(std::vector<HOp>& ops) {
  int last[kRoundQubits];
  std::fill(last, last + kRoundQubits, -1);
  for (size_t i = 0; i < ops.size(); i++) {
    HOp& g = ops[i];
    const bool plain = g.kind == HOp::M1 && g.nc == 0;
    if (plain && last[g.q0] >= 0) {
      HOp& p = ops[last[g.q0]];
      if (p.kind == HOp::M1 && p.nc == 0 && (p.diag || g.diag) && p.factors.size() < 64) {
        if (g.diag) {
          p.factors.insert(p.factors.end(), g.factors.begin(), g.factors.end());
          p.real = p.real && g.real;
          g.dead = true;
          continue;
        }
        g.factors.insert(g.factors.begin(), p.factors.begin(), p.factors.end());
        g.real = g.real && p.real;
        p.dead = true;
      }
    }
    last[g.q0] = (int)i;
    if (g.kind == HOp::M2 || g.kind == HOp::SWAP) last[g.q1] = (int)i;
    for (int c = 0; c < g.nc; c++) last[g.cs[c]] = (int)i;
  }
}

// The device form of the templates.
struct BImage {
  std::vector<BTmpl> tmpl;
  std::vector<BChunk> chunks;
  std::vector<BRound> rounds;
  std::vector<BRoundGate> gates;
  std::vector<BMat> matv;
  std::vector<BFactor> factors;
  std::vector<PauliTileGroup> groups;
  std::vector<BTerm> terms;
};

// Lower one template's ops to rounds, and its Pauli terms to physical masks.
// Returns the work of one instance (gates x amplitudes).
int64_t lower_template(std::vector<HOp>& ops, const std::vector<PauliTerm>& terms, BTmpl& T, BImage& im) {
  fold_ops(ops);
  RoundPlan rp(T.n);
  for (size_t i = 0; i < ops.size(); i++) {
    const HOp& o = ops[i];
    if (o.dead) continue;
    switch (o.kind) {
      case HOp::M1: rp.gate(o.q0, o.cs, o.nc, false, (int)i); break;
      case HOp::M2: {
        const int qs[2] = {o.q0, o.q1};
        rp.dense(qs, 2, o.cs, o.nc, (int)i);
        break;
      }
      case HOp::X:
        if (o.nc == 1) rp.cnot(o.cs[0], o.q0);
        else rp.gate(o.q0, o.cs, o.nc, true, (int)i);
        break;
      case HOp::SWAP:
        if (o.nc == 0) {
          rp.swap(o.q0, o.q1);
        } else {  // cswap(c, a, b) = cnot(b, a) toffoli(c, a, b) cnot(b, a)
          const int cs[2] = {o.cs[0], o.q0};
          rp.cnot(o.q1, o.q0);
          rp.gate(o.q1, cs, 2, true, (int)i);
          rp.cnot(o.q1, o.q0);
        }
        break;
    }
  }
  rp.close();
  int64_t work = 0;
  T.chunk_first = (int64_t)im.chunks.size();
  const int room = kVqeSlots >> T.lgpack;
  int slot = 0;
  BChunk C;
  auto new_chunk = [&]() {
    C = BChunk{(int32_t)im.rounds.size(), 0, (int32_t)im.gates.size(), 0, (int32_t)im.matv.size(), 0, slot, 0};
  };
  auto end_chunk = [&]() {
    C.nslots = slot - C.slot0;
    if (C.nrounds) im.chunks.push_back(C);
    new_chunk();
  };
  new_chunk();
  for (const Round& r : rp.rounds) {
    int need = 0;
    for (int k = 0; k < r.ngates; k++) need += rp.gates[r.gate0 + k].x ? 0 : r.dense ? 4 : 1;
    if (slot + need - C.slot0 > room || C.nrounds == kVqeRounds || C.ngates + r.ngates > kVqeGates) end_chunk();
    BRound R = {};
    std::copy(r.slot, r.slot + 16, R.slot);
    std::copy(r.piv, r.piv + 4, R.piv);
    R.k = r.k;
    R.two = r.dense;
    R.r2[0] = r.rd[0];
    R.r2[1] = r.rd[1];
    R.ngates = (uint16_t)r.ngates;
    R.gate0 = C.ngates;
    im.rounds.push_back(R);
    C.nrounds++;
    C.ngates += r.ngates;
    for (int k = 0; k < r.ngates; k++) {
      const RoundGate& g = rp.gates[r.gate0 + k];
      BRoundGate G = {};
      G.form = g.x ? 2 : !r.dense && ops[g.op].real ? 1 : 0;
      G.bit = g.bit;
      G.nc = g.nc;
      G.r = g.r;
      std::copy(g.cj, g.cj + 3, G.cj);
      std::copy(g.rc, g.rc + 3, G.rc);
      G.slot = slot - C.slot0;
      if (!g.x) {
        const std::vector<BFactor>& f = ops[g.op].factors;
        im.matv.push_back(BMat{(int32_t)im.factors.size(), (int16_t)f.size(), (int16_t)r.dense, slot});
        im.factors.insert(im.factors.end(), f.begin(), f.end());
        slot += r.dense ? 4 : 1;
        C.nmats++;
      }
      im.gates.push_back(G);
    }
    work += int64_t(1 + r.ngates) << T.n;
  }
  end_chunk();
  T.nchunks = (int)((int64_t)im.chunks.size() - T.chunk_first);
  // Pauli terms
  std::map<std::pair<uint32_t, int>, std::vector<BTerm>> groups;
  for (const PauliTerm& t : terms) {
    uint32_t flip = 0, z = 0;
    for (int q = 0; q < T.n; q++) {
      if ((t.flip >> q) & 1) flip ^= rp.col[q];
      if ((t.zm >> q) & 1) z ^= rp.row[q];
    }
    // index 16 t + j: j is the register index, whose bit `out` the pairs leave out
    const int top = flip ? 31 - __builtin_clz(flip) : 0, out = flip ? std::min(top, 3) : 4;
    uint32_t zthr = z >> 4, zidx = z & 15u;
    if (top >= 4 && (zidx & 8u) && !(flip & 8u)) zthr ^= 1u << (top - 4);
    if (flip) zidx = ((zidx >> (out + 1)) << out) | (zidx & ((1u << out) - 1));
    const double w = ((t.ny & 3) == 1 || (t.ny & 3) == 2 ? -1.0 : 1.0) * (flip ? 2.0 : 1.0);
    groups[{flip, t.ny & 3}].push_back(BTerm{w * t.coeff, zthr | zidx << 16, 0});
  }
  T.group_first = (int64_t)im.groups.size();
  T.ngroups = 0;
  for (auto& kv : groups) {
    std::vector<BTerm>& v = kv.second;
    std::stable_sort(v.begin(), v.end(), [](const BTerm& x, const BTerm& y) { return (x.zm >> 16) < (y.zm >> 16); });
    for (size_t o = 0; o < v.size(); o += 0xffff) {
      const size_t cnt = std::min<size_t>(0xffff, v.size() - o);
      PauliTileGroup G = {};
      G.flip = kv.first.first;
      G.top = G.flip ? (uint8_t)(31 - __builtin_clz(G.flip)) : 0;
      G.odd = (uint8_t)(kv.first.second & 1);
      G.nterms = (uint16_t)cnt;
      G.first = (int32_t)im.terms.size();
      im.terms.insert(im.terms.end(), v.begin() + o, v.begin() + o + cnt);
      im.groups.push_back(G);
      T.ngroups++;
    }
    work += int64_t(1 + v.size() / 4) << T.n;
  }
  return work;
}

}  // namespace
}  // namespace ket

using namespace ket;

extern "C" int ket_batch_vqe(ket_ctx* c, int ntmpl, const ket_batch_template* tp, const ket_op* ops,
                             const double* mats, size_t nmat, const ket_param_binding* binds, const double* coeffs,
                             const char* pauli, int ninst, const int* inst_tmpl, const double* theta, int nparams,
                             int use_graph, double* energy) {
  if (!c || ntmpl < 0 || ninst < 0 || nparams < 0) return fail(KET_ERR_TYPE, "null context or negative count");
  if (ninst == 0) return KET_OK;
  if (!tp || !ops || !inst_tmpl || !energy || (nparams > 0 && !theta)) return fail(KET_ERR_TYPE, "null argument");
  cudaSetDevice(c->device);
  // ---- templates: validate and encode
  std::vector<std::vector<HOp>> hops(ntmpl);
  std::vector<std::vector<PauliTerm>> hterms(ntmpl);
  BImage im;
  im.tmpl.resize(ntmpl);
  const int64_t csr_off = (int64_t)nmat;  // the csrswap block, appended to the matrices
  for (int j = 0; j < ntmpl; j++) {
    const ket_batch_template& T = tp[j];
    const int n = T.nqubits;
    if (n < 1 || n > kVqeMaxQubits)
      return fail(KET_ERR_UNSUPPORTED, "batch templates take 1.." + std::to_string(kVqeMaxQubits) +
                                           " qubits (one instance's state lives in shared memory)");
    if (T.nops < 0 || T.nbinds < 0 || T.nterms < 0 || T.op_first < 0 || T.bind_first < 0 || T.term_first < 0 ||
        T.pauli_first < 0)
      return fail(KET_ERR_TYPE, "template " + std::to_string(j) + ": negative count or offset");
    if (T.nterms > 0 && (!coeffs || !pauli)) return fail(KET_ERR_TYPE, "null Hamiltonian");
    if (T.nbinds > 0 && !binds) return fail(KET_ERR_TYPE, "null bindings");
    const ket_op* to = ops + T.op_first;
    {  // RangeError / TypeError as the reference's builder (circuit.ts:1113-1146)
      std::vector<Gate> chk;
      std::string err;
      const int rc = lower_ops(n, to, (size_t)T.nops, mats, nmat, true, chk, err);
      if (rc) return fail(rc, "template " + std::to_string(j) + ": " + err);
    }
    std::vector<int> bind_of(T.nops, -1);
    for (int b = 0; b < T.nbinds; b++) {
      const ket_param_binding& pb = binds[T.bind_first + b];
      if (pb.op < 0 || pb.op >= T.nops) return fail(KET_ERR_RANGE, "binding op index out of range");
      if (pb.param < 0 || pb.param >= nparams) return fail(KET_ERR_RANGE, "binding parameter index out of range");
      if (pb.gate < KET_PG_RX || pb.gate > KET_PG_XY) return fail(KET_ERR_TYPE, "unknown parametric gate");
      const int want = (pb.gate >= KET_PG_CRX && pb.gate <= KET_PG_CU1) ? KET_OP_CONTROLLED
                       : pb.gate >= KET_PG_XX                           ? KET_OP_TWO
                                                                        : KET_OP_SINGLE;
      if (to[pb.op].kind != want) return fail(KET_ERR_TYPE, "binding gate does not match the op kind");
      if (bind_of[pb.op] >= 0) return fail(KET_ERR_TYPE, "an op has two bindings");
      bind_of[pb.op] = b;
    }
    BTmpl& B = im.tmpl[j];
    memset(&B, 0, sizeof(B));
    B.n = std::max(n, kVqeMinQubits);
    std::vector<HOp>& out = hops[j];
    for (int k = 0; k < T.nops; k++) {
      const ket_op& op = to[k];
      HOp o;
      int64_t moff = op.mat;
      const int* q = op.q;
      auto controls = [&](std::initializer_list<int> cs) {
        for (int c : cs) o.cs[o.nc++] = c;
      };
      switch (op.kind) {
        case KET_OP_BARRIER: continue;
        case KET_OP_SINGLE: o.q0 = q[0]; break;
        case KET_OP_CONTROLLED: o.q0 = q[1]; controls({q[0]}); break;
        case KET_OP_TWO: o.kind = HOp::M2; o.q0 = q[0]; o.q1 = q[1]; break;
        case KET_OP_CNOT: o.kind = HOp::X; o.q0 = q[1]; controls({q[0]}); break;
        case KET_OP_TOFFOLI: o.kind = HOp::X; o.q0 = q[2]; controls({q[0], q[1]}); break;
        case KET_OP_SWAP: o.kind = HOp::SWAP; o.q0 = q[0]; o.q1 = q[1]; break;
        case KET_OP_CSWAP: o.kind = HOp::SWAP; o.q0 = q[1]; o.q1 = q[2]; controls({q[0]}); break;
        case KET_OP_CSRSWAP:  // sqrt(iSWAP) on (q1, q2) when q0 is set (applyCsrSwap, statevector.ts:177-207)
          o.kind = HOp::M2; o.q0 = q[1]; o.q1 = q[2]; controls({q[0]}); moff = csr_off; break;
        case KET_OP_UNITARY:
          if (op.nq == 1) { o.q0 = q[0]; break; }
          if (op.nq == 2) { o.kind = HOp::M2; o.q0 = q[0]; o.q1 = q[1]; break; }
          return fail(KET_ERR_UNSUPPORTED, "batch templates take unitaries of 1 or 2 qubits");
        default:
          return fail(KET_ERR_UNSUPPORTED, "batch templates take pure gate ops only (no measure, reset or if)");
      }
      if (o.kind == HOp::M1 || o.kind == HOp::M2) {
        BFactor f = {};
        f.fam = -1;
        f.two = o.kind == HOp::M2;
        f.moff = moff;
        const int b = bind_of[k];
        if (b >= 0) {
          const ket_param_binding& pb = binds[T.bind_first + b];
          f.fam = (int16_t)pb.gate;
          f.param = pb.param;
          f.scale = pb.scale;
          f.shift = pb.shift;
          o.diag = pb.gate == KET_PG_RZ || pb.gate == KET_PG_U1;
          o.real = pb.gate == KET_PG_RY || pb.gate == KET_PG_CRY;
        } else if (moff != csr_off) {
          const int64_t need = f.two ? 16 : 4;
          if (moff < 0 || (size_t)(moff + need) > nmat) return fail(KET_ERR_TYPE, "op matrix offset out of bounds");
          const double* m = mats + 2 * moff;
          o.diag = !f.two && m[2] == 0 && m[3] == 0 && m[4] == 0 && m[5] == 0;
          o.real = !f.two && m[1] == 0 && m[3] == 0 && m[5] == 0 && m[7] == 0;
        }
        o.factors.push_back(f);
      }
      out.push_back(std::move(o));
    }
    // Hamiltonian (PauliTerm convention: ops[0] acts on qubit n-1; |coeff| < 1e-15 skipped,
    // identity terms add their coeff, algorithms.ts:283-336)
    B.ident = 0.0;
    for (int t = 0; t < T.nterms; t++) {
      const double cf = coeffs[T.term_first + t];
      const char* ps = pauli + T.pauli_first + (int64_t)t * n;
      for (int q = 0; q < n; q++)
        if (ps[q] == 0) return fail(KET_ERR_TYPE, "ops length must equal ansatz.qubits (" + std::to_string(n) + ")");
      if (std::fabs(cf) < 1e-15) continue;
      PauliTerm tm{cf, 0, 0, 0};
      bool any = false;
      for (int q = 0; q < n; q++) {
        const char ch = (char)toupper((unsigned char)ps[n - 1 - q]);
        if (ch == 'I') continue;
        any = true;
        if (ch == 'X' || ch == 'Y') tm.flip |= uint64_t(1) << q;
        if (ch != 'X') tm.zm |= uint64_t(1) << q;
        if (ch == 'Y') tm.ny++;
      }
      if (!any) { B.ident += cf; continue; }
      hterms[j].push_back(tm);
    }
  }
  std::vector<double> dm(mats ? mats : nullptr, mats ? mats + 2 * nmat : nullptr);
  dm.resize(2 * nmat);
  {
    const double h = 1.0 / std::sqrt(2.0);
    double blk[32] = {0};
    blk[0] = 1; blk[2 * 5] = h; blk[2 * 6 + 1] = h; blk[2 * 9 + 1] = h; blk[2 * 10] = h; blk[2 * 15] = 1;
    dm.insert(dm.end(), blk, blk + 32);
  }
  // ---- packs: instances by template, as few to a pack as lets all packs run at once, and
  // where no size does, as many as a pack takes
  std::vector<int64_t> count(ntmpl, 0);
  for (int i = 0; i < ninst; i++) {
    if (inst_tmpl[i] < 0 || inst_tmpl[i] >= ntmpl) return fail(KET_ERR_RANGE, "instance template index out of range");
    count[inst_tmpl[i]]++;
  }
  auto pack_bits = [&](int j, int cap) { return std::min(cap, kVqeMaxQubits - im.tmpl[j].n); };
  constexpr size_t kVqeFixed = 64 * kVqeSlots + sizeof(BRound) * kVqeRounds + sizeof(BRoundGate) * kVqeGates;
  int cap = 0;
  for (; cap < kVqePackBits; cap++) {
    int64_t packs = 0;
    int widest = kVqeMinQubits;
    for (int j = 0; j < ntmpl; j++) {
      if (count[j] == 0) continue;
      packs += (count[j] + (1 << pack_bits(j, cap)) - 1) >> pack_bits(j, cap);
      widest = std::max(widest, im.tmpl[j].n + pack_bits(j, cap));
    }
    const int by_regs = kVqeMaxThreads / vqe_threads(widest);
    const int by_smem = (int)(size_t(227 * 1024) / ((size_t(16) << widest) + kVqeFixed + 1024));
    if (packs <= (int64_t)num_sms() * std::max(1, std::min(by_regs, by_smem))) break;
  }
  std::vector<int> order(ninst);
  std::vector<BItem> items;
  std::vector<int64_t> work;
  int tile = kVqeMinQubits;
  {
    std::vector<int> at(ntmpl + 1, 0);
    for (int j = 0; j < ntmpl; j++) at[j + 1] = at[j] + (int)count[j];
    std::vector<int> fill(at.begin(), at.end() - 1);
    for (int i = 0; i < ninst; i++) order[fill[inst_tmpl[i]]++] = i;
    for (int j = 0; j < ntmpl; j++) {
      if (count[j] == 0) continue;
      im.tmpl[j].lgpack = pack_bits(j, cap);
      const int pack = 1 << im.tmpl[j].lgpack;
      const int64_t w = lower_template(hops[j], hterms[j], im.tmpl[j], im) << im.tmpl[j].lgpack;
      for (int f = at[j]; f < at[j + 1]; f += pack) {
        items.push_back(BItem{j, f, std::min(pack, at[j + 1] - f)});
        work.push_back(w);
      }
      tile = std::max(tile, im.tmpl[j].n + im.tmpl[j].lgpack);
    }
    // the heaviest first
    std::vector<int> by(items.size());
    for (size_t i = 0; i < by.size(); i++) by[i] = (int)i;
    std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return work[x] > work[y]; });
    std::vector<BItem> sorted;
    for (int i : by) sorted.push_back(items[i]);
    items.swap(sorted);
  }
  // ---- workspace: the templates' image, then parameters, energies and the queue
  size_t total = 0;
  auto place = [&](size_t bytes) {
    const size_t at = total;
    total += (std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
    return at;
  };
  struct Part { const void* src; size_t bytes, at; };
  std::vector<Part> parts;
  auto part = [&](const auto& v) {
    const size_t bytes = v.size() * sizeof(v[0]);
    parts.push_back(Part{v.data(), bytes, place(bytes)});
    return parts.back().at;
  };
  const size_t o_tmpl = part(im.tmpl), o_chunks = part(im.chunks), o_rounds = part(im.rounds), o_gates = part(im.gates),
               o_matv = part(im.matv), o_factors = part(im.factors), o_mats = part(dm), o_groups = part(im.groups),
               o_terms = part(im.terms), o_items = part(items), o_order = part(order);
  const size_t image = total;
  const size_t o_theta = place(8 * (size_t)ninst * nparams), o_energy = place(8 * (size_t)ninst), o_next = place(256);
  if (c->vqe_work_bytes < total) {
    int rc = ctx_wait(c);
    if (rc) return rc;
    if (c->vqe_graph_exec) { cudaGraphExecDestroy(c->vqe_graph_exec); c->vqe_graph_exec = nullptr; }
    c->vqe_graph_key = 0;
    if (c->vqe_work) cudaFree(c->vqe_work);
    c->vqe_work = nullptr;
    c->vqe_work_bytes = 0;
    rc = dev_alloc(&c->vqe_work, total);
    if (rc) return rc;
    c->vqe_work_bytes = total;
  }
  char* base = (char*)c->vqe_work;
  // One copy for everything before the parameters, and for those where they are few
  const size_t theta_bytes = 8 * (size_t)ninst * nparams, with = theta_bytes <= (64 << 10) ? theta_bytes : 0;
  std::vector<unsigned char> img(image + with, 0);
  for (const Part& p : parts)
    if (p.bytes) memcpy(img.data() + p.at, p.src, p.bytes);
  if (with) memcpy(img.data() + o_theta, theta, with);
  cudaError_t e = cudaMemcpyAsync(base, img.data(), img.size(), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess && with != theta_bytes)
    e = cudaMemcpyAsync(base + o_theta, theta, theta_bytes, cudaMemcpyHostToDevice, c->stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(batch)");
  c->h2d_bytes += image + theta_bytes;
  BArgs a;
  memset(&a, 0, sizeof(a));  // its bytes are the graph's key
  a.tmpl = (const BTmpl*)(base + o_tmpl);
  a.chunks = (const BChunk*)(base + o_chunks);
  a.rounds = (const BRound*)(base + o_rounds);
  a.gates = (const BRoundGate*)(base + o_gates);
  a.matv = (const BMat*)(base + o_matv);
  a.factors = (const BFactor*)(base + o_factors);
  a.mats = (const double2*)(base + o_mats);
  a.groups = (const PauliTileGroup*)(base + o_groups);
  a.terms = (const BTerm*)(base + o_terms);
  a.items = (const BItem*)(base + o_items);
  a.order = (const int*)(base + o_order);
  a.theta = (const double*)(base + o_theta);
  a.energy = (double*)(base + o_energy);
  a.next = (unsigned int*)(base + o_next);
  a.nitems = (int)items.size();
  a.nparams = nparams;
  a.tile = tile;
  // ---- launch: a resident grid sized for the widest pack's shared memory and the
  // largest chunk
  int gates_max = 1;
  a.slots = a.rounds_max = 1;
  for (const BTmpl& T : im.tmpl)
    for (int k = 0; k < T.nchunks; k++) {
      const BChunk& C = im.chunks[T.chunk_first + k];
      a.slots = std::max(a.slots, C.nslots << T.lgpack);
      a.rounds_max = std::max(a.rounds_max, (int)C.nrounds);
      gates_max = std::max(gates_max, (int)C.ngates);
    }
  // (where every SM has one CTA at most, all the threads that share the Hamiltonian's groups)
  const int threads = (int)items.size() <= num_sms() ? kVqeMaxThreads : vqe_threads(tile);
  const size_t smem = (size_t(16) << tile) + 64 * (size_t)a.slots + sizeof(BRound) * a.rounds_max + sizeof(BRoundGate) * gates_max;
  static std::atomic<uint64_t> attr_set{0};
  const uint64_t bit = uint64_t(1) << (c->device & 63);
  if (!(attr_set.load() & bit)) {
    e = cudaFuncSetAttribute(k_batch_vqe, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)((size_t(16) << kVqeMaxQubits) + kVqeFixed));
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_batch_vqe)");
    attr_set.fetch_or(bit);
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_vqe, threads, smem);
  const int grid = std::max(1, std::min(num_sms() * std::max(1, per_sm), a.nitems));
  auto record = [&]() -> cudaError_t {
    cudaMemsetAsync(a.next, 0, 4, c->stream);
    k_batch_vqe<<<grid, threads, smem, c->stream>>>(a);
    return cudaGetLastError();
  };
  prof_begin(c);
  if (!use_graph) {
    e = record();
  } else {
    uint64_t key = 1469598103934665603ull;
    auto mix = [&](const void* p, size_t nb) {
      for (size_t i = 0; i < nb; i++) key = (key ^ ((const unsigned char*)p)[i]) * 1099511628211ull;
    };
    mix(&a, sizeof(a));
    mix(&smem, sizeof(smem));
    mix(&grid, sizeof(grid));
    mix(&threads, sizeof(threads));
    if (c->vqe_graph_exec && c->vqe_graph_key == key) {
      e = cudaGraphLaunch(c->vqe_graph_exec, c->stream);
    } else {
      cudaGraph_t graph;
      e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
      if (e == cudaSuccess) {
        cudaError_t er = record();
        e = cudaStreamEndCapture(c->stream, &graph);
        if (er != cudaSuccess) e = er;
      }
      if (e == cudaSuccess) {
        if (c->vqe_graph_exec) { cudaGraphExecDestroy(c->vqe_graph_exec); c->vqe_graph_exec = nullptr; }
        c->vqe_graph_key = 0;
        e = cudaGraphInstantiate(&c->vqe_graph_exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e == cudaSuccess) {
          c->vqe_graph_key = key;
          e = cudaGraphLaunch(c->vqe_graph_exec, c->stream);
        }
      }
    }
  }
  prof_end(c, PK_BATCH);
  if (e != cudaSuccess) return cuda_fail(e, "batch vqe launch");
  e = cudaMemcpyAsync(energy, a.energy, 8 * (size_t)ninst, cudaMemcpyDeviceToHost, c->stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(energy)");
  c->d2h_bytes += 8 * (size_t)ninst;
  return ctx_wait(c);
}
