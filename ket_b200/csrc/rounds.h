// rounds.h -- planning of in-shared-memory simulation: gates on a state of at
// most 13 qubits grouped into rounds, with CNOTs and swaps as relabellings.
//
// The state sits in shared memory at physical indices p; the logical index is
// B p over GF(2).  A CNOT or an uncontrolled swap only changes B, so it moves
// nothing.  A gate on logical qubit q pairs p with p ^ col[q], and p's logical bit
// q is the parity of p & row[q].
//
// A round is a run of consecutive one-qubit gates whose pair masks span at most
// four dimensions (the span is filled up to four, so that one form of the code
// serves all rounds): each thread loads the 16 amplitudes of one coset of the span into
// registers, applies every gate of the round there, in program order, and stores
// them back -- one pass over shared memory and one barrier for the whole run.  A
// coset is closed under the round's gates, so each amplitude sees them in program
// order, pruning after every gate included.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <utility>
#include <vector>

namespace ket {

constexpr int kRoundBits = 4;        // dimension of a round's span, at most
constexpr int kRoundGates = 16;      // gates in a round, at most
constexpr int kRoundQubits = 13;

// Shared-memory slot of amplitude i: the low three bits XORed with every higher
// group of three, so that eight threads on any of the usual index patterns touch
// eight 16-byte banks.  Linear over GF(2): slot(p ^ m) = slot(p) ^ slot(m).
#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t round_slot(uint32_t i) {
  return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9) ^ (i >> 12)) & 7u);
}

#ifdef __CUDACC__
// A round's 16 slot offsets, two a register, from shared memory (16-byte aligned).
// Read before the loads and again before the stores: kept across the gates, the 16
// addresses spilled as many amplitudes.
struct RoundSlots {
  uint32_t w[8];
  __device__ __forceinline__ void read(const uint16_t* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(a));
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "r"(a + 16));
  }
  __device__ __forceinline__ uint32_t operator()(int j) const { return j & 1 ? w[j >> 1] >> 16 : w[j >> 1] & 0xffffu; }
};
#endif

struct RoundGate {
  uint8_t x;         // 1: X under its controls, 0: a 2x2 under its controls
  uint8_t diag;      // 1: diagonal on the functional r, 2: on (r, r2); it has no mask
  uint8_t bit;       // the gate's mask = basis mask `bit` of the round
  uint8_t nc;        // controls
  uint8_t cj[3];     // per control: the basis masks that flip it
  uint8_t rj[2];     // diagonal: the basis masks that flip r, r2
  uint16_t r, r2;    // row functional of the target
  uint16_t m;        // pair mask of the target
  uint16_t rc[3];    // row functionals of the controls
  int32_t op;        // the caller's op
};

struct Round {
  uint8_t k;                     // dimension: the builder's, or that of a dense round
  uint8_t dense;                 // 1: one 2^k x 2^k, local index bit i on mask i
  uint8_t piv[kRoundBits];       // pivot bits of the span, ascending
  uint16_t m[kRoundBits];        // basis masks
  uint16_t slot[1 << kRoundBits];  // round_slot of the XOR of the masks in j
  uint16_t rd[kRoundBits];       // dense: row functional of local index bit i
  int32_t gate0, ngates;
};

// Rounds from gates given by their masks and functionals.
class RoundBuilder {
 public:
  std::vector<Round> rounds;
  std::vector<RoundGate> gates;

  // n: bits of an index, at least `bits`; bits: the dimension of the rounds.
  explicit RoundBuilder(int n, int bits = kRoundBits) : n_(n), bits_(bits) {}

  // A one-qubit gate (or X) on the target (m, r) under controls rc.
  void add(uint16_t m, uint16_t r, const uint16_t* rc, int nc, bool x, int op) {
    RoundGate g = {};
    g.x = x;
    g.nc = (uint8_t)nc;
    g.r = r;
    g.m = m;
    std::copy(rc, rc + nc, g.rc);
    g.op = op;
    if (!join(g)) {
      close();
      join(g);
    }
  }
  // A diagonal on the functional r, or with two set on (r, r2): it pairs nothing, so
  // it takes no dimension of the round.
  void add_diag(uint16_t r, uint16_t r2, bool two, const uint16_t* rc, int nc, int op) {
    if ((int)cur_.size() >= kRoundGates) close();
    RoundGate g = {};
    g.diag = two ? 2 : 1;
    g.nc = (uint8_t)nc;
    g.r = r;
    g.r2 = r2;
    std::copy(rc, rc + nc, g.rc);
    g.op = op;
    cur_.push_back(g);
  }
  // A 2^k x 2^k, local index bit i on (ms[i], rs[i]), under controls: a round of its own.
  void add_dense(const uint16_t* ms, const uint16_t* rs, int k, const uint16_t* rc, int nc, int op) {
    close();
    RoundGate g = {};
    g.nc = (uint8_t)nc;
    std::copy(rc, rc + nc, g.rc);
    g.op = op;
    cur_ = {g};
    basis_.assign(ms, ms + k);
    std::copy(rs, rs + k, rd_);
    dense_ = true;
    close();
  }
  // End the round under construction (before anything that is not a gate).
  void close() {
    if (!cur_.empty()) {
      if (!dense_) fill();
      Round R = {};
      R.k = (uint8_t)basis_.size();
      R.dense = dense_;
      std::vector<uint16_t> e = basis_;
      for (size_t i = 0; i < e.size(); i++) {  // echelon form: pivot = highest set bit
        const int h = 31 - __builtin_clz((unsigned)e[i]);
        R.piv[i] = (uint8_t)h;
        for (size_t j = i + 1; j < e.size(); j++)
          if ((e[j] >> h) & 1) e[j] ^= e[i];
      }
      std::sort(R.piv, R.piv + R.k);
      for (int i = 0; i < R.k; i++) R.m[i] = basis_[i];
      for (int j = 0; j < (1 << R.k); j++) {
        uint32_t x = 0;
        for (int i = 0; i < R.k; i++)
          if ((j >> i) & 1) x ^= basis_[i];
        R.slot[j] = (uint16_t)round_slot(x);
      }
      for (int i = 0; i < kRoundBits; i++) R.rd[i] = rd_[i];
      R.gate0 = (int32_t)gates.size();
      R.ngates = (int32_t)cur_.size();
      for (RoundGate& g : cur_) {
        for (int c = 0; c < g.nc; c++) g.cj[c] = flipped_by(g.rc[c]);
        g.rj[0] = flipped_by(g.r);
        g.rj[1] = flipped_by(g.r2);
        gates.push_back(g);
      }
      rounds.push_back(R);
    }
    cur_.clear();
    basis_.clear();
    brow_.clear();
    dense_ = false;
  }

 private:
  int n_, bits_;
  std::vector<RoundGate> cur_;
  std::vector<uint16_t> basis_, brow_;  // masks, and the targets' row functionals: brow_[i] . basis_[j] = (i == j)
  uint16_t rd_[kRoundBits] = {};
  bool dense_ = false;

  uint8_t flipped_by(uint16_t r) const {
    uint8_t f = 0;
    for (size_t i = 0; i < basis_.size(); i++)
      if (odd(basis_[i] & r)) f |= (uint8_t)(1u << i);
    return f;
  }
  static bool odd(uint32_t x) { return __builtin_popcount(x) & 1; }
  bool independent(uint16_t m) const {
    uint32_t x = m;
    std::vector<uint16_t> e = basis_;
    for (size_t i = 0; i < e.size(); i++) {
      const int h = 31 - __builtin_clz((unsigned)e[i]);
      for (size_t j = i + 1; j < e.size(); j++)
        if ((e[j] >> h) & 1) e[j] ^= e[i];
      if ((x >> h) & 1) x ^= e[i];
    }
    return x != 0;
  }
  // Every target's logical bit is fixed by its own mask alone across a coset, so
  // one test on the coset's base gives a thread's role for all its pairs.
  bool join(RoundGate& g) {
    if ((int)cur_.size() >= kRoundGates) return false;
    size_t at = 0;
    while (at < basis_.size() && basis_[at] != g.m) at++;
    if (at < basis_.size()) {
      if (brow_[at] != g.r) return false;
    } else {
      if ((int)at >= bits_ || !independent(g.m)) return false;
      for (size_t i = 0; i < at; i++)
        if (odd(basis_[i] & g.r) || odd(g.m & brow_[i])) return false;
      basis_.push_back(g.m);
      brow_.push_back(g.r);
    }
    g.bit = (uint8_t)at;
    cur_.push_back(g);
    return true;
  }
  // Masks that complete the span and flip none of the round's targets: unit
  // vectors, each made orthogonal to the targets' functionals.
  void fill() {
    const size_t k = brow_.size();
    for (int b = n_ - 1; b >= 0 && (int)basis_.size() < bits_; b--) {
      uint16_t m = (uint16_t)(1u << b);
      for (size_t i = 0; i < k; i++)
        if (odd(m & brow_[i])) m ^= basis_[i];
      if (m && independent(m)) basis_.push_back(m);
    }
  }
};

// Rounds of gates on logical qubits, with the relabelling.
class RoundPlan : public RoundBuilder {
 public:
  uint16_t row[kRoundQubits], col[kRoundQubits];

  explicit RoundPlan(int n) : RoundBuilder(n) {
    for (int q = 0; q < kRoundQubits; q++) row[q] = col[q] = (uint16_t)(1u << q);
  }
  void cnot(int c, int t) { row[t] ^= row[c]; col[c] ^= col[t]; }
  void swap(int a, int b) { std::swap(row[a], row[b]); std::swap(col[a], col[b]); }
  // A one-qubit gate (or X) on q under controls cs.
  void gate(int q, const int* cs, int nc, bool x, int op) {
    uint16_t rc[3];
    for (int i = 0; i < nc; i++) rc[i] = row[cs[i]];
    add(col[q], row[q], rc, nc, x, op);
  }
  // A 2^k x 2^k on qs (qs[0] = MSB) under controls cs.
  void dense(const int* qs, int k, const int* cs, int nc, int op) {
    uint16_t rc[3], ms[kRoundBits], rs[kRoundBits];
    for (int i = 0; i < nc; i++) rc[i] = row[cs[i]];
    for (int i = 0; i < k; i++) {
      ms[i] = col[qs[k - 1 - i]];
      rs[i] = row[qs[k - 1 - i]];
    }
    add_dense(ms, rs, k, rc, nc, op);
  }
};

}  // namespace ket
