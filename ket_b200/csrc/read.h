// read.h -- read-out kernel launchers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <map>
#include <utility>
#include <vector>

#include "ket_sv.h"

namespace ket {

#define KET_MAX_MARGINAL_QUBITS 12
#define KET_PAULI_GROUP_TERMS 64

struct MarginalSpec {
  int m;
  int q[KET_MAX_MARGINAL_QUBITS];
  uint64_t mask;
};

struct PauliGroup {
  uint64_t flip;                        // X|Y positions
  int ny;                               // number of Y factors (mod 4 phase i^ny)
  int nterms;
  uint64_t zm[KET_PAULI_GROUP_TERMS];   // Z|Y positions of each term
  double coeff[KET_PAULI_GROUP_TERMS];
};

// Tiled Pauli sums: a tile is 2^12 amplitudes, tile bit b = qubit bits[b].
#define KET_PAULI_TILE_BITS 12
#define KET_PAULI_TILE_LOW 4     // qubits 0-3 stay tile bits 0-3: 256 contiguous bytes at c128, 128 at c64
#define KET_PAULI_TILE_TERMS 512 // terms (so groups) of one pass
struct PauliTileArgs {
  uint64_t ntiles;
  int ngroups, nterms, flips;    // flips: whether any group flips a qubit
  int nctx;
  int bits[KET_PAULI_TILE_BITS];
  int ctxbits[KET_MAX_QUBITS];   // qubits outside the tile, ascending
};
struct PauliTileGroup {          // terms sharing a flip mask and i^ny
  uint32_t flip;                 // tile bits
  uint8_t top, odd;              // highest flipped tile bit; whether the imaginary part counts
  uint16_t nterms;
  int32_t first;
};
struct PauliTileTerm {
  double coeff;                  // with the sign of i^ny folded in, and 2 for a pair
  uint64_t zctx;                 // Z|Y qubits outside the tile
  uint32_t zm;                   // thread mask | mask over the products' index << 16
  uint32_t pad;
};

// A Pauli string: it flips the X|Y qubits, signs by the Z|Y qubits, times i^ny.
struct PauliTerm {
  double coeff;
  uint64_t flip, zm;
  int ny;
};
typedef std::map<std::pair<uint64_t, int>, std::vector<const PauliTerm*>> PauliGroups;  // by (flip, ny mod 4)

// One pass of a tiled Pauli kernel: its tile, and its groups and terms in tile bits.
struct PauliTilePass {
  PauliTileArgs args;
  std::vector<PauliTileGroup> groups;
  std::vector<PauliTileTerm> terms;
};
std::vector<PauliTilePass> plan_pauli_tiles(int n, const std::vector<PauliTerm>& terms, bool expectation,
                                            PauliGroups& wide);

int num_sms();

cudaError_t launch_norm2(const void* amp, int n, int prec, double* scratch, double* out, cudaStream_t s);
size_t norm2_scratch(int n);
cudaError_t launch_probs_dense(const void* amp, int prec, uint64_t off, uint64_t cnt, double thr, double* out,
                               cudaStream_t s);
uint64_t kept_chunk(int n);
cudaError_t launch_count_kept(const void* amp, int n, int prec, double thr, uint64_t* counts, cudaStream_t s);
cudaError_t launch_compact_kept(const void* amp, int n, int prec, double thr, const uint64_t* offs, uint64_t cap,
                                uint64_t* oidx, double* op, cudaStream_t s);
uint64_t marg_chunk(int n);
cudaError_t launch_marginals(const void* amp, int n, int prec, double* partial, double* out, cudaStream_t s);
size_t mdist_partials(int n, uint64_t mask);  // doubles of scratch
cudaError_t launch_marginal_dist(const void* amp, int n, int prec, const MarginalSpec& spec, double* partial,
                                 double* out, cudaStream_t s);
// Sampling: the reference's running FP64 sum over kept entries in ascending
// index order, bit for bit, kept as one checkpoint per 32 entries; each draw
// (0 <= r <= 1) searches the checkpoints and adds inside one sub-chunk.
size_t sample_scratch(int n);
int sample_launches();
cudaError_t launch_sample(const void* amp, int n, int prec, double thr, const double* r, uint64_t shots, void* scratch,
                          uint64_t* out, cudaStream_t s);
cudaError_t launch_gather(const void* amp, int prec, const uint64_t* idx, uint64_t k, double* out, cudaStream_t s);
cudaError_t launch_pauli_group(const void* amp, int n, int prec, const PauliGroup& g, double* partial, double* out,
                               cudaStream_t s);
size_t pauli_scratch(int n);
// One pass of tiled Pauli sums: pauli_tile_grid(n) partials.
unsigned pauli_tile_grid(int n);
cudaError_t launch_pauli_tile(const void* amp, int n, int prec, const PauliTileArgs& g, const PauliTileGroup* groups,
                              const PauliTileTerm* terms, double* partial, cudaStream_t s);
// lam (+)= the pass's terms applied to psi (first: lam = ident * psi + ...); last:
// pauli_tile_grid(n) partials of Re <psi|lam>.
cudaError_t launch_hpsi_tile(const void* psi, void* lam, int n, const PauliTileArgs& g, const PauliTileGroup* groups,
                             const PauliTileTerm* terms, double ident, bool first, bool last, double* partial,
                             cudaStream_t s);
// Fixed-order sum of `count` partials.
cudaError_t launch_sum(const double* partial, uint64_t count, double* out, cudaStream_t s);

// <a|b> (re, im) and max |a_i - b_i| of two states of the same size, any precisions.
cudaError_t launch_compare(const void* a, int pa, const void* b, int pb, int n, double* scratch, double* out,
                           cudaStream_t s);
size_t compare_scratch(int n);

}  // namespace ket
