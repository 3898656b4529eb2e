// pauli_tile.cpp -- host side of the tiled Pauli kernels (k_pauli_tile,
// k_hpsi_tile): which terms share a pass over the state, and their masks in
// the pass's tile bits.
#include <algorithm>
#include <cstring>

#include "read.h"

namespace ket {

// Tile passes for the groups, first fit in ascending flip order, each pass with
// as many flipped qubits (and terms) as its tile takes; groups that flip more
// qubits above the low ones than a tile holds are left in `wide`.
std::vector<PauliTilePass> plan_pauli_tiles(int n, const std::vector<PauliTerm>& terms, bool expectation,
                                            PauliGroups& wide) {
  PauliGroups all;
  for (const PauliTerm& t : terms) all[{t.flip, t.ny & 3}].push_back(&t);
  const uint64_t low = (uint64_t(1) << KET_PAULI_TILE_LOW) - 1;
  std::vector<PauliTilePass> passes;
  PauliGroups left;
  for (auto& kv : all)
    (__builtin_popcountll(kv.first.first | low) <= KET_PAULI_TILE_BITS ? left : wide).insert(kv);
  while (!left.empty()) {
    uint64_t S = low;
    size_t room = KET_PAULI_TILE_TERMS;
    PauliGroups now, rest;
    for (auto& kv : left) {
      const size_t take = __builtin_popcountll(S | kv.first.first) <= KET_PAULI_TILE_BITS
                              ? std::min(room, kv.second.size()) : 0;
      const auto cut = kv.second.begin() + take;
      if (take) now[kv.first].assign(kv.second.begin(), cut);
      if (cut != kv.second.end()) rest[kv.first].assign(cut, kv.second.end());
      if (take) S |= kv.first.first;
      room -= take;
    }
    for (int q = 0; __builtin_popcountll(S) < KET_PAULI_TILE_BITS; q++) S |= uint64_t(1) << q;
    PauliTilePass P;
    memset(&P.args, 0, sizeof(P.args));
    int nb = 0;
    for (int q = 0; q < n; q++) {
      if ((S >> q) & 1) P.args.bits[nb++] = q;
      else P.args.ctxbits[P.args.nctx++] = q;
    }
    P.args.ntiles = uint64_t(1) << (n - KET_PAULI_TILE_BITS);
    auto tile_mask = [&](uint64_t m) {
      uint32_t r = 0;
      for (int b = 0; b < KET_PAULI_TILE_BITS; b++)
        if ((m >> P.args.bits[b]) & 1) r |= 1u << b;
      return r;
    };
    for (auto& kv : now) {
      const int ny = kv.first.second;
      PauliTileGroup G;
      G.flip = tile_mask(kv.first.first);
      G.top = G.flip ? (uint8_t)(31 - __builtin_clz(G.flip)) : 0;
      G.odd = (uint8_t)(ny & 1);
      G.first = (int)P.terms.size();
      G.nterms = (uint16_t)kv.second.size();
      // expectation: Re(i^ny z) = Re z, -Im z, -Re z, Im z with z = psi_y conj(psi_x),
      // and a pair counts twice; H psi: (-i)^ny, the sign of x being that of y
      // times (-1)^ny
      const double w = (ny == 1 || ny == 2 ? -1.0 : 1.0) * (expectation && G.flip ? 2.0 : 1.0);
      for (const PauliTerm* t : kv.second) {
        const uint32_t z = tile_mask(t->zm);
        uint32_t zthr = z & 0x1ffu, zidx = z >> 9;
        if (expectation && G.flip) {
          // the products' index leaves out register bit p: clear in a register
          // flip, equal to the thread's bit `top` in a thread flip
          const int p = G.top >= 9 ? G.top - 9 : 2;
          if (G.top < 9 && ((zidx >> p) & 1)) zthr ^= 1u << G.top;
          zidx = ((zidx >> (p + 1)) << p) | (zidx & ((1u << p) - 1));
        }
        P.terms.push_back(PauliTileTerm{w * t->coeff, t->zm & ~S, zthr | zidx << 16, 0});
      }
      std::stable_sort(P.terms.begin() + G.first, P.terms.end(), [](const PauliTileTerm& x, const PauliTileTerm& y) {
        return (x.zm >> 16) < (y.zm >> 16);
      });
      P.groups.push_back(G);
      P.args.flips |= G.flip != 0;
    }
    P.args.ngroups = (int)P.groups.size();
    P.args.nterms = (int)P.terms.size();
    passes.push_back(std::move(P));
    left.swap(rest);
  }
  return passes;
}

}  // namespace ket
