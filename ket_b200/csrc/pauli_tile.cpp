// pauli_tile.cpp -- host side of the tiled Pauli kernels (k_pauli_tile,
// k_hpsi_tile): which terms share a pass over the state, and their masks in
// the pass's tile bits.
#include <algorithm>
#include <cstring>

#include "read.h"

namespace ket {

// Tile passes for the groups, first fit in ascending flip order, each pass with
// as many flipped qubits (and terms) as its tile takes among the next kPauliWindow
// groups; groups that flip more qubits above the low ones than a tile holds are left
// in `wide`.  The window bounds the planning of Hamiltonians of many flips: without it
// 3000 random strings on 20 qubits took 50 ms here, more than their passes.
//
// An expectation's pass that holds one group gains nothing from the tile.  Up to
// kPauliGroupQubits qubits such a group goes to `wide` as well: its own pass takes the
// terms as kernel parameters, where a tile's tables are a copy first (one string on 12
// to 20 qubits 31.6 us by its own pass, 34.4 by a tile; on 24 qubits 98 and 85).
constexpr size_t kPauliWindow = 1024;
constexpr int kPauliGroupQubits = 20;
std::vector<PauliTilePass> plan_pauli_tiles(int n, const std::vector<PauliTerm>& terms, bool expectation,
                                            PauliGroups& wide) {
  PauliGroups all;
  for (const PauliTerm& t : terms) all[{t.flip, t.ny & 3}].push_back(&t);
  const uint64_t low = (uint64_t(1) << KET_PAULI_TILE_LOW) - 1;
  std::vector<PauliTilePass> passes;
  typedef std::vector<const PauliTerm*> Members;
  struct Left {
    uint64_t flip;
    int ny;
    Members* v;
    size_t from;  // members before it are placed
    int next;     // the next group with members left, or -1
  };
  std::vector<Left> left;
  for (auto& kv : all) {
    if (__builtin_popcountll(kv.first.first | low) <= KET_PAULI_TILE_BITS)
      left.push_back(Left{kv.first.first, kv.first.second, &kv.second, 0, (int)left.size() + 1});
    else
      wide[kv.first] = std::move(kv.second);
  }
  if (!left.empty()) left.back().next = -1;
  int head = left.empty() ? -1 : 0;
  struct Taken {
    Left* g;
    size_t from, count;
  };
  std::vector<Taken> now;
  while (head >= 0) {
    uint64_t S = low;
    size_t room = KET_PAULI_TILE_TERMS, seen = 0;
    now.clear();
    for (int i = head, before = -1; i >= 0 && room && seen < kPauliWindow; seen++) {
      Left& g = left[i];
      const size_t take = __builtin_popcountll(S | g.flip) <= KET_PAULI_TILE_BITS ? std::min(room, g.v->size() - g.from) : 0;
      if (take) {
        now.push_back(Taken{&g, g.from, take});
        S |= g.flip;
        room -= take;
        g.from += take;
      }
      if (g.from == g.v->size()) (before < 0 ? head : left[before].next) = g.next;
      else before = i;
      i = g.next;
    }
    if (expectation && n <= kPauliGroupQubits && now.size() == 1 && now[0].count == now[0].g->v->size() &&
        now[0].count <= KET_PAULI_GROUP_TERMS) {
      wide[{now[0].g->flip, now[0].g->ny}] = std::move(*now[0].g->v);
      continue;
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
    for (const Taken& tk : now) {
      const int ny = tk.g->ny;
      PauliTileGroup G;
      G.flip = tile_mask(tk.g->flip);
      G.top = G.flip ? (uint8_t)(31 - __builtin_clz(G.flip)) : 0;
      G.odd = (uint8_t)(ny & 1);
      G.first = (int)P.terms.size();
      G.nterms = (uint16_t)tk.count;
      // expectation: Re(i^ny z) = Re z, -Im z, -Re z, Im z with z = psi_y conj(psi_x),
      // and a pair counts twice; H psi: (-i)^ny, the sign of x being that of y
      // times (-1)^ny
      const double w = (ny == 1 || ny == 2 ? -1.0 : 1.0) * (expectation && G.flip ? 2.0 : 1.0);
      for (size_t i = tk.from; i < tk.from + tk.count; i++) {
        const PauliTerm* t = (*tk.g->v)[i];
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
  }
  return passes;
}

}  // namespace ket
