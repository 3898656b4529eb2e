// pauli_terms.cuh -- signed sums over a thread's products, shared by the kernels
// that evaluate Pauli terms (kernels_read.cu, batch_vqe.cu).
#pragma once

#include <stdint.h>

namespace ket {

__device__ __forceinline__ double flip_sign(double v, uint32_t odd) {  // odd: 0 or 1
  return __hiloint2double(__double2hiint(v) ^ (int)(odd << 31), __double2loint(v));
}

// One sum over a group's NB products b: the signs of its terms [first, first +
// nterms) are a thread part, parity(t & thread mask), times a parity of the
// products' index.  coeff(i) and zm(i) give a term's coefficient and its masks
// (thread mask | index mask << 16); the terms are sorted by index mask.  One term
// signs the products; several share a Walsh transform over the index, after which
// a term costs one addition.
template <int NB, typename C, typename Z>
__device__ __forceinline__ double pauli_terms(double (&b)[NB], C coeff, Z zm, int first, int nterms, int t) {
  static_assert(NB <= 16, "parities of up to four index bits");
  if (nterms == 1) {
    const uint32_t z = zm(first), zi = z >> 16;
    if (zi) {
#pragma unroll
      for (int j = 1; j < NB; j++) b[j] = flip_sign(b[j], (0x6996u >> (j & zi)) & 1u);
    }
#pragma unroll
    for (int st = NB / 2; st > 0; st >>= 1)
#pragma unroll
      for (int j = 0; j < st; j++) b[j] += b[j + st];
    return flip_sign(coeff(first), __popc(t & z & 0xffffu) & 1) * b[0];
  }
#pragma unroll
  for (int st = 1; st < NB; st <<= 1)
#pragma unroll
    for (int j = 0; j < NB; j++)
      if (!(j & st)) {
        const double x = b[j], y = b[j | st];
        b[j] = x + y;
        b[j | st] = x - y;
      }
  double acc = 0.0;
  int i = first;
#pragma unroll
  for (int w = 0; w < NB; w++) {
    double c = 0.0;
    for (; i < first + nterms; i++) {
      const uint32_t z = zm(i);
      if ((z >> 16) != w) break;
      c += flip_sign(coeff(i), __popc(t & z & 0xffffu) & 1);
    }
    acc += c * b[w];
  }
  return acc;
}

}  // namespace ket
