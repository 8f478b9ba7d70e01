// The serial double sum of 1 - x over a box (the neutral fraction's numerator,
// get_HIIbubbles.c:473-477), bit for bit, from chunks of NEUTRAL_CHUNK terms
// that are prepared in parallel (kernels_elem.cu).
//
// While the running sum S stays in [2^E, 2^(E+1)) an addition rounds its term
// t to a multiple of u = 2^(E-52), whatever S is, except for ties (t an odd
// multiple of u / 2), which go to the even multiple and so depend on the
// parity of S / u alone.  A run of terms is therefore a pair: the multiples
// of u that it adds to an even and to an odd S / u.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace sf21 {

constexpr int NEUTRAL_CHUNK = 4096;

// Exponent of a double that is zero (-1023) or normal and positive.
inline int neutral_exponent(double s) {
  uint64_t b;
  memcpy(&b, &s, 8);
  return (int)(b >> 52) - 1023;
}

// S after all chunks.  E[c]: the binade that chunk c's pair (even[c], odd[c] at
// stride 2 from step) was made for, below 0 if it has none; x(i): the box.  E
// is an estimate: a pair is used only if S has that exponent before the chunk
// and after it.  The terms of a chunk that has a pair are not negative, so S
// was in the binade throughout and the addition is exact; any other chunk is
// added term by term.
template <class X>
double neutral_serial(long n3, const long long* step, const int* E, const X& x) {
  double S = 0.;
  for (long c = 0; c * NEUTRAL_CHUNK < n3; ++c) {
    if (E[c] >= 0 && neutral_exponent(S) == E[c]) {
      uint64_t b;
      memcpy(&b, &S, 8);
      const double T = S + ldexp((double)step[2 * c + (b & 1)], E[c] - 52);
      if (neutral_exponent(T) == E[c]) {
        S = T;
        continue;
      }
    }
    const long end = n3 < (c + 1) * NEUTRAL_CHUNK ? n3 : (c + 1) * NEUTRAL_CHUNK;
    for (long i = c * NEUTRAL_CHUNK; i < end; ++i) S += 1.0 - x(i);
  }
  return S;
}

}  // namespace sf21
