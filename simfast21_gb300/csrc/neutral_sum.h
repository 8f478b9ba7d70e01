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

#if defined(__CUDACC__)
#define NEU_HD __host__ __device__ __forceinline__
#else
#define NEU_HD static inline
#endif

// 1.0 - x in double, for a float x in [0, 1], as a multiple of 2^-53: doubles
// of [0, 1] are such multiples from 1/2 up, and below 1/2 the difference is
// exact, a multiple of 2^-24.  x is rounded to one (ties to even: the
// difference from 2^53 has the same parity).
NEU_HD uint64_t neutral_units(float x) {
  union {
    float f;
    uint32_t u;
  } c;
  c.f = x;
  const int ex = (int)((c.u >> 23) & 255);
  const uint64_t m = (c.u & 0x7FFFFFu) | (ex ? 0x800000u : 0u);
  uint64_t X = 0;  // x 2^53 = m 2^(ex - 97)
  if (ex >= 97) {
    X = m << (ex - 97 < 30 ? ex - 97 : 30);
  } else if (ex >= 72) {
    const int s = 97 - ex;
    const uint64_t rem = m & ((1ull << s) - 1), half = 1ull << (s - 1);
    X = m >> s;
    X += rem > half || (rem == half && (X & 1));
  }
  return (1ull << 53) - X;
}

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
