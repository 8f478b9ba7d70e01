// Host-side check of neutral_sum.h: the sum composed from chunk pairs against
// the serial sum, for a box of one value x everywhere.
// Usage: neutral_check <n3> <x> ...
// Prints "<x> <composed> <serial>" in hexadecimal floats.
//        neutral_check units <n>
// Prints "units <cases> <mismatches>": neutral_units against 1.0 - x, n floats
// of each exponent of [0, 1] and those next to the powers of two.
//
// The pairs are made by their definition: the serial additions of a chunk to
// 2^E and to the next double.  The binades come from the exact sums (n times a
// double of at most 53 bits, in 128-bit integers), which the serial sum drifts
// away from, since equal terms are rounded the same way every time.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "neutral_sum.h"

using namespace sf21;

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  if (!strcmp(argv[1], "units")) {
    const long n = atol(argv[2]);
    long cases = 0, bad = 0;
    uint32_t r = 1;
    auto check = [&](uint32_t bits) {
      float x;
      memcpy(&x, &bits, 4);
      if (!(x >= 0.0f && x <= 1.0f)) return;
      ++cases;
      bad += ldexp((double)neutral_units(x), -53) != 1.0 - x;
    };
    for (uint32_t ex = 0; ex <= 127; ++ex) {
      for (int d = -3; d <= 3; ++d) check((ex << 23) + (uint32_t)d);
      for (long i = 0; i < n; ++i) check(ex << 23 | ((r = r * 1664525u + 1013904223u) >> 9));
      for (int k = 0; k < 23; ++k) check(ex << 23 | 1u << k);  // ties among them
      for (int k = 0; k < 23; ++k) check(ex << 23 | (0x7FFFFFu >> k << k));
    }
    printf("units %ld %ld\n", cases, bad);
    return 0;
  }
  const long n3 = atol(argv[1]), chunks = (n3 + NEUTRAL_CHUNK - 1) / NEUTRAL_CHUNK;
  for (int a = 2; a < argc; ++a) {
    const float x = strtof(argv[a], nullptr);
    const double t = 1.0 - x;
    const auto units = (unsigned __int128)ldexp(t, 53);  // t in [0, 1] as a multiple of 2^-53
    auto binade = [&](long n) {                          // of n t
      unsigned __int128 v = units * (unsigned __int128)n;
      int e = -54;
      for (; v; v >>= 1) ++e;
      return e;
    };
    std::vector<int> E(chunks, -1);
    std::vector<long long> step(2 * chunks, 0);
    std::map<int, std::pair<long long, long long>> made;
    for (long c = 0; c < chunks; ++c) {
      const long i0 = c * NEUTRAL_CHUNK, i1 = i0 + NEUTRAL_CHUNK < n3 ? i0 + NEUTRAL_CHUNK : n3;
      if (i1 - i0 < NEUTRAL_CHUNK || binade(i0) < 0 || binade(i0) != binade(i1)) continue;
      E[c] = binade(i0);
      if (!made.count(E[c])) {
        const double lo = ldexp(1.0, E[c]), u = ldexp(1.0, E[c] - 52);
        double s0 = lo, s1 = lo + u;
        for (int k = 0; k < NEUTRAL_CHUNK; ++k) {
          s0 += t;
          s1 += t;
        }
        made[E[c]] = {(long long)((s0 - lo) / u), (long long)((s1 - (lo + u)) / u)};
      }
      step[2 * c] = made[E[c]].first;
      step[2 * c + 1] = made[E[c]].second;
    }
    const double got = neutral_serial(n3, step.data(), E.data(), [x](long) { return x; });
    double want = 0.;
    for (long i = 0; i < n3; ++i) want += 1.0 - x;
    printf("%a %a %a\n", x, got, want);
  }
  return 0;
}
