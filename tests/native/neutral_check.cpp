// Host-side check of neutral_sum.h: the sum composed from chunk pairs against
// the serial sum, for a box of one value x everywhere.
// Usage: neutral_check <n3> <x> ...
// Prints "<x> <composed> <serial>" in hexadecimal floats.
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
