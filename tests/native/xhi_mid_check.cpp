// xhi_fast between 2^-5 and 1: every 8th float of the octaves against the
// exact chain.  Prints, per octave, floats checked, mismatches, floats that
// the fast path left to the chain.
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "prologue_fast.h"

int main() {
  for (int e = -5; e <= 0; ++e) {
    long n = 0, bad = 0, left = 0;
    for (uint32_t m = 0; m < (1u << 23); m += 8) {
      const uint32_t u = ((uint32_t)(127 + e) << 23) | m;
      float r, got;
      memcpy(&r, &u, 4);
      ++n;
      if (!xhi_fast(r, &got)) {
        ++left;
        continue;
      }
      const float want = sd_to_float(xhi_exact(sd_from_float(r)));
      bad += memcmp(&got, &want, 4) != 0;
    }
    printf("%d %ld %ld %ld\n", e, n, bad, left);
  }
  return 0;
}
