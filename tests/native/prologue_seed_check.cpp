// Host-side check of prologue_fast.h with the float seeds of its Newton
// iterations at the edge of their stated error (compile with -DPF_SEED_ERR=e,
// |e| at most 2^-21): every path still returns the float of the exact chain, or
// of the path below it that has no such seed.
// Usage: prologue_seed_check <n> <seed>
// Prints "<name> <cases> <mismatches> <fallbacks>".
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "prologue_fast.h"

static uint64_t d2bits(double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; }
static uint32_t f2bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static float bits2f(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static uint64_t rng_state;
static uint64_t rnd64() {
  rng_state ^= rng_state << 13; rng_state ^= rng_state >> 7; rng_state ^= rng_state << 17;
  return rng_state;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 100000;
  rng_state = argc > 2 ? strtoull(argv[2], 0, 10) : 1;
  long cases = 0, bad = 0, left = 0;
  uint64_t tab[384];
  for (int i = 0; i < 384; ++i) tab[i] = rrec_table(i);
  const double zs[3] = {6.0, 8.5, 15.0};
  for (double z : zs) {
    const sd_t rec1 = d2bits(1.e-24 * 9.84815696 * std::pow(1.0 + z, 5.06773134));
    const sd_t dvv = d2bits(std::pow(150.0 * 3.0856775807e24 / 256 / 0.7 / (1. + z), 3.0));
    const sd_t r2 = d2bits(1.76105133), r3 = d2bits(0.81722878), vn = d2bits(1.e+45);
    const sd_divc r2c = sd_divc_prepare(r2), vnc = sd_divc_prepare(vn);
    const RrecFast rf = rrec_fast_prepare(rec1, dvv, vn, r2, r3);
    if (!rf.ok) return 2;
    for (long i = 0; i < n; ++i) {
      const float od = bits2f((uint32_t)(119 + rnd64() % 16) << 23 | ((uint32_t)rnd64() & 0x7FFFFFu));
      float got = 0.f, want = 0.f;
      ++cases;
      if (!rrec_quick(od, rf, tab, &got)) {
        ++left;
        continue;
      }
      if (!rrec_fast(od, rf, &want)) want = sd_to_float(rrec_exact(od, r2c, r3, rec1, dvv, vnc));
      if (f2bits(got) != f2bits(want)) {
        if (bad++ < 5) printf("# rrec z=%g 1 + d=%a quick=%a exact=%a\n", z, od, got, want);
      }
    }
  }
  printf("rrec %ld %ld %ld\n", cases, bad, left);
  cases = bad = left = 0;
  for (long i = 0; i < n / 4; ++i) {
    const float r = bits2f((uint32_t)(127 - 30 + rnd64() % 29) << 23 | ((uint32_t)rnd64() & 0x7FFFFFu));
    float got = 0.f;
    ++cases;
    if (!xhi_fast(r, &got)) {
      ++left;
      continue;
    }
    const float want = sd_to_float(xhi_exact(sd_from_float(r)));
    if (f2bits(got) != f2bits(want)) {
      if (bad++ < 5) printf("# xhi ratio=%a fast=%a exact=%a\n", r, got, want);
    }
  }
  printf("xhi %ld %ld %ld\n", cases, bad, left);
  return 0;
}
