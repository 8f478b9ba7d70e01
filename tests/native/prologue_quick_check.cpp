// Host-side check of the shorter paths of prologue_fast.h: each returns the
// float of the exact soft-double chain whenever it returns.
// Usage: prologue_quick_check <n_random> <seed>
// Prints "<name> <cases> <mismatches> <fallbacks>" for
//   xhi_octaves: XHI of every 16th float of the octaves at both ends and in the middle of xhi_fast's range;
//   xhi:         random floats with binary exponents in [-32, -3] (the range and both outsides);
//   rrec:        rrec_quick, lognormal 1 + d and floats with exponents in [-60, 60], six redshifts, four boxes;
//   one_minus:   1 - f and the largest float below it, random floats in [0, 1] and floats near 0, 1/2 and 1.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>

#include "prologue_fast.h"

static uint64_t d2bits(double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; }
static uint32_t f2bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static float bits2f(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static uint64_t rng_state;
static uint64_t rnd64() {
  rng_state ^= rng_state << 13; rng_state ^= rng_state >> 7; rng_state ^= rng_state << 17;
  return rng_state;
}
static double rnd_unit() { return (double)(rnd64() >> 11) * 0x1p-53; }
static float rnd_float_exp(int emin, int emax) {
  const uint32_t e = (uint32_t)(127 + emin) + (uint32_t)(rnd64() % (uint64_t)(emax - emin + 1));
  return bits2f((e << 23) | ((uint32_t)rnd64() & 0x7FFFFFu));
}

struct Stat { const char* name; long n = 0, bad = 0, fallback = 0; };
static void tally(Stat& s, bool fast, float got, float want, double arg) {
  s.n++;
  if (!fast) { s.fallback++; return; }
  if (f2bits(got) != f2bits(want)) {
    if (s.bad < 5) printf("# %s mismatch arg=%a fast=%a exact=%a\n", s.name, arg, got, want);
    s.bad++;
  }
}
static void check_xhi(Stat& s, float r) {
  float got = 0.f;
  const bool fast = xhi_fast(r, &got);
  tally(s, fast, got, sd_to_float(xhi_exact(sd_from_float(r))), r);
}
static void check_one_minus(Stat& s, float f) {
  float lo, rn;
  one_minus(f, &lo, &rn);
  const sd_t o = sd_sub(0x3FF0000000000000ULL, sd_from_float(f));
  const float wrn = sd_to_float(o);
  const float wlo = sd_gt(sd_from_float(wrn), o) ? nextafterf(wrn, -INFINITY) : wrn;
  tally(s, true, rn, wrn, f);
  tally(s, true, lo, wlo, f);
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 100000;
  rng_state = argc > 2 ? strtoull(argv[2], 0, 10) : 88172645463325252ULL;
  Stat xo{"xhi_octaves"}, xr{"xhi"}, rr{"rrec"}, om{"one_minus"};
  for (int e : {-30, -12, -11, -5})
    for (uint32_t m = 0; m < (1u << 23); m += 16) check_xhi(xo, bits2f(((uint32_t)(127 + e) << 23) | m));
  for (long i = 0; i < 8 * n; ++i) check_xhi(xr, rnd_float_exp(-32, -3));
  uint64_t tab[384];
  for (int i = 0; i < 384; ++i) tab[i] = rrec_table(i);
  const double zs[6] = {5.0, 7.0, 8.5, 11.0, 15.0, 20.0};
  const double Ls[4] = {300.0, 106.5, 50.0, 1000.0};
  const int Ns[4] = {512, 600, 128, 1200};
  for (double z : zs)
    for (int bx = 0; bx < 4; ++bx) {
      const sd_t rec1 = d2bits(1.e-24 * 9.84815696 * std::pow(1.0 + z, 5.06773134));
      const sd_t dvv = d2bits(std::pow(Ls[bx] * 3.0856775807e24 / Ns[bx] / 0.7 / (1. + z), 3.0));
      const sd_t r2 = d2bits(1.76105133), r3 = d2bits(0.81722878), vn = d2bits(1.e+45);
      const sd_divc r2c = sd_divc_prepare(r2), vnc = sd_divc_prepare(vn);
      const RrecFast rf = rrec_fast_prepare(rec1, dvv, vn, r2, r3);
      if (!rf.ok) return 2;
      for (long i = 0; i < n; ++i) {
        const double gs = std::sqrt(-2.0 * std::log(1.0 - rnd_unit())) * std::cos(6.283185307179586 * rnd_unit());
        const float od = (i % 4) ? (float)std::exp(1.5 * gs) : rnd_float_exp(-60, 60);
        float got = 0.f;
        const bool fast = rrec_quick(od, rf, tab, &got);
        tally(rr, fast, got, fast ? sd_to_float(rrec_exact(od, r2c, r3, rec1, dvv, vnc)) : 0.f, od);
      }
    }
  for (long i = 0; i < 8 * n; ++i) {
    check_one_minus(om, (float)rnd_unit());
    check_one_minus(om, rnd_float_exp(-70, -1));
  }
  for (float f : {0.0f, 0.5f, 1.0f, 0x1p-24f, 0x1p-25f, 0x1p-53f, 0x1p-54f, 0x1p-55f, 0x1.8p-54f, 0x1.000002p-54f})
    for (int d = -3; d <= 3; ++d) {
      const float v = bits2f(f2bits(f) + (uint32_t)(f == 0.0f && d < 0 ? 0 : d));
      if (v >= 0.0f && v <= 1.0f) check_one_minus(om, v);
    }
  for (const Stat* s : {&xo, &xr, &rr, &om}) printf("%s %ld %ld %ld\n", s->name, s->n, s->bad, s->fallback);
  return 0;
}
