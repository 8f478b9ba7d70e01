// Fast paths for the HII prologue's per-voxel double chains, each returning
// the float that the exact chain would return (get_HIIbubbles.c:216-225,
// 272-274; user_functions.c:58-65, 101-106).
//
// The reference computes each per-voxel quantity as a chain of double
// operations and keeps only the result rounded to float.  softdouble.h
// reproduces every double operation bit for bit in integer arithmetic.  That
// is exact but long: a 124-bit fixed-point pow, a 212-bit fourth power, and
// 128/64-bit integer divisions.  The fast paths here evaluate the chain's
// real-number value F in 64-bit fixed point, with a proven relative error
// bound e_F.  The exact chain's double result D lies within a bound e_D of the
// same real number; each function states both bounds.  With e_D + e_F below
// 2^-48 and F further than 2^-46 (relative) from every float rounding
// midpoint, D and F round to the same float, which is returned
// (pf_round_guard).  Otherwise, or when an operand is outside the path's
// range, the function returns false and the caller evaluates the exact
// chain.  Float midpoints are 2^-23 apart (relative), so the guard band
// catches about one input in 2^21.
//
// Host and device compile the same code, so the CPU tests can compare every
// fast path with its exact chain on any number of inputs.
#pragma once
#include <math.h>

#include "softdouble.h"

// ---- shared pieces ----------------------------------------------------------

// floor(a b / 2^62) for signed Q.62 values whose product stays below 2^125.
SD_HD int64_t pf_mulq62(int64_t a, int64_t b) { return (int64_t)(((sd_i128)a * b) >> 62); }

// Float seeds of the Newton iterations: relative error up to 2^-21.  The
// iterations and guard bands allow for all of it (checked on the host with
// seeds at both ends, PF_SEED_ERR), so host and device may differ.
SD_HD float pf_seed_recip(float x) {
#ifdef __CUDA_ARCH__
  return __fdividef(1.0f, x);
#elif defined(PF_SEED_ERR)  // tests: a seed at the edge of its error
  return 1.0f / x * (1.0f + PF_SEED_ERR);
#else
  return 1.0f / x;
#endif
}

// Product of two significands with bit 63 set, normalised so that bit 63 is
// set again.  *e gains the product's binary exponent change.  Relative
// truncation error below 2^-62.
SD_HD uint64_t pf_mulnorm(uint64_t a, uint64_t b, int* e) {
  const sd_u128 p = (sd_u128)a * b;  // in [2^126, 2^128)
  if (p >> 127) return (uint64_t)(p >> 64);
  *e -= 1;
  return (uint64_t)(p >> 63);
}

// 1 / S for S in Q.62, [1, 2): two Newton steps from a float reciprocal
// (relative error 2^-23 -> 2^-46 -> below 3 units of 2^-62).  Newton's
// iterates for the reciprocal approach 1/S from below, up to the
// truncations, so the result is in (2^61, 2^62 + 1].
SD_HD int64_t pf_recip_q62(uint64_t S) {
  const float sf = (float)(S >> 32) * (1.0f / 1073741824.0f);  // S 2^-62 in float
  const float yf = 1.0f / sf;
  int64_t Y = (int64_t)(yf * 4611686018427387904.0f);           // Q.62
  const int64_t S62 = (int64_t)S;
  for (int it = 0; it < 2; ++it)  // 2 - S Y in Q.62 (2 = 2^63 as unsigned)
    Y = pf_mulq62(Y, (int64_t)((1ULL << 63) - (uint64_t)pf_mulq62(S62, Y)));
  return Y;
}

SD_HD float pf_bits_float(uint32_t u) {
  union {
    uint32_t u;
    float f;
  } c;
  c.u = u;
  return c.f;
}

// Round F = Fm 2^(eF - 64) (bit 63 of Fm set) to float, with sign bit `sign`
// (bit 31).  Returns false when F lies within `band` units of Fm (2^18:
// relative 2^-46) of a float rounding midpoint, or when the float would not be normal.
SD_HD bool pf_round_guard(uint64_t Fm, int eF, uint32_t sign, float* out, uint64_t band = 1ULL << 18) {
  const uint64_t rem = Fm & ((1ULL << 40) - 1);  // the dropped bits; midpoint 2^39
  const uint64_t half = 1ULL << 39;
  const uint64_t dist = rem > half ? rem - half : half - rem;
  if (dist <= band) return false;
  uint32_t sig = (uint32_t)(Fm >> 40) + (rem > half ? 1u : 0u);
  int E = eF - 1;  // F = (Fm / 2^63) 2^(eF - 1)
  if (sig >> 24) {
    sig >>= 1;
    E += 1;
  }
  if (E < -126 || E > 127) return false;
  *out = pf_bits_float(sign | ((uint32_t)(E + 127) << 23) | (sig & 0x7FFFFFu));
  return true;
}

// ---- products by constants: (..((x k0) k1)..) k[n-1] -----------------------
// The source conversion (:272-274, or :258 for the halo branch) and the
// residual-fraction argument (1 + d) 1.881e-7 (1+z)^3 G_H(z) (:220).
// e_D: n roundings, n u (u = 2^-53, n <= 6).  e_F: the constants' product
// kept to 64 bits (n - 1 truncations) and the final product, below 2^-60.
struct ProdFast {
  uint64_t km;     // K = k0 k1 .. = km 2^(kx - 64), bit 63 of km set
  int kx;
  int emin, emax;  // range of the partial products' exponents relative to x's
  int ok;          // 0: constants outside the path's range (exact chain always)
};

SD_HD bool prod_fast(sd_t x, const ProdFast& k, float* out) {
  if (!k.ok) return false;
  const uint32_t sign = (uint32_t)(x >> 63) << 31;
  const int ex = (int)((x >> 52) & 0x7FF);
  if (ex == 0x7FF) return false;
  if (ex == 0) {
    if ((x << 1) != 0) return false;  // subnormal
    *out = pf_bits_float(sign);       // +-0 k = +-0 for positive constants
    return true;
  }
  const int e = ex - 1023;
  // every partial product stays a normal double, as the n u bound assumes
  if (e + k.emin < -1000 || e + k.emax > 1000) return false;
  const uint64_t mx = ((x & 0xFFFFFFFFFFFFFULL) | (1ULL << 52)) << 11;  // x = mx 2^(e + 1 - 64)
  int eF = e + 1 + k.kx;
  const uint64_t Fm = pf_mulnorm(mx, k.km, &eF);
  return pf_round_guard(Fm, eF, sign, out);
}

// ---- one division: a / b rounded to double, then to float --------------------
// XHI's last step (user_functions.c:105).  e_D: u/2.  e_F: the reciprocal
// (2^-59.4) and the product (2^-62), below 2^-59.
SD_HD bool div_fast(sd_t a, sd_t b, float* out) {
  const uint32_t sign = (uint32_t)((a ^ b) >> 63) << 31;
  const int ea = (int)((a >> 52) & 0x7FF), eb = (int)((b >> 52) & 0x7FF);
  if (eb == 0 || eb == 0x7FF || ea == 0x7FF) return false;
  if (ea == 0) {
    if ((a << 1) != 0) return false;
    *out = pf_bits_float(sign);
    return true;
  }
  const uint64_t ma = ((a & 0xFFFFFFFFFFFFFULL) | (1ULL << 52)) << 11;  // a = ma 2^(ea - 1023 + 1 - 64)
  const uint64_t S = ((b & 0xFFFFFFFFFFFFFULL) | (1ULL << 52)) << 10;   // b's significand, Q.62
  const int64_t Y = pf_recip_q62(S);
  if (Y <= 0) return false;
  const int lz = sd_clz64((uint64_t)Y);
  // 1 / b = (Y << lz) 2^(2 - lz - 64) 2^-(eb - 1023)
  int eF = (ea - 1023 + 1) + (2 - lz) - (eb - 1023);
  const uint64_t Fm = pf_mulnorm(ma, (uint64_t)Y << lz, &eF);
  return pf_round_guard(Fm, eF, sign, out);
}

// ---- the recombination rate -------------------------------------------------
// density_map[i] = (float)Rrec((float)(1 + d), z) (:222, user_functions.c:58-65):
//   Rrec = rec1 * pow(rec2 / (1 + rec2), 4) * dvv / v_norm,  rec2 = pow(od / r2, r3).
// Real value: V = C (1 + 2^-w)^-4, w = r3 (log2 od - log2 r2), C = rec1 dvv / v_norm.
// e_D: od / r2 adds u, amplified by r3 < 1.  pow adds u plus at most 2^-59.
// 1 + rec2 and the division add 2u.  The fourth power multiplies that sum
// (3.9 u) by 4 and adds u.  The two products and the division by v_norm add
// 3u more: 19.4 u < 2^-48.6.  e_F: below 2^-56 (each step's bound is written
// at the step).
struct RrecFast {
  int64_t l2r2;  // log2(r2), Q.62
  uint64_t r3;   // r3, Q.63 (2^-11 <= r3 < 1)
  uint64_t cm;   // C = cm 2^(cx - 64), bit 63 of cm set
  int cx;
  int ok;        // 0: constants outside the path's range (exact chain always)
};

// The exact chain, operation by operation as user_functions.c:58-65.
SD_HD sd_t rrec_exact(float od, const sd_divc& r2c, sd_t r3, sd_t rec1, sd_t dvv, const sd_divc& v_normc) {
  const sd_t rec2 = sd_pow(sd_div_c(sd_from_float(od), r2c), r3);
  const sd_t q = sd_div(rec2, sd_add(0x3FF0000000000000ULL, rec2));
  const sd_t rec3 = sd_pow4(q);  // pow(.., 4.): correctly rounded like sd_pow
  return sd_div_c(sd_mul(sd_mul(rec1, rec3), dvv), v_normc);
}

// Float value of Rrec(od) in *out and true, or false (guard band, od outside
// [2^-60, 2^61), a result outside the normal float range, or constants out of
// range): the caller then uses rrec_exact.
SD_HD bool rrec_fast(float od, const RrecFast& k, float* out) {
  union {
    float f;
    uint32_t u;
  } cv;
  cv.f = od;
  const uint32_t fb = cv.u;
  const int eo = (int)((fb >> 23) & 255);
  if (!k.ok || (fb >> 31) || eo == 0 || eo == 255) return false;
  const int e = eo - 127;
  if (e < -60 || e > 60) return false;

  // log2(od) = e + log2(c_j) + ln(1 + t) / ln 2, c_j = 2^62 / SD_POW_INV[j]
  // (the table of sd_pow, j = top 7 fraction bits), t = m / c_j - 1 with
  // |t| <= 2^-8.  t is taken exactly from the 86-bit product and truncated to
  // Q.62.  The series to t^7 leaves |t|^8 / 8 < 2^-67.  The Horner steps,
  // 1/ln 2 and the two tables add at most 6 units of 2^-62.
  const uint64_t mo = (fb & 0x7FFFFFu) | 0x800000u;  // m 2^23
  const int j = (int)((mo >> 16) & 127);
  const sd_u128 P = (sd_u128)mo * SD_POW_INV[j];     // (m / c_j) 2^85
  const int64_t T = (int64_t)(((sd_i128)P - ((sd_i128)1 << 85)) >> 23);
  const int64_t Q1 = (int64_t)1 << 62;
  int64_t acc = Q1 / 7;
  acc = -(Q1 / 6) + pf_mulq62(T, acc);
  acc = Q1 / 5 + pf_mulq62(T, acc);
  acc = -(Q1 / 4) + pf_mulq62(T, acc);
  acc = Q1 / 3 + pf_mulq62(T, acc);
  acc = -(Q1 / 2) + pf_mulq62(T, acc);
  acc = Q1 + pf_mulq62(T, acc);
  const int64_t lnp = pf_mulq62(T, acc);  // ln(1 + t)
  const int64_t inv_ln2 = (int64_t)((SD_POW_INV_LN2_HI << 2) | (SD_POW_INV_LN2_LO >> 62));
  const int64_t l2c = (int64_t)((SD_POW_L2C_HI[j] << 30) | (SD_POW_L2C_LO[j] >> 34));
  const int64_t dfrac = l2c + pf_mulq62(lnp, inv_ln2) - k.l2r2;  // |dfrac| < 2

  // w = r3 (e + dfrac) in Q.63; error at most r3 6 + 1/2 units of 2^-62, under
  // 2^-59.6.  v = -w = nv + f with f in [0, 1).
  const sd_i128 W = (sd_i128)k.r3 * e + (((sd_i128)k.r3 * dfrac) >> 62);
  const sd_i128 V = -W;
  const int nv = (int)(V >> 63);
  const uint64_t f = (uint64_t)(V - (sd_i128)nv * ((sd_i128)1 << 63));  // Q.63 (nv may be negative)

  // 2^f = 2^(j2/128) e^x, x = (f - j2/128) ln 2 < 2^-7.5, series to x^6
  // (remainder < 2^-65).  U in Q.62, [1, 2); relative error (the error of w
  // included) below 2^-59.2.
  const int j2 = (int)(f >> 56);
  const int64_t ln2 = (int64_t)((SD_POW_LN2_HI << 2) | (SD_POW_LN2_LO >> 62));
  const int64_t X = pf_mulq62((int64_t)((f & ((1ULL << 56) - 1)) >> 1), ln2);
  int64_t ex = Q1 / 720;
  ex = Q1 / 120 + pf_mulq62(X, ex);
  ex = Q1 / 24 + pf_mulq62(X, ex);
  ex = Q1 / 6 + pf_mulq62(X, ex);
  ex = Q1 / 2 + pf_mulq62(X, ex);
  ex = Q1 + pf_mulq62(X, ex);
  ex = Q1 + pf_mulq62(X, ex);
  const int64_t e2t = (int64_t)((SD_POW_EXP2T_HI[j2] << 2) | (SD_POW_EXP2T_LO[j2] >> 62));
  const uint64_t U = (uint64_t)pf_mulq62(e2t, ex);

  // s = 1 + 2^-w = 1 + U 2^nv = S 2^es, S in Q.62, [1, 2); two truncations.
  uint64_t S;
  int es;
  if (nv >= 0) {
    S = U + (nv < 63 ? (1ULL << 62) >> nv : 0);
    es = nv;
  } else {
    S = (1ULL << 62) + (nv > -64 ? U >> (-nv) : 0);
    es = 0;
  }
  if (S >> 63) {
    S >>= 1;
    es += 1;
  }

  // y = 1 / S (3 units of 2^-62).  F = C y^4 2^(-4 es): three normalised
  // products (relative error < 2^-62 each).  Relative error of F: 4 x 2^-58.5
  // (s and y) plus the products and C, below 2^-56.
  const int64_t Y = pf_recip_q62(S);
  if (Y <= 0) return false;
  const int lz = sd_clz64((uint64_t)Y);
  const uint64_t ym = (uint64_t)Y << lz;  // y = ym 2^(2 - lz - 64)
  int e2 = 2 * (2 - lz);
  const uint64_t y2 = pf_mulnorm(ym, ym, &e2);
  int e4 = 2 * e2;
  const uint64_t y4 = pf_mulnorm(y2, y2, &e4);
  int eF = e4 + k.cx - 4 * es;
  const uint64_t Fm = pf_mulnorm(y4, k.cm, &eF);  // F = Fm 2^(eF - 64)
  return pf_round_guard(Fm, eF, 0u, out);
}

// The same value, with a guard band of 2^25 units (2^-39 or more): it declines
// for about one input in 2^14, which then takes rrec_fast.  The error is that
// of 1 / S four times over: the seed's 2^-21 and the rounding of its argument
// (2^-24) give 2^-41.6 after the Newton step and 2^-39.6 in the fourth power,
// which leaves a third of the band to the series (2^-44 each, four times over).
// The series' terms of third and higher order (below 2^-25) are evaluated in
// float, the squares from 31-bit factors.  tab: rrec_table's 3 x 128 words.
SD_HD bool rrec_quick(float od, const RrecFast& k, const uint64_t* tab, float* out) {
  union {
    float f;
    uint32_t u;
  } cv;
  cv.f = od;
  const uint32_t fb = cv.u;
  const int eo = (int)((fb >> 23) & 255);
  const int e = eo - 127;
  if (!k.ok || (fb >> 31) || e < -60 || e > 60) return false;
  const uint64_t mo = (fb & 0x7FFFFFu) | 0x800000u;
  const int j = (int)((mo >> 16) & 127);
  // t = m / c_j - 1 in Q.52 (|t| <= 2^-8), ln(1 + t): error below 2^-45
  const sd_u128 P = (sd_u128)mo * tab[j];
  const int64_t T = (int64_t)(uint64_t)(P >> 33) - ((int64_t)1 << 52);
  const int32_t th = (int32_t)(T >> 14);  // Q.38
  const float tf = (float)th * 3.637978807091713e-12f;
  const float tc = tf * tf * tf * (0.33333333f + tf * (-0.25f + tf * (0.2f - tf * 0.16666667f)));
  const int64_t lnp = T - (((int64_t)th * th) >> 25) + (int32_t)(tc * 4503599627370496.0f);
  // w = r3 (e + log2 parts) in Q.52
  const int64_t inv_ln2 = (int64_t)((SD_POW_INV_LN2_HI << 2) | (SD_POW_INV_LN2_LO >> 62));
  const int64_t L = ((int64_t)e << 52) + (int64_t)(tab[128 + j] >> 10) + pf_mulq62(lnp, inv_ln2) - (k.l2r2 >> 10);
  const int64_t v = -(int64_t)(((sd_i128)L * (int64_t)k.r3) >> 63);
  const int nv = (int)(v >> 52);
  const uint64_t f = (uint64_t)v & ((1ULL << 52) - 1);
  // 2^f = 2^(j2/128) e^x, x < 2^-7.5 in Q.52: error below 2^-44
  const int j2 = (int)(f >> 45);
  const uint64_t X = sd_mulhi64(f & ((1ULL << 45) - 1), SD_POW_LN2_HI << 4);
  const uint32_t xh = (uint32_t)(X >> 14);  // Q.38
  const float xf = (float)xh * 3.637978807091713e-12f;
  const float xc = xf * xf * xf * (0.16666667f + xf * (0.041666667f + xf * 0.0083333333f));
  const uint64_t ex = (1ULL << 52) + X + (((uint64_t)xh * xh) >> 25) + (uint32_t)(xc * 4503599627370496.0f);
  const uint64_t U = sd_mulhi64(tab[256 + j2] << 1, ex << 11);  // Q.62, [1, 2)
  uint64_t S;
  int es;
  if (nv >= 0) {
    S = U + (nv < 63 ? (1ULL << 62) >> nv : 0);
    es = nv;
  } else {
    S = (1ULL << 62) + (nv > -64 ? U >> (-nv) : 0);
    es = 0;
  }
  if (S >> 63) {
    S >>= 1;
    es += 1;
  }
  // 1 / S by one Newton step from a float seed: error below 2^-41.6
  const float yf = pf_seed_recip((float)(uint32_t)(S >> 32) * (1.0f / 1073741824.0f));
  const uint64_t Y0 = (uint64_t)(uint32_t)(yf * 1073741824.0f) << 32;           // Q.62
  const uint64_t t1 = (1ULL << 61) - sd_mulhi64(S, Y0);                         // 2 - S Y0, Q.60
  const uint64_t Y = sd_mulhi64(Y0, t1) << 4;                                   // Q.62
  if (Y == 0) return false;
  const int lz = sd_clz64(Y);
  const uint64_t ym = Y << lz;
  int e2 = 2 * (2 - lz);
  const uint64_t y2 = pf_mulnorm(ym, ym, &e2);
  int e4 = 2 * e2;
  const uint64_t y4 = pf_mulnorm(y2, y2, &e4);
  int eF = e4 + k.cx - 4 * es;
  const uint64_t Fm = pf_mulnorm(y4, k.cm, &eF);
  return pf_round_guard(Fm, eF, 0u, out, 1ULL << 25);
}
// Word i of the table: 2^62 / c_j, log2 c_j (Q.62), 2^(j/128) (Q.62).
SD_HD uint64_t rrec_table(int i) {
  const int j = i & 127;
  if (i < 128) return SD_POW_INV[j];
  if (i < 256) return (SD_POW_L2C_HI[j] << 30) | (SD_POW_L2C_LO[j] >> 34);
  return (SD_POW_EXP2T_HI[j] << 2) | (SD_POW_EXP2T_LO[j] >> 62);
}

// ---- the residual neutral fraction -----------------------------------------
// XHI(ratio), user_functions.c:101-106, operation by operation in double.
SD_HD sd_t xhi_exact(sd_t r) {
  if (sd_is_zero(r)) return 0;
  const sd_t two_r = sd_ldexp(r, 1);                        // 2.*ratio (exact)
  const sd_t b = sd_add(two_r, 0x3FF0000000000000ULL);      // 2.*ratio + 1.
  const sd_t c = sd_mul(b, b);                              // (..)*(..)
  const sd_t e = sd_mul(sd_ldexp(r, 2), r);                 // 4.*ratio*ratio
  const sd_t g = sd_sqrt_fast(sd_sub(c, e));
  const sd_t num = sd_sub(b, g);                            // 2.*ratio + 1. - sqrt(..)
  return sd_div(num, two_r);                                // /(2.*ratio)
}

// (float)XHI(ratio) for 2^-30 <= ratio < 1/2.  Below 2^-4, with b = 2 ratio, 1 + b
// and 1 + 2 b are exact doubles, and the reference's c = (1 + b)^2 rounded,
// minus 4 ratio^2 = b^2 (exact), rounds back to exactly 1 + 2 b: the rounding
// error of c is at most 2^-53, 1 + 2 b is a multiple of 2^-51.  So its
// numerator is 1 + b - g with g = sqrt(1 + 2 b) rounded to a multiple of
// 2^-52, i.e. n 2^-52 with n the integer nearest to
//   2^52 (1 + b - sqrt(1 + 2 b)) = 2^52 b^2 u,  u = 1 / (1 + b + sqrt(1 + 2 b)),
// u the root of b^2 u^2 - 2 (1 + b) u + 1 = 0: two Newton steps from a float
// seed, with the derivative -2 sqrt(1 + 2 b) in float (error of u below 2^-60).
// Then n 2^-52 / b, whose two roundings give the float unless the quotient
// lies near a midpoint.  False: outside the range, n undecided (its fraction
// within 64 units of one half), or the quotient in the guard band.
// For 2^-4 <= ratio < 1/2 (b < 1), the bulk of a box from redshift 11 up, c
// and c - 4 ratio^2 (< 4) are rounded by 2^-52 at most each and g by 2^-53, so
// the numerator (exact, 2^-7.2 at least) is within 1.4 2^-52 of 1 + b - g, a
// relative 2^-44.3, and the quotient is b u to that: the same u, and a guard
// band of 2^-42 at least (256^3 at redshift 12, 60 % of the cells there: 1.9 -> 0.5 ms).
SD_HD bool xhi_fast(float ratio, float* out) {
  union {
    float f;
    uint32_t u;
  } cv;
  cv.f = ratio;
  const int er = (int)(cv.u >> 23) - 127;  // a sign bit makes it large
  if (er < -30 || er > -2) return false;
  const uint64_t M = (cv.u & 0x7FFFFFu) | 0x800000u;
  const int k = 22 - er;  // b = M 2^-k, 24 <= k <= 52
  const uint64_t M2 = M * M;
  const int s2 = 64 - 2 * k;
  const uint64_t B2 = s2 >= 0 ? M2 << s2 : M2 >> -s2;           // b^2, Q.64
  const uint64_t A = (1ULL << 63) + (M << (63 - k));            // 2 (1 + b), Q.62
  const float bf = 2.0f * ratio;
  const float sf = sqrtf(1.0f + 2.0f * bf);
  const float g2 = pf_seed_recip(sf) * 2.0f;                     // 4 / (2 sqrt(1 + 2 b))
  uint64_t U = (uint64_t)(uint32_t)(pf_seed_recip(1.0f + bf + sf) * 4294967296.0f) << 32;  // u, Q.64
  // residual 1 - u (2 (1 + b) - b^2 u) in Q.62; the correction in Q.64 is residual x g2
  int64_t f = (int64_t)((1ULL << 62) - sd_mulhi64(A - (sd_mulhi64(B2, U) >> 2), U));
  U += (uint64_t)((int64_t)(int32_t)((float)(int32_t)(f >> 14) * g2) * 16384);
  f = (int64_t)((1ULL << 62) - sd_mulhi64(A - (sd_mulhi64(B2, U) >> 2), U));
  U += (uint64_t)(int64_t)(int32_t)((float)(int32_t)f * g2);
  if (er > -5) {
    const int lu = sd_clz64(U);
    int eF = 24 - k - lu;
    const uint64_t Fm = pf_mulnorm(M << 40, U << lu, &eF);
    return pf_round_guard(Fm, eF, 0u, out, 1ULL << 22);
  }
  const uint64_t V = sd_mulhi64(M2 << 16, U);                    // M^2 u 2^16; n = V 2^-(2k - 36)
  const int sh = 2 * k - 36;
  if (sh >= 64) {  // V < 2^63: n = 0
    *out = 0.0f;
    return true;
  }
  const uint64_t rem = V & ((1ULL << sh) - 1), half = 1ULL << (sh - 1);
  if ((rem > half ? rem - half : half - rem) < 64) return false;
  const uint64_t n = (V >> sh) + (rem > half ? 1 : 0);
  if (n == 0) {
    *out = 0.0f;
    return true;
  }
  // F = n 2^(k - 52) / M, 1 / M by one Newton step from a float seed (error
  // below 2^-42; band 2^23 units)
  const float mf = (float)(uint32_t)M * 1.1920928955078125e-07f;  // M 2^-23, exact
  const uint32_t y0 = (uint32_t)(pf_seed_recip(mf) * 2147483648.0f);  // Q.31
  const uint64_t Y0 = (uint64_t)y0 << 32;                             // Q.63
  const uint64_t t1 = (1ULL << 63) - sd_mulhi64(M << 40, Y0);         // 2 - m y0, Q.62
  uint64_t Y = sd_mulhi64(Y0, t1);                                    // Q.61
  const int lz2 = sd_clz64(Y);                                        // 1/m in (1/2, 1]: 2 or 3
  Y <<= lz2;
  const int lz = sd_clz64(n);
  int eF = k - 10 - lz - (lz2 - 2);
  const uint64_t Fm = pf_mulnorm(n << lz, Y, &eF);
  return pf_round_guard(Fm, eF, 0u, out, 1ULL << 23);
}

// (float)XHI(ratio).  The subtraction 2 ratio + 1 - sqrt(..) cancels most
// digits for small ratios, so outside xhi_fast every step before the division
// stays exact; the division takes the fast path (div_fast).
SD_HD float xhi_float(float ratio) {
  float q;
  if (xhi_fast(ratio, &q)) return q;
  const sd_t r = sd_from_float(ratio);
  if (sd_is_zero(r)) return 0.0f;
  const sd_t two_r = sd_ldexp(r, 1);
  const sd_t b = sd_add(two_r, 0x3FF0000000000000ULL);
  const sd_t c = sd_mul(b, b);
  const sd_t e = sd_mul(sd_ldexp(r, 2), r);
  const sd_t g = sd_sqrt_fast(sd_sub(c, e));
  const sd_t num = sd_sub(b, g);
  float x;
  if (!div_fast(num, two_r, &x)) x = sd_to_float(sd_div(num, two_r));
  return x;
}

// ---- the cap 1 - fresid (:469-471) -------------------------------------------
// o = 1.0 - f in double for a float f in [0, 1]: *lo = the largest float <= o,
// *rn = the float nearest to o.  1 - f rounded once to float equals the double
// rounded to float (53 >= 2 24 + 1), and o < rn exactly when 1 - f lies more
// than half a double ulp (2^-54 below 1; a tie goes to rn) under rn; for
// f >= 1/2 the float difference is exact.
SD_HD void one_minus(float f, float* lo, float* rn) {
  const float r = 1.0f - f;
  union {
    float f;
    uint32_t u;
  } cv;
  cv.f = r;
  if (f < 0.5f && f - (1.0f - r) > 5.5511151231257827e-17f) cv.u -= 1;
  *rn = r;
  *lo = cv.f;
}

// ---- host preparation of the constants (host code; visible to both nvcc passes) ---------------------------------------
static inline bool pf_normal_pos(sd_t x) {
  const int ex = (int)((x >> 52) & 0x7FF);
  return !(x >> 63) && ex != 0 && ex != 0x7FF;
}

// K = k0 k1 .. k[n-1] for positive normal doubles, kept to 64 bits after each
// product (truncation below 2^-63 per product).
static inline ProdFast prod_fast_prepare(const sd_t* ks, int n) {
  ProdFast k = {};
  if (n < 1 || n > 6) return k;
  uint64_t m = 1ULL << 63;
  int x = 1;  // value 1 = 2^63 2^(1 - 64)
  int pe = 0;
  k.emin = k.emax = 0;
  for (int i = 0; i < n; ++i) {
    if (!pf_normal_pos(ks[i])) return k;
    const int ei = (int)((ks[i] >> 52) & 0x7FF) - 1023;
    const uint64_t mi = ((ks[i] & 0xFFFFFFFFFFFFFULL) | (1ULL << 52)) << 11;
    x += ei + 1;
    m = pf_mulnorm(m, mi, &x);
    pe += ei;  // the i + 1 significands' product adds 0 .. i + 1 more
    if (pe < k.emin) k.emin = pe;
    if (pe + i + 1 > k.emax) k.emax = pe + i + 1;
  }
  k.km = m;
  k.kx = x;
  k.ok = 1;
  return k;
}

// log2 r2 from sd_pow's own fixed-point logarithm (error far below 2^-62);
// C from the exact 106-bit product rec1 dvv divided by v_norm in 128-bit
// integers (truncation below 2^-62 relative).
static inline RrecFast rrec_fast_prepare(sd_t rec1, sd_t dvv, sd_t v_norm, sd_t r2, sd_t r3) {
  RrecFast k = {};
  if (!pf_normal_pos(rec1) || !pf_normal_pos(dvv) || !pf_normal_pos(v_norm) || !pf_normal_pos(r2) ||
      !pf_normal_pos(r3))
    return k;
  const int e3 = (int)((r3 >> 52) & 0x7FF) - 1023;
  const int e2 = (int)((r2 >> 52) & 0x7FF) - 1023;
  if (e3 > -1 || e3 < -11 || e2 < -60 || e2 > 60) return k;
  const uint64_t m3 = (r3 & 0xFFFFFFFFFFFFFULL) | (1ULL << 52);
  k.r3 = m3 << (11 + e3);  // r3 = m3 2^(e3 - 52) in Q.63
  k.l2r2 = (int64_t)(sd_log2_q96(r2) >> 34);
  const uint64_t ma = (rec1 & 0xFFFFFFFFFFFFFULL) | (1ULL << 52);
  const uint64_t mb = (dvv & 0xFFFFFFFFFFFFFULL) | (1ULL << 52);
  const uint64_t mv = (v_norm & 0xFFFFFFFFFFFFFULL) | (1ULL << 52);
  const int ea = (int)((rec1 >> 52) & 0x7FF) - 1023;
  const int eb = (int)((dvv >> 52) & 0x7FF) - 1023;
  const int ev = (int)((v_norm >> 52) & 0x7FF) - 1023;
  // C = (ma mb / mv) 2^(ea + eb - ev - 52); q = floor(ma mb 2^22 / mv) in [2^73, 2^76)
  const sd_u128 q = (((sd_u128)ma * mb) << 22) / mv;
  const int lead = 127 - sd_clz128(q);
  k.cm = (uint64_t)(q >> (lead - 63));
  // C = q 2^(ea + eb - ev - 74) = (cm 2^-64) 2^(lead + 1 + ea + eb - ev - 74)
  k.cx = lead + 1 + ea + eb - ev - 74;
  k.ok = 1;
  return k;
}
