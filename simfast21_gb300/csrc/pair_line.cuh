// Line FFTs of two radii at once.
//
// Pairs.  A value of a radius pair is a cpair: the real parts of radii 2p and
// 2p + 1 in one 64-bit register pair, the imaginary parts in another.
// sm_103a has packed single-precision add, multiply and fused multiply-add
// (f32x2), each lane rounded on its own exactly as the scalar instruction
// rounds, so one instruction advances both radii and every radius keeps the
// bits of the scalar transform.
//
// Groups.  A line of N points runs the Stockham stages of fft_line.cuh (N a
// power of two) or kernels_gen.cu (2-3-5 sides) in the same order, in two or
// three groups of consecutive stages.  A thread holds all the elements that
// a group's stages combine, so inside a group the Stockham reordering is a
// renaming of registers; shared memory is crossed only between groups.  Where
// the radices give no good cut, a radix-8 stage is cut inside: its first one
// or two levels (S8A2, S8A4) end a group, the others (S8B4, S8B2) begin the
// next; the butterfly graph is that of dft8, so the bits are too.
//
// Why: the scalar passes take 59 / 37 / 45 instructions per voxel and radius
// (filter / ky / kx pass, 512^3) and the 2-3-5 sides went through shared
// memory at every stage.  Pairs halve the arithmetic, twiddle and address
// instructions; groups of 5 to 16 elements keep the exchanges at one or two
// per line with enough threads per SM to hide the latencies.
#pragma once
#include "fft_line.cuh"
#include "sf21_device.cuh"

namespace sf21 {

struct __align__(16) cpair {
  float2 re, im;  // lanes x, y: radii 2p, 2p + 1
};

// Written as PTX with the rounding named: the two-wide intrinsics (__fmul2_rn
// followed by __fadd2_rn) were seen to be contracted into one fused
// multiply-add (first hits that differed from the scalar pipelines').
#define SF21_F32X2(NAME)                                                                                       \
  __device__ __forceinline__ float2 NAME##2(float2 a, float2 b) {                                              \
    float2 d;                                                                                                  \
    asm("{.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t" #NAME                       \
        ".rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;}"                                                          \
        : "=f"(d.x), "=f"(d.y)                                                                                 \
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                             \
    return d;                                                                                                  \
  }
SF21_F32X2(add)
SF21_F32X2(sub)
SF21_F32X2(mul)
#undef SF21_F32X2
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }

__device__ __forceinline__ cpair padd(cpair a, cpair b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ cpair psub(cpair a, cpair b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a + (-i b) forward, a + i b inverse; and the difference
template <bool INV>
__device__ __forceinline__ cpair padd_mi(cpair a, cpair b) {
  return INV ? cpair{sub2(a.re, b.im), add2(a.im, b.re)} : cpair{add2(a.re, b.im), sub2(a.im, b.re)};
}
template <bool INV>
__device__ __forceinline__ cpair psub_mi(cpair a, cpair b) {
  return INV ? cpair{add2(a.re, b.im), sub2(a.im, b.re)} : cpair{sub2(a.re, b.im), add2(a.im, b.re)};
}
// a w of both radii by one twiddle: cmul's products and roundings per lane
// (the product that cmul negates is formed with the negated factor)
__device__ __forceinline__ cpair pcmul(cpair a, float2 w) {
  const float2 wx = dup2(w.x), wy = dup2(w.y), wn = dup2(-w.y);
  return {fma2(a.re, wx, mul2(a.im, wn)), fma2(a.re, wy, mul2(a.im, wx))};
}

template <bool INV>
__device__ __forceinline__ void pdft2(cpair& a, cpair& b) {
  const cpair t = a;
  a = padd(t, b);
  b = psub(t, b);
}

template <bool INV>
__device__ __forceinline__ void pdft4(cpair& a0, cpair& a1, cpair& a2, cpair& a3) {
  const cpair t0 = padd(a0, a2), t1 = psub(a0, a2);
  const cpair t2 = padd(a1, a3), t3 = psub(a1, a3);
  a0 = padd(t0, t2);
  a2 = psub(t0, t2);
  a1 = padd_mi<INV>(t1, t3);
  a3 = psub_mi<INV>(t1, t3);
}

// Last level of dft8 for output k of 0..3: e + w8^k o and e - w8^k o, with
// w8 o = h s, s a sum of the parts of o (a negated sum is kept positive and
// its sign moves to h).
template <bool INV, int KK>
__device__ __forceinline__ void p8_last(cpair& e, cpair& o) {
  const float2 h = dup2(0.70710678118654752440f), hn = dup2(-0.70710678118654752440f);
  cpair s, d;
  if constexpr (KK == 0) {
    s = padd(e, o);
    d = psub(e, o);
  } else if constexpr (KK == 2) {
    s = padd_mi<INV>(e, o);
    d = psub_mi<INV>(e, o);
  } else {
    const float2 df = sub2(o.re, o.im), sm = add2(o.re, o.im);
    if constexpr ((KK == 1) == INV) {
      if constexpr (KK == 1) {  // inverse, k = 1: s = (re - im, re + im)
        s = {fma2(h, df, e.re), fma2(h, sm, e.im)};
        d = {fma2(hn, df, e.re), fma2(hn, sm, e.im)};
      } else {  // forward, k = 3: s = (im - re, -(re + im))
        s = {fma2(hn, df, e.re), fma2(hn, sm, e.im)};
        d = {fma2(h, df, e.re), fma2(h, sm, e.im)};
      }
    } else {
      if constexpr (KK == 1) {  // forward, k = 1: s = (re + im, im - re)
        s = {fma2(h, sm, e.re), fma2(hn, df, e.im)};
        d = {fma2(hn, sm, e.re), fma2(h, df, e.im)};
      } else {  // inverse, k = 3: s = (-(re + im), re - im)
        s = {fma2(hn, sm, e.re), fma2(h, df, e.im)};
        d = {fma2(h, sm, e.re), fma2(hn, df, e.im)};
      }
    }
  }
  e = s;
  o = d;
}

// The second and third level of dft8 on the differences D_0..D_3 of its
// first: outputs 1, 3, 5, 7 (in a0..a3).  On the sums S they are pdft4.
template <bool INV>
__device__ __forceinline__ void pdft4_odd(cpair& a0, cpair& a1, cpair& a2, cpair& a3) {
  cpair e1 = padd_mi<INV>(a0, a2), e3 = psub_mi<INV>(a0, a2);
  cpair o1 = padd_mi<INV>(a1, a3), o3 = psub_mi<INV>(a1, a3);
  p8_last<INV, 1>(e1, o1);  // e1: output 1, o1: output 5
  p8_last<INV, 3>(e3, o3);  // e3: output 3, o3: output 7
  a0 = e1;
  a1 = e3;
  a2 = o1;
  a3 = o3;
}

template <bool INV>
__device__ __forceinline__ void pdft8(cpair* v) {
  cpair e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  cpair o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  pdft4<INV>(e0, e1, e2, e3);
  pdft4<INV>(o0, o1, o2, o3);
  p8_last<INV, 0>(e0, o0);
  p8_last<INV, 1>(e1, o1);
  p8_last<INV, 2>(e2, o2);
  p8_last<INV, 3>(e3, o3);
  v[0] = e0;
  v[1] = e1;
  v[2] = e2;
  v[3] = e3;
  v[4] = o0;
  v[5] = o1;
  v[6] = o2;
  v[7] = o3;
}

// dft3 and dft5 of kernels_gen.cu with the fused multiply-adds that the
// compiler forms there, written out; G600: those of kernels_gen600.cu, whose
// source fixes other roundings (the products of dft3 are scalar, so that they
// are not fused with the additions that they feed).
template <bool INV, bool G600>
__device__ __forceinline__ void pdft3(cpair& x0, cpair& x1, cpair& x2) {
  const float s = INV ? -0.86602540378443864676f : 0.86602540378443864676f;
  const float2 s2 = dup2(s), sn = dup2(-s), mh = dup2(-0.5f);
  const cpair t1 = padd(x1, x2), t2 = psub(x1, x2);
  const cpair m = {fma2(mh, t1.re, x0.re), fma2(mh, t1.im, x0.im)};
  x0 = padd(x0, t1);
  if constexpr (G600) {
    const cpair b = {make_float2(__fmul_rn(s, t2.re.x), __fmul_rn(s, t2.re.y)),
                     make_float2(__fmul_rn(s, t2.im.x), __fmul_rn(s, t2.im.y))};
    x1 = padd_mi<false>(m, b);  // the sign of the direction is in s
    x2 = psub_mi<false>(m, b);
  } else {
    x1 = {fma2(s2, t2.im, m.re), fma2(sn, t2.re, m.im)};
    x2 = {fma2(sn, t2.im, m.re), fma2(s2, t2.re, m.im)};
  }
}

template <bool INV, bool G600>
__device__ __forceinline__ void pdft5(cpair& x0, cpair& x1, cpair& x2, cpair& x3, cpair& x4) {
  const float2 c1 = dup2(0.30901699437494742410f), c2 = dup2(-0.80901699437494742410f);
  const float f1 = INV ? -0.95105651629515357212f : 0.95105651629515357212f;
  const float f2 = INV ? -0.58778525229247312917f : 0.58778525229247312917f;
  const float2 s1 = dup2(f1), s2 = dup2(f2), s1n = dup2(-f1);
  const cpair p1 = padd(x1, x4), m1 = psub(x1, x4), p2 = padd(x2, x3), m2 = psub(x2, x3);
  const cpair a1 = {fma2(c2, p2.re, fma2(c1, p1.re, x0.re)), fma2(c2, p2.im, fma2(c1, p1.im, x0.im))};
  const cpair a2 = {fma2(c1, p2.re, fma2(c2, p1.re, x0.re)), fma2(c1, p2.im, fma2(c2, p1.im, x0.im))};
  cpair b1, b2;
  if constexpr (G600) {
    b1 = {fma2(s2, m2.re, mul2(s1, m1.re)), fma2(s2, m2.im, mul2(s1, m1.im))};
    b2 = {fma2(s1n, m2.re, mul2(s2, m1.re)), fma2(s1n, m2.im, mul2(s2, m1.im))};
  } else {
    b1 = {fma2(s1, m1.re, mul2(s2, m2.re)), fma2(s1, m1.im, mul2(s2, m2.im))};
    b2 = {fma2(s2, m1.re, mul2(s1n, m2.re)), fma2(s2, m1.im, mul2(s1n, m2.im))};
  }
  x0 = padd(x0, padd(p1, p2));
  x1 = padd_mi<false>(a1, b1);  // the sign of the direction is in s1, s2
  x4 = psub_mi<false>(a1, b1);
  x2 = padd_mi<false>(a2, b2);
  x3 = psub_mi<false>(a2, b2);
}

// ---- plans --------------------------------------------------------------------
// Stage codes: a radix, or a part of a radix-8 stage.
constexpr int S8A2 = 12;  // first level of a radix-8 stage (radix 2, the stage's twiddles)
constexpr int S8B4 = 14;  // its second and third level (radix 4, no twiddles)
constexpr int S8A4 = 24;  // first and second level (radix 4, the stage's twiddles)
constexpr int S8B2 = 22;  // its third level (radix 2, no twiddles)
constexpr int CUT = 0;    // ends a group
__host__ __device__ constexpr int stage_radix(int c) { return c == CUT ? 1 : c > 10 ? c % 10 : c; }

// A line: its length, the threads that share it, and the stage codes of its
// groups, CUT between groups.
template <int N_, int T_, int... CODES>
struct PairLine {
  static constexpr int N = N_;
  static constexpr int T = T_;
  static constexpr int n = sizeof...(CODES);
  __host__ __device__ static constexpr int code(int i) {
    const int c[] = {CODES...};
    return c[i];
  }
  // group g (0, 1, 2): its first code, elements per thread, the span before it
  __host__ __device__ static constexpr int first(int g) {
    int i = 0;
    for (; i < n && g > 0; ++i)
      if (code(i) == CUT) --g;
    return g > 0 ? n : i;
  }
  __host__ __device__ static constexpr int elems(int g) {
    int e = 1;
    for (int i = first(g); i < n && code(i) != CUT; ++i) e *= stage_radix(code(i));
    return e;
  }
  __host__ __device__ static constexpr int cut_span() {  // span before the radix-8 stage that is cut, 0 if none
    int ns = 1;
    for (int i = 0; i < n; ++i) {
      if (code(i) == S8A2 || code(i) == S8A4) return ns;
      ns *= stage_radix(code(i));
    }
    return 0;
  }
  static constexpr int E1 = elems(0), E2 = elems(1), E3 = elems(2);
  static constexpr int GROUPS = E3 > 1 ? 3 : 2;
  static constexpr int EL = GROUPS == 3 ? E3 : E2;             // last group
  static constexpr int Q1 = N / E1, Q2 = N / E2, QL = N / EL;  // subsets of the groups
  static constexpr int IT1 = (Q1 + T - 1) / T, IT2 = (Q2 + T - 1) / T, ITL = (QL + T - 1) / T;
  static constexpr int TW = N + (N == 600 ? 600 : 8 * cut_span());  // twiddle entries in shared memory
  // cpairs of a row's exchange: padded by one in eight when group 1 writes with an even stride
  static constexpr int XR = E1 % 2 == 0 ? N + N / 8 : N;
  static_assert(E1 * E2 * E3 == N, "the codes do not cover the line");
};

// Twiddle tables in shared memory.  The stage of span Ns and radix R has its
// factors w^(k r N/(Ns R)), k < Ns, 1 <= r < R, at (r - 1) Ns + k from Ns on
// (consecutive k on consecutive banks; the stages' tables [Ns, Ns R) follow one
// another).  A radix-8 stage that is cut has them for r = 0 too (ones), at
// N + r Ns + k.
// N = 600 follows kernels_gen600.cu, 600 = 25 x 24: radices 5, 5, 8, 3, where
// the values that enter the radix-8 stage take the whole twiddle w^(n1 k) of
// their position k + 25 n1 (at N + 25 n1 + k) and the radix-3 stage only
// w24^(r (k / 25)).
// plain: w^t = exp(-2 pi i t / N), t < N
template <class L, int I = 0, int NS = 1>
__device__ __forceinline__ void pair_tw_load(float2* st, const float2* __restrict__ plain) {
  if constexpr (I < L::n) {
    constexpr int N = L::N, C = L::code(I), R = stage_radix(C);
    if constexpr (N == 600 && NS == 25 && C != CUT) {
      for (int i = threadIdx.x; i < 600; i += blockDim.x) st[N + i] = plain[(i % 25) * (i / 25)];
    } else if constexpr (N == 600 && C == 3) {
      for (int i = threadIdx.x; i < 400; i += blockDim.x) st[NS + i] = plain[25 * (1 + i / 200) * (i % 200 / 25)];
    } else if constexpr (C == S8A2 || C == S8A4) {
      for (int i = threadIdx.x; i < 8 * NS; i += blockDim.x) st[N + i] = plain[(i % NS) * (i / NS) * (N / (8 * NS))];
    } else if constexpr (C != CUT && C < 10 && NS > 1) {
      for (int i = threadIdx.x; i < NS * (R - 1); i += blockDim.x)
        st[NS + i] = plain[(i % NS) * (1 + i / NS) * (N / (NS * R))];
    }
    pair_tw_load<L, I + 1, NS * R>(st, plain);
  }
}

// ---- the groups ----------------------------------------------------------------
// The stages of one group on the E elements of subset q, from code I on; NS0
// is the span before the group, NSL the span inside it.  On entry element m
// is at position q + m N/E of the line, on return at
//   (q / NS0) NS0 E + q mod NS0 + NS0 m.
// The stage's twiddle index k is q mod NS0 + NS0 (m mod NSL).
template <class L, bool INV, int I, int NS0, int NSL, int E>
__device__ __forceinline__ void pair_stages(cpair (&v)[E], const float2* tw, int q) {
  constexpr int N = L::N;
  constexpr bool DONE = I >= L::n || L::code(I < L::n ? I : 0) == CUT;
  if constexpr (!DONE) {
    constexpr int C = L::code(I);
    constexpr int R = stage_radix(C);
    constexpr int NS = NS0 * NSL;
    constexpr int MU = E / (NSL * R);
    const int k0 = NS0 == 1 ? 0 : q % NS0;
    cpair o[E];
    // S8B4, S8B2 (the first stage of their group): the output digit of the cut stage's first part
    [[maybe_unused]] int digit = 0;
    if constexpr (C == S8B4) digit = k0 / (NS0 / 2);
    if constexpr (C == S8B2) digit = k0 / (NS0 / 4);
#pragma unroll
    for (int mu = 0; mu < MU; ++mu)
#pragma unroll
      for (int ka = 0; ka < NSL; ++ka) {
        cpair u[R];
#pragma unroll
        for (int r = 0; r < R; ++r) u[r] = v[ka + NSL * (mu + r * MU)];
        if constexpr (N == 600 && NS == 25) {
          const int pos = (q / NS0) * NS0 * NSL + k0 + NS0 * ka + NSL * (N / E) * mu;
          const float2* t = tw + N + (pos / 25) * 25 + k0 + NS0 * ka;
#pragma unroll
          for (int r = 0; r < R; ++r) u[r] = pcmul(u[r], twid<INV>(t, r * NSL * (N / E) * MU));
        } else if constexpr (C == S8A2 || C == S8A4) {
          // index in the radix-8 stage: the position divided by N/8
          const int pos = (q / NS0) * NS0 * NSL + k0 + NS0 * ka + NSL * (N / E) * mu;
          const float2* t = tw + N + (pos / (N / 8)) * NS + k0 + NS0 * ka;
#pragma unroll
          for (int r = 0; r < R; ++r) u[r] = pcmul(u[r], twid<INV>(t, (8 / R) * r * NS));
        } else if constexpr (C < 10 && NS > 1) {
          const float2* t = tw + NS + k0 + NS0 * ka;
#pragma unroll
          for (int r = 1; r < R; ++r) u[r] = pcmul(u[r], twid<INV>(t, (r - 1) * NS));
        }
        if constexpr (C == 8) pdft8<INV>(u);
        if constexpr (C == 5) pdft5<INV, N == 600>(u[0], u[1], u[2], u[3], u[4]);
        if constexpr (C == 4 || C == S8A4) pdft4<INV>(u[0], u[1], u[2], u[3]);
        if constexpr (C == 3) pdft3<INV, N == 600>(u[0], u[1], u[2]);
        if constexpr (C == 2 || C == S8A2) pdft2<INV>(u[0], u[1]);
        if constexpr (C == S8B4) {
          if (digit == 0) pdft4<INV>(u[0], u[1], u[2], u[3]);
          else pdft4_odd<INV>(u[0], u[1], u[2], u[3]);
        }
        if constexpr (C == S8B2) {
          if (digit == 0) p8_last<INV, 0>(u[0], u[1]);
          else if (digit == 1) p8_last<INV, 1>(u[0], u[1]);
          else if (digit == 2) p8_last<INV, 2>(u[0], u[1]);
          else p8_last<INV, 3>(u[0], u[1]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) o[ka + r * NSL + NSL * R * mu] = u[r];
      }
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = o[m];
    pair_stages<L, INV, I + 1, NS0, NSL * R>(v, tw, q);
  }
}

__device__ __forceinline__ cpair ld_pair(const cpair* p) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  return {make_float2(t.x, t.y), make_float2(t.z, t.w)};
}
__device__ __forceinline__ void st_pair(cpair* p, const cpair& v) {
  *reinterpret_cast<float4*>(p) = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}

// Where position p of a line lies in its exchange buffer, in cpairs: as
// [p][8 columns] in a column tile (S = 8: a quarter warp's 8 lanes are the 8
// columns of one p), padded by one in eight for a row when group 1 writes
// with an even stride.
template <class L, int S>
__device__ __forceinline__ int pair_at(int p) {
  if constexpr (S == 8) return p * 8;
  else if constexpr (L::E1 % 2 == 0) return p + (p >> 3);
  else return p;
}

// One line after its elements are in v (subset q = t + i T of group 1 in
// v[i]); ex: the line's exchange buffer.  out(q, m, value) takes the line's
// element q + m QL.  sync() is a barrier over the line's threads at least; the
// caller puts one between the last use of ex and this call.  With three
// groups the middle one writes its results back to the places it read (no
// barrier between), and the last one reads them from there.
template <class L, bool INV, int S, class Sync, class Out>
__device__ __forceinline__ void pair_line(cpair (&v)[L::IT1][L::E1], cpair* ex, const float2* tw, int t, Sync sync,
                                          Out out) {
#pragma unroll
  for (int i = 0; i < L::IT1; ++i) {
    const int q = t + i * L::T;
    if (L::Q1 % L::T == 0 || q < L::Q1) {
      pair_stages<L, INV, 0, 1, 1>(v[i], tw, q);
#pragma unroll
      for (int m = 0; m < L::E1; ++m) st_pair(ex + pair_at<L, S>(q * L::E1 + m), v[i][m]);
    }
  }
  sync();
  if constexpr (L::GROUPS == 3) {
#pragma unroll
    for (int i = 0; i < L::IT2; ++i) {
      const int q = t + i * L::T;
      if (L::Q2 % L::T == 0 || q < L::Q2) {
        cpair u[L::E2];
#pragma unroll
        for (int m = 0; m < L::E2; ++m) u[m] = ld_pair(ex + pair_at<L, S>(q + m * L::Q2));
        pair_stages<L, INV, L::first(1), L::E1, 1>(u, tw, q);
#pragma unroll
        for (int m = 0; m < L::E2; ++m) st_pair(ex + pair_at<L, S>(q + m * L::Q2), u[m]);
      }
    }
    sync();
  }
#pragma unroll
  for (int i = 0; i < L::ITL; ++i) {
    const int q = t + i * L::T;
    if (L::QL % L::T == 0 || q < L::QL) {
      cpair u[L::EL];
      // two groups: position q + m QL; three: output m' = (q / E1) of the
      // middle group's subset m E1 + q mod E1
      const int from = L::GROUPS == 3 ? q % L::E1 + (q / L::E1) * L::Q2 : q;
#pragma unroll
      for (int m = 0; m < L::EL; ++m)
        u[m] = ld_pair(ex + pair_at<L, S>(from + m * (L::GROUPS == 3 ? L::E1 : L::QL)));
      pair_stages<L, INV, L::first(L::GROUPS - 1), L::QL, 1>(u, tw, q);
#pragma unroll
      for (int m = 0; m < L::EL; ++m) out(q, m, i, u[m]);
    }
  }
}

}  // namespace sf21
