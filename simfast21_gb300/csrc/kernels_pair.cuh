// Inverse transform of a batch of radii, two radii at a time: the kernels of
// one box side (instantiated by the kernels_pair_*.cu units).
//
// The work boxes of a batch are private, so a pair of radii shares a box of
// 16-byte values {rec_2p, rec_2p+1, ion_2p, ion_2p+1}, column-block major with
// blocks of 8 columns:
//     index(a, b, c) = ((c / 8) N + a) N + b) 8 + c mod 8,
// one slab of 8 N^2 values per column block: a b-axis tile (fixed a, one
// block) is one contiguous run, an a-axis tile (fixed b) reads 128-byte runs
// inside one slab.  A batch with an odd number of radii (the last one of a set)
// carries its last radius twice (the centre test of a radius is idempotent).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pair_line.cuh"
#include "sf21_kernels.h"

namespace sf21 {

__host__ __device__ constexpr int pair_min(int a, int b) { return a < b ? a : b; }
__host__ __device__ constexpr int pair_max(int a, int b) { return a > b ? a : b; }

// Column tiles: 8 columns of one line set, small boxes several tiles per CTA.
// REGS: registers per thread that the occupancy is planned for.
template <class L, int REGS>
struct PairCol {
  static constexpr int N = L::N;
  static constexpr int LT = 8 * L::T;
  static constexpr int TPC = LT >= 128 ? 1 : (N * (N / 8)) % (128 / LT) == 0 ? 128 / LT : 1;
  static constexpr int THREADS = LT * TPC;
  static constexpr int NTILES = N * (N / 8);
  static constexpr size_t SMEM = (size_t)TPC * N * 8 * sizeof(cpair) + L::TW * sizeof(float2);
  static constexpr int PER_SM = pair_max(1, pair_min(pair_min(32, 65536 / ((THREADS + 31) / 32 * 32 * REGS)),
                                                     (int)(230000 / (SMEM + 1024))));
};

// Largest side whose radii may go to several grid rows.  Larger boxes fill the
// device with one row, and the code that lets rows meet costs them registers
// (96^3: 390 -> 411 us with it in the kernels).
constexpr int PAIR_MULTI_N = 80;
// The kernels' argument: the 1 KB of RADII_MAX entries only where they are used
// (it costs a launch 2 us)
template <int N>
using PairBatch = BatchOf<N <= PAIR_MULTI_N ? RADII_MAX : KMAX>;
template <int N>
PairBatch<N> pair_batch(const Batch& bt) {
  PairBatch<N> b;
  b.K = bt.K;
  b.set = bt.set;
  b.zmul = bt.zmul;
  for (int k = 0; k < (int)(sizeof(b.r) / sizeof(b.r[0])); ++k) b.r[k] = bt.r[k];
  return b;
}

// Rows: RW rows per CTA.
template <class L, int RW_, int REGS>
struct PairRow {
  static constexpr int N = L::N;
  static constexpr int RW = RW_;
  static constexpr int THREADS = RW * L::T;
  static constexpr int NW = (N / 2 + L::T) / L::T;  // window values per thread
  static constexpr int WS = (N / 2 + 2) / 2 * 2;    // float2 of a row's windows
  static constexpr size_t SMEM =
      (size_t)RW * (L::XR * sizeof(cpair) + WS * sizeof(float2)) + L::TW * sizeof(float2);
  static constexpr int PER_SM = pair_max(1, pair_min(pair_min(32, 65536 / ((THREADS + 31) / 32 * 32 * REGS)),
                                                     (int)(230000 / (SMEM + 1024))));
  static_assert((N * N) % RW == 0, "rows per CTA");
};

// ---- c axis: the top-hat filter of the batch's radii, inverse transform -------
// (get_HIIbubbles.c:305-322.)  Persistent: a CTA takes row groups blockIdx.x,
// blockIdx.x + gridDim.x, ...; the next group's spectrum rows are asked into
// L2 while the current one is transformed.  c and N - c share |k|, so per pair
// the row's threads evaluate the N/2 + 1 distinct windows once into shared
// memory.
template <class L, int RW, int REGS>
__global__ void __launch_bounds__(PairRow<L, RW, REGS>::THREADS, PairRow<L, RW, REGS>::PER_SM)
k_pair_rows_filter(const float2* __restrict__ spec, const __grid_constant__ PairBatch<L::N> bt, int per,
                   const float2* __restrict__ plain) {
  using R = PairRow<L, RW, REGS>;
  constexpr int N = L::N;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float2* ws = reinterpret_cast<float2*>(exs + RW * L::XR);
  float2* tw = ws + RW * R::WS;
  constexpr int NG = N * N / RW;  // row groups
  const int row = threadIdx.x / L::T, t = threadIdx.x % L::T;
  cpair* ex = exs + row * L::XR;
  float2* wrow = ws + row * R::WS;
  auto sync = [] {
    if constexpr (R::THREADS <= 32) __syncwarp();
    else __syncthreads();
  };
  auto load = [&](float2 (&z)[L::IT1][L::E1], int group) {
    const float2* src = spec + ((long)group * RW + row) * N;
#pragma unroll
    for (int i = 0; i < L::IT1; ++i) {
      const int q = t + i * L::T;
      if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
        for (int m = 0; m < L::E1; ++m) z[i][m] = __ldg(src + q + m * L::Q1);
      }
    }
  };
  constexpr bool MULTI = N <= PAIR_MULTI_N;  // this grid row's radii
  const int k0 = MULTI ? blockIdx.y * per : 0, k1 = MULTI ? min(bt.K, k0 + per) : bt.K;
  pair_tw_load<L>(tw, plain);
  __syncthreads();
  for (int group = blockIdx.x; group < NG; group += gridDim.x) {
    const int rid = group * RW + row;
    float kmag[R::NW];
    {
      const int a = rid / N, b = rid % N;
      const int ka = kfreq(a, N), kb = kfreq(b, N);
      const int kab = ka * ka + kb * kb;
#pragma unroll
      for (int i = 0; i < R::NW; ++i) {
        const int kc = t + i * L::T;
        kmag[i] = sqrtf((float)(kab + kc * kc));
      }
    }
    float2 z[L::IT1][L::E1];
    load(z, group);
    if (group + gridDim.x < NG)  // the next group's rows on their way into L2
      for (int i = threadIdx.x; i < RW * N / 16; i += R::THREADS)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(spec + (long)(group + gridDim.x) * RW * N + 16 * i));
    for (int k = k0; k < k1; k += 2) {
      const float d0 = bt.r[k].dkR, d1 = bt.r[k + 1].dkR;
#pragma unroll
      for (int i = 0; i < R::NW; ++i) {
        const int kc = t + i * L::T;
        if (kc <= N / 2) wrow[kc] = make_float2(w_tophat(d0 * kmag[i]), w_tophat(d1 * kmag[i]));
      }
      sync();  // the windows are in; the previous pair's exchange has been read
      cpair v[L::IT1][L::E1];
#pragma unroll
      for (int i = 0; i < L::IT1; ++i) {
        const int q = t + i * L::T;
        if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
          for (int m = 0; m < L::E1; ++m) {
            const int c = q + m * L::Q1;
            const float2 x = z[i][m], w = wrow[c <= N / 2 ? c : N - c];
            // scalar products: a packed product that feeds a packed addition
            // was seen to be fused with it, which loses the scalar bits
            v[i][m].re = make_float2(__fmul_rn(x.x, w.x), __fmul_rn(x.x, w.y));
            v[i][m].im = make_float2(__fmul_rn(x.y, w.x), __fmul_rn(x.y, w.y));
          }
        }
      }
      cpair* box = reinterpret_cast<cpair*>(bt.r[k].work) + (long)rid * 8;
      pair_line<L, true, 1>(v, ex, tw, t, sync, [&](int q, int m, int, const cpair& u) {
        if constexpr (L::QL % 8 == 0) {
          st_pair(box + (long)(q / 8) * N * N * 8 + q % 8 + (long)m * (L::QL / 8) * N * N * 8, u);
        } else {
          const int c = q + m * L::QL;
          st_pair(box + (long)(c / 8) * N * N * 8 + c % 8, u);
        }
      });
    }
  }
}

// ---- strided axes ---------------------------------------------------------------
// EPI 0: b axis, in place.  EPI 1: a axis, then the centre test and the
// first-hit update (get_HIIbubbles.c:335-352; is_centre on both lanes).
// EPI 2: a axis, then the running maximum of ion_R / rec_R and its radius (the
// rule of k_cols_a_crit, in the order of the radii).
// One CTA per tile (group); no prefetch into registers: several CTAs per SM
// overlap one tile's loads with another's transform, and the next pair's
// lines are asked into L2 a pair ahead.
template <class L, bool INV, int EPI, int REGS>
__global__ void __launch_bounds__(PairCol<L, REGS>::THREADS, PairCol<L, REGS>::PER_SM)
k_pair_cols(const __grid_constant__ PairBatch<L::N> bt, int per, uint8_t* __restrict__ rc, float* __restrict__ Cbuf, const float* __restrict__ alpha_ptr,
            const float2* __restrict__ plain, int ahead) {
  using C = PairCol<L, REGS>;
  constexpr int N = L::N;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float2* tw = reinterpret_cast<float2*>(exs + C::TPC * N * 8);
  pair_tw_load<L>(tw, plain);
  const int sub = threadIdx.x / C::LT;
  const int col = threadIdx.x % 8;
  const int t = (threadIdx.x % C::LT) / 8;
  const int tile = blockIdx.x * C::TPC + sub;
  cpair* ex = exs + sub * N * 8 + col;
  constexpr long RS = EPI >= 1 ? (long)N * 8 : 8;  // from one element of a line to the next
  const long base = (EPI >= 1 ? ((long)(tile / N) * N * N + tile % N) * 8 : (long)tile * N * 8) + col;
  float alpha = 0.0f;
  if (EPI >= 1) alpha = *alpha_ptr;
  auto sync = [] { __syncthreads(); };
  // EPI 1: bit 8 (m & 3) + k - k0 of hit[m / 4]: output m is a centre at radius k of
  // the batch (radius indices increase with k: the lowest bit is the first hit)
  constexpr int HW = (L::EL + 3) / 4;
  uint32_t hit[EPI >= 1 ? L::ITL : 1][HW];
#pragma unroll
  for (int i = 0; i < (EPI >= 1 ? L::ITL : 1); ++i)
#pragma unroll
    for (int h = 0; h < HW; ++h) hit[i][h] = EPI == 2 ? 0xFFFFFFFFu : 0u;
  // EPI 2: the batch's best ratio of each output; byte m & 3 of hit[m / 4] is its radius index
  float best[EPI == 2 ? L::ITL : 1][L::EL];
#pragma unroll
  for (int i = 0; i < (EPI == 2 ? L::ITL : 1); ++i)
#pragma unroll
    for (int m = 0; m < L::EL; ++m) best[i][m] = -INFINITY;
  // no source anywhere (alpha < 0): ion_R is exactly zero
  const float crit_zeta = alpha > 0.0f ? bt.zmul : 0.0f, crit_alpha = fabsf(alpha);
  constexpr bool MULTI = N <= PAIR_MULTI_N;  // this grid row's radii
  const int k0 = MULTI ? blockIdx.y * per : 0, k1 = MULTI ? min(bt.K, k0 + per) : bt.K;
  for (int k = k0; k < k1; k += 2) {
    cpair* box = reinterpret_cast<cpair*>(bt.r[k].work) + base;
    cpair v[L::IT1][L::E1];
#pragma unroll
    for (int i = 0; i < L::IT1; ++i) {
      const int q = t + i * L::T;
      if (L::Q1 % L::T == 0 || q < L::Q1) {
        const cpair* src = box + q * RS;
#pragma unroll
        for (int m = 0; m < L::E1; ++m) v[i][m] = ld_pair(src + m * L::Q1 * RS);
      }
    }
    if (ahead > 0) {  // the next pair's lines on their way into L2 (the last pair: those of a tile that comes later)
      const bool more = k + 2 < k1;
      const int ntile = tile + (more ? 0 : ahead * C::TPC);
      if (ntile < C::NTILES) {
        const cpair* nx = reinterpret_cast<const cpair*>(bt.r[more ? k + 2 : k0].work) +
                          (EPI >= 1 ? ((long)(ntile / N) * N * N + ntile % N) * 8 : (long)ntile * N * 8);
        for (int r = threadIdx.x % C::LT; r < N; r += C::LT)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + r * RS));
      }
    }
    __syncthreads();  // the previous pair's exchange has been read (k = 0: twiddles)
    const float2 al2 = dup2(alpha), zm2 = dup2(bt.zmul);
    const uint32_t bit = 1u << (k - k0);
    pair_line<L, INV, 8>(v, ex, tw, t, sync, [&](int q, int m, int i, const cpair& u) {
      if constexpr (EPI == 0) {
        st_pair(box + (q + m * L::QL) * RS, u);
      } else if constexpr (EPI == 2) {
#pragma unroll
        for (int lane = 0; lane < 2; ++lane) {
          const float den = (lane ? u.re.y : u.re.x) * crit_alpha;  // alpha * rec_R
          if (den > 0.0f) {
            const float ratio = __fdiv_rn((lane ? u.im.y : u.im.x) * crit_zeta, den);
            if (ratio > best[i][m]) {
              best[i][m] = ratio;
              hit[i][m >> 2] = __byte_perm(hit[i][m >> 2], (uint32_t)bt.r[k + lane].ridx,
                                           (0x3210u & ~(0xFu << (4 * (m & 3)))) | (4u << (4 * (m & 3))));
            }
          }
        }
      } else {
        const float2 y = mul2(u.im, zm2), x = mul2(u.re, al2);
        if (u.im.x > 0.0f && y.x >= x.x) hit[i][m >> 2] |= bit << (8 * (m & 3));
        if (u.im.y > 0.0f && y.y >= x.y) hit[i][m >> 2] |= bit << (8 * (m & 3) + 1);
      }
    });
  }
  if constexpr (EPI == 2) {
    const int b = tile % N;
    const int c = (tile / N) * 8 + col;
#pragma unroll
    for (int i = 0; i < L::ITL; ++i) {
      const int q = t + i * L::T;
      if (L::QL % L::T == 0 || q < L::QL) {
        float old[L::EL];
#pragma unroll
        for (int m = 0; m < L::EL; ++m) old[m] = Cbuf[((long)(q + m * L::QL) * N + b) * N + c];
#pragma unroll
        for (int m = 0; m < L::EL; ++m) {
          if (best[i][m] > old[m]) {
            const long idx = ((long)(q + m * L::QL) * N + b) * N + c;
            Cbuf[idx] = best[i][m];
            rc[idx] = (uint8_t)(hit[i][m >> 2] >> (8 * (m & 3)));
          }
        }
      }
    }
  }
  if (EPI == 1 && alpha > 0.0f) {  // alpha <= 0: no source anywhere, no centre
    const int b = tile % N;
    const int c = (tile / N) * 8 + col;
#pragma unroll
    for (int i = 0; i < L::ITL; ++i) {
      const int q = t + i * L::T;
      if (L::QL % L::T == 0 || q < L::QL) {
        if constexpr (N <= PAIR_MULTI_N) {
          if (gridDim.y > 1) {
            // several grid rows meet in a cell: four lanes' bytes to a word, the
            // smaller of each by compare-and-swap, all words' first tries (no
            // hit yet) in flight together
            const unsigned lanes = 0xFFu << (threadIdx.x & 24);
            uint32_t w[L::EL], seen[L::EL];
            uint32_t* dst = reinterpret_cast<uint32_t*>(rc + ((long)q * N + b) * N + (c & ~3));
            constexpr long MS = (long)L::QL * N * N / 4;
#pragma unroll
            for (int m = 0; m < L::EL; ++m) {
              const uint32_t byte = (hit[i][m >> 2] >> (8 * (m & 3))) & 0xFFu;
              const uint32_t none = ~(0xFFu << (8 * (col & 3)));
              w[m] = byte ? none | (uint32_t)(bt.r[k0].ridx + __ffs(byte) - 1) << (8 * (col & 3)) : 0xFFFFFFFFu;
              w[m] &= __shfl_xor_sync(lanes, w[m], 1);
              w[m] &= __shfl_xor_sync(lanes, w[m], 2);
              if (col & 3) w[m] = 0xFFFFFFFFu;
            }
#pragma unroll
            for (int m = 0; m < L::EL; ++m)
              seen[m] = w[m] != 0xFFFFFFFFu ? atomicCAS(dst + m * MS, 0xFFFFFFFFu, w[m]) : 0xFFFFFFFFu;
#pragma unroll
            for (int m = 0; m < L::EL; ++m) {
              uint32_t old = seen[m];
              if (old == 0xFFFFFFFFu) continue;  // nothing to write, or written
              for (uint32_t now = __vminu4(old, w[m]); now != old; now = __vminu4(old, w[m])) {
                const uint32_t s = atomicCAS(dst + m * MS, old, now);
                if (s == old) break;
                old = s;
              }
            }
            continue;
          }
        }
        // all the reads first (independent), then the updates; the radius
        // indices of a batch are consecutive
        uint32_t old[L::EL];
#pragma unroll
        for (int m = 0; m < L::EL; ++m) {
          const uint32_t byte = (hit[i][m >> 2] >> (8 * (m & 3))) & 0xFFu;
          old[m] = byte ? rc[((long)(q + m * L::QL) * N + b) * N + c] : 0u;
        }
#pragma unroll
        for (int m = 0; m < L::EL; ++m) {
          const uint32_t byte = (hit[i][m >> 2] >> (8 * (m & 3))) & 0xFFu;
          const uint32_t h = (uint32_t)(bt.r[k0].ridx + __ffs(byte) - 1);
          if (byte && h < old[m]) rc[((long)(q + m * L::QL) * N + b) * N + c] = (uint8_t)h;
        }
      }
    }
  }
}

// ---- adjoint of the criterion -----------------------------------------------------
// a axis: fields -> masked cotangents (the rule of k_cols_a_adj) -> forward a
// axis, in place in the pair boxes; per-CTA partial sums of g C / zeta.  The
// argmax bytes of the tile are read once; a slot with ridx < 0 (the one that
// fills an odd batch) takes no voxel.
template <class L, int REGS>
__global__ void __launch_bounds__(PairCol<L, REGS>::THREADS, PairCol<L, REGS>::PER_SM)
k_pair_cols_a_adj(const __grid_constant__ PairBatch<L::N> bt, const float* __restrict__ g, const uint8_t* __restrict__ Abuf,
                  const float* __restrict__ alpha_ptr, float* __restrict__ zpart, const float2* __restrict__ plain) {
  using C = PairCol<L, REGS>;
  constexpr int N = L::N;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float2* tw = reinterpret_cast<float2*>(exs + C::TPC * N * 8);
  __shared__ float red[32];
  pair_tw_load<L>(tw, plain);
  const int sub = threadIdx.x / C::LT;
  const int col = threadIdx.x % 8;
  const int t = (threadIdx.x % C::LT) / 8;
  const int tile = blockIdx.x * C::TPC + sub;
  cpair* ex = exs + sub * N * 8 + col;
  constexpr long RS = (long)N * 8;
  const long base = ((long)(tile / N) * N * N + tile % N) * 8 + col;
  const long vox = (long)(tile % N) * N + (tile / N) * 8 + col;  // natural index of (a = 0, b, c)
  const float alpha = fabsf(*alpha_ptr);  // sign: the no-source mark
  const float inv_alpha = 1.0f / alpha;   // exact: alpha is a power of two
  auto sync = [] { __syncthreads(); };
  uint32_t arg[L::ITL][(L::EL + 3) / 4];
#pragma unroll
  for (int i = 0; i < L::ITL; ++i) {
    const int q = t + i * L::T;
#pragma unroll
    for (int m = 0; m < L::EL; ++m) {
      uint32_t a = RC_NONE;
      if (L::QL % L::T == 0 || q < L::QL) a = Abuf[vox + (long)(q + m * L::QL) * N * N];
      arg[i][m >> 2] = (m & 3) ? arg[i][m >> 2] | a << (8 * (m & 3)) : a;
    }
  }
  float zacc = 0.0f;
  for (int k = 0; k < bt.K; k += 2) {
    cpair* box = reinterpret_cast<cpair*>(bt.r[k].work) + base;
    const int r0 = bt.r[k].ridx, r1 = bt.r[k + 1].ridx;
    cpair v[L::IT1][L::E1], o[L::ITL][L::EL];
#pragma unroll
    for (int i = 0; i < L::IT1; ++i) {
      const int q = t + i * L::T;
      if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
        for (int m = 0; m < L::E1; ++m) v[i][m] = ld_pair(box + (q + m * L::Q1) * RS);
      }
    }
    __syncthreads();  // the previous pair's exchange has been read (k = 0: twiddles)
    pair_line<L, true, 8>(v, ex, tw, t, sync, [&](int q, int m, int i, const cpair& u) {
      const int a = (arg[i][m >> 2] >> (8 * (m & 3))) & 0xFF;
      cpair c = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
      if (a == r0 || a == r1) {
        const float rec = a == r0 ? u.re.x : u.re.y;  // rec_R (> 0 where A = R)
        const float h = (a == r0 ? u.im.x : u.im.y) * inv_alpha;
        const float Cr = __fdiv_rn(bt.zmul * h, rec);
        const float gg = g[vox + (long)(q + m * L::QL) * N * N];
        const float ginv = __fdiv_rn(gg, rec);
        const float2 w = make_float2(-ginv * Cr, ginv * bt.zmul * inv_alpha);
        if (a == r0) {
          c.re.x = w.x;
          c.im.x = w.y;
        } else {
          c.re.y = w.x;
          c.im.y = w.y;
        }
        zacc += gg * __fdiv_rn(Cr, bt.zmul);
      }
      o[i][m] = c;
    });
    __syncthreads();  // the inverse line's exchange has been read
#pragma unroll
    for (int i = 0; i < L::ITL; ++i) {
      const int q = t + i * L::T;
      if (L::QL % L::T == 0 || q < L::QL) {
#pragma unroll
        for (int m = 0; m < L::EL; ++m) st_pair(ex + (q + m * L::QL) * 8, o[i][m]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < L::IT1; ++i) {
      const int q = t + i * L::T;
      if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
        for (int m = 0; m < L::E1; ++m) v[i][m] = ld_pair(ex + (q + m * L::Q1) * 8);
      }
    }
    __syncthreads();
    pair_line<L, false, 8>(v, ex, tw, t, sync,
                           [&](int q, int m, int, const cpair& u) { st_pair(box + (q + m * L::QL) * RS, u); });
  }
  // deterministic partial of the CTA (accumulated over the batches in stream order)
  for (int s = 16; s > 0; s >>= 1) zacc += __shfl_xor_sync(0xffffffffu, zacc, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = zacc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.0f;
    for (int w = 0; w < (C::THREADS + 31) / 32; ++w) s += red[w];
    zpart[blockIdx.x] += s;
  }
}

// c axis, forward, of the batch's cotangent pairs, times W_R, summed over the
// batch in the order of its radii and added to the k-space accumulator
// (k_rows_adj_acc).  The windows of a row lie in two buffers used in turn.
template <class L, int RW, int REGS>
__global__ void __launch_bounds__(PairRow<L, RW, REGS>::THREADS, PairRow<L, RW, REGS>::PER_SM)
k_pair_rows_adj(const __grid_constant__ PairBatch<L::N> bt, float2* __restrict__ acc, const float2* __restrict__ plain) {
  using R = PairRow<L, RW, REGS>;
  constexpr int N = L::N;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float2* ws = reinterpret_cast<float2*>(exs + RW * L::XR);
  float2* tw = ws + 2 * RW * R::WS;
  constexpr int NG = N * N / RW;  // row groups
  const int row = threadIdx.x / L::T, t = threadIdx.x % L::T;
  cpair* ex = exs + row * L::XR;
  auto sync = [] {
    if constexpr (R::THREADS <= 32) __syncwarp();
    else __syncthreads();
  };
  pair_tw_load<L>(tw, plain);
  __syncthreads();
  int buf = 0;
  for (int group = blockIdx.x; group < NG; group += gridDim.x) {
    const int rid = group * RW + row;
    float kmag[R::NW];
    {
      const int a = rid / N, b = rid % N;
      const int ka = kfreq(a, N), kb = kfreq(b, N);
      const int kab = ka * ka + kb * kb;
#pragma unroll
      for (int i = 0; i < R::NW; ++i) {
        const int kc = t + i * L::T;
        kmag[i] = sqrtf((float)(kab + kc * kc));
      }
    }
    float2 sum[L::ITL][L::EL];
#pragma unroll
    for (int i = 0; i < L::ITL; ++i)
#pragma unroll
      for (int m = 0; m < L::EL; ++m) sum[i][m] = make_float2(0.0f, 0.0f);
    for (int k = 0; k < bt.K; k += 2, buf ^= 1) {
      const cpair* box = reinterpret_cast<const cpair*>(bt.r[k].work) + (long)rid * 8;
      cpair v[L::IT1][L::E1];
#pragma unroll
      for (int i = 0; i < L::IT1; ++i) {
        const int q = t + i * L::T;
        if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
          for (int m = 0; m < L::E1; ++m) {
            const int c = q + m * L::Q1;
            v[i][m] = ld_pair(box + (long)(c / 8) * N * N * 8 + c % 8);
          }
        }
      }
      float2* wrow = ws + (buf * RW + row) * R::WS;
      const float d0 = bt.r[k].dkR, d1 = bt.r[k + 1].dkR;
#pragma unroll
      for (int i = 0; i < R::NW; ++i) {
        const int kc = t + i * L::T;
        if (kc <= N / 2) wrow[kc] = make_float2(w_tophat(d0 * kmag[i]), w_tophat(d1 * kmag[i]));
      }
      sync();  // the windows are in; the previous pair's exchange has been read
      const bool both = k + 1 < bt.K;
      pair_line<L, false, 1>(v, ex, tw, t, sync, [&](int q, int m, int i, const cpair& u) {
        const int c = q + m * L::QL;
        const float2 w = wrow[c <= N / 2 ? c : N - c];
        float2 s = sum[i][m];
        s.x = fmaf(w.x, u.re.x, s.x);
        s.y = fmaf(w.x, u.im.x, s.y);
        if (both) {
          s.x = fmaf(w.y, u.re.y, s.x);
          s.y = fmaf(w.y, u.im.y, s.y);
        }
        sum[i][m] = s;
      });
    }
    float2* dst = acc + (long)rid * N;
#pragma unroll
    for (int i = 0; i < L::ITL; ++i) {
      const int q = t + i * L::T;
      if (L::QL % L::T == 0 || q < L::QL) {
#pragma unroll
        for (int m = 0; m < L::EL; ++m) {
          const int c = q + m * L::QL;
          const float2 old = dst[c];
          dst[c] = make_float2(old.x + sum[i][m].x, old.y + sum[i][m].y);
        }
      }
    }
  }
}

// ---- the halo finder's filter bank ---------------------------------------------------
// Two complex transforms (of two masses each: F (s W_a + i s W_b), kernels_hf.cu)
// as the lanes of a pair.  Slot K of a batch with an odd number of transforms
// repeats the last one.
// The product is written with the fused multiply-adds that the compiler forms
// for z.x wa - z.y wb and z.x wb + z.y wa in the one-transform kernels
// (kernels_hf.cu at the powers of two, kernels_gen.cu at the other sides; the
// other three forms differ from them in more than half of the values).
template <bool POW2>
__device__ __forceinline__ float2 hf_mul(float2 z, float wa, float wb) {
  return make_float2(fmaf(z.x, wa, -__fmul_rn(z.y, wb)),
                     POW2 ? fmaf(z.x, wb, __fmul_rn(z.y, wa)) : fmaf(z.y, wa, __fmul_rn(z.x, wb)));
}

template <class L, int RW, int REGS>
__global__ void __launch_bounds__(PairRow<L, RW, REGS>::THREADS, PairRow<L, RW, REGS>::PER_SM)
k_pair_hf_rows(const float2* __restrict__ spec, HfBatch hb, const float2* __restrict__ plain) {
  using R = PairRow<L, RW, REGS>;
  constexpr int N = L::N;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float4* ws = reinterpret_cast<float4*>(exs + RW * L::XR);  // the four masses' windows of a row
  float2* tw = reinterpret_cast<float2*>(ws + RW * R::WS);
  constexpr int NG = N * N / RW;  // row groups
  const int row = threadIdx.x / L::T, t = threadIdx.x % L::T;
  cpair* ex = exs + row * L::XR;
  float4* wrow = ws + row * R::WS;
  auto sync = [] {
    if constexpr (R::THREADS <= 32) __syncwarp();
    else __syncthreads();
  };
  pair_tw_load<L>(tw, plain);
  __syncthreads();
  for (int group = blockIdx.x; group < NG; group += gridDim.x) {
    const int rid = group * RW + row;
    const int a = rid / N, b = rid % N;
    const int ka = kfreq(a, N), kb = kfreq(b, N);
    const int kab = ka * ka + kb * kb;
    float2 z[L::IT1][L::E1];
    const float2* src = spec + (long)rid * N;
#pragma unroll
    for (int i = 0; i < L::IT1; ++i) {
      const int q = t + i * L::T;
      if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
        for (int m = 0; m < L::E1; ++m) z[i][m] = __ldg(src + q + m * L::Q1);
      }
    }
    if (group + gridDim.x < NG)  // the next group's rows on their way into L2
      for (int i = threadIdx.x; i < RW * N / 16; i += R::THREADS)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(spec + (long)(group + gridDim.x) * RW * N + 16 * i));
    for (int k = 0; k < hb.K; k += 2) {
      const HfPair &p0 = hb.p[k], &p1 = hb.p[k + 1];
      sync();  // the previous windows and exchange have been read
      for (int kc = t; kc <= N / 2; kc += L::T) {
        const float kmag = sqrtf((float)(kab + kc * kc));
        float4 w;
        w.x = __fmul_rn(hb.scale, w_tophat(p0.dkRa * kmag));
        w.y = p0.bits_b ? __fmul_rn(hb.scale, w_tophat(p0.dkRb * kmag)) : 0.0f;
        w.z = __fmul_rn(hb.scale, w_tophat(p1.dkRa * kmag));
        w.w = p1.bits_b ? __fmul_rn(hb.scale, w_tophat(p1.dkRb * kmag)) : 0.0f;
        wrow[kc] = w;
      }
      sync();
      cpair v[L::IT1][L::E1];
#pragma unroll
      for (int i = 0; i < L::IT1; ++i) {
        const int q = t + i * L::T;
        if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
          for (int m = 0; m < L::E1; ++m) {
            const int c = q + m * L::Q1;
            const float4 w = wrow[c <= N / 2 ? c : N - c];
            constexpr bool POW2 = (N & (N - 1)) == 0;
            const float2 x = hf_mul<POW2>(z[i][m], w.x, w.y), y = hf_mul<POW2>(z[i][m], w.z, w.w);
            v[i][m].re = make_float2(x.x, y.x);
            v[i][m].im = make_float2(x.y, y.y);
          }
        }
      }
      cpair* box = reinterpret_cast<cpair*>(p0.work) + (long)rid * 8;
      pair_line<L, true, 1>(v, ex, tw, t, sync, [&](int q, int m, int, const cpair& u) {
        const int c = q + m * L::QL;
        st_pair(box + (long)(c / 8) * N * N * 8 + c % 8, u);
      });
    }
  }
}

// a axis + the four thresholds: one bit per cell and mass.  A CTA takes up to
// four tiles in a row of cells, one after the other, and stores their bytes as
// one word: with a byte per tile row the stores' sectors took as long as the
// transform's exchanges (512^3, two transforms: 880 us; 550 us with words, the
// radius passes' a axis with its test 520 us).  The bits of eight outputs and
// four masses are gathered by one 8 x 8 transposition among the columns' lanes.

// Tiles of eight columns that a CTA takes one after the other along a row of
// the bit sets, to store their bytes as one word (whole words in every row)
template <class C>
__host__ __device__ constexpr int pair_hf_run() {
  for (int j = 4; j > 1; j /= 2)
    if (C::N / 8 % j == 0 && C::NTILES / j % C::TPC == 0) return j;
  return 1;
}
template <class L, int REGS>
__global__ void __launch_bounds__(PairCol<L, REGS>::THREADS, PairCol<L, REGS>::PER_SM)
k_pair_hf_cols_a(HfBatch hb, const float2* __restrict__ plain, int ahead) {
  using C = PairCol<L, REGS>;
  constexpr int N = L::N;
  constexpr int J = pair_hf_run<C>();
  constexpr int NB = N / 8 / J;  // runs per row of the bit sets
  constexpr int H = (L::EL + 7) / 8;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float2* tw = reinterpret_cast<float2*>(exs + C::TPC * N * 8);
  pair_tw_load<L>(tw, plain);
  const int sub = threadIdx.x / C::LT;
  const int col = threadIdx.x % 8;
  const int t = (threadIdx.x % C::LT) / 8;
  const int run = blockIdx.x * C::TPC + sub;
  const int cb0 = run % NB * J, b = run / NB;
  cpair* ex = exs + sub * N * 8 + col;
  constexpr long RS = (long)N * 8, CBS = (long)N * N * 8;
  const long base = (long)cb0 * CBS + (long)b * 8;
  const unsigned wmask =
      C::THREADS % 32 && threadIdx.x / 32 == C::THREADS / 32 ? (1u << (C::THREADS % 32)) - 1u : 0xffffffffu;
  auto sync = [] { __syncthreads(); };
  for (int k = 0; k < hb.K; k += 2) {
    const HfPair &p0 = hb.p[k], &p1 = hb.p[k + 1];
    uint32_t run_bits[4][L::ITL][H];  // mass, then the lane's output: its run's bytes, tile j in byte j
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int i = 0; i < L::ITL; ++i)
#pragma unroll
        for (int h = 0; h < H; ++h) run_bits[s][i][h] = 0u;
    for (int j = 0; j < J; ++j) {
      const cpair* box = reinterpret_cast<const cpair*>(p0.work) + base + j * CBS + col;
      cpair v[L::IT1][L::E1];
#pragma unroll
      for (int i = 0; i < L::IT1; ++i) {
        const int q = t + i * L::T;
        if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
          for (int m = 0; m < L::E1; ++m) v[i][m] = ld_pair(box + (q + m * L::Q1) * RS);
        }
      }
      const int nrun = run + ahead * C::TPC;
      if (j + 1 < J || nrun < N * NB) {  // a later tile's lines on their way into L2
        const cpair* nx = reinterpret_cast<const cpair*>(p0.work) +
                          (j + 1 < J ? base + (j + 1) * CBS : (long)(nrun % NB * J) * CBS + (long)(nrun / NB) * 8);
        for (int r = threadIdx.x % C::LT; r < N; r += C::LT)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + r * RS));
      }
      __syncthreads();  // the previous tile's exchange has been read (the first: twiddles)
      uint32_t over[L::ITL][H];  // bit 8 s + (m & 7) of word m / 8: output m of mass s above its threshold
#pragma unroll
      for (int i = 0; i < L::ITL; ++i)
#pragma unroll
        for (int h = 0; h < H; ++h) over[i][h] = 0u;
      pair_line<L, true, 8>(v, ex, tw, t, sync, [&](int q, int m, int i, const cpair& u) {
        const uint32_t o = (u.re.x > p0.thr_a ? 1u : 0u) | (u.im.x > p0.thr_b ? 1u << 8 : 0u) |
                           (u.re.y > p1.thr_a ? 1u << 16 : 0u) | (u.im.y > p1.thr_b ? 1u << 24 : 0u);
        over[i][m >> 3] |= o << (m & 7);
      });
#pragma unroll
      for (int i = 0; i < L::ITL; ++i)
#pragma unroll
        for (int h = 0; h < H; ++h) {
          // the eight columns' lanes transpose the bits of eight outputs, all
          // masses at once: then lane m has output 8 h + m, bit c is column c
          uint32_t w = over[i][h];
#pragma unroll
          for (int s = 4; s > 0; s >>= 1) {
            const uint32_t keep = s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u : 0x55555555u;
            const uint32_t x = __shfl_xor_sync(wmask, w, s);
            w = col & s ? (w & ~keep) | ((x & ~keep) >> s) : (w & keep) | ((x & keep) << s);
          }
#pragma unroll
          for (int s = 0; s < 4; ++s) run_bits[s][i][h] |= (w >> (8 * s) & 0xffu) << (8 * j);
        }
    }
#pragma unroll
    for (int i = 0; i < L::ITL; ++i) {
      const int q = t + i * L::T;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int m = 8 * h + col;
        if ((L::QL % L::T == 0 || q < L::QL) && (L::EL % 8 == 0 || m < L::EL)) {
          const long byte = (((long)(q + m * L::QL) * N + b) * N >> 3) + cb0;  // 8 cells per byte
          auto put = [&](uint32_t* bits, uint32_t w) {
            unsigned char* dst = reinterpret_cast<unsigned char*>(bits) + byte;
            if constexpr (J == 4) *reinterpret_cast<uint32_t*>(dst) = w;
            else if constexpr (J == 2) *reinterpret_cast<uint16_t*>(dst) = (uint16_t)w;
            else *dst = (unsigned char)w;
          };
          put(p0.bits_a, run_bits[0][i][h]);
          if (p0.bits_b) put(p0.bits_b, run_bits[1][i][h]);
          if (k + 1 < hb.K) {
            put(p1.bits_a, run_bits[2][i][h]);
            if (p1.bits_b) put(p1.bits_b, run_bits[3][i][h]);
          }
        }
      }
    }
  }
}

// ---- one natural-layout box: pairs of rows, pairs of columns ------------------------
// The same lines on one complex box a N^2 + b N + c, the lanes being two rows
// (2r, 2r + 1) or two adjacent columns.
//
// c axis, forward or inverse.  in: complex rows (the imaginary part times
// |*alpha|), or real rows times the axis windows (real: wax of N values, or null).
// Only the columns c < ncol of the result are stored.
template <class L, int RW, int REGS, bool INV>
__global__ void __launch_bounds__(PairRow<L, RW, REGS>::THREADS, PairRow<L, RW, REGS>::PER_SM)
k_pair_nat_rows(const float2* in, const float* __restrict__ real, const float* __restrict__ wax, float2* out, int ncol,
                const float* __restrict__ alpha_ptr, const float2* __restrict__ plain) {
  using R = PairRow<L, RW, REGS>;
  constexpr int N = L::N;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float2* tw = reinterpret_cast<float2*>(exs + RW * L::XR);
  constexpr int NG = N * N / 2 / RW;  // groups of row pairs
  const int row = threadIdx.x / L::T, t = threadIdx.x % L::T;
  cpair* ex = exs + row * L::XR;
  auto sync = [] {
    if constexpr (R::THREADS <= 32) __syncwarp();
    else __syncthreads();
  };
  pair_tw_load<L>(tw, plain);
  const float alpha = alpha_ptr ? fabsf(*alpha_ptr) : 1.0f;
  for (int group = blockIdx.x; group < NG; group += gridDim.x) {
    const long r0 = 2 * ((long)group * RW + row);
    cpair v[L::IT1][L::E1];
    float w0 = 1.0f, w1 = 1.0f;  // the windows of the a and b axes
    if (real && wax) {
      const float wa = wax[r0 / N];  // N is even: both rows have the same a
      w0 = __fmul_rn(wa, wax[r0 % N]);
      w1 = __fmul_rn(wa, wax[r0 % N + 1]);
    }
#pragma unroll
    for (int i = 0; i < L::IT1; ++i) {
      const int q = t + i * L::T;
      if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
        for (int m = 0; m < L::E1; ++m) {
          const int c = q + m * L::Q1;
          if (real) {
            float x0 = real[r0 * N + c], x1 = real[(r0 + 1) * N + c];
            if (wax) {
              x0 = __fmul_rn(x0, __fmul_rn(w0, wax[c]));
              x1 = __fmul_rn(x1, __fmul_rn(w1, wax[c]));
            }
            v[i][m] = {make_float2(x0, x1), make_float2(0.0f, 0.0f)};
          } else {
            const float2 x0 = in[r0 * N + c], x1 = in[(r0 + 1) * N + c];
            v[i][m] = {make_float2(x0.x, x1.x), make_float2(x0.y * alpha, x1.y * alpha)};
          }
        }
      }
    }
    sync();  // twiddles; the previous group's exchange has been read
    pair_line<L, INV, 1>(v, ex, tw, t, sync, [&](int q, int m, int, const cpair& u) {
      const int c = q + m * L::QL;
      if (c < ncol) {
        out[r0 * N + c] = make_float2(u.re.x, u.im.x);
        out[(r0 + 1) * N + c] = make_float2(u.re.y, u.im.y);
      }
    });
  }
}

// b (AXIS 1) or a (AXIS 0) axis in place: tiles of 16 columns, as 8 pairs.
// blockIdx.x = column block + nblk outer index (nblk blocks cover the columns
// that are wanted; a block past the side is cut).
template <class L, bool INV, int AXIS, int REGS>
__global__ void __launch_bounds__(PairCol<L, REGS>::LT, PairCol<L, REGS>::PER_SM)
k_pair_nat_cols(float2* box, int nblk, const float2* __restrict__ plain) {
  constexpr int N = L::N;
  extern __shared__ __align__(16) unsigned char psm[];
  cpair* exs = reinterpret_cast<cpair*>(psm);
  float2* tw = reinterpret_cast<float2*>(exs + N * 8);
  pair_tw_load<L>(tw, plain);
  const int col = threadIdx.x % 8, t = threadIdx.x / 8;
  const int outer = blockIdx.x / nblk, c = (blockIdx.x % nblk) * 16 + 2 * col;
  constexpr long RS = AXIS == 1 ? N : (long)N * N;
  const bool on = N % 16 == 0 || c < N;
  float4* line = reinterpret_cast<float4*>(box + (AXIS == 1 ? (long)outer * N * N : (long)outer * N) + (on ? c : 0));
  constexpr long RS2 = RS / 2;  // float4 from one element of a line to the next
  cpair v[L::IT1][L::E1];
#pragma unroll
  for (int i = 0; i < L::IT1; ++i) {
    const int q = t + i * L::T;
    if (L::Q1 % L::T == 0 || q < L::Q1) {
#pragma unroll
      for (int m = 0; m < L::E1; ++m) {
        const float4 x = line[(q + m * L::Q1) * RS2];
        v[i][m] = {make_float2(x.x, x.z), make_float2(x.y, x.w)};
      }
    }
  }
  __syncthreads();
  auto sync = [] { __syncthreads(); };
  pair_line<L, INV, 8>(v, exs + col, tw, t, sync, [&](int q, int m, int, const cpair& u) {
    if (on) line[(q + m * L::QL) * RS2] = make_float4(u.re.x, u.im.x, u.re.y, u.im.y);
  });
}

// ---- the lines of each side ----------------------------------------------------------
// Column tiles: threads per line, codes, planned registers.  Rows: threads per
// line, rows per CTA, planned registers, codes.  Chosen by timing candidates
// of each kind on the GPU (8 radii; SM clocks per voxel and radius, where
// DRAM's copy rate allows 0.42 / 0.74 / 0.37 for the filter / ky / kx pass):
// tiles want few exchanges as long as two or more CTAs fit an SM (two groups at
// 256: kx 0.40, three 0.47; at 512 0.53 and 0.53, but ky 0.86 and 0.74), rows
// want many threads (512: three groups 0.56, two 0.80), and threads per line
// that fill whole warps (400: 40 threads 0.58, 50 threads 0.76).  600 follows
// kernels_gen600.cu.  720, 1000, 1080, 1152, 1200 and 1280 have no line here yet,
// though their radices have such cuts (1200 = 25 x 6 x 8): they stay with the
// shared-memory lines of kernels_gen.cu.
template <int N> struct PairSide;
#define SF21_SIDE(N_, CT, CREGS, RT, RW_, RREGS, COLS, ROWS)          \
  template <> struct PairSide<N_> {                                  \
    using Col = PairLine<N_, CT, SF21_CODES COLS>;                   \
    using Row = PairLine<N_, RT, SF21_CODES ROWS>;                   \
    static constexpr int CR = CREGS, RW = RW_, RR = RREGS;           \
  };
#define SF21_CODES(...) __VA_ARGS__
SF21_SIDE(16, 2, 64, 2, 16, 96, (8, CUT, 2), (8, CUT, 2))
SF21_SIDE(24, 8, 64, 8, 8, 96, (3, CUT, 8), (3, CUT, 8))
SF21_SIDE(32, 4, 64, 4, 16, 96, (8, CUT, 4), (8, CUT, 4))
SF21_SIDE(40, 8, 80, 8, 8, 96, (5, CUT, 8), (5, CUT, 8))
SF21_SIDE(48, 8, 80, 8, 8, 96, (3, S8A2, CUT, S8B4, 2), (3, S8A2, CUT, S8B4, 2))
SF21_SIDE(64, 8, 64, 8, 8, 96, (8, CUT, 8), (8, CUT, 8))
SF21_SIDE(72, 9, 80, 9, 8, 112, (3, 3, CUT, 8), (3, 3, CUT, 8))
SF21_SIDE(80, 10, 96, 10, 8, 112, (5, S8A2, CUT, S8B4, 2), (5, S8A2, CUT, S8B4, 2))
SF21_SIDE(96, 12, 96, 12, 8, 128, (3, S8A4, CUT, S8B2, 4), (3, S8A4, CUT, S8B2, 4))
SF21_SIDE(120, 16, 128, 16, 4, 168, (5, 3, CUT, 8), (5, 3, CUT, 8))
SF21_SIDE(128, 16, 64, 16, 4, 128, (8, CUT, 8, CUT, 2), (8, CUT, 8, CUT, 2))
SF21_SIDE(144, 16, 112, 16, 4, 128, (3, 3, CUT, 8, 2), (3, 3, CUT, 8, 2))
SF21_SIDE(160, 16, 112, 16, 4, 128, (5, S8A2, CUT, S8B4, 4), (5, S8A2, CUT, S8B4, 4))
SF21_SIDE(192, 16, 128, 16, 4, 168, (3, S8A4, CUT, S8B2, 8), (3, S8A4, CUT, S8B2, 8))
SF21_SIDE(200, 40, 64, 40, 4, 64, (5, CUT, 5, CUT, 8), (5, CUT, 5, CUT, 8))
SF21_SIDE(216, 24, 128, 24, 4, 168, (3, 3, CUT, 3, 8), (3, 3, CUT, 3, 8))
SF21_SIDE(240, 16, 128, 16, 2, 168, (5, 3, CUT, 8, 2), (5, 3, CUT, 8, 2))
SF21_SIDE(256, 16, 128, 32, 2, 96, (8, S8A2, CUT, S8B4, 4), (8, CUT, 8, CUT, 4))
SF21_SIDE(288, 32, 64, 32, 2, 80, (3, 3, CUT, 8, CUT, 4), (3, 3, CUT, 8, CUT, 4))
SF21_SIDE(320, 40, 80, 64, 1, 64, (5, CUT, 8, CUT, 8), (5, CUT, 8, CUT, 8))
SF21_SIDE(360, 24, 128, 48, 2, 128, (5, 3, CUT, 3, 8), (5, CUT, 3, 3, CUT, 8))
SF21_SIDE(384, 24, 128, 24, 4, 168, (3, 8, CUT, 8, 2), (3, 8, CUT, 8, 2))
SF21_SIDE(400, 40, 80, 40, 4, 96, (5, CUT, 5, S8A2, CUT, S8B4, 2), (5, CUT, 5, S8A2, CUT, S8B4, 2))
SF21_SIDE(432, 48, 80, 48, 2, 80, (3, 3, CUT, 3, S8A2, CUT, S8B4, 2), (3, 3, CUT, 3, S8A2, CUT, S8B4, 2))
SF21_SIDE(480, 32, 128, 64, 1, 128, (5, 3, CUT, 8, 4), (5, 3, CUT, 8, CUT, 4))
SF21_SIDE(512, 64, 64, 64, 1, 96, (8, CUT, 8, CUT, 8), (8, CUT, 8, CUT, 8))
SF21_SIDE(576, 64, 64, 64, 1, 80, (3, 3, CUT, 8, CUT, 8), (3, 3, CUT, 8, CUT, 8))
SF21_SIDE(600, 24, 128, 60, 1, 128, (5, 5, CUT, 8, 3), (5, CUT, 5, S8A2, CUT, S8B4, 3))
SF21_SIDE(640, 64, 128, 64, 1, 128, (5, CUT, 8, CUT, 8, 2), (5, CUT, 8, CUT, 8, 2))
SF21_SIDE(648, 48, 80, 81, 1, 96, (3, 3, CUT, 3, 3, CUT, 8), (3, 3, CUT, 3, 3, CUT, 8))
SF21_SIDE(768, 64, 128, 64, 1, 128, (3, S8A4, CUT, S8B2, 8, CUT, 4), (3, S8A4, CUT, S8B2, 8, CUT, 4))
SF21_SIDE(800, 80, 96, 80, 2, 128, (5, CUT, 5, S8A2, CUT, S8B4, 4), (5, CUT, 5, S8A2, CUT, S8B4, 4))
SF21_SIDE(864, 48, 128, 108, 1, 128, (3, 3, CUT, 3, S8A4, CUT, S8B2, 4), (3, 3, CUT, 3, S8A4, CUT, S8B2, 4))
SF21_SIDE(960, 64, 128, 64, 1, 128, (5, 3, CUT, 8, CUT, 8), (5, 3, CUT, 8, CUT, 8))
SF21_SIDE(1024, 64, 128, 128, 1, 128, (8, CUT, 8, CUT, 8, 2), (8, CUT, 8, CUT, 8, 2))
#undef SF21_CODES
#undef SF21_SIDE

// ---- host side: the launches of one side ------------------------------------------
template <class L, int RW, int REGS>
cudaError_t pair_rows_setup() {
  return cudaFuncSetAttribute(k_pair_rows_filter<L, RW, REGS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)PairRow<L, RW, REGS>::SMEM);
}
// Radii to a grid row: as few as fit the device at once (x CTAs per grid row),
// since a CTA takes its pairs one after the other; KMAX where the tiles fill it.
inline int pair_per(int K, int x, int most) {
  int per = 2;
  while (per < KMAX && (long)x * ((K + per - 1) / per) > most) per *= 2;
  return per;
}
template <class L, int RW, int REGS>
cudaError_t pair_rows_launch(const float2* spec, const Batch& bt, const float2* tw, int nsm, cudaStream_t st) {
  using R = PairRow<L, RW, REGS>;
  const int ng = L::N * L::N / RW, most = nsm * R::PER_SM;
  const int x = pair_min(ng, most), per = L::N > PAIR_MULTI_N ? KMAX : pair_per(bt.K, x, most);
  k_pair_rows_filter<L, RW, REGS><<<dim3(x, (bt.K + per - 1) / per), R::THREADS, R::SMEM, st>>>(
      spec, pair_batch<L::N>(bt), per, tw);
  return cudaGetLastError();
}
template <class L, bool INV, int EPI, int REGS>
cudaError_t pair_cols_setup() {
  return cudaFuncSetAttribute(k_pair_cols<L, INV, EPI, REGS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)PairCol<L, REGS>::SMEM);
}
template <class L, bool INV, int EPI, int REGS, bool AHEAD>
cudaError_t pair_cols_launch(const Batch& bt, uint8_t* rc, float* C, const float* alpha, const float2* tw, int nsm,
                             cudaStream_t st) {
  using G = PairCol<L, REGS>;
  const int x = G::NTILES / G::TPC, per = EPI == 2 || L::N > PAIR_MULTI_N ? KMAX : pair_per(bt.K, x, nsm * G::PER_SM);
  k_pair_cols<L, INV, EPI, REGS><<<dim3(x, (bt.K + per - 1) / per), G::THREADS, G::SMEM, st>>>(
      pair_batch<L::N>(bt), per, rc, C, alpha, tw, AHEAD ? nsm * G::PER_SM : 0);
  return cudaGetLastError();
}

template <int N>
struct PairLaunch {
  using S = PairSide<N>;
  using Row = typename S::Row;
  using Col = typename S::Col;
  // the next pair's lines asked into L2 ahead: faster in the kx pass at every
  // side, in the ky pass where an SM holds two CTAs (512: 0.74 against 0.78 clk),
  // not at the small sides (240: 0.78 against 0.75)
  static constexpr bool AHEAD_B = N >= 300;
  // the criterion and the adjoint hold more per thread than the centre test
  static constexpr int CRA = S::CR <= 80 ? 112 : S::CR <= 112 ? 128 : 168;
  static constexpr size_t ADJ_ROW_SMEM =
      PairRow<Row, S::RW, S::RR>::SMEM + (size_t)S::RW * PairRow<Row, S::RW, S::RR>::WS * sizeof(float2);
  static cudaError_t setup() {
    cudaError_t e = pair_rows_setup<Row, S::RW, S::RR>();
    if (!e) e = pair_cols_setup<Col, true, 0, S::CR>();
    if (!e) e = pair_cols_setup<Col, true, 1, S::CR>();
    if (!e) e = pair_cols_setup<Col, true, 2, CRA>();
    if (!e) e = pair_cols_setup<Col, false, 0, S::CR>();
    if (!e)
      e = cudaFuncSetAttribute(k_pair_cols_a_adj<Col, CRA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)PairCol<Col, CRA>::SMEM);
    if (!e)
      e = cudaFuncSetAttribute(k_pair_rows_adj<Row, S::RW, S::RR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)ADJ_ROW_SMEM);
    if (!e) e = nat_setup();
    if (!e)
      e = cudaFuncSetAttribute(k_pair_hf_rows<Row, S::RW, S::RR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)HF_ROW_SMEM);
    if (!e)
      e = cudaFuncSetAttribute(k_pair_hf_cols_a<Col, S::CR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)PairCol<Col, S::CR>::SMEM);
    return e;
  }
  // the halo finder's filter bank
  static constexpr size_t HF_ROW_SMEM =
      PairRow<Row, S::RW, S::RR>::SMEM + (size_t)S::RW * PairRow<Row, S::RW, S::RR>::WS * sizeof(float2);
  static cudaError_t hf_rows(const float2* spec, const HfBatch& hb, const float2* tw, int nsm, cudaStream_t st) {
    using R = PairRow<Row, S::RW, S::RR>;
    const int ng = N * N / S::RW, most = nsm * R::PER_SM;
    k_pair_hf_rows<Row, S::RW, S::RR><<<pair_min(ng, most), R::THREADS, HF_ROW_SMEM, st>>>(spec, hb, tw);
    return cudaGetLastError();
  }
  static cudaError_t hf_cols_a(const HfBatch& hb, const float2* tw, int nsm, cudaStream_t st) {
    using G = PairCol<Col, S::CR>;
    k_pair_hf_cols_a<Col, S::CR><<<G::NTILES / pair_hf_run<G>() / G::TPC, G::THREADS, G::SMEM, st>>>(hb, tw, nsm * G::PER_SM);
    return cudaGetLastError();
  }
  // one natural-layout box
  static constexpr size_t NAT_COL_SMEM = (size_t)N * 8 * sizeof(cpair) + Col::TW * sizeof(float2);
  static cudaError_t nat_setup() {
    cudaError_t e = cudaSuccess;
    for (auto f : {k_pair_nat_rows<Row, S::RW, S::RR, false>, k_pair_nat_rows<Row, S::RW, S::RR, true>})
      if (!e)
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairRow<Row, S::RW, S::RR>::SMEM);
    for (auto f : {k_pair_nat_cols<Col, false, 0, S::CR>, k_pair_nat_cols<Col, false, 1, S::CR>,
                   k_pair_nat_cols<Col, true, 0, S::CR>, k_pair_nat_cols<Col, true, 1, S::CR>})
      if (!e) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NAT_COL_SMEM);
    return e;
  }
  static cudaError_t nat_rows(const float2* in, const float* real, const float* wax, float2* out, int ncol, bool inverse,
                              const float* alpha, const float2* tw, int nsm, cudaStream_t st) {
    using R = PairRow<Row, S::RW, S::RR>;
    const int ng = N * N / 2 / S::RW, most = nsm * R::PER_SM;
    auto f = inverse ? k_pair_nat_rows<Row, S::RW, S::RR, true> : k_pair_nat_rows<Row, S::RW, S::RR, false>;
    f<<<pair_min(ng, most), R::THREADS, R::SMEM, st>>>(in, real, wax, out, ncol, alpha, tw);
    return cudaGetLastError();
  }
  static cudaError_t nat_cols(float2* box, int axis, bool inverse, int ncol, const float2* tw, cudaStream_t st) {
    auto f = inverse ? (axis ? k_pair_nat_cols<Col, true, 1, S::CR> : k_pair_nat_cols<Col, true, 0, S::CR>)
                     : (axis ? k_pair_nat_cols<Col, false, 1, S::CR> : k_pair_nat_cols<Col, false, 0, S::CR>);
    const int nblk = (ncol + 15) / 16;
    f<<<N * nblk, PairCol<Col, S::CR>::LT, NAT_COL_SMEM, st>>>(box, nblk, tw);
    return cudaGetLastError();
  }
  static cudaError_t cols_b(const Batch& bt, bool inverse, const float2* tw, int nsm, cudaStream_t st) {
    return inverse ? pair_cols_launch<Col, true, 0, S::CR, AHEAD_B>(bt, nullptr, nullptr, nullptr, tw, nsm, st)
                   : pair_cols_launch<Col, false, 0, S::CR, AHEAD_B>(bt, nullptr, nullptr, nullptr, tw, nsm, st);
  }
  static cudaError_t cols_a_test(const Batch& bt, uint8_t* rc, const float* alpha, const float2* tw, int nsm,
                                 cudaStream_t st) {
    return pair_cols_launch<Col, true, 1, S::CR, true>(bt, rc, nullptr, alpha, tw, nsm, st);
  }
  static cudaError_t cols_a_crit(const Batch& bt, float* C, uint8_t* A, const float* alpha, const float2* tw, int nsm,
                                 cudaStream_t st) {
    return pair_cols_launch<Col, true, 2, CRA, true>(bt, A, C, alpha, tw, nsm, st);
  }
  static cudaError_t cols_a_adj(const Batch& bt, const float* g, const uint8_t* A, const float* alpha, float* zpart,
                                const float2* tw, cudaStream_t st) {
    using G = PairCol<Col, CRA>;
    k_pair_cols_a_adj<Col, CRA><<<G::NTILES / G::TPC, G::THREADS, G::SMEM, st>>>(pair_batch<N>(bt), g, A, alpha, zpart, tw);
    return cudaGetLastError();
  }
  static cudaError_t rows_adj(const Batch& bt, float2* acc, const float2* tw, int nsm, cudaStream_t st) {
    using R = PairRow<Row, S::RW, S::RR>;
    const int ng = N * N / S::RW, most = nsm * R::PER_SM;
    k_pair_rows_adj<Row, S::RW, S::RR><<<pair_min(ng, most), R::THREADS, ADJ_ROW_SMEM, st>>>(pair_batch<N>(bt), acc, tw);
    return cudaGetLastError();
  }
  static constexpr PairOps ops() {
    return {N <= PAIR_MULTI_N ? RADII_MAX : KMAX,
            setup,       pair_rows_launch<Row, S::RW, S::RR>, cols_b,   cols_a_test,
            cols_a_crit, cols_a_adj,                          rows_adj, PairCol<Col, CRA>::NTILES / PairCol<Col, CRA>::TPC,
            nat_rows,    nat_cols,                            hf_rows,  hf_cols_a};
  }
};

}  // namespace sf21
