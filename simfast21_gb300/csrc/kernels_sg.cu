// Subgrid Poisson cycle of the halo finder on the GPU (get_halos.c:326-371).
//
// The reference walks the unflagged cells in index order and draws one
// Poisson deviate per cell from a single taus generator (gsl_ran_poisson,
// the product-of-uniforms method for means <= 10): a draw that starts at
// stream position s consumes L(s) uniforms, L(s) = the first L with
// u_s u_{s+1} ... u_{s+L-1} <= exp(-mu) (products in double), and returns
// k = L(s) - 1.  Draw n starts at s_n, s_{n+1} = s_n + L(s_n).  The GPU form
// reproduces that stream exactly:
//   A  per block of SG_B positions: the generator's state is jumped to the
//      block (the generator is linear over GF(2): 32x32 bit matrices of its
//      powers), a warp's lanes step 32 consecutive positions each, L(s) is
//      computed for every position (one integer compare decides L = 1; longer
//      chains multiply in float, and with the IEEE double rounding done in
//      integers where the float product is too close to exp(-mu)), and the
//      segments' tables compose to, for every entry offset e < SG_LMAX, the
//      block's exit offset and draw count;
//   B  the entries of all blocks follow by composing those tables (groups of
//      SG_G blocks, supergroups of SG_G groups, in parallel; the supergroups
//      in order; then down to the groups and the blocks);
//   C  each block replays its chain from its entry and lists the draws with
//      k >= 1 (k = 0 writes nothing) with their draw index;
//   D  draw n belongs to the n-th unflagged cell (binary search in the
//      per-word prefix counts of the unflagged bit set); nn = (int)
//      round(k (1 + delta growth hbias)) in soft-double; the records follow
//      from a prefix sum over nn.
// No FP64 unit is used: sg_dmul.h (the draw products) and softdouble.h (the
// halo counts) give the IEEE results in integer arithmetic.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sf21_kernels.h"
#include "sg_dmul.h"
#include "softdouble.h"

namespace sf21 {

__device__ __forceinline__ uint32_t gf2_apply(const uint32_t* __restrict__ col, uint32_t v) {
  uint32_t r = 0;
#pragma unroll
  for (int k = 0; k < 32; ++k) r ^= (0u - ((v >> k) & 1u)) & __ldg(col + k);
  return r;
}

// the same with the columns SG_LOCAL words apart
__device__ __forceinline__ uint32_t gf2_apply_strided(const uint32_t* __restrict__ col, uint32_t v) {
  uint32_t r = 0;
#pragma unroll
  for (int k = 0; k < 32; ++k) r ^= (0u - ((v >> k) & 1u)) & __ldg(col + (size_t)k * SG_LOCAL);
  return r;
}

__device__ __forceinline__ void taus_step(uint32_t& a, uint32_t& b, uint32_t& c) {
  a = ((a & 4294967294u) << 12) ^ (((a << 13) ^ a) >> 19);
  b = ((b & 4294967288u) << 4) ^ (((b << 2) ^ b) >> 25);
  c = ((c & 4294967280u) << 17) ^ (((c << 3) ^ c) >> 11);
}

// Access checks of the draw and record kernels: an index outside its buffer
// is recorded (err[1] = site, err[2] = low 31 bits of the index) and the
// access skipped; the host turns a record into an error return.
__device__ __forceinline__ void sg_bad(int* err, int site, uint64_t idx) {
  if (atomicCAS(err + 1, 0, site) == 0) err[2] = (int)(idx & 0x7fffffff);
}

// A ------------------------------------------------------------------------
// jumps: pow2[(k 3 + c) 32 + col] = column col of component c of T^(2^k)
// (k < SG_POW2); local[(c 32 + col) SG_LOCAL + i] = the same of T^(SG_SEG i)
// (i < SG_LOCAL), stored so that the lanes of a warp, each applying its own
// power, read consecutive words.  S0: the state whose next step gives
// position 0.
// The state at the start of every block, T^(b SG_B) S0: one thread per
// component and run of SG_RUN blocks, the first by its bits, the others by
// one T^SG_B each.
constexpr int SG_RUN = 4;
static_assert(SG_WARPS % SG_RUN == 0, "runs of blocks");
__global__ void k_sg_start(SgArgs a, const uint32_t* __restrict__ pow2, long nblocks, uint32_t* __restrict__ start) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nblocks / SG_RUN * 3) return;
  const long b = t / 3 * SG_RUN;
  const int c = (int)(t % 3);
  const uint64_t base = (uint64_t)b * SG_B;
  uint32_t v = a.s0[c];
  for (int k = 0; k < SG_POW2; ++k)
    if ((base >> k) & 1u) v = gf2_apply(pow2 + ((size_t)k * 3 + c) * 32, v);
  for (int r = 0;; ++r) {
    start[(b + r) * 3 + c] = v;
    if (r + 1 == SG_RUN) break;
    v = gf2_apply(pow2 + ((size_t)SG_LOG2B * 3 + c) * 32, v);
  }
}

// Where word j of a segment's row lies: rows of 33 words, so that the lanes'
// rows start on different banks; j may run on into the rows that follow.
__device__ __forceinline__ int sg_at(int row, int j) { return row * 33 + j + (j >> 5); }

// Draw length at a position whose first uniform exceeds exp(-mu), in the
// reference's arithmetic (products in double).
__device__ __noinline__ int sg_draw_exact(const uint32_t* sx, int row, int p, uint64_t emu_bits) {
  const DMant emu = dm_from_bits(emu_bits);
  DMant prod = dm_from_u32(sx[sg_at(row, p)]);
  int L = 2;
  for (; L <= SG_LMAX; ++L) {
    const uint32_t xn = sx[sg_at(row, p + L - 1)];
    if (xn == 0) break;  // a zero factor ends the draw
    prod = dm_mul_u32(prod, xn);
    if (dm_le(prod, emu)) break;
  }
  return L;
}

// One warp per block of SG_B positions, one lane per segment of SG_SEG = 32.
//   1  each lane jumps to its segment and steps through it, the outputs into
//      shared memory and the positions with L >= 2 into a mask;
//   2  L at the positions of the mask, by products in float: their error is
//      under 2 SG_LMAX 2^-24 = 2^-17 of the value, so a product outside
//      (lo, hi) = exp(-mu) (1 -+ 2^-15) is on its side of exp(-mu) in double
//      too, and only the others (one in 2^14) take sg_draw_exact;
//   3  for every position of the mask, from the last back to the first: where
//      the chain from it leaves the segment and after how many draws (between
//      the positions of the mask every draw takes one uniform);
//   4  the block's table: the chains of all SG_LMAX entries, two per lane, go
//      through the segments until they have met (two or three segments, as a
//      rule); for the rest every lane walks its own segment, from entry 0
//      first and then from its neighbour's exit until nothing changes (the
//      exits settle from the left, mostly after two or three rounds).
// What bounds it: the integer pipe, about 17 operations per position for the
// generator itself and 10 for the jump.  512^3 cells, mean 0.03 per cell (138 M
// positions): 0.225 ms, 2.32 ms when every position took part in ten rounds of
// pointer jumping in shared memory and four positions shared a jump.
__global__ void __launch_bounds__(SG_THREADS)
k_sg_len(SgArgs a, long nblocks, const uint32_t* __restrict__ start, const uint32_t* __restrict__ local,
         uint8_t* __restrict__ Lout, uint32_t* __restrict__ LB, uint8_t* __restrict__ X, uint16_t* __restrict__ D,
         int* __restrict__ err) {
  __shared__ uint32_t sx[(SG_WARPS * 32 + SG_LMAX / 32) * 33];
  __shared__ uint32_t sl[SG_WARPS * 32 * 9];  // draw lengths, rows of 32 bytes and a word between
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32, row = threadIdx.x;
  const long b = (long)blockIdx.x * SG_WARPS + w;
  uint32_t mask = 0;
  // the segments of the CTA's blocks, and (warp 0) those that its last draws run into
  for (int pass = 0; pass < (w ? 1 : 2); ++pass) {
    if (pass && lane >= SG_LMAX / 32) break;
    const uint32_t* s = start + 3 * (pass ? b + SG_WARPS - 1 : b);
    const uint32_t* J = local + (pass ? 32 + lane : lane);
    const int r0 = pass ? SG_WARPS * 32 + lane : row;
    uint32_t x = gf2_apply_strided(J, __ldg(s)), y = gf2_apply_strided(J + 32 * SG_LOCAL, __ldg(s + 1)),
             z = gf2_apply_strided(J + 64 * SG_LOCAL, __ldg(s + 2));
    uint32_t mk = 0;
#pragma unroll
    for (int r = 0; r < SG_SEG; ++r) {
      taus_step(x, y, z);
      const uint32_t u = x ^ y ^ z;
      sx[r0 * 33 + r] = u;
      // x <= X1 <=> u = x 2^-32 <= exp(-mu) <=> one uniform
      if (u > a.x1) mk |= 1u << r;
    }
    if (!pass) mask = mk;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) sl[row * 9 + k] = 0x01010101u;
  __syncthreads();
  uint8_t* lrow = reinterpret_cast<uint8_t*>(sl + row * 9);
  for (uint32_t m = mask; m; m &= m - 1) {
    const int p = __ffs(m) - 1;
    float prod = __uint2float_rn(sx[row * 33 + p]) * 0x1p-32f;
    int L = 2;
    for (; L <= SG_LMAX; ++L) {
      prod *= __uint2float_rn(sx[sg_at(row, p + L - 1)]) * 0x1p-32f;
      if (prod <= a.hi) break;
    }
    if (L > SG_LMAX || prod > a.lo) L = sg_draw_exact(sx, row, p, a.emu);
    if (L > SG_LMAX) {
      atomicOr(err, 1);
      L = SG_LMAX;
    }
    lrow[p] = (uint8_t)L;
  }
  __syncthreads();  // the outputs have been read: the rows take the chains, exit | draws << 8
  for (uint32_t m = mask; m;) {
    const int p = 31 - __clz(m);
    m ^= 1u << p;
    const int n = p + lrow[p];
    uint32_t v;
    if (n >= SG_SEG) {
      v = (uint32_t)(n - SG_SEG) | 1u << 8;
    } else {
      const uint32_t mm = mask & (0xffffffffu << n);
      if (!mm) {
        v = (uint32_t)(1 + SG_SEG - n) << 8;
      } else {
        const int q = __ffs(mm) - 1;
        v = sx[row * 33 + q] + ((uint32_t)(1 + q - n) << 8);
      }
    }
    sx[row * 33 + p] = v;
  }
  __syncwarp();
  if (b >= nblocks) return;
  uint32_t* Lw = reinterpret_cast<uint32_t*>(Lout + (uint64_t)b * SG_B);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int i = k * 32 + lane;
    Lw[i] = sl[(w * 32 + i / 8) * 9 + i % 8];
  }
  LB[(size_t)b * (SG_B / 32) + lane] = mask;
  // entry e of the segment in row r with mask mk: its exit in place of e, its draws added to c
  auto walk = [&](int& e, uint32_t& c, uint32_t mk, int r) {
    if (e >= SG_SEG) {
      e -= SG_SEG;
      return;
    }
    const uint32_t mm = mk & (0xffffffffu << e);
    if (!mm) {
      c += (uint32_t)(SG_SEG - e);
      e = 0;
    } else {
      const int p = __ffs(mm) - 1;
      const uint32_t v = sx[r * 33 + p];
      c += (uint32_t)(p - e) + (v >> 8);
      e = (int)(v & 0xffu);
    }
  };
  int e0 = lane, e1 = lane + 32, j = 0;
  uint32_t c0 = 0, c1 = 0;
  bool met = false;
  while (j < 32 && !met) {
    const uint32_t mk = __shfl_sync(0xffffffffu, mask, j);
    walk(e0, c0, mk, w * 32 + j);
    walk(e1, c1, mk, w * 32 + j);
    ++j;
    const int f = __shfl_sync(0xffffffffu, e0, 0);
    met = __all_sync(0xffffffffu, e0 == f && e1 == f);
  }
  if (j < 32) {  // all at entry e0 of segment j
    int entry = lane == j ? e0 : 0, x;
    uint32_t c;
    for (int round = 0; round < 32; ++round) {
      x = entry;
      c = 0;
      walk(x, c, mask, row);
      int next = __shfl_up_sync(0xffffffffu, x, 1);
      if (lane <= j) next = entry;
      const bool same = __all_sync(0xffffffffu, next == entry);
      entry = next;
      if (same) break;
    }
    const uint32_t rest = __reduce_add_sync(0xffffffffu, lane >= j ? c : 0u);
    c0 += rest;
    c1 += rest;
    e0 = e1 = __shfl_sync(0xffffffffu, x, 31);
  }
  X[(size_t)b * SG_LMAX + lane] = (uint8_t)e0;
  X[(size_t)b * SG_LMAX + 32 + lane] = (uint8_t)e1;
  D[(size_t)b * SG_LMAX + lane] = (uint16_t)c0;
  D[(size_t)b * SG_LMAX + 32 + lane] = (uint16_t)c1;
}

// B ------------------------------------------------------------------------
// Entries of all blocks, by composing the per-block tables (exit offset X,
// draws D for each entry offset e < SG_LMAX) in groups of SG_G: blocks ->
// groups -> supergroups (SG_LMAX threads per parent, each walking one entry
// through the SG_G children), one thread over the supergroups, then down again
// (one thread per parent walking its children from the parent's entry).
template <class TD>
__global__ void k_sg_compose(const uint8_t* __restrict__ X, const TD* __restrict__ D, long n,
                             uint8_t* __restrict__ PX, uint32_t* __restrict__ PD) {
  const long g = blockIdx.x;
  const int e0 = threadIdx.x;  // SG_LMAX threads
  int e = e0;
  uint32_t tot = 0;
  const long c1 = (g + 1) * SG_G < n ? (g + 1) * SG_G : n;
  for (long c = g * SG_G; c < c1; ++c) {
    tot += D[(size_t)c * SG_LMAX + e];
    e = X[(size_t)c * SG_LMAX + e];
  }
  PX[(size_t)g * SG_LMAX + e0] = (uint8_t)e;
  PD[(size_t)g * SG_LMAX + e0] = tot;
}

__global__ void k_sg_top(const uint8_t* __restrict__ X, const uint32_t* __restrict__ D, long n,
                         uint8_t* __restrict__ entry, uint64_t* __restrict__ base_out) {
  if (threadIdx.x || blockIdx.x) return;
  int e = 0;
  uint64_t base = 0;
  for (long c = 0; c < n; ++c) {
    entry[c] = (uint8_t)e;
    base_out[c] = base;
    base += D[(size_t)c * SG_LMAX + e];
    e = X[(size_t)c * SG_LMAX + e];
  }
  base_out[n] = base;  // draws available in all generated positions
}

template <class TD>
__global__ void k_sg_descend(const uint8_t* __restrict__ X, const TD* __restrict__ D, long n, long nparents,
                             const uint8_t* __restrict__ pentry, const uint64_t* __restrict__ pbase,
                             uint8_t* __restrict__ entry, uint64_t* __restrict__ base_out) {
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nparents) return;
  int e = pentry[g];
  uint64_t base = pbase[g];
  const long c1 = (g + 1) * SG_G < n ? (g + 1) * SG_G : n;
  for (long c = g * SG_G; c < c1; ++c) {
    entry[c] = (uint8_t)e;
    base_out[c] = base;
    base += D[(size_t)c * SG_LMAX + e];
    e = X[(size_t)c * SG_LMAX + e];
  }
}

// C ------------------------------------------------------------------------
// mode 0: count the draws with k >= 1 among draws < U per block, and record
// the position after draw U - 1; mode 1: write them (draw index, k).
constexpr int WALK_THREADS = 128;
// Each thread walks one block.  Between two long draws (k >= 1) every draw
// takes one uniform, so the walk jumps from long position to long position
// with the block's bit set of long positions (LB) and counts the one-uniform
// draws in between; it touches the draw lengths (L) only at long positions.
__global__ void __launch_bounds__(WALK_THREADS)
k_sg_walk(int mode, const uint8_t* __restrict__ Lb, const uint32_t* __restrict__ LB, long nblocks,
          const uint8_t* __restrict__ bentry, const uint64_t* __restrict__ bbase, uint64_t U,
          uint32_t* __restrict__ cnt, uint64_t* __restrict__ consumed, uint64_t* __restrict__ dn,
          uint8_t* __restrict__ dk, uint64_t cap, int* __restrict__ err) {
  const long b = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nblocks) return;
  uint64_t n = bbase[b];
  if (n >= U) {
    if (mode == 0) cnt[b] = 0;
    return;
  }
  const uint64_t base = (uint64_t)b * SG_B;
  const uint32_t* lb = LB + (size_t)b * (SG_B / 32);
  int s = bentry[b];
  uint32_t c = 0;
  const uint32_t off = mode ? cnt[b] : 0;
  while (s < SG_B && n < U) {
    // next long position p >= s (SG_B if none)
    int w = s >> 5;
    uint32_t m = __ldg(lb + w) & (0xffffffffu << (s & 31));
    while (!m && ++w < SG_B / 32) m = __ldg(lb + w);
    const int p = m ? w * 32 + __ffs(m) - 1 : SG_B;
    // draws at s .. p-1 take one uniform each
    const uint64_t steps = (uint64_t)(p - s);
    if (n + steps >= U) {  // draw U - 1 is one of them
      if (mode == 0) *consumed = base + s + (U - 1 - n) + 1;
      n = U;
      break;
    }
    n += steps;
    s = p;
    if (s >= SG_B) break;
    const int L = Lb[base + s];
    if (mode) {
      if ((uint64_t)off + c < cap) {
        dn[off + c] = n;
        dk[off + c] = (uint8_t)(L - 1);
      } else {
        sg_bad(err, 1, (uint64_t)off + c);
      }
    }
    ++c;
    if (mode == 0 && n == U - 1) *consumed = base + s + L;
    s += L;
    ++n;
  }
  if (mode == 0) cnt[b] = c;
}

// D ------------------------------------------------------------------------
__device__ __forceinline__ int64_t sd_round_half_away(sd_t x) {
  if (sd_is_zero(x)) return 0;
  const int e = (int)((x >> 52) & 0x7FF) - 1023;
  const uint64_t m = (x & 0xFFFFFFFFFFFFFULL) | (1ULL << 52);  // value = m 2^(e-52)
  int64_t q;
  if (e < -1) {
    q = 0;
  } else if (e >= 52) {
    q = (int64_t)(m << (e - 52 < 11 ? e - 52 : 10));
  } else {
    const int sh = 52 - e;  // 1..53
    const uint64_t r = m & ((1ULL << sh) - 1);
    q = (int64_t)(m >> sh) + (r >= (1ULL << (sh - 1)) ? 1 : 0);
  }
  return (x >> 63) ? -q : q;
}

// cell of draw n: the n-th zero bit of FL; wpre[w] = zero bits of words < w
__device__ __forceinline__ uint32_t select_unflagged(const uint32_t* __restrict__ FL,
                                                     const uint32_t* __restrict__ wpre, long nwords, uint64_t n) {
  long lo = 0, hi = nwords - 1;  // last w with wpre[w] <= n
  while (lo < hi) {
    const long mid = (lo + hi + 1) >> 1;
    if (wpre[mid] <= n) lo = mid; else hi = mid - 1;
  }
  uint32_t free_bits = ~FL[lo];
  uint32_t r = (uint32_t)(n - wpre[lo]);
  while (r-- && free_bits) free_bits &= free_bits - 1;
  return (uint32_t)(lo * 32 + (free_bits ? __ffs(free_bits) - 1 : 0));  // n < free cells: never the 0 case
}

__global__ void k_sg_nn(const uint64_t* __restrict__ dn, const uint8_t* __restrict__ dk, long nd,
                        const uint32_t* __restrict__ FL, const uint32_t* __restrict__ wpre, long nwords,
                        const float* __restrict__ delta, uint64_t growth, uint64_t hbias, uint32_t* __restrict__ cell,
                        uint32_t* __restrict__ nn, int* __restrict__ err) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nd; i += (long)gridDim.x * blockDim.x) {
    const uint32_t t = select_unflagged(FL, wpre, nwords, dn[i]);
    if ((long)t >= nwords * 32) {
      sg_bad(err, 2, t);
      cell[i] = 0;
      nn[i] = 0;
      continue;
    }
    // tempv = map_in_f[index] * growth * hbias; nn = (int) round(Pn (1 + tempv))  (:351-354)
    const sd_t tempv = sd_mul(sd_mul(sd_from_float(delta[t]), growth), hbias);
    const sd_t v = sd_mul(sd_from_int(dk[i]), sd_add(0x3FF0000000000000ULL, tempv));
    int64_t q = sd_round_half_away(v);
    if (q > (1 << 24)) {  // a finite density and k <= 63 stay far below
      sg_bad(err, 3, (uint64_t)i);
      q = 0;
    }
    cell[i] = t;
    nn[i] = q > 0 ? (uint32_t)q : 0u;
  }
}

__global__ void k_sg_records(const uint32_t* __restrict__ cell, const uint32_t* __restrict__ nn,
                             const uint32_t* __restrict__ off, long nd, int N, float mass,
                             float4* __restrict__ out, uint64_t cap, int* __restrict__ err) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nd; i += (long)gridDim.x * blockDim.x) {
    const uint32_t t = cell[i];
    const uint32_t q = t / (uint32_t)N, a = q / (uint32_t)N;
    const float4 rec = make_float4(mass, (float)a, (float)(q - a * (uint32_t)N), (float)(t - q * (uint32_t)N));
    const uint32_t o = off[i];
    for (uint32_t r = 0; r < nn[i]; ++r) {
      if ((uint64_t)o + r < cap)
        out[o + r] = rec;
      else
        sg_bad(err, 4, (uint64_t)o + r);
    }
  }
}

// zero bits per word of FL
__global__ void k_sg_free_count(const uint32_t* __restrict__ FL, long nwords, uint32_t* __restrict__ c) {
  for (long w = (long)blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += (long)gridDim.x * blockDim.x)
    c[w] = 32u - (uint32_t)__popc(FL[w]);
}

// ---------------------------------------------------------------------------
// Exclusive prefix sums of a uint32 array (chunk sums, one CTA over the
// chunk sums, per-chunk scans with the chunk's offset).  Totals < 2^32.
constexpr int SC_THREADS = 256;
constexpr long SC_CHUNK = 8192;

__global__ void __launch_bounds__(SC_THREADS) k_chunk_sum(const uint32_t* __restrict__ a, long n,
                                                          uint32_t* __restrict__ sums) {
  const long c0 = blockIdx.x * SC_CHUNK;
  uint32_t s = 0;
  for (long i = c0 + threadIdx.x; i < c0 + SC_CHUNK && i < n; i += SC_THREADS) s += a[i];
  s = __reduce_add_sync(0xffffffffu, s);
  __shared__ uint32_t red[SC_THREADS / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int k = 0; k < SC_THREADS / 32; ++k) t += red[k];
    sums[blockIdx.x] = t;
  }
}

// a and out may be the same array (in-place scans): no __restrict__ on them,
// and a CTA's elements are all loaded before the first slot is overwritten.
// A warp owns SC_CHUNK / 8 consecutive elements, 128 at a time, four per lane
// (32 consecutive ones per thread: 46 us for the words of 512^3 cells, 8 us so).
__global__ void __launch_bounds__(SC_THREADS) k_chunk_scan(const uint32_t* a, long n,
                                                           const uint32_t* __restrict__ off, uint32_t* out) {
  constexpr int WARPS = SC_THREADS / 32, IT = (int)(SC_CHUNK / SC_THREADS / 4);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long i0 = blockIdx.x * SC_CHUNK + (long)w * (SC_CHUNK / WARPS) + 4 * lane;
  uint4 v[IT];
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const long p = i0 + 128 * i;
    if (p + 3 < n) {
      v[i] = *reinterpret_cast<const uint4*>(a + p);
    } else {
      v[i].x = p < n ? a[p] : 0u;
      v[i].y = p + 1 < n ? a[p + 1] : 0u;
      v[i].z = p + 2 < n ? a[p + 2] : 0u;
      v[i].w = 0u;
    }
  }
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < IT; ++i) s += v[i].x + v[i].y + v[i].z + v[i].w;
  __shared__ uint32_t wsum[WARPS];
  s = __reduce_add_sync(0xffffffffu, s);
  if (lane == 0) wsum[w] = s;
  __syncthreads();
  uint32_t pos = off[blockIdx.x];
  for (int k = 0; k < w; ++k) pos += wsum[k];
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const uint32_t t = v[i].x + v[i].y + v[i].z + v[i].w;
    uint32_t x = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const long p = i0 + 128 * i;
    uint4 r;
    r.x = pos + x - t;
    r.y = r.x + v[i].x;
    r.z = r.y + v[i].y;
    r.w = r.z + v[i].z;
    if (p + 3 < n) {
      *reinterpret_cast<uint4*>(out + p) = r;
    } else {
      if (p < n) out[p] = r.x;
      if (p + 1 < n) out[p + 1] = r.y;
      if (p + 2 < n) out[p + 2] = r.z;
    }
    pos += __shfl_sync(0xffffffffu, x, 31);
  }
}

long scan_chunks(long n) { return (n + SC_CHUNK - 1) / SC_CHUNK; }

cudaError_t launch_scan_u32(const uint32_t* a, long n, uint32_t* out, uint32_t* chunk, uint32_t* total,
                            cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const long nc = scan_chunks(n);
  k_chunk_sum<<<(unsigned)nc, SC_THREADS, 0, st>>>(a, n, chunk);
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  if ((e = launch_scan_counts(chunk, nc, total, st))) return e;
  k_chunk_scan<<<(unsigned)nc, SC_THREADS, 0, st>>>(a, n, chunk, out);
  return cudaGetLastError();
}

static unsigned grid_for(long n, int threads) {
  long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 152 * 32) b = 152 * 32;
  return (unsigned)b;
}

cudaError_t launch_sg_len(long nblocks, const SgArgs& a, const uint32_t* pow2, const uint32_t* local, uint32_t* start,
                          uint8_t* L, uint32_t* LB, uint8_t* X, uint16_t* D, int* err, cudaStream_t st) {
  const long padded = sg_padded(nblocks);
  k_sg_start<<<(unsigned)((padded / SG_RUN * 3 + 255) / 256), 256, 0, st>>>(a, pow2, padded, start);
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  k_sg_len<<<(unsigned)(padded / SG_WARPS), SG_THREADS, 0, st>>>(a, nblocks, start, local, L, LB, X, D, err);
  return cudaGetLastError();
}

long sg_padded(long nblocks) { return (nblocks + SG_WARPS - 1) / SG_WARPS * SG_WARPS; }
long sg_groups(long n) { return (n + SG_G - 1) / SG_G; }

cudaError_t launch_sg_entries(const uint8_t* X, const uint16_t* D, long nblocks, const SgEntryBufs& eb,
                              cudaStream_t st) {
  const long ng = sg_groups(nblocks), ns = sg_groups(ng);
  k_sg_compose<uint16_t><<<(unsigned)ng, SG_LMAX, 0, st>>>(X, D, nblocks, eb.gx, eb.gd);
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  k_sg_compose<uint32_t><<<(unsigned)ns, SG_LMAX, 0, st>>>(eb.gx, eb.gd, ng, eb.sx, eb.sd);
  if ((e = cudaGetLastError())) return e;
  k_sg_top<<<1, 32, 0, st>>>(eb.sx, eb.sd, ns, eb.sentry, eb.sbase);
  if ((e = cudaGetLastError())) return e;
  k_sg_descend<uint32_t><<<(unsigned)((ns + 127) / 128), 128, 0, st>>>(eb.gx, eb.gd, ng, ns, eb.sentry, eb.sbase,
                                                                        eb.gentry, eb.gbase);
  if ((e = cudaGetLastError())) return e;
  k_sg_descend<uint16_t><<<(unsigned)((ng + 127) / 128), 128, 0, st>>>(X, D, nblocks, ng, eb.gentry, eb.gbase,
                                                                        eb.bentry, eb.bbase);
  return cudaGetLastError();
}

cudaError_t launch_sg_walk(int mode, const uint8_t* L, const uint32_t* LB, long nblocks, const uint8_t* bentry,
                           const uint64_t* bbase, uint64_t U, uint32_t* cnt, uint64_t* consumed, uint64_t* dn,
                           uint8_t* dk, uint64_t cap, int* err, cudaStream_t st) {
  k_sg_walk<<<(unsigned)((nblocks + WALK_THREADS - 1) / WALK_THREADS), WALK_THREADS, 0, st>>>(
      mode, L, LB, nblocks, bentry, bbase, U, cnt, consumed, dn, dk, cap, err);
  return cudaGetLastError();
}

cudaError_t launch_sg_free_count(const uint32_t* FL, long nwords, uint32_t* c, cudaStream_t st) {
  k_sg_free_count<<<grid_for(nwords, 256), 256, 0, st>>>(FL, nwords, c);
  return cudaGetLastError();
}

cudaError_t launch_sg_nn(const uint64_t* dn, const uint8_t* dk, long nd, const uint32_t* FL, const uint32_t* wpre,
                         long nwords, const float* delta, uint64_t growth, uint64_t hbias, uint32_t* cell,
                         uint32_t* nn, int* err, cudaStream_t st) {
  if (nd <= 0) return cudaSuccess;
  k_sg_nn<<<grid_for(nd, 256), 256, 0, st>>>(dn, dk, nd, FL, wpre, nwords, delta, growth, hbias, cell, nn, err);
  return cudaGetLastError();
}

cudaError_t launch_sg_records(const uint32_t* cell, const uint32_t* nn, const uint32_t* off, long nd, int N,
                              float mass, float4* out, uint64_t cap, int* err, cudaStream_t st) {
  if (nd <= 0) return cudaSuccess;
  k_sg_records<<<grid_for(nd, 256), 256, 0, st>>>(cell, nn, off, nd, N, mass, out, cap, err);
  return cudaGetLastError();
}

}  // namespace sf21
