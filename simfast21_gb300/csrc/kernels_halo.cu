// Halo-catalogue source box on the GPU (use_SFR = F branch of the stage,
// get_HIIbubbles.c:229-253): Rion(M, z) of every halo (user_functions.c:40-47),
// cloud-in-cell deposit on the N_halo^3 grid (auxiliary.c:761-808) and the
// block average to N_smooth^3 (auxiliary.c:643-684) -- bit-identical with the
// reference's serial loop.  The star-formation-rate stage (get_SFR.c:114-131)
// is the same deposit with the weight sfr(M, z) = Rion(M, z) / Qion(z)
// (user_functions.c:71-75) and each smoothed cell divided by dx_halo^3.
//
// The reference adds the 8 CIC contributions of halo 0, then halo 1, ... into
// a float box (float += double each time), so a cell's value depends on the
// order of its contributions.  Here every contribution is computed in
// parallel (same float/double steps, integer soft-double for the double
// ones) and written at its serial position, the (cell, weight) entries are
// grouped by cell with a stable radix sort (the serial order survives inside
// each cell), and each cell's chain is replayed in that order.  The block
// average gives the reference's serial double sum (exactly, by an integer sum
// when no partial sum rounds, else by the soft-double chain).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <mutex>

#include "../../include/sf21_hii.h"

#include "sf21_kernels.h"
#include "softdouble.h"

namespace sf21 {

struct HaloRec {  // Halo_t, auxiliary.h:13-17
  float Mass, x, y, z;
};

__device__ __forceinline__ long wrap_cell(long x, long n) {  // check_borders, auxiliary.c:537-544
  if (x >= 0 && x < n) return x;  // the usual cases without a 64-bit division
  if (x >= n && x < 2 * n) return x - n;
  if (x < 0 && x >= -n) return x + n;
  x = x % n;
  if (x < 0) x += n;
  return x;
}

// Constants of Rion (user_functions.c:33-38) and pow(1+z, c4), as double bit
// patterns set on the host; qion = Qion(z) for the sfr weight, 0 for Rion.
struct RionConst {
  sd_t c1, c2, c3, three, vnorm, p1, qion;
};

// Rion(hmass, z) = c1 hmass (1+z)^c4 (hmass/c2)^c3 exp(-(c2/hmass)^3) / V_norm
// in double; the value CIC receives is that double (or sfr = Rion / Qion,
// user_functions.c:71-75) rounded to its float parameter (auxiliary.c:761).
__device__ __forceinline__ float weight_sd(float m, const RionConst& k) {
  const sd_t M = sd_from_float(m);
  const sd_t t1 = sd_mul(sd_mul(k.c1, M), k.p1);
  const sd_t t2 = sd_pow(sd_div(M, k.c2), k.c3);
  const sd_t t3 = sd_exp(sd_neg(sd_pow(sd_div(k.c2, M), k.three)));
  const sd_t rion = sd_div(sd_mul(sd_mul(t1, t2), t3), k.vnorm);
  return sd_to_float(k.qion ? sd_div(rion, k.qion) : rion);
}

// Weights per distinct mass.  A catalogue of the halo finder holds a few
// distinct masses (one per mass of its schedule), so the soft-double
// pow/exp of the weight runs once per distinct mass: the mass bit patterns
// are sorted and made unique, their weights computed, and each halo finds
// its mass by binary search.
__global__ void k_mass_keys(long nh, const HaloRec* __restrict__ halos, uint32_t* __restrict__ keys) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += (long)gridDim.x * blockDim.x)
    keys[i] = __float_as_uint(halos[i].Mass);
}

__global__ void k_mass_weights(long nh, const uint32_t* __restrict__ uniq, const int* __restrict__ n_uniq,
                               RionConst rk, float* __restrict__ w) {
  const long n = *n_uniq;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n && i < nh; i += (long)gridDim.x * blockDim.x)
    w[i] = weight_sd(__uint_as_float(uniq[i]), rk);
}

struct MassTable {
  const uint32_t* uniq;  // sorted distinct mass bit patterns (nullptr: compute per halo)
  const int* n_uniq;
  const float* w;
};

// weight of a halo's mass: the lower bound of its bits in uq[0, nu) (it is
// there), or computed
__device__ __forceinline__ float mass_weight(float mass, const uint32_t* uq, const float* wq, int nu,
                                             const RionConst& rk) {
  if (!uq) return weight_sd(mass, rk);
  const uint32_t key = __float_as_uint(mass);
  int lo = 0, hi = nu - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (uq[mid] < key)
      lo = mid + 1;
    else
      hi = mid;
  }
  return wq[lo];
}

// Cell below a coordinate and the fraction above it (auxiliary.c:769-780)
__device__ __forceinline__ long cic_cell(float f, float* frac) {
  long c = (long)f;
  float q = f - (float)c;
  if (q < 0.0f) {
    c = c - 1;
    q = fabsf(q);
  }
  *frac = q;
  return c;
}

// The reference's corner loop (auxiliary.c:769-806) moves a negative
// fraction f to the cell below at its first corner, then for each upper
// corner flips f to (float)(1.0 - f) and back again after the deposit.
// The flip back is not exact for f < 1/2: it leaves f' = 1 - fl(1 - f),
// and later corners see f'.  Along each axis the cells are wrap(c0) and
// wrap(c0 + 1); the factors, in the loop's corner order (a, b, c), are
//   x: a = 0: 1 - x;  a = 1: 1 - fl(1 - x)
//   y: b = 0: 1 - y for a = 0, 1 - y' for a = 1;  b = 1: 1 - fl(1 - y)
//   z: c = 0: 1 - z for (a, b) = (0, 0), 1 - z' after;  c = 1: 1 - fl(1 - z)
// (1 - v in double, as the reference's (1.0 - x1)), multiplied in the
// reference's order ((fx * fy) * fz) * map_in.
struct Cic {
  long cx[2], cy[2], cz[2];
  sd_t FX[2], FY0[2], FY1, FZ0, FZ0p, FZ1;
  __device__ __forceinline__ sd_t xy(int a, int b) const { return sd_mul(FX[a], b ? FY1 : FY0[a]); }
  __device__ __forceinline__ sd_t z(int a, int b, int c) const { return c ? FZ1 : ((a == 0 && b == 0) ? FZ0 : FZ0p); }
};
__device__ __forceinline__ Cic cic_of(float x, float y, float z, long N) {
  const sd_t one = 0x3FF0000000000000ULL;
  const float f[3] = {x, y, z};
  long c0[3];
  float fr[3];
#pragma unroll
  for (int d = 0; d < 3; d++) c0[d] = cic_cell(f[d], &fr[d]);
  const float fx1 = 1.0f - fr[0], fy1 = 1.0f - fr[1], fz1 = 1.0f - fr[2];  // fl(1 - f)
  const float yp = 1.0f - fy1, zp = 1.0f - fz1;                              // f' (exact differences)
  Cic q;
  q.FX[0] = sd_sub(one, sd_from_float(fr[0]));
  q.FX[1] = sd_sub(one, sd_from_float(fx1));
  q.FY0[0] = sd_sub(one, sd_from_float(fr[1]));
  q.FY0[1] = sd_sub(one, sd_from_float(yp));
  q.FY1 = sd_sub(one, sd_from_float(fy1));
  q.FZ0 = sd_sub(one, sd_from_float(fr[2]));
  q.FZ0p = sd_sub(one, sd_from_float(zp));
  q.FZ1 = sd_sub(one, sd_from_float(fz1));
#pragma unroll
  for (int d = 0; d < 2; d++) {
    q.cx[d] = wrap_cell(c0[0] + d, N);
    q.cy[d] = wrap_cell(c0[1] + d, N);
    q.cz[d] = wrap_cell(c0[2] + d, N);
  }
  return q;
}

// 8 contributions per halo, in the reference's corner order: entry 8 i + c
// holds the cell key and the double weight of corner c of halo i, so the
// entries are in the serial order of the reference's deposit loop.
constexpr int CONTRIB_THREADS = 256;
constexpr int MASS_SMEM = 1024;  // distinct masses held in shared memory

template <typename K>
__global__ void __launch_bounds__(CONTRIB_THREADS)
k_halo_contrib(long nh, const HaloRec* __restrict__ halos, RionConst rk, MassTable mt, long N,
               K* __restrict__ keys, sd_t* __restrict__ vals) {
  __shared__ K skey[8 * CONTRIB_THREADS];
  __shared__ sd_t sval[8 * CONTRIB_THREADS];
  __shared__ uint32_t suniq[MASS_SMEM];
  __shared__ float sw[MASS_SMEM];
  const int nu = mt.uniq ? *mt.n_uniq : 0;
  const bool in_smem = nu > 0 && nu <= MASS_SMEM;
  if (in_smem)
    for (int t = threadIdx.x; t < nu; t += blockDim.x) {
      suniq[t] = mt.uniq[t];
      sw[t] = mt.w[t];
    }
  const uint32_t* uq = in_smem ? suniq : mt.uniq;
  const float* wq = in_smem ? sw : mt.w;
  __syncthreads();
  // one chunk of CONTRIB_THREADS halos per block and step (uniform trip count:
  // the staging barriers are reached by every thread)
  for (long b0 = (long)blockIdx.x * CONTRIB_THREADS; b0 < nh; b0 += (long)gridDim.x * CONTRIB_THREADS) {
    const long i = b0 + threadIdx.x;
    if (i < nh) {
      const HaloRec h = halos[i];
      const float map_in = mass_weight(h.Mass, uq, wq, nu, rk);
      const sd_t mw = sd_from_float(map_in);
      const Cic q = cic_of(h.x, h.y, h.z, N);
#pragma unroll
      for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
          const sd_t xy = q.xy(a, b);
          const long kxy = (q.cx[a] * N + q.cy[b]) * N;
#pragma unroll
          for (int c = 0; c < 2; c++) {
            const int slot = 8 * threadIdx.x + 4 * a + 2 * b + c;
            skey[slot] = (K)(kxy + q.cz[c]);
            sval[slot] = sd_mul(sd_mul(xy, q.z(a, b, c)), mw);
          }
        }
    }
    __syncthreads();
    // entry 8 i + c of the chunk, written with consecutive threads on
    // consecutive entries
    const long e0 = 8 * b0, ne = 8 * nh;
    for (int t = threadIdx.x; t < 8 * CONTRIB_THREADS; t += CONTRIB_THREADS)
      if (e0 + t < ne) {
        keys[e0 + t] = skey[t];
        vals[e0 + t] = sval[t];
      }
    __syncthreads();
  }
}

// Replay each cell's chain map = (float)((double)map + w) in serial order:
// the entries were sorted by cell with a stable sort, so each cell's run
// keeps the deposit order.
template <typename K>
__global__ void k_halo_accumulate(long ne, const K* __restrict__ keys, const sd_t* __restrict__ vals,
                                  float* __restrict__ fine) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += (long)gridDim.x * blockDim.x) {
    const K key = keys[i];
    if (i > 0 && keys[i - 1] == key) continue;  // not the first entry of its cell
    float acc = 0.0f;
    long k = i;
    do {
      acc = sd_to_float(sd_add(sd_from_float(acc), vals[k]));
      ++k;
    } while (k < ne && keys[k] == key);
    fine[key] = acc;
  }
}

static unsigned grid_for(long n);

static int key_bits(long Nh3) {
  int end_bit = 1;
  while (end_bit < 64 && ((unsigned long long)1 << end_bit) < (unsigned long long)Nh3) ++end_bit;
  return end_bit;
}

// Deposit of nh halos into the zeroed fine grid: contributions, stable sort
// by cell (keys K: 32 bits when N^3 <= 2^32), replay.
template <typename K>
static cudaError_t deposit(long nh, const HaloRec* halos, RionConst rk, MassTable mt, long N, K* k0, K* k1,
                           sd_t* v0, sd_t* v1, void* tmp, size_t tmp_bytes, float* fine, cudaStream_t st) {
  const long ne = 8 * nh;
  k_halo_contrib<K><<<grid_for(nh), CONTRIB_THREADS, 0, st>>>(nh, halos, rk, mt, N, k0, v0);
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  if ((e = cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, k0, k1, v0, v1, (int)ne, 0, key_bits(N * N * N), st)))
    return e;
  k_halo_accumulate<K><<<grid_for(ne), 256, 0, st>>>(ne, k1, v1, fine);
  return cudaGetLastError();
}

// Block average (smooth_box): av = sum of the sm^3 fine values in double in
// the reference's loop order, / sm^3, rounded to float; a post divisor then
// divides that float by a double and rounds again (get_SFR.c:129-131).
//
// Fast exact path: when the block's values are non-negative and their
// significands, aligned to the smallest one, sum to less than 2^53, every
// partial sum of the serial double loop is exact, so the loop's result is the
// integer sum; av is then that integer times a power of two.  Otherwise the
// serial soft-double chain runs.  Divisions by sm^3 (when not a power of two)
// and by the post divisor use precomputed reciprocals (sd_div_c).
struct SmoothArgs {
  long N, Ns, sm;
  int sm3_log2;    // log2(sm^3) when a power of two, else -1
  sd_divc sm3;     // sm^3 as a divisor
  int post;        // 1: divide by post_div
  sd_divc post_div;
  float inv_sm3_hi, inv_sm3_lo;  // 1 / sm^3
  float inv_hi, inv_lo;  // 1 / post divisor, where it is of a moderate size (else 0: never sure)
  float zero;            // the average of a block of zeros
};

// Exact-path step: adds float bits u to the running sum S * 2^emin;
// returns false when the sum leaves the exact range (or u is negative,
// infinite or NaN).
__device__ __forceinline__ bool exact_add(uint32_t u, uint64_t& S, int& emin) {
  if (u == 0) return true;
  const uint32_t ex = u >> 23;  // sign bit included: negative values leave the fast path
  if (ex >= 0xFF) return false;
  const uint64_t m = ex ? ((u & 0x7FFFFFu) | 0x800000u) : u;
  const int e = ex ? (int)ex - 150 : -149;
  if (S == 0) {
    S = m;
    emin = e;
    return true;
  }
  if (e < emin) {  // rebase the sum on the smaller exponent
    const int d = emin - e;
    if (d > 29 || (S >> (53 - d)) != 0) return false;
    S <<= d;
    emin = e;
  }
  const int sh = e - emin;
  if (sh > 29) return false;
  S += m << sh;
  return (S >> 53) == 0;
}

__device__ __forceinline__ sd_t exact_pack(uint64_t S, int emin) {
  if (S == 0) return 0;
  const int lz = sd_clz64(S);
  const uint64_t m = S << (lz - 11);  // leading one at bit 52
  const int e = emin + (63 - lz);     // S * 2^emin = (m / 2^52) * 2^e
  return ((uint64_t)(e + 1023) << 52) | (m & 0xFFFFFFFFFFFFFULL);
}

// Sum of the n values v[0..n) (loop order) in double, serial semantics.
__device__ __forceinline__ sd_t block_sum(const float* v, int n) {
  uint64_t S = 0;
  int emin = 0;
  bool ok = true;
  for (int k = 0; k < n && ok; k++) ok = exact_add(__float_as_uint(v[k]), S, emin);
  if (ok) return exact_pack(S, emin);
  sd_t av = 0;
  for (int k = 0; k < n; k++) av = sd_add(av, sd_from_float(v[k]));
  return av;
}

// The same over a block of sm^3 cells in memory, one row of sm values at a
// time: planes and rows sx and sy values apart.
__device__ __forceinline__ sd_t rows_sum(const float* v, long sx, long sy, int sm) {
  uint64_t S = 0;
  int emin = 0;
  bool ok = true;
  for (int x = 0; x < sm && ok; x++)
    for (int y = 0; y < sm && ok; y++) {
      const float* row = v + x * sx + y * sy;
      for (int z = 0; z < sm && ok; z++) ok = exact_add(__float_as_uint(row[z]), S, emin);
    }
  if (ok) return exact_pack(S, emin);
  sd_t av = 0;
  for (int x = 0; x < sm; x++)
    for (int y = 0; y < sm; y++)
      for (int z = 0; z < sm; z++) av = sd_add(av, sd_from_float(v[x * sx + y * sy + z]));
  return av;
}

__device__ __forceinline__ sd_t smooth_sum(const float* __restrict__ fine, long base, const SmoothArgs& a) {
  const long N = a.N;
  const int sm = (int)a.sm;
  if (sm == 2) {  // the usual case (N_halo = 2 N_smoothed): all eight loads issued together
    float v[8];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float* row = fine + base + (long)(k >> 1) * N * N + (long)(k & 1) * N;
      v[2 * k] = __ldg(row);
      v[2 * k + 1] = __ldg(row + 1);
    }
    return block_sum(v, 8);
  }
  if (sm == 1) return sd_from_float(fine[base]);
  return rows_sum(fine + base, N * N, N, sm);
}

__device__ __forceinline__ float smooth_value(sd_t av, const SmoothArgs& a) {
  sd_t q;
  if (a.sm3_log2 >= 0)
    // exact: av / 2^k stays normal (a NaN from non-finite input stays NaN)
    q = (sd_is_zero(av) || ((av >> 52) & 0x7FF) == 0x7FF) ? av : av - ((uint64_t)a.sm3_log2 << 52);
  else
    q = sd_div_c(av, a.sm3);
  float v = sd_to_float(q);
  if (a.post) v = sd_to_float(sd_div_c(sd_from_float(v), a.post_div));
  return v;
}

// One CTA row per (i, j) of the smoothed box (blockIdx.x = i * Ns + j),
// threads over p.
__global__ void k_smooth_box(const float* __restrict__ fine, float* __restrict__ out, const SmoothArgs a) {
  const long N = a.N, sm = a.sm;
  const int Ns = (int)a.Ns;
  const int p = blockIdx.y * blockDim.x + threadIdx.x;
  if (p >= Ns) return;
  const int i = blockIdx.x / Ns, j = blockIdx.x % Ns;
  out[(long)blockIdx.x * Ns + p] =
      smooth_value(smooth_sum(fine, ((long)i * sm) * N * N + ((long)j * sm) * N + (long)p * sm, a), a);
}

static long block_side(long N_halo, long N_smooth) {  // smooth_box's sm
  const long sm = (long)roundf((float)((1.0 * N_halo) / N_smooth));
  return N_smooth * sm > N_halo ? sm - 1 : sm;
}

static SmoothArgs smooth_args(long N_halo, long N_smooth, double post_div) {
  SmoothArgs a;
  const long sm = block_side(N_halo, N_smooth);
  a.N = N_halo;
  a.Ns = N_smooth;
  a.sm = sm;
  const double sm3 = 1.0 * sm * sm * sm;
  int k = 0;
  while ((1L << k) < sm * sm * sm) ++k;
  a.sm3_log2 = ((1L << k) == sm * sm * sm) ? k : -1;
  uint64_t b;
  memcpy(&b, &sm3, 8);
  a.sm3 = sd_divc_prepare(b);
  a.post = post_div != 0.0;
  memcpy(&b, &post_div, 8);
  a.post_div = sd_divc_prepare(a.post ? b : 0x3FF0000000000000ULL);
  a.inv_sm3_hi = (float)(1.0 / sm3);
  a.inv_sm3_lo = (float)(1.0 / sm3 - (double)a.inv_sm3_hi);
  const bool moderate = a.post && post_div > 0x1p-50 && post_div < 0x1p50;
  a.inv_hi = moderate ? (float)(1.0 / post_div) : 0.f;
  a.inv_lo = moderate ? (float)(1.0 / post_div - (double)a.inv_hi) : 0.f;
  a.zero = (float)(a.post ? 0.0 / post_div : 0.0);
  return a;
}

static cudaError_t launch_smooth(const float* fine, float* out, long N_halo, long N_smooth, double post_div,
                                 cudaStream_t st) {
  const int T = 128;
  const dim3 grid((unsigned)(N_smooth * N_smooth), (unsigned)((N_smooth + T - 1) / T));
  k_smooth_box<<<grid, T, 0, st>>>(fine, out, smooth_args(N_halo, N_smooth, post_div));
  return cudaGetLastError();
}

static unsigned grid_for(long n) {
  long b = (n + 255) / 256;
  return (unsigned)(b < 152 * 32 ? b : 152 * 32);
}

// ---------------------------------------------------------------------------
// Deposit and block average by tiles of the fine grid, for blocks of up to 4
// cells a side.
//
// The entries above are eight per halo, sorted as (cell, double) pairs, and
// the fine grid goes to memory and back (N_halo = 1200, 2 10^7 halos: 13 GB
// through the sort, 14 GB of grid for 0.9 GB of result).  Here the halos
// themselves are sorted, by the tile of their lowest cell and by the axes
// along which their upper cells lie in the next tile (three bits), and one CTA
// takes a tile: its halos are 27 runs of the sorted list (per axis: own and
// not over the edge, own and over it, the previous tile's over the edge).  The
// tile's cells are in shared memory, so a chain never leaves the CTA, and its
// order is made there: every waiting contribution puts its serial number
// 8 i + corner into its cell's slot by atomicMin, the smallest one is added,
// and the others go again, until none waits (in a crowd: tile_crowd).  Within a
// run the halos keep their order (the sort is stable); when a tile has more of
// them than the CTA has threads, it takes those below a serial number that
// leaves no run behind.
// The block average follows from shared memory, for the blocks that have a
// contribution, in pairs of floats; no grid is stored.
//
// 1200^3 cells, 2 10^7 halos: 14.6 -> 7.4 ms, of which the two sorts take 1.0.
// It is bound by its instructions (the pairs of floats below) and by the
// barriers of the rounds: 64 to 256 threads, tiles of 1024 to 8192
// cells and 24 to 64 KB were within 10 %, a tile of 4096 cells and 96 threads
// (47 halos in it on average, 60 with those of its neighbours) the fastest.
constexpr int TILE_THREADS = 96;
constexpr int TILE_CTAS = 6;
constexpr int TILE_ROUNDS = 24;  // more of them for 96 halos: a crowd (24 and tile_crowd for 96 take about the same)
constexpr int TILE_MAX_SM = 4;  // block sides that have tiles
// Cells of a tile: whole blocks of sm cells, about 8 x 16 x 32, long in z for
// the result's rows; 32 KB of shared memory, and a halo is in 1.27 tiles on
// average
__host__ __device__ constexpr int tile_x(int sm) { return sm == 3 ? 9 : 8; }
__host__ __device__ constexpr int tile_y(int sm) { return 16 / sm * sm; }
__host__ __device__ constexpr int tile_z(int sm) { return 32 / sm * sm; }

struct HaloTiles {
  int N, tx, ty, tz;     // cells of the fine grid and of a tile: whole blocks of sm
  int nx, ny, nz;        // tiles
  long keys() const { return 8L * nx * ny * nz; }
};

static HaloTiles halo_tiles(long N_halo, long sm) {
  HaloTiles t;
  t.N = (int)N_halo;
  t.tx = tile_x((int)sm);
  t.ty = tile_y((int)sm);
  t.tz = tile_z((int)sm);
  t.nx = (t.N + t.tx - 1) / t.tx;
  t.ny = (t.N + t.ty - 1) / t.ty;
  t.nz = (t.N + t.tz - 1) / t.tz;
  return t;
}

// Sort key 8 tile + class, the halo's index, and its record with the weight in
// the mass's place.
__global__ void __launch_bounds__(CONTRIB_THREADS)
k_halo_keys(long nh, const HaloRec* __restrict__ halos, RionConst rk, MassTable mt, HaloTiles t,
            uint32_t* __restrict__ keys, uint32_t* __restrict__ idx, float4* __restrict__ rec) {
  __shared__ uint32_t suniq[MASS_SMEM];
  __shared__ float sw[MASS_SMEM];
  const int nu = *mt.n_uniq;
  const bool in_smem = nu > 0 && nu <= MASS_SMEM;
  if (in_smem)
    for (int k = threadIdx.x; k < nu; k += blockDim.x) {
      suniq[k] = mt.uniq[k];
      sw[k] = mt.w[k];
    }
  const uint32_t* uq = in_smem ? suniq : mt.uniq;
  const float* wq = in_smem ? sw : mt.w;
  __syncthreads();
  for (long i = (long)blockIdx.x * CONTRIB_THREADS + threadIdx.x; i < nh; i += (long)gridDim.x * CONTRIB_THREADS) {
    const HaloRec h = halos[i];
    const float f[3] = {h.x, h.y, h.z};
    const int side[3] = {t.tx, t.ty, t.tz}, n[3] = {t.nx, t.ny, t.nz};
    uint32_t tile = 0, over = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      float fr;
      const long c = cic_cell(f[d], &fr);
      const int t0 = (int)wrap_cell(c, t.N) / side[d], t1 = (int)wrap_cell(c + 1, t.N) / side[d];
      tile = tile * (uint32_t)n[d] + (uint32_t)t0;
      over = 2 * over + (t1 != t0 ? 1u : 0u);
    }
    keys[i] = 8 * tile + over;
    idx[i] = (uint32_t)i;
    rec[i] = make_float4(mass_weight(h.Mass, uq, wq, nu, rk), h.x, h.y, h.z);
  }
}

// start[k] = first entry of the sorted keys that is not below k, k <= nkeys
__global__ void k_halo_starts(long nh, const uint32_t* __restrict__ keys, long nkeys, uint32_t* __restrict__ start) {
  for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k <= nkeys; k += (long)gridDim.x * blockDim.x) {
    long lo = 0, hi = nh;
    while (lo < hi) {
      const long mid = (lo + hi) >> 1;
      if (keys[mid] < (unsigned long long)k)
        lo = mid + 1;
      else
        hi = mid;
    }
    start[k] = (uint32_t)lo;
  }
}

// Pairs of floats (hi + lo, |lo| at most half an ulp of hi) for the doubles of
// the deposit and the block average.  Their relative error stays under 2^-43
// in the uses below, so the float that a double chain would round to is known
// unless the pair lies within 2^-40 of the middle between two floats; then,
// and where a value is not finite, negative or so small that a low part could
// be lost, the soft-double chain runs.  (All of it in soft double: 24 000
// instructions a tile and half of the time waiting for instructions, 33 ms for
// 1200^3 cells and 2 10^7 halos.)
struct FPair {
  float hi, lo;
};
__device__ __forceinline__ FPair fp_norm(float hi, float lo) {
  const float s = __fadd_rn(hi, lo);
  return {s, __fsub_rn(lo, __fsub_rn(s, hi))};
}
__device__ __forceinline__ FPair fp_mul(FPair a, FPair b) {
  const float p = __fmul_rn(a.hi, b.hi);
  const float e = fmaf(a.lo, b.hi, fmaf(a.hi, b.lo, fmaf(a.hi, b.hi, -p)));
  return fp_norm(p, e);
}
__device__ __forceinline__ FPair fp_scale(FPair a, float b) {
  const float p = __fmul_rn(a.hi, b);
  return fp_norm(p, fmaf(a.lo, b, fmaf(a.hi, b, -p)));
}
// v + a for a float v >= 0
__device__ __forceinline__ FPair fp_add(FPair a, float v) {
  const float s = __fadd_rn(a.hi, v), t = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, t)), __fsub_rn(v, t));
  return fp_norm(s, __fadd_rn(e, a.lo));
}
__device__ __forceinline__ FPair fp_add2(FPair a, FPair b) {
  const FPair s = fp_add(a, b.hi);
  return fp_norm(s.hi, __fadd_rn(s.lo, b.lo));
}
// a.hi is the float nearest to every value within 2^-40 of a (and a is of a
// size at which no low part was lost)
__device__ __forceinline__ bool fp_sure(FPair a) {
  const float d = a.hi * 0x1p-40f;
  return a.hi > 0x1p-60f && a.hi < 0x1p100f && __fadd_rn(a.hi, a.lo + d) == a.hi && __fadd_rn(a.hi, a.lo - d) == a.hi;
}
__device__ __forceinline__ FPair fp_one_minus(float f) {  // exact for f in [0, 1)
  const float h = __fsub_rn(1.0f, f);
  return {h, __fsub_rn(__fsub_rn(1.0f, h), f)};
}

// The weight of the corner (a, b, c) of a halo of mass weight m at the
// fractions fx, fy, fz, by the factors of Cic (the upper ones are floats); true
// where the pair holds
__device__ __forceinline__ bool cic_pair(float m, float fx, float fy, float fz, int a, int b, int c, FPair* w) {
  const float fx1 = __fsub_rn(1.0f, fx);
  const float yp = __fsub_rn(1.0f, __fsub_rn(1.0f, fy)), zp = __fsub_rn(1.0f, __fsub_rn(1.0f, fz));
  const FPair X = a ? FPair{__fsub_rn(1.0f, fx1), 0.f} : fp_one_minus(fx);
  const FPair Y = b ? FPair{yp, 0.f} : fp_one_minus(a ? yp : fy);
  const FPair Z = c ? FPair{zp, 0.f} : fp_one_minus(a || b ? zp : fz);
  *w = fp_scale(fp_mul(fp_mul(X, Y), Z), m);
  return fx >= 0.f && fx < 1.f && fy >= 0.f && fy < 1.f && fz >= 0.f && fz < 1.f && m >= 0x1p-50f && m < 0x1p60f;
}

// acc + the contribution of corner k of a halo, as the reference adds it
__device__ __noinline__ float corner_exact(float acc, float4 h, int N, int k) {
  const Cic q = cic_of(h.y, h.z, h.w, N);
  const int a = k >> 2, b = k >> 1 & 1, c = k & 1;
  const sd_t w = sd_mul(sd_mul(q.xy(a, b), q.z(a, b, c)), sd_from_float(h.x));
  return sd_to_float(sd_add(sd_from_float(acc), w));
}

// A row of a block
template <int SM>
__device__ __forceinline__ void block_row(const float* p, float (&v)[SM]) {
  if constexpr (SM == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else if constexpr (SM == 2) {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x, v[1] = q.y;
  } else {
#pragma unroll
    for (int k = 0; k < SM; k++) v[k] = p[k];
  }
}

// The block average of sm^3 cells in shared memory, rows and planes sy and sx apart
__device__ __noinline__ float block_exact(const float* v, int sx, int sy, int sm, const SmoothArgs& a) {
  return smooth_value(rows_sum(v, sx, sy, sm), a);
}

// How many of each of a tile's runs go now (warp 0; lane = run, which stands at
// cur[run] and ends at end): take = their numbers, summed up to each run
__device__ __forceinline__ void tile_take(uint32_t more, uint32_t end, const uint32_t* __restrict__ idx,
                                          const uint32_t* cur, uint32_t* take) {
  const int lane = threadIdx.x & 31;
  const uint32_t b = cur[lane], n = end - b;
  uint32_t m = n;
  if (more > TILE_THREADS) {
    // a share of the threads in proportion to what is left, one at least
    // (27 runs: 69 + 27 = 96), then only what lies below the first entry
    // that some run would keep back
    const uint32_t share = n ? 1 + (uint32_t)((unsigned long long)n * (TILE_THREADS - 27) / more) : 0;
    m = min(n, share);
    const uint32_t limit = __reduce_min_sync(0xffffffffu, m < n ? idx[b + m] : 0xffffffffu);
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (idx[b + mid] < limit)
        lo = mid + 1;
      else
        hi = mid;
    }
    m = lo;
  }
  uint32_t incl = m;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  take[lane] = incl;
}
// The halo of this thread, one of the taken
__device__ __forceinline__ uint32_t tile_taken(const uint32_t* __restrict__ idx, const uint32_t* cur, const uint32_t* take) {
  int r = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1)
    if (take[r + s - 1] <= threadIdx.x) r += s;
  return idx[cur[r] + threadIdx.x - (r ? take[r - 1] : 0)];
}

// The rest of a tile that has a crowd, many halos in a cell: the contributions
// of 96 halos at a time are worked out by all threads, and eight lanes, one to
// a corner, add them halo by halo in the catalogue's order.  A round of
// k_halo_tiles adds one of a cell's contributions, and the posts to a slot are
// served in turn: 1.3 us a round.  10^6 halos, 97 532 of them in one cell of
// 480^3: 123 ms by rounds alone, 44 by the fine grid, 20 so.  A function of its
// own, so that the tiles without a crowd (all of them, as a rule) keep their
// registers.  (The cells of a halo differ: N > 1.)
__device__ __noinline__ void tile_crowd(int N, int tx, int ty, int tz, const uint32_t* __restrict__ idx,
                                        const float4* __restrict__ rec, int x0, int y0, int z0, uint32_t more,
                                        uint32_t end, uint32_t* cur, uint32_t* take, uint32_t* work, float* fine) {
  uint32_t* halo = work;                                           // [TILE_THREADS], in the catalogue's order
  int* cells = reinterpret_cast<int*>(work + TILE_THREADS);        // [8 TILE_THREADS]: 2 cell + (the pair holds), or -1
  float2* pairs = reinterpret_cast<float2*>(cells + 8 * TILE_THREADS);
  const int lane = threadIdx.x & 31;
  while (more) {
    if (threadIdx.x < 32) tile_take(more, end, idx, cur, take);
    __syncthreads();
    const uint32_t taken = take[31], i = threadIdx.x < taken ? tile_taken(idx, cur, take) : ~0u;
    cells[threadIdx.x] = (int)i;
    __syncthreads();
    int rank = 0;
    for (int k = 0; k < TILE_THREADS; k++) rank += (uint32_t)cells[k] < i;
    if (threadIdx.x < taken) halo[rank] = i;
    __syncthreads();
    for (int e = threadIdx.x; e < 8 * (int)taken; e += TILE_THREADS) {
      const float4 h = rec[halo[e >> 3]];
      const int a = e >> 2 & 1, b = e >> 1 & 1, c = e & 1;
      float fx, fy, fz;
      const int lx = (int)wrap_cell(cic_cell(h.y, &fx) + a, N) - x0;
      const int ly = (int)wrap_cell(cic_cell(h.z, &fy) + b, N) - y0;
      const int lz = (int)wrap_cell(cic_cell(h.w, &fz) + c, N) - z0;
      const bool in = (unsigned)lx < (unsigned)tx && (unsigned)ly < (unsigned)ty && (unsigned)lz < (unsigned)tz;
      FPair w;
      const bool plain = cic_pair(h.x, fx, fy, fz, a, b, c, &w);
      cells[e] = in ? 2 * ((lx * ty + ly) * tz + lz) + plain : -1;
      pairs[e] = make_float2(w.hi, w.lo);
    }
    __syncthreads();
    if (threadIdx.x < 8) {
      int c = cells[threadIdx.x];
      float2 w = pairs[threadIdx.x];
      for (int r = 0; r < (int)taken; r++) {
        const int c1 = c, e = 8 * min(r + 1, (int)taken - 1) + threadIdx.x;
        const FPair w1 = {w.x, w.y};
        c = cells[e];
        w = pairs[e];
        if (c1 >= 0) {
          const FPair v = fp_add(w1, fine[c1 >> 1]);
          if ((c1 & 1) && fp_sure(v))
            fine[c1 >> 1] = v.hi;
          else if (!(c1 & 1) || w1.hi != 0.0f)
            fine[c1 >> 1] = corner_exact(fine[c1 >> 1], rec[halo[r]], N, threadIdx.x);
        }
        __syncwarp(0xffu);
      }
    }
    if (threadIdx.x < 32) cur[lane] += take[lane] - (lane ? take[lane - 1] : 0);
    more -= taken;
    __syncthreads();
  }
}

template <int SM>
__global__ void __launch_bounds__(TILE_THREADS, TILE_CTAS)
k_halo_tiles(HaloTiles t, const uint32_t* __restrict__ start, const uint32_t* __restrict__ idx,
             const float4* __restrict__ rec, float* __restrict__ out, const __grid_constant__ SmoothArgs a) {
  extern __shared__ __align__(16) float tile_fine[];
  __shared__ uint32_t cur[32], take[32];
  __shared__ uint32_t left;  // halos that have not been taken
  __shared__ int rounds;     // of the batch
  __shared__ bool crowd;
  constexpr int TX = tile_x(SM), TY = tile_y(SM), TZ = tile_z(SM);
  constexpr int cells = (TX * TY * TZ + 3) & ~3;  // whole float4
  uint32_t* slot = reinterpret_cast<uint32_t*>(tile_fine + cells);
  const int tz = blockIdx.x % t.nz, ty = blockIdx.x / t.nz % t.ny, tx = blockIdx.x / t.nz / t.ny;
  const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
  const int Ns = (int)a.Ns;
  const int ox = x0 / SM, oy = y0 / SM, oz = z0 / SM;  // the tile's part of the result
  constexpr int MX = TX / SM, MY = TY / SM, MZ = TZ / SM;
  if (ox >= Ns || oy >= Ns || oz >= Ns) return;  // cells beyond the last block
  const int lane = threadIdx.x & 31;
  uint32_t end = 0;  // of the lane's run (warp 0)
  if (threadIdx.x < 32) {
    uint32_t b = 0;
    if (start && lane < 27) {  // per axis: 0 own, inside; 1 own, over the edge; 2 the previous tile's, over the edge
      const int dx = lane / 9, dy = lane / 3 % 3, dz = lane % 3;
      const int sx = dx < 2 ? tx : (tx ? tx : t.nx) - 1, sy = dy < 2 ? ty : (ty ? ty : t.ny) - 1,
                sz = dz < 2 ? tz : (tz ? tz : t.nz) - 1;
      const long key = 8L * (((long)sx * t.ny + sy) * t.nz + sz) + (dx ? 4 : 0) + (dy ? 2 : 0) + (dz ? 1 : 0);
      b = start[key];
      end = start[key + 1];
    }
    cur[lane] = b;
    const uint32_t n = __reduce_add_sync(0xffffffffu, end - b);
    if (lane == 0) left = n, rounds = 0;
  }
  __syncthreads();
  uint32_t more = left;
  const bool any = more != 0;
  if (any)
    for (int k = 4 * threadIdx.x; k < cells; k += 4 * TILE_THREADS) {
      *reinterpret_cast<float4*>(tile_fine + k) = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<uint4*>(slot + k) = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
  while (more) {
    if (threadIdx.x < 32) tile_take(more, end, idx, cur, take);
    __syncthreads();
    const uint32_t taken = take[31];
    uint32_t wait = 0;  // bit k = 4 a + 2 b + c: that corner's contribution waits
    uint32_t order = 0;
    int base = 0;      // corner k's cell is base + dx (k >> 2) + dy (k >> 1 & 1) + dz (k & 1)
    int dx = 0, dy = 0, dz = 0;
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
    FPair w[8];
    bool plain = false;  // the pairs hold
    if (threadIdx.x < taken) {
      const uint32_t i = tile_taken(idx, cur, take);
      h = rec[i];
      order = 8 * i;
      float fx, fy, fz;
      const long cx = cic_cell(h.y, &fx), cy = cic_cell(h.z, &fy), cz = cic_cell(h.w, &fz);
      const int lx0 = (int)wrap_cell(cx, t.N) - x0, lx1 = (int)wrap_cell(cx + 1, t.N) - x0;
      const int ly0 = (int)wrap_cell(cy, t.N) - y0, ly1 = (int)wrap_cell(cy + 1, t.N) - y0;
      const int lz0 = (int)wrap_cell(cz, t.N) - z0, lz1 = (int)wrap_cell(cz + 1, t.N) - z0;
      const uint32_t in = ((unsigned)lx0 < (unsigned)TX ? 0x0fu : 0u) | ((unsigned)lx1 < (unsigned)TX ? 0xf0u : 0u);
      const uint32_t iny = ((unsigned)ly0 < (unsigned)TY ? 0x33u : 0u) | ((unsigned)ly1 < (unsigned)TY ? 0xccu : 0u);
      const uint32_t inz = ((unsigned)lz0 < (unsigned)TZ ? 0x55u : 0u) | ((unsigned)lz1 < (unsigned)TZ ? 0xaau : 0u);
      wait = in & iny & inz;
      base = (lx0 * TY + ly0) * TZ + lz0;
      dx = (lx1 - lx0) * TY * TZ;
      dy = (ly1 - ly0) * TZ;
      dz = lz1 - lz0;
      // the factors of Cic, as pairs (the upper ones are floats)
      plain = fx >= 0.f && fx < 1.f && fy >= 0.f && fy < 1.f && fz >= 0.f && fz < 1.f && h.x >= 0x1p-50f &&
              h.x < 0x1p60f;
      const float fx1 = __fsub_rn(1.0f, fx), fy1 = __fsub_rn(1.0f, fy), fz1 = __fsub_rn(1.0f, fz);
      const float yp = __fsub_rn(1.0f, fy1), zp = __fsub_rn(1.0f, fz1);
      const FPair X[2] = {fp_one_minus(fx), {__fsub_rn(1.0f, fx1), 0.f}};
      const FPair Y0[2] = {fp_one_minus(fy), fp_one_minus(yp)};
      const FPair Y1 = {yp, 0.f}, Z0 = fp_one_minus(fz), Z0p = fp_one_minus(zp), Z1 = {zp, 0.f};
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int ca = k >> 2, cb = k >> 1 & 1, cc = k & 1;
        const FPair xy = fp_mul(X[ca], cb ? Y1 : Y0[ca]);
        w[k] = fp_scale(fp_mul(xy, cc ? Z1 : k == 0 ? Z0 : Z0p), h.x);
      }
    }
    do {
      if (threadIdx.x == 0) rounds++;
      if (wait) {
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (wait >> k & 1u) atomicMin(slot + base + (k >> 2) * dx + (k >> 1 & 1) * dy + (k & 1) * dz, order + k);
      }
      __syncthreads();
      if (wait) {
        uint32_t exact = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int cell = base + (k >> 2) * dx + (k >> 1 & 1) * dy + (k & 1) * dz;
          if ((wait >> k & 1u) && slot[cell] == order + k) {
            const FPair v = fp_add(w[k], tile_fine[cell]);
            if (plain && fp_sure(v)) {
              tile_fine[cell] = v.hi;
            } else if (!plain || w[k].hi != 0.0f) {  // a factor of zero (a halo on a cell's face): the cell stays
              exact |= 1u << k;
            }
            slot[cell] = 0xffffffffu;
            wait &= ~(1u << k);
          }
        }
        for (; exact; exact &= exact - 1) {
          const int k = __ffs(exact) - 1;
          const int cell = base + (k >> 2) * dx + (k >> 1 & 1) * dy + (k & 1) * dz;
          tile_fine[cell] = corner_exact(tile_fine[cell], h, t.N, k);
        }
      }
    } while (__syncthreads_or(wait != 0));
    if (threadIdx.x < 32) {
      cur[lane] += take[lane] - (lane ? take[lane - 1] : 0);
      if (lane == 0) {
        left = more - taken;
        crowd = rounds > TILE_ROUNDS;
        rounds = 0;
      }
    }
    __syncthreads();
    more = left;
    if (crowd && more && t.N > 1) {
      tile_crowd(t.N, TX, TY, TZ, idx, rec, x0, y0, z0, more, end, cur, take, slot, tile_fine);
      break;
    }
  }
  // Blocks without a contribution first (most of them, at a halo per hundred
  // cells); the others into a list, so that whole warps work on them
  uint16_t* list = reinterpret_cast<uint16_t*>(slot);  // the slots have been used
  __shared__ uint32_t listed;
  if (threadIdx.x == 0) listed = 0;
  __syncthreads();
  const auto where = [&](int o, int* b) {  // block o's cells, and its place in the result (-1: outside)
    const int p = o % MZ, j = o / MZ % MY, i = o / MZ / MY;
    *b = ((i * SM) * TY + j * SM) * TZ + p * SM;
    return ox + i < Ns && oy + j < Ns && oz + p < Ns ? ((long)(ox + i) * Ns + oy + j) * Ns + oz + p : -1L;
  };
  for (int o0 = threadIdx.x - lane; o0 < MX * MY * MZ; o0 += TILE_THREADS) {
    const int o = o0 + lane;
    int b;
    long dst = o < MX * MY * MZ ? where(o, &b) : -1;
    bool zero = true;
    if (dst >= 0 && any) {
      uint32_t bits = 0;  // (comparisons chained by && wait for one load after the other)
#pragma unroll
      for (int r = 0; r < SM * SM; r++) {
        float v[SM];
        block_row<SM>(tile_fine + b + (r / SM) * TY * TZ + (r % SM) * TZ, v);
#pragma unroll
        for (int k = 0; k < SM; k++) bits |= __float_as_uint(v[k]);
      }
      zero = bits << 1 == 0;
    }
    if (dst >= 0 && zero) out[dst] = a.zero;
    const uint32_t m = __ballot_sync(0xffffffffu, !zero);
    uint32_t at = 0;
    if (lane == 0 && m) at = atomicAdd(&listed, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (!zero) list[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)o;
  }
  __syncthreads();
  // Side 4: a block's planes to four lanes, since a tile has few blocks then
  // and the chain of 64 cells would be longer than all the rest
  constexpr int LANES = SM == 4 ? 4 : 1, PLANES = SM / LANES;
  for (int k0 = threadIdx.x - lane; k0 < (int)listed * LANES; k0 += TILE_THREADS) {
    const int k = (k0 + lane) / LANES;
    int b = 0;
    const long dst = k < (int)listed ? where(list[k], &b) : -1;
    const float* c = tile_fine + b;
    float v = 0.f;
    bool sure = false;
    FPair part[PLANES];  // each plane's sum: the chains run side by side
#pragma unroll
    for (int y = 0; y < SM; y++) {
      float u[PLANES][SM];
#pragma unroll
      for (int x = 0; x < PLANES; x++) block_row<SM>(c + (lane % LANES + x) * TY * TZ + y * TZ, u[x]);
#pragma unroll
      for (int z = 0; z < SM; z++)
#pragma unroll
        for (int x = 0; x < PLANES; x++) part[x] = y + z ? fp_add(part[x], u[x][z]) : FPair{u[x][0], 0.f};
    }
    FPair q = part[0];
#pragma unroll
    for (int x = 1; x < PLANES; x++) q = fp_add2(q, part[x]);
#pragma unroll
    for (int o = 1; o < LANES; o <<= 1)
      q = fp_add2(q, {__shfl_xor_sync(0xffffffffu, q.hi, o), __shfl_xor_sync(0xffffffffu, q.lo, o)});
    if (dst < 0 || lane % LANES) continue;
    // the average of 1, 8 or 64 cells is a power of two away from the sum; the
    // quotient by the post divisor is that of the rounded average
    if constexpr (SM == 3) q = fp_mul(q, {a.inv_sm3_hi, a.inv_sm3_lo});
    if (fp_sure(q)) {
      v = SM == 3 ? q.hi : q.hi * (1.0f / (SM * SM * SM));
      sure = true;
      if (a.post) {
        const FPair d = fp_scale({a.inv_hi, a.inv_lo}, v);
        sure = fp_sure(d);
        v = d.hi;
      }
    }
    if (!sure) v = block_exact(c, TY * TZ, TZ, SM, a);
    out[dst] = v;
  }
}

// Which deposit takes a catalogue (fine: the fine grid in memory, tiles: the
// kernel above; ms a call).
//
// Block sides up to 4 have tiles.  0.0001, 0.001 and 0.01 halos per cell:
//   480 -> 160   fine 0.39, 0.48, 1.05   tiles 0.25, 0.36, 0.53
//   480 -> 120   fine 0.36, 0.44, 1.02   tiles 0.24, 0.40, 0.67
//   1200 -> 300  fine 2.69, 3.84, 12.3   tiles 1.59, 3.87, 8.32
// From 5 up a tile has too few blocks for its threads (with the blocks' cells in
// a loop: 480 -> 96, fine 0.36, 0.44, 1.04, tiles 0.40, 0.90, 1.51; 480 -> 30,
// fine 1.27, 1.49, 2.83, tiles 4.2, 7.6, 18.9).
//
// Where the tiles are fewer than two an SM (up to about 100^3 cells), they wait
// for the rounds of their halos, and many halos a tile go faster through the
// sort of the contributions, the sooner the fewer the tiles are (us a call among
// others, by halos a tile):
//   48^3, side 1, 36 tiles    140: fine 65, tiles 65;  250: 66, 75
//   64^3, side 1, 64 tiles    140: 67, 64;  200: 68, 70;  300: 70, 77
//   96^3, side 1, 216 tiles   140: 78, 69;  250: 85, 81
//   64^3, side 2, 64 tiles    150: 66, 62;  250: 69, 70
//   72^3, side 3, 120 tiles   250: 77, 73
//   96^3, side 4, 216 tiles   350: 98, 82
// so the line lies at 95 halos a tile and one more for every tile, half as much
// again for sides above 1 (less to average and store).  Up to 2000 halos the
// tiles are ahead in any case: eight contributions a halo are long enough for
// the larger form of the sort then, the halos are not (32^3, 8 tiles, 200 a
// tile: 40, 35).
// Grids beyond 2048 keep the fine grid.
static bool has_tiles(long N_halo, long N_smooth) {
  const long sm = block_side(N_halo, N_smooth);
  return sm >= 1 && sm <= TILE_MAX_SM && N_halo <= 2048;
}
constexpr long FEW_TILES = 300;
static bool few_tiles(long N_halo, long N_smooth) {
  return halo_tiles(N_halo, block_side(N_halo, N_smooth)).keys() / 8 < FEW_TILES;
}
static bool by_tiles(long nh, long N_halo, long N_smooth) {
  if (!has_tiles(N_halo, N_smooth)) return false;
  const long sm = block_side(N_halo, N_smooth), tiles = halo_tiles(N_halo, sm).keys() / 8;
  return tiles >= FEW_TILES || nh < 2000 || 2 * nh < (sm > 1 ? 3 : 2) * (95 + tiles) * tiles;
}
bool halo_needs_grid(long N_halo, long N_smooth) {
  return !has_tiles(N_halo, N_smooth) || few_tiles(N_halo, N_smooth);
}

size_t halo_scratch_bytes(long nh, long N_halo, long N_smooth) {
  size_t key_tmp = 0, uniq_tmp = 0;
  cub::DeviceRadixSort::SortKeys(nullptr, key_tmp, (uint32_t*)nullptr, (uint32_t*)nullptr, (int)nh);
  cub::DeviceSelect::Unique(nullptr, uniq_tmp, (uint32_t*)nullptr, (uint32_t*)nullptr, (int*)nullptr, (int)nh);
  size_t tmp = std::max(key_tmp, uniq_tmp);
  size_t bytes = 0;
  if (has_tiles(N_halo, N_smooth)) {
    size_t pairs = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, pairs, (uint32_t*)nullptr, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (uint32_t*)nullptr, (int)nh);
    // records | keys and indices, twice | masses and weights | starts | CUB temporary storage
    bytes = (size_t)nh * 40 + 4 * (size_t)(halo_tiles(N_halo, block_side(N_halo, N_smooth)).keys() + 1) +
            std::max(tmp, pairs) + 4096;
    if (!few_tiles(N_halo, N_smooth)) return bytes;
  }
  const long ne = 8 * nh;
  size_t t64 = 0, t32 = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, t64, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                  (sd_t*)nullptr, (sd_t*)nullptr, (int)ne);
  cub::DeviceRadixSort::SortPairs(nullptr, t32, (uint32_t*)nullptr, (uint32_t*)nullptr, (sd_t*)nullptr,
                                  (sd_t*)nullptr, (int)ne);
  tmp = std::max(tmp, std::max(t64, t32));
  // k0 | k1 (8 B each) | v0 | v1 (8 B each) | CUB temporary storage
  return std::max(bytes, (size_t)ne * 32 + tmp + 4096);
}

static uint64_t bits_of(double d) {
  uint64_t u;
  memcpy(&u, &d, 8);
  return u;
}

static RionConst rion_const(double z, double qion) {
  RionConst rk;
  rk.c1 = bits_of(1.575e39);
  rk.c2 = bits_of(9.367608e+07);
  rk.c3 = bits_of(0.44);
  rk.three = bits_of(3.0);
  rk.vnorm = bits_of(1.e+45);
  rk.p1 = bits_of(pow((1.0 + z), 2.27044695e+00));
  rk.qion = qion != 0.0 ? bits_of(qion) : 0;
  return rk;
}

// Sorted distinct masses and their weights; 4 nh bytes each at mk0, mk1, uniq
// and w, an int at n_uniq.
static cudaError_t mass_table(long nh, const HaloRec* halos, const RionConst& rk, uint32_t* mk0, uint32_t* mk1,
                              uint32_t* uniq, float* w, int* n_uniq, void* tmp, size_t tmp_bytes, MassTable* mt,
                              cudaStream_t st) {
  k_mass_keys<<<grid_for(nh), 256, 0, st>>>(nh, halos, mk0);
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  size_t tb = tmp_bytes;
  if ((e = cub::DeviceRadixSort::SortKeys(tmp, tb, mk0, mk1, (int)nh, 0, 32, st))) return e;
  tb = tmp_bytes;
  if ((e = cub::DeviceSelect::Unique(tmp, tb, mk1, uniq, n_uniq, (int)nh, st))) return e;
  k_mass_weights<<<grid_for(nh), 256, 0, st>>>(nh, uniq, n_uniq, rk, w);
  *mt = {uniq, n_uniq, w};
  return cudaGetLastError();
}

template <int SM>
static cudaError_t tiles_launch(const HaloTiles& t, const uint32_t* start, const uint32_t* idx, const float4* rec,
                                float* out, const SmoothArgs& a, cudaStream_t st) {
  const size_t smem = 8 * (((size_t)t.tx * t.ty * t.tz + 3) & ~(size_t)3);
  cudaError_t e = cudaFuncSetAttribute(k_halo_tiles<SM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e) return e;
  k_halo_tiles<SM><<<(unsigned)((long)t.nx * t.ny * t.nz), TILE_THREADS, smem, st>>>(t, start, idx, rec, out, a);
  return cudaGetLastError();
}

static cudaError_t source_by_tiles(long nh, const HaloRec* halos, const RionConst& rk, long N_halo, long N_smooth,
                                   float* out, void* scratch, size_t scratch_bytes, double post_div,
                                   cudaStream_t st) {
  const SmoothArgs a = smooth_args(N_halo, N_smooth, post_div);
  const HaloTiles t = halo_tiles(N_halo, a.sm);
  float4* rec = (float4*)scratch;
  uint32_t* k0 = (uint32_t*)(rec + nh);
  uint32_t *k1 = k0 + nh, *i0 = k1 + nh, *i1 = i0 + nh, *uniq = i1 + nh;
  float* wts = (float*)(uniq + nh);
  uint32_t* start = (uint32_t*)(wts + nh);
  int* n_uniq = (int*)(start + t.keys() + 1);
  unsigned char* p = (unsigned char*)(((uintptr_t)(n_uniq + 1) + 255) & ~(uintptr_t)255);
  const size_t tmp_bytes = scratch_bytes - (size_t)(p - (unsigned char*)scratch);
  cudaError_t e = cudaSuccess;
  if (nh > 0) {
    MassTable mt;
    if ((e = mass_table(nh, halos, rk, k1, i1, uniq, wts, n_uniq, p, tmp_bytes, &mt, st))) return e;
    k_halo_keys<<<grid_for(nh), CONTRIB_THREADS, 0, st>>>(nh, halos, rk, mt, t, k0, i0, rec);
    if ((e = cudaGetLastError())) return e;
    size_t tb = tmp_bytes;
    if ((e = cub::DeviceRadixSort::SortPairs(p, tb, k0, k1, i0, i1, (int)nh, 0, key_bits(t.keys()), st))) return e;
    k_halo_starts<<<grid_for(t.keys() + 1), 256, 0, st>>>(nh, k1, t.keys(), start);
    if ((e = cudaGetLastError())) return e;
  } else {
    start = nullptr;  // no runs (and no scratch, maybe)
  }
  if (a.sm == 1) return tiles_launch<1>(t, start, i1, rec, out, a, st);
  if (a.sm == 2) return tiles_launch<2>(t, start, i1, rec, out, a, st);
  if (a.sm == 3) return tiles_launch<3>(t, start, i1, rec, out, a, st);
  return tiles_launch<4>(t, start, i1, rec, out, a, st);
}

// fine: N_halo^3 floats, used only if halo_needs_grid
cudaError_t launch_halo_source(long nh, const void* halos_dev, double z, long N_halo, long N_smooth, float* fine,
                               float* out, void* scratch, size_t scratch_bytes, cudaStream_t st, double qion,
                               double post_div) {
  const RionConst rk = rion_const(z, qion);
  const HaloRec* hrec = (const HaloRec*)halos_dev;
  if (by_tiles(nh, N_halo, N_smooth))
    return source_by_tiles(nh, hrec, rk, N_halo, N_smooth, out, scratch, scratch_bytes, post_div, st);
  const long ne = 8 * nh;
  const long Nh3 = N_halo * N_halo * N_halo;
  cudaError_t e;
  if ((e = cudaMemsetAsync(fine, 0, sizeof(float) * Nh3, st))) return e;
  if (nh > 0) {
    unsigned char* p = (unsigned char*)scratch;
    void* k0 = p;
    p += ne * 8;
    void* k1 = p;
    p += ne * 8;
    sd_t* v0 = (sd_t*)p;
    p += ne * sizeof(sd_t);
    sd_t* v1 = (sd_t*)p;
    p += ne * sizeof(sd_t);
    p = (unsigned char*)(((uintptr_t)p + 255) & ~(uintptr_t)255);
    const size_t tmp_bytes = scratch_bytes - (size_t)(p - (unsigned char*)scratch);
    // distinct-mass table (16 nh bytes) and its count in v1, free until the
    // cell sort writes it (64 nh bytes); CUB's temporary storage is the cell
    // sort's
    uint32_t* mk0 = (uint32_t*)v1;
    uint32_t* uniq = mk0 + 2 * nh;
    float* wts = (float*)(uniq + nh);
    MassTable mt;
    if ((e = mass_table(nh, hrec, rk, mk0, mk0 + nh, uniq, wts, (int*)(wts + nh), p, tmp_bytes, &mt, st))) return e;
    if (key_bits(Nh3) <= 32)
      e = deposit<uint32_t>(nh, hrec, rk, mt, N_halo, (uint32_t*)k0, (uint32_t*)k1, v0, v1, p, tmp_bytes, fine, st);
    else
      e = deposit<unsigned long long>(nh, hrec, rk, mt, N_halo, (unsigned long long*)k0, (unsigned long long*)k1, v0,
                                      v1, p, tmp_bytes, fine, st);
    if (e) return e;
  }
  return launch_smooth(fine, out, N_halo, N_smooth, post_div, st);
}

// ---------------------------------------------------------------------------
// Allocation-free variant (sf21_hii_halo_source_noalloc).  Some callers cannot
// call cudaMalloc at the point where they need the source box: a host
// application that owns a fixed device-memory budget and forbids allocations
// after start-up, a caller running between CUDA graph launches that must not
// change the device heap, or one that calls from inside a memory pool's
// callbacks.  For them the fine grid, the sort keys/values and CUB's temporary
// storage live in this fixed file-scope array instead of cudaMalloc'd scratch,
// which caps the sizes (kNoAllocMaxNHalo, kNoAllocMaxHalos).  One array per
// device: calls that overlap on the same device (two streams, two threads)
// share it and race; the caller serialises them.
//
// The array's device address belongs to the CUDA context the module is loaded
// in.  It is looked up with cudaGetSymbolAddress once per context (the first
// call in a context does it, so that call should come before any stream
// capture) and cached under the context's process-unique id (cuCtxGetId):
// after cudaDeviceReset, or under another context, the next call looks it up
// again instead of reusing a stale address.
constexpr size_t kNoAllocScratchBytes = (size_t)16 << 20;  // 16 MiB
constexpr long kNoAllocMaxNHalo = 128;                     // fine grid <= 8 MiB
constexpr long kNoAllocMaxHalos = 16384;                   // 131072 CIC entries, 4 MiB
constexpr int kNoAllocCacheSlots = 64;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

static std::mutex g_noalloc_mu;
static struct {
  unsigned long long ctx_id;
  void* ptr;
} g_noalloc_cache[kNoAllocCacheSlots];
static int g_noalloc_next = 0;

// Process-unique id of the current context (driver entry points, so the
// library needs no link against libcuda).
static cudaError_t current_context_id(unsigned long long* id) {
  typedef int (*CtxGetCurrent)(void**);
  typedef int (*CtxGetId)(void*, unsigned long long*);
  static CtxGetCurrent get_current = nullptr;
  static CtxGetId get_id = nullptr;
  if (!get_current || !get_id) {
    void* f = nullptr;
    void* g = nullptr;
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q1) != cudaSuccess ||
        q1 != cudaDriverEntryPointSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetId", &g, 12000, cudaEnableDefault, &q2) != cudaSuccess ||
        q2 != cudaDriverEntryPointSuccess)
      return cudaErrorNotSupported;
    get_current = (CtxGetCurrent)f;
    get_id = (CtxGetId)g;
  }
  void* ctx = nullptr;
  if (get_current(&ctx) != 0 || !ctx) return cudaErrorDeviceUninitialized;
  return get_id(ctx, id) == 0 ? cudaSuccess : cudaErrorDeviceUninitialized;
}

// Set-up, once per context with its device current: the device address of
// the array.  Nothing is allocated (the array belongs to the loaded module).
static cudaError_t noalloc_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaSetDevice(dev);  // makes the device's primary context current
  unsigned long long id = 0;
  if (e == cudaSuccess) e = current_context_id(&id);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  for (int i = 0; i < kNoAllocCacheSlots; ++i)
    if (g_noalloc_cache[i].ptr && g_noalloc_cache[i].ctx_id == id) {
      *out = g_noalloc_cache[i].ptr;
      return cudaSuccess;
    }
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  g_noalloc_cache[g_noalloc_next] = {id, p};
  g_noalloc_next = (g_noalloc_next + 1) % kNoAllocCacheSlots;
  *out = p;
  return cudaSuccess;
}

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

int halo_source_noalloc(double z, long N_halo, long N_smooth, long nh, const void* halos_dev, float* out,
                        cudaStream_t st, char* err, size_t errlen) {
  if (nh < 0 || (nh > 0 && !halos_dev) || !out || N_smooth < 1 || N_halo < 1) {
    snprintf(err, errlen, "bad arguments");
    return SF21_E_ARG;
  }
  if (N_halo < N_smooth) {
    snprintf(err, errlen, "N_halo < N_smoothed (smooth_box, auxiliary.c:651-654)");
    return SF21_E_ARG;
  }
  if (N_halo > kNoAllocMaxNHalo || nh > kNoAllocMaxHalos) {
    snprintf(err, errlen, "no-alloc halo source limited to N_halo <= %ld and <= %ld halos (got N_halo %ld, %ld halos)",
             kNoAllocMaxNHalo, kNoAllocMaxHalos, N_halo, nh);
    return SF21_E_UNSUPPORTED;
  }
  const long ne = 8 * nh;
  const long Nh3 = N_halo * N_halo * N_halo;
  size_t sort_tmp = 0;
  if (ne > 0) {
    const cudaError_t q = cub::DeviceRadixSort::SortPairs(nullptr, sort_tmp, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                                          (sd_t*)nullptr, (sd_t*)nullptr, (int)ne);
    if (q != cudaSuccess) {
      snprintf(err, errlen, "no-alloc halo source: sort size query failed: %s", cudaGetErrorString(q));
      return SF21_E_CUDA;
    }
  }
  // layout: fine | k0 | k1 | v0 | v1 | CUB temp, each 256-byte aligned (N_halo <= 128: 32-bit keys)
  const size_t o_k0 = align256(sizeof(float) * Nh3);
  const size_t o_k1 = o_k0 + align256(ne * sizeof(uint32_t));
  const size_t o_v0 = o_k1 + align256(ne * sizeof(uint32_t));
  const size_t o_v1 = o_v0 + align256(ne * sizeof(sd_t));
  const size_t o_t = o_v1 + align256(ne * sizeof(sd_t));
  if (o_t + sort_tmp > kNoAllocScratchBytes) {
    snprintf(err, errlen, "no-alloc halo source needs %zu scratch bytes, has %zu", o_t + sort_tmp,
             kNoAllocScratchBytes);
    return SF21_E_UNSUPPORTED;
  }
  void* base = nullptr;
  cudaError_t e = noalloc_scratch(&base);
  if (e != cudaSuccess) {
    snprintf(err, errlen, "scratch set-up failed: %s", cudaGetErrorString(e));
    return SF21_E_CUDA;
  }
  unsigned char* p = (unsigned char*)base;
  float* fine = (float*)p;
  const RionConst rk = rion_const(z, 0.0);
  // The fine grid is the only part that must start at zero (the CIC chains
  // write each touched cell once, untouched cells stay 0); keys and values
  // are written in full before they are read, and CUB initialises its own
  // temporary storage.
  if ((e = cudaMemsetAsync(fine, 0, sizeof(float) * Nh3, st)) == cudaSuccess && nh > 0) {
    const MassTable direct = {nullptr, nullptr, nullptr};
    e = deposit<uint32_t>(nh, (const HaloRec*)halos_dev, rk, direct, N_halo, (uint32_t*)(p + o_k0),
                          (uint32_t*)(p + o_k1), (sd_t*)(p + o_v0), (sd_t*)(p + o_v1), p + o_t, sort_tmp, fine, st);
  }
  if (e == cudaSuccess) {
    e = launch_smooth(fine, out, N_halo, N_smooth, 0.0, st);
  }
  if (e != cudaSuccess) {
    snprintf(err, errlen, "no-alloc halo source: %s", cudaGetErrorString(e));
    return SF21_E_CUDA;
  }
  return SF21_OK;
}

}  // namespace sf21

// Context-free, allocation-free halo source box (declared in sf21_hii.h).
extern "C" int sf21_hii_halo_source_noalloc(double z, long N_halo, long N_smoothed, long nhalos,
                                            const void* halos_dev, float* rion_box_dev, void* stream) {
  char err[256] = {0};
  const int rc = sf21::halo_source_noalloc(z, N_halo, N_smoothed, nhalos, halos_dev, rion_box_dev,
                                           (cudaStream_t)stream, err, sizeof err);
  if (rc != SF21_OK) sf21::set_global_error(err);
  return rc;
}
