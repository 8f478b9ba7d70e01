// Element-wise kernels of the HII stage: the prologue
// (get_HIIbubbles.c:216-225, 272-274), the norm balance of the packed
// transform and the single-cell fill check hook (:281-288).  All per-voxel
// double arithmetic of the reference is reproduced bit for bit with the
// integer soft-double routines.  The dilation and the per-set finish are in
// kernels_dt.cu.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "neutral_sum.h"
#include "sf21_kernels.h"
#include "softdouble.h"

namespace sf21 {

#define SD_ONE (0x3FF0000000000000ULL)

// Source chain before zeta, left to right as the reference multiplies.
__device__ __forceinline__ sd_t src_chain(float s, const PrologueArgs& pa) {
  sd_t t = sd_from_float(s);
  for (int m = 0; m < pa.n_src_mul; ++m) t = sd_mul(t, pa.src_mul[m]);
  return t;
}

constexpr int PRO_THREADS = 256;

// alpha = 2^round(log2(|rec| / |ion|)), so that the two halves of the packed
// transform have comparable norms.  An ionisation box that is zero in every
// cell gets alpha = -1: the reference's filtered ionisation field is then
// exactly zero and no cell is a centre (its test wants ion_R > 0,
// get_HIIbubbles.c:339-348), while the packed transform's imaginary half
// holds rounding cross-talk from the recombination half; is_centre reads
// alpha <= 0 as "no centre", and the other users take |alpha|.
// By the prologue's last block to finish (a launch of its own took as long as
// a small box's whole pass), over all blocks' partial sums in their order.
__device__ __forceinline__ void alpha_of(const float* partials, int nblocks, float* __restrict__ alpha) {
  __shared__ float sa[PRO_THREADS], sb[PRO_THREADS];
  float a = 0.f, b = 0.f;
  for (int i = threadIdx.x; i < nblocks; i += PRO_THREADS) {
    a += __ldcg(partials + 2 * i);
    b += __ldcg(partials + 2 * i + 1);
  }
  sa[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int s = PRO_THREADS / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sa[threadIdx.x] += sa[threadIdx.x + s];
      sb[threadIdx.x] += sb[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    float r = 1.0f;
    if (sb[0] == 0.f) {
      r = -1.0f;
    } else if (sa[0] > 0.f && sb[0] > 0.f && isfinite(sa[0]) && isfinite(sb[0])) {
      float e = rintf(0.5f * log2f(sa[0] / sb[0]));
      e = fminf(fmaxf(e, -60.f), 60.f);
      r = exp2f(e);
    }
    *alpha = r;
  }
}

__global__ void __launch_bounds__(PRO_THREADS)
k_prologue(long n3, const float* __restrict__ delta, const float* __restrict__ src,
           const PrologueArgs pa, float* __restrict__ rec0, float* __restrict__ fres,
           float2* __restrict__ packed, float* partials, uint8_t* __restrict__ rc, unsigned int* __restrict__ done,
           float* __restrict__ alpha) {
  // rrec_quick's tables: lanes index them by their own densities
  __shared__ uint64_t tab[384];
  for (int t = threadIdx.x; t < 384; t += blockDim.x) tab[t] = rrec_table(t);
  __syncthreads();
  float sd2 = 0.f, sh2 = 0.f;
  int nz = 0;  // some ionisation rate is not exactly zero
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += (long)gridDim.x * blockDim.x) {
    const float d = delta[i];
    const sd_t one_d = sd_add(SD_ONE, sd_from_float(d));  // 1. + density_map[i]
    // Each quantity takes its fast path (prologue_fast.h), which returns the
    // exact chain's float for all but about one voxel in 2^18 (Rrec: the
    // quick path for all but one in 2^14, then the fast one); those voxels
    // evaluate the exact chain.
    // fresid = XHI((float)((1+d) * 1.881e-7 * pow(1+z,3) * G_H(z)))      (:220-221)
    float fr;
    if (!prod_fast(one_d, pa.pf_resid, &fr))
      fr = sd_to_float(sd_mul(sd_mul(sd_mul(one_d, pa.c_resid), pa.one_plus_z_cubed), pa.g_h));
    const float fx = xhi_float(fr);
    // density_map = (float)Rrec((float)(1 + d), z)                          (:222)
    const float od = 1.0f + d;  // one_d rounded to float: rounding it twice is innocuous (53 >= 2 24 + 1)
    float rr;
    if (!rrec_quick(od, pa.rf, tab, &rr) && !rrec_fast(od, pa.rf, &rr))
      rr = sd_to_float(rrec_exact(od, pa.r2c, pa.r3, pa.rec1, pa.dvv, pa.v_normc));
    // source before zeta                                                   (:272-274)
    const float s = src[i];
    float h1;
    if (!prod_fast(sd_from_float(s), pa.pf_src, &h1)) h1 = sd_to_float(src_chain(s, pa));
    rec0[i] = rr;
    fres[i] = fx;
    packed[i] = make_float2(rr, h1);
    rc[i] = RC_NONE;
    sd2 += rr * rr;
    sh2 += h1 * h1;
    nz |= (h1 != 0.0f);
  }
  nz = __syncthreads_or(nz);
  // block reduction of the two sums of squares (only their ratio is used)
  __shared__ float red[2][PRO_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) {
    sd2 += __shfl_xor_sync(0xffffffffu, sd2, o);
    sh2 += __shfl_xor_sync(0xffffffffu, sh2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = sd2;
    red[1][threadIdx.x >> 5] = sh2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float a = 0.f, b = 0.f;
    for (int w = 0; w < PRO_THREADS / 32; ++w) {
      a += red[0][w];
      b += red[1][w];
    }
    // a block with a nonzero rate reports a nonzero sum even when every
    // square underflows, so that an all-zero box is told apart exactly
    if (nz && b == 0.f) b = __int_as_float(1);
    partials[2 * blockIdx.x] = a;
    partials[2 * blockIdx.x + 1] = b;
  }
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(done, 1u) + 1 == gridDim.x;
    if (last) *done = 0;  // for the next launch on the stream
    __threadfence();
  }
  __syncthreads();
  if (last) alpha_of(partials, gridDim.x, alpha);
}

int prologue_blocks(long n3) {
  long b = (n3 + PRO_THREADS - 1) / PRO_THREADS;
  return (int)(b < 152 * 16 ? b : 152 * 16);
}

cudaError_t launch_prologue(long n3, const float* delta, const float* src, const PrologueArgs& pa,
                            float* rec0, float* fres, float2* packed, float* partials, int nblocks, uint8_t* rc,
                            unsigned int* done, float* alpha, cudaStream_t st) {
  k_prologue<<<nblocks, PRO_THREADS, 0, st>>>(n3, delta, src, pa, rec0, fres, packed, partials, rc, done, alpha);
  return cudaGetLastError();
}

// Single-cell fill alone (check hook): :281-288 without dilation and cap.
__global__ void k_fill0(long n3, sd_t zeta, const float* __restrict__ src, const float* __restrict__ rec0,
                        const PrologueArgs pa, float* __restrict__ fill) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += (long)gridDim.x * blockDim.x) {
    const float h = sd_to_float(sd_mul(src_chain(src[i], pa), zeta));
    const float d = rec0[i];
    float f;
    if (h > 0.0f)
      f = (d > 0.0f) ? ((h >= d) ? 1.0f : __fdiv_rn(h, d)) : 1.0f;
    else
      f = 0.0f;
    fill[i] = f;
  }
}

cudaError_t launch_fill0(long n3, uint64_t zeta, const float* src, const float* rec0,
                         const PrologueArgs& pa, float* fill, cudaStream_t st) {
  k_fill0<<<prologue_blocks(n3), PRO_THREADS, 0, st>>>(n3, zeta, src, rec0, pa, fill);
  return cudaGetLastError();
}

// Neutral fraction (:473-477): the serial double sum of 1 - x from chunks, each
// a pair of multiples of u (neutral_sum.h).  Pairs compose.  Everything here is
// in integers: a term is a multiple of 2^-53 (neutral_units), and while S is in
// [2^E, 2^(E+1)) an addition rounds it to a multiple of 2^(E+1) of those.  E of
// a chunk follows from the chunks' sums; a chunk in which S may leave its
// binade (about one per binade), starts below 1 or has a term outside [0, 1]
// is left to the host's serial loop (E = -1).
// A call with host boxes and four sets, neutral fractions included: 16^3 0.52
// ms with the sums as loops on host threads, 0.99 when one block added the
// chunks' sums in FP64, each thread all that come before its own, 0.26 so;
// 64^3 0.81, 1.19, 0.53; 256^3 20.4, 9.0, 8.0.
constexpr int NEU_THREADS = 256, NEU_PER = NEUTRAL_CHUNK / NEU_THREADS;  // consecutive terms per thread
static_assert(NEU_PER == 16, "four float4 per thread");
constexpr uint64_t NEU_BAD = ~0ull;  // sum of a chunk with a term outside [0, 1]

// false: a term is outside [0, 1]
__device__ __forceinline__ bool neutral_terms(const float* __restrict__ x, long n3, uint64_t (&t)[NEU_PER]) {
  const long i0 = (long)blockIdx.x * NEUTRAL_CHUNK + (long)threadIdx.x * NEU_PER;
  bool ok = true;
#pragma unroll
  for (int k = 0; k < NEU_PER; k += 4) {
    const float4 v = i0 + k < n3 ? __ldg(reinterpret_cast<const float4*>(x + i0 + k)) : make_float4(1.f, 1.f, 1.f, 1.f);
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      ok = ok && f[j] >= 0.0f && f[j] <= 1.0f;
      t[k + j] = neutral_units(f[j]);
    }
  }
  return ok;
}

// sum[chunk]: its terms' sum in units of 2^-32, 256 of them too small at most
// (a thread's 16 terms are below 2^58 units of 2^-53)
__global__ void __launch_bounds__(NEU_THREADS)
k_neutral_sums(const float* __restrict__ x, long n3, uint64_t* __restrict__ sum) {
  uint64_t t[NEU_PER], s = 0;
  const bool ok = neutral_terms(x, n3, t);
#pragma unroll
  for (int k = 0; k < NEU_PER; ++k) s += t[k];
  s >>= 21;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ uint64_t sh[NEU_THREADS / 32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  const bool good = __syncthreads_and(ok);
  if (threadIdx.x == 0) {
    for (int w = 1; w < NEU_THREADS / 32; ++w) s += sh[w];
    sum[blockIdx.x] = good ? s : NEU_BAD;
  }
}

// E of every chunk, from the sums before and after it.  One block scans the
// chunks, four to a thread: 4096 of them at a time, 8 times at 512^3.
constexpr int NEU_SCAN = 1024;
__global__ void __launch_bounds__(NEU_SCAN) k_neutral_binades(int nchunk, const uint64_t* __restrict__ sum, int* __restrict__ E) {
  __shared__ uint64_t sh[NEU_SCAN / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t carry = 0;
  for (int c0 = 0; c0 < nchunk; c0 += 4 * NEU_SCAN) {
    const int c = c0 + 4 * threadIdx.x;
    uint64_t v[4], t = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = c + k < nchunk ? sum[c + k] : 0;
      t += v[k] == NEU_BAD ? 0 : v[k];
    }
    uint64_t x = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    uint64_t y = sh[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    uint64_t before = carry + x - t;
    const uint64_t below = __shfl_sync(0xffffffffu, y, w ? w - 1 : 0);
    if (w) before += below;
    carry += __shfl_sync(0xffffffffu, y, 31);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (c + k >= nchunk) break;
      const uint64_t after = before + (v[k] == NEU_BAD ? 0 : v[k]);
      const int el = 31 - __clzll((long long)before), eh = 31 - __clzll((long long)after);  // in units of 2^-32
      E[c + k] = el >= 0 && el == eh && v[k] != NEU_BAD ? el : -1;
      before = after;
    }
    __syncthreads();  // sh has been read
  }
}

__global__ void __launch_bounds__(NEU_THREADS)
k_neutral_steps(const float* __restrict__ x, long n3, const int* __restrict__ binade, longlong2* __restrict__ step) {
  const int E = binade[blockIdx.x];
  if (E < 0) return;
  uint64_t t[NEU_PER];
  neutral_terms(x, n3, t);
  long long d0 = 0, d1 = 0;  // added to an even and an odd S / u
  const int sh = E + 1;      // u = 2^(E-52)
  const uint64_t half = 1ull << E;
#pragma unroll
  for (int k = 0; k < NEU_PER; ++k) {
    const long long q = (long long)(t[k] >> sh);
    const uint64_t rem = t[k] & (2 * half - 1);
    const long long up = rem > half;
    const bool tie = rem == half;
    d0 += q + (tie ? (d0 + q) & 1 : up);
    d1 += q + (tie ? (1 + d1 + q) & 1 : up);
  }
  // neighbours in order: within a warp, then the warps
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto then = [](longlong2 f, longlong2 g) {
    return make_longlong2(f.x + (f.x & 1 ? g.y : g.x), f.y + ((1 + f.y) & 1 ? g.y : g.x));
  };
  longlong2 f = make_longlong2(d0, d1);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const longlong2 g = make_longlong2(__shfl_down_sync(0xffffffffu, f.x, o), __shfl_down_sync(0xffffffffu, f.y, o));
    if ((lane & (2 * o - 1)) == 0) f = then(f, g);
  }
  __shared__ longlong2 sh2[NEU_THREADS / 32];
  if (lane == 0) sh2[w] = f;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < NEU_THREADS / 32; ++k) f = then(f, sh2[k]);
    step[blockIdx.x] = f;
  }
}

int neutral_chunks(long n3) { return (int)((n3 + NEUTRAL_CHUNK - 1) / NEUTRAL_CHUNK); }
size_t neutral_bytes(long n3) {  // whole longlong2, so that the sets' buffers can follow one another
  return ((size_t)neutral_chunks(n3) * (sizeof(longlong2) + sizeof(uint64_t) + sizeof(int)) + 15) / 16 * 16;
}
cudaError_t launch_neutral(long n3, const float* x, void* buf, cudaStream_t st) {
  const int n = neutral_chunks(n3);
  longlong2* step = static_cast<longlong2*>(buf);
  uint64_t* sum = reinterpret_cast<uint64_t*>(step + n);
  int* E = reinterpret_cast<int*>(sum + n);
  k_neutral_sums<<<n, NEU_THREADS, 0, st>>>(x, n3, sum);
  k_neutral_binades<<<1, NEU_SCAN, 0, st>>>(n, sum, E);
  k_neutral_steps<<<n, NEU_THREADS, 0, st>>>(x, n3, E, step);
  return cudaGetLastError();
}

// The serial sum from the chunks' pairs (buf: launch_neutral's, on the host; null: none) and the box x
double neutral_sum(long n3, const void* buf, const float* x) {
  if (!buf) {
    double S = 0.;
    for (long i = 0; i < n3; ++i) S += 1.0 - x[i];
    return S;
  }
  const int n = neutral_chunks(n3);
  const longlong2* step = static_cast<const longlong2*>(buf);
  const int* E = reinterpret_cast<const int*>(reinterpret_cast<const uint64_t*>(step + n) + n);
  return neutral_serial(n3, &step->x, E, [x](long i) { return x[i]; });
}

}  // namespace sf21
