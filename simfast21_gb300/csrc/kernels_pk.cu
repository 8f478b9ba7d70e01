// Power spectrum of a cubic box on the GPU (tools/power3d_f.c:124-194):
// window, forward transform (the filter bank's own FFT passes), and the
// spherical binning of |F(k)|^2 over the r2c half-spectrum.
//
//   k_pk_pack: (float)(value * w(i) w(j) w(p)) as the real part of a complex
//     box (imaginary part 0), the window given per axis;
//   k_pk_bin: one CTA per PK_ROWS rows (i, j), threads over p = 0..N/2:
//     bin = round(|k| / dk) = round(sqrt(i'^2 + j'^2 + p^2)) in integers
//     (i', j' the signed indices; for a cube every axis has the same dk),
//     power = re^2 + im^2 in float as the tool computes it; per-CTA sums in
//     shared memory, written out per CTA, counts added exactly with integer
//     atomics;
//   k_pk_reduce: adds the CTAs' sums exactly, in integers, so a few
//     kilobytes go to the host instead of the 14.6 MB of partial sums at 512^3,
//     which took most of the call there.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sf21_device.cuh"
#include "sf21_kernels.h"
#include "softdouble.h"

namespace sf21 {

constexpr int PK_THREADS = 256;
constexpr int PK_ROWS = 32;

int pk_nbins(int N) {
  const long h = N / 2;
  long m = 0;
  const long n = 3 * h * h;
  while ((m + 1) * (m + 1) <= n) ++m;
  return (int)((n - m * m > m) ? m + 1 : m) + 1;  // round(sqrt(3 (N/2)^2)) + 1, :83
}

int pk_bin_grid(int N) { return (int)(((long)N * N + PK_ROWS - 1) / PK_ROWS); }

__global__ void k_pk_pack(long n3, int N, const float* __restrict__ box, const float* __restrict__ wax,
                          float2* __restrict__ out) {
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n3; t += (long)gridDim.x * blockDim.x) {
    const int p = (int)(t % N), j = (int)((t / N) % N), i = (int)(t / ((long)N * N));
    const float w = __fmul_rn(__fmul_rn(wax[i], wax[j]), wax[p]);
    out[t] = make_float2(__fmul_rn(box[t], w), 0.0f);
  }
}

__device__ __forceinline__ int round_sqrt(int n) {
  int m = (int)sqrtf((float)n);
  while (m * m > n) --m;
  while ((m + 1) * (m + 1) <= n) ++m;
  return (n - m * m > m) ? m + 1 : m;  // sqrt(n) >= m + 1/2  <=>  n > m^2 + m
}

__global__ void __launch_bounds__(PK_THREADS)
k_pk_bin(int N, const float2* __restrict__ spec, int nk, float* __restrict__ partials,
         unsigned long long* __restrict__ counts) {
  extern __shared__ float pk_smem[];
  float* sums = pk_smem;
  int* cnt = reinterpret_cast<int*>(pk_smem + nk);
  for (int b = threadIdx.x; b < nk; b += blockDim.x) {
    sums[b] = 0.0f;
    cnt[b] = 0;
  }
  __syncthreads();
  const int half = N / 2 + 1;
  const long row0 = (long)blockIdx.x * PK_ROWS;
  for (int t = threadIdx.x; t < PK_ROWS * half; t += blockDim.x) {
    const long row = row0 + t / half;
    if (row >= (long)N * N) break;
    const int p = t % half;
    const int i = (int)(row / N), j = (int)(row % N);
    const int si = kfreq(i, N), sj = kfreq(j, N);
    const int b = round_sqrt(si * si + sj * sj + p * p);
    const float2 z = spec[row * N + p];
    const float pw = __fadd_rn(__fmul_rn(z.x, z.x), __fmul_rn(z.y, z.y));
    atomicAdd(&sums[b], pw);
    atomicAdd(&cnt[b], 1);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nk; b += blockDim.x) {
    partials[(long)blockIdx.x * nk + b] = sums[b];
    if (cnt[b]) atomicAdd(&counts[b], (unsigned long long)cnt[b]);
  }
}

// partials: [ncta][nk], not negative; sums[b]: bin b's sum, rounded to double
// once, as bits.  Terms are 128-bit integers in units of 2^-103 of the largest
// one's exponent (2^16 CTAs at most: 120 bits), which a first pass over the
// partials finds: sums of integers are two instructions a term and shuffles
// after that.  (Chains and a tree of soft doubles made a call 6 us longer at
// 64^3, 128 partial sums a bin, 73 us for 67, and 12 at 512^3, 8192 a bin.)  A
// sum with an infinity is infinite, one with a NaN is NaN.
// threadIdx.x = bin of the CTA's PKR_BINS, the threadIdx.y rows share the CTAs.
constexpr int PKR_BINS = 4, PKR_ROWS = 256, PKR_WARPS = PKR_BINS * PKR_ROWS / 32;
static_assert(PKR_WARPS == 32, "the last step is one warp, four sums to a lane");

__device__ __forceinline__ sd_u128 pk_lanes(sd_u128 v) {  // over the warp's lanes of one bin
#pragma unroll
  for (int o = PKR_BINS; o < 32; o <<= 1)
    v += (sd_u128)__shfl_xor_sync(0xffffffffu, (unsigned long long)(v >> 64), o) << 64 |
         __shfl_xor_sync(0xffffffffu, (unsigned long long)v, o);
  return v;
}

// v 2^e as a double's bits, to nearest even (its exponent is a normal one)
__device__ __forceinline__ uint64_t pk_double(sd_u128 v, int e) {
  if (!v) return 0;
  const uint64_t hi = (uint64_t)(v >> 64);
  const int top = hi ? 127 - __clzll((long long)hi) : 63 - __clzll((long long)(uint64_t)v);
  uint64_t q;
  if (top <= 52) {
    q = (uint64_t)v << (52 - top);
  } else {
    const int s = top - 52;
    const sd_u128 rem = v & (((sd_u128)1 << s) - 1), half = (sd_u128)1 << (s - 1);
    q = (uint64_t)(v >> s);
    q += rem > half || (rem == half && (q & 1));
  }
  return ((uint64_t)(top + e + 1022) << 52) + q;  // q has bit 52 (or is 2^53: the next exponent)
}

__global__ void __launch_bounds__(PKR_BINS * PKR_ROWS)
k_pk_reduce(int ncta, int nk, const float* __restrict__ partials, uint64_t* __restrict__ sums) {
  __shared__ uint32_t most[PKR_BINS];
  __shared__ unsigned long long part[PKR_WARPS][PKR_BINS][2];
  const int x = threadIdx.x, b = blockIdx.x * PKR_BINS + x, tid = threadIdx.y * PKR_BINS + x;
  const int lane = tid & 31, w = tid >> 5;
  if (tid < PKR_BINS) most[tid] = 0;
  __syncthreads();
  const int g0 = b < nk ? threadIdx.y : ncta;
  uint32_t m = 0;  // of the bits: floats that are not negative are in their order, infinity and NaNs above them
#pragma unroll 8
  for (int g = g0; g < ncta; g += PKR_ROWS) m = max(m, __float_as_uint(partials[(long)g * nk + b]) & 0x7FFFFFFFu);
#pragma unroll
  for (int o = PKR_BINS; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane < PKR_BINS) atomicMax(&most[x], m);
  __syncthreads();
  m = most[x];
  const int E = max((int)(m >> 23), 1);
  sd_u128 s = 0;
  if (m < 0x7F800000u) {
#pragma unroll 8
    for (int g = g0; g < ncta; g += PKR_ROWS) {
      const uint32_t u = __float_as_uint(partials[(long)g * nk + b]) & 0x7FFFFFFFu;
      const int e = max((int)(u >> 23), 1);
      const uint32_t f = (u & 0x7FFFFFu) | (u >> 23 ? 0x800000u : 0u);  // value f 2^(e - 150)
      s += (sd_u128)f << 80 >> min(E - e, 127);
    }
  }
  s = pk_lanes(s);
  if (lane < PKR_BINS) {
    part[w][x][0] = (unsigned long long)(s >> 64);
    part[w][x][1] = (unsigned long long)s;
  }
  __syncthreads();
  if (w == 0) {
    s = 0;
#pragma unroll
    for (int k = lane / PKR_BINS; k < PKR_WARPS; k += 32 / PKR_BINS) s += (sd_u128)part[k][x][0] << 64 | part[k][x][1];
    s = pk_lanes(s);
    if (lane < PKR_BINS && b < nk)
      sums[b] = m > 0x7F800000u ? SD_QNAN : m == 0x7F800000u ? 0x7FF0000000000000ULL : pk_double(s, E - 230);
  }
}

cudaError_t launch_pk_reduce(int N, int nk, const float* partials, uint64_t* sums, cudaStream_t st) {
  k_pk_reduce<<<(nk + PKR_BINS - 1) / PKR_BINS, dim3(PKR_BINS, PKR_ROWS), 0, st>>>(pk_bin_grid(N), nk, partials, sums);
  return cudaGetLastError();
}

cudaError_t launch_pk_pack(int N, const float* box, const float* wax, float2* out, cudaStream_t st) {
  const long n3 = (long)N * N * N;
  long blocks = (n3 + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  k_pk_pack<<<(unsigned)blocks, 256, 0, st>>>(n3, N, box, wax, out);
  return cudaGetLastError();
}

cudaError_t launch_pk_bin(int N, const float2* spec, int nk, float* partials, unsigned long long* counts,
                          cudaStream_t st) {
  const size_t smem = (size_t)nk * (sizeof(float) + sizeof(int));
  k_pk_bin<<<pk_bin_grid(N), PK_THREADS, smem, st>>>(N, spec, nk, partials, counts);
  return cudaGetLastError();
}

}  // namespace sf21
