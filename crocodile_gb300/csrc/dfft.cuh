// Double-float FFT building blocks shared by the transforms of dfft.cu and
// the fused recombination passes of recombine.cu: the radix-2 / radix-4
// Stockham transform of a pair (dfft.cu has the algorithm), the row-transform
// kernel over an element I/O policy, and its launcher.
//
// An I/O policy is a small struct passed by value with
//   __device__ cdf ld(int64_t row, int i) const;            // element i of row
//   __device__ void st(int64_t row, int i, const cdf &v) const;
// so a transform can gather its input (a window, a crop, a conversion) and
// scatter its output (a crop, a transpose, a weighting) without a separate
// pass over HBM.
#pragma once

#include <algorithm>

#include "cg_internal.cuh"
#include "df.cuh"

namespace cg {

bool dfft_supported(int n);
// device table of w^k = exp(sign 2 pi i k / n), k < 3n/4, as double-float
// (cached per device, n and sign)
int dfft_twiddles(int n, int sign, const float4 **out);

namespace dfk {

__device__ __forceinline__ cdf cdf_mul_j(const cdf &v, bool inverse) {  // times -i (+i)
  return inverse ? cdf{df_neg(v.im), v.re} : cdf{v.im, df_neg(v.re)};
}

// ---------------------------------------------------------------- pair transforms
// A thread carries a pair of transforms (two rows, or two adjacent columns)
// in the halves of packed registers (df.cuh): thread t of N/4 holds elements
// t + k N/4 (k < 4) of both.  That is what the first stage of either kind
// reads and what the last radix-4 stage leaves, so elements go from the load
// policy into registers and from registers to the store policy, and only the
// exchanges between stages pass through shared memory: one plane of real and
// one of imaginary parts per pair (16 bytes: hi and lo of both), the index
// padded by one in eight, which spreads the strided writes of the first
// exchanges over the banks.  Bound by FP32 issue; 484 planes of 512^2, both
// passes, and the recombination around them (four facets to 22 x 22 subgrids
// and back): 12.07 ms against 12.78 with scalar butterflies and every stage
// through shared memory, bit-identical.
//
// The radix-2 stage (odd log2 N, first) has stride 1; the radix-4 stage of
// stride s takes t = p s + q to y[q + s (4p + k)] with twiddles w^(k p s)
// (k p s < 3N/4).  Outputs 1 and 3 differ by the sign of i only, so they are
// formed as u = a1 + (i d) and v = a1 - (i d) and the direction decides which
// of the two is output 1: no operand is negated or selected.
__device__ __forceinline__ int pad8(int i) { return i + (i >> 3); }
// 256 threads per CTA (up to 1024-point transforms) and registers for 1024
// threads per SM: at 768 per SM the loads' latency shows (12.65 against 12.07
// ms for four facets to 22 x 22 subgrids and back), and smaller CTAs narrow
// the column passes' rows (13.1 ms with 128 threads).
constexpr int DFFT_THREADS = 256, DFFT_SM_THREADS = 1024;
constexpr int pairs_for(int logn) {
  const int q = (1 << logn) / 4;
  return DFFT_THREADS / q > 0 ? DFFT_THREADS / q : 1;
}
constexpr int pair_plane(int n) { return n + n / 8; }  // float4 per plane

__device__ __forceinline__ void pair_put(float4 *re, float4 *im, int i, const cdf2 &v) {
  const ulonglong2 a = make_ulonglong2(v.re.hi.v, v.re.lo.v);
  const ulonglong2 b = make_ulonglong2(v.im.hi.v, v.im.lo.v);
  ((ulonglong2 *)re)[pad8(i)] = a;
  ((ulonglong2 *)im)[pad8(i)] = b;
}
__device__ __forceinline__ cdf2 pair_get(const float4 *re, const float4 *im, int i) {
  const ulonglong2 a = ((const ulonglong2 *)re)[pad8(i)];
  const ulonglong2 b = ((const ulonglong2 *)im)[pad8(i)];
  return {{{a.x}, {a.y}}, {{b.x}, {b.y}}};
}

// The transform of the pair held in e; every thread of the block calls it.
// Leaves element t + k N/4 in e[k] for k = 0 and 2; e[1] and e[3] hold
// elements t + k1 N/4 and t + k3 N/4, (k1, k3) = (1, 3) for an inverse
// transform and (3, 1) for a forward one.  re, im: the pair's exchange planes.
template <int LOGN>
__device__ __forceinline__ void pair_fft(cdf2 (&e)[4], float4 *re, float4 *im,
                                         const float4 *stw, int t, bool inverse) {
  constexpr int N = 1 << LOGN, Q = N / 4;
  const int k1 = inverse ? 1 : 3, k3 = inverse ? 3 : 1;
  if (LOGN & 1) {
    const cdf2 d0 = cdf2_sub_f(e[0], e[2]), d1 = cdf2_sub_f(e[1], e[3]);
    pair_put(re, im, 2 * t, cdf2_add_f(e[0], e[2]));
    pair_put(re, im, 2 * t + 1, t == 0 ? d0 : cdf2_mul_f(d0, stw[t]));
    pair_put(re, im, 2 * (t + Q), cdf2_add_f(e[1], e[3]));
    pair_put(re, im, 2 * (t + Q) + 1, cdf2_mul_f(d1, stw[t + Q]));
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = pair_get(re, im, t + k * Q);
    __syncthreads();
  }
#pragma unroll
  for (int ls = (LOGN & 1); ls < LOGN; ls += 2) {
    const int s = 1 << ls;
    const int q = t & (s - 1), ps = t - q;  // p s
    const cdf2 a0 = cdf2_add_f(e[0], e[2]), a1 = cdf2_sub_f(e[0], e[2]);
    const cdf2 b0 = cdf2_add_f(e[1], e[3]), d = cdf2_sub_f(e[1], e[3]);
    cdf2 y0 = cdf2_add_f(a0, b0), y2 = cdf2_sub_f(a0, b0);
    cdf2 u = {df2_sub_fast(a1.re, d.im), df2_add_fast(a1.im, d.re)};  // a1 + i d
    cdf2 v = {df2_add_fast(a1.re, d.im), df2_sub_fast(a1.im, d.re)};  // a1 - i d
    if (ls + 2 >= LOGN) {  // last stage: p = 0, the outputs are this thread's elements
      e[0] = y0;
      e[1] = u;
      e[2] = y2;
      e[3] = v;
      return;
    }
    if (ps != 0) {
      u = cdf2_mul_f(u, stw[k1 * ps]);
      y2 = cdf2_mul_f(y2, stw[2 * ps]);
      v = cdf2_mul_f(v, stw[k3 * ps]);
    }
    const int o = q + 4 * ps;
    pair_put(re, im, o, y0);
    pair_put(re, im, o + k1 * s, u);
    pair_put(re, im, o + 2 * s, y2);
    pair_put(re, im, o + k3 * s, v);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = pair_get(re, im, t + k * Q);
    __syncthreads();
  }
}

// ---------------------------------------------------------------- row transforms
// PAIRS pairs of rows of length N per CTA, N/4 threads per pair.
template <int LOGN, int PAIRS, class IO>
__global__ void __launch_bounds__((1 << LOGN) / 4 * PAIRS, DFFT_SM_THREADS / ((1 << LOGN) / 4 * PAIRS))
    k_dfft_rows(IO io, int64_t batch, const float4 *__restrict__ tw, int inverse) {
  constexpr int N = 1 << LOGN;
  constexpr int Q = N / 4;
  constexpr int PL = pair_plane(N);
  extern __shared__ __align__(16) unsigned char dsm_raw[];
  float4 *planes = (float4 *)dsm_raw;       // [PAIRS][2][PL]
  float4 *stw = planes + PAIRS * 2 * PL;    // [3N/4] twiddles
  const int r = threadIdx.x / Q, t = threadIdx.x - (threadIdx.x / Q) * Q;
  float4 *re = planes + r * 2 * PL, *im = re + PL;
  for (int k = threadIdx.x; k < 3 * Q; k += blockDim.x) stw[k] = tw[k];
  const bool inv = inverse != 0;
  __syncthreads();
  for (int64_t row0 = (int64_t)blockIdx.x * (2 * PAIRS); row0 < batch;
       row0 += (int64_t)gridDim.x * (2 * PAIRS)) {
    const int64_t row = row0 + 2 * r;
    const bool live0 = row < batch, live1 = row + 1 < batch;
    const cdf zero = {{0.f, 0.f}, {0.f, 0.f}};
    cdf2 e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      e[k] = cdf2_pack(live0 ? io.ld(row, t + k * Q) : zero,
                       live1 ? io.ld(row + 1, t + k * Q) : zero);
    pair_fft<LOGN>(e, re, im, stw, t, inv);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = t + ((k & 1) && !inv ? 4 - k : k) * Q;
      cdf a, b;
      cdf2_unpack(e[k], a, b);
      if (live0) io.st(row, i, a);
      if (live1) io.st(row + 1, i, b);
    }
  }
}

template <int LOGN, int PAIRS, class IO>
int launch_rows(IO io, int64_t batch, const float4 *tw, int inverse, cudaStream_t st) {
  constexpr int N = 1 << LOGN;
  const size_t smem = (size_t)(2 * PAIRS * pair_plane(N) + 3 * N / 4) * sizeof(float4);
  if (smem > 48 * 1024)  // set on every launch: the attribute is per device
    CG_CUDA(cudaFuncSetAttribute(k_dfft_rows<LOGN, PAIRS, IO>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t ctas = (batch + 2 * PAIRS - 1) / (2 * PAIRS);
  const unsigned grid = (unsigned)std::min<int64_t>(ctas, (int64_t)num_sms() * 8);
  k_dfft_rows<LOGN, PAIRS, IO><<<grid, N / 4 * PAIRS, smem, st>>>(io, batch, tw, inverse);
  CG_LAUNCH("double-float FFT");
  return CG_OK;
}

template <class IO>
int launch_any(IO io, int64_t batch, int n, int inverse, cudaStream_t st) {
  CG_REQUIRE(dfft_supported(n), "double-float FFT lengths are powers of two 64..2048");
  if (batch <= 0) return CG_OK;
  const float4 *tw;
  int rc = dfft_twiddles(n, inverse ? 1 : -1, &tw);
  if (rc) return rc;
  switch (n) {  // N/4 threads per pair of rows, 256 threads per CTA up to 1024
    case 64: return launch_rows<6, pairs_for(6)>(io, batch, tw, inverse, st);
    case 128: return launch_rows<7, pairs_for(7)>(io, batch, tw, inverse, st);
    case 256: return launch_rows<8, pairs_for(8)>(io, batch, tw, inverse, st);
    case 512: return launch_rows<9, pairs_for(9)>(io, batch, tw, inverse, st);
    case 1024: return launch_rows<10, pairs_for(10)>(io, batch, tw, inverse, st);
    case 2048: return launch_rows<11, pairs_for(11)>(io, batch, tw, inverse, st);
  }
  return set_error(CG_ERR_ARG, "unsupported double-float FFT length %d", n);
}

}  // namespace dfk

// In-place batched transforms of `batch` rows of length n (a power of two,
// 64..2048) through the I/O policy io; inverse: exp(+2 pi i), unnormalised.
template <class IO>
int dfft_rows_io(IO io, int64_t batch, int n, int inverse, cudaStream_t st) {
  return dfk::launch_any(io, batch, n, inverse, st);
}

}  // namespace cg
