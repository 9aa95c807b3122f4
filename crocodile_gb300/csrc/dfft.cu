// Batched complex FFTs computed in double-float arithmetic.
//
// GB300 runs FP64 at a small fraction of its FP32 rate, and a batched FP64
// FFT is bound by that rate, not by memory.  Here each complex value is
// carried as two unevaluated float sums (hi + lo, about 48 significant bits)
// and every butterfly uses error-free transformations on the FP32 units
// (df.cuh; sloppy pair sums in the butterflies, normwise error about 2u^2
// per stage, u = 2^-24).  Transforms are power-of-two lengths 64 .. 2048 in
// shared memory by the Stockham (self-sorting) algorithm in radix 4, with one
// radix-2 stage first when log2 n is odd: the stage with stride s reads
// x[q + s (p + k m)] (m = n/(4s), k < 4, t = p s + q) and writes
// y[q + s (4p + k)] = (the 4-point DFT of those four)_k w^(k p s), so the
// output is in natural order; half the shared-memory passes and a quarter
// fewer twiddle products than radix 2.  Twiddles w^k = exp(-+2 pi i k / n),
// k < 3n/4, come from an FP64 host table split into hi + lo.
// Unnormalised, as cuFFT.
//
// Elements reach the kernels through an I/O policy, so one transform serves
//   - complex128 rows in place (converted on load and store),
//   - double-float rows (float4 = re.hi, re.lo, im.hi, im.lo) in place,
//   - the two passes of a centred 2-D transform of complex128 planes: rows
//     with the (-1)^(i+j) pre-modulation, complex128 in and double-float out;
//     then columns, double-float in and complex128 out with the post-
//     modulation and the 1 / (H W) of an inverse.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "cg_internal.cuh"
#include "df.cuh"
#include "dfft.cuh"

namespace cg {

namespace {

// ---------------------------------------------------------------- I/O policies
// ld(row, i) / st(row, i, v): element i of transform row `row`

struct IoC128 {
  double2 *d;
  int n;
  __device__ cdf ld(int64_t row, int i) const { return cdf_from(d[row * n + i]); }
  __device__ void st(int64_t row, int i, const cdf &v) const { d[row * n + i] = cdf_to(v); }
};

struct IoDF {
  float4 *d;
  int n;
  __device__ cdf ld(int64_t row, int i) const { return cdf_load(d[row * n + i]); }
  __device__ void st(int64_t row, int i, const cdf &v) const { d[row * n + i] = cdf_store(v); }
};

__device__ __forceinline__ cdf cdf_neg(const cdf &v) { return {df_neg(v.re), df_neg(v.im)}; }

// centred 2-D, pass over rows: rows of h x w complex128 planes (element
// strides plane, pitch) standing in the middle of zero H x n planes, row
// r0 + i and column c0 + j of the plane being element (i, j); the sign
// (-1)^(r + c) of the pre-modulation; double-float out, to the same rows of
// the H x n planes at d (same 16 bytes per element; d may be the source when
// the planes are whole).
struct IoRowsCentred {
  const double2 *src;
  float4 *d;
  int64_t plane, pitch;
  int n, H, h, w, r0, c0;
  __device__ cdf ld(int64_t row, int i) const {
    const int p = (int)row / h, r = (int)row - p * h, j = i - c0;
    if ((unsigned)j >= (unsigned)w) return {{0.f, 0.f}, {0.f, 0.f}};
    const cdf v = cdf_from(src[p * plane + r * pitch + j]);
    return ((r + r0 + i) & 1) ? cdf_neg(v) : v;
  }
  __device__ void st(int64_t row, int i, const cdf &v) const {
    const int p = (int)row / h, r = (int)row - p * h;
    d[((int64_t)p * H + r + r0) * n + i] = cdf_store(v);
  }
};

// The block of a centred 2-D transform: input rows that hold data (the others
// are zeros that no pass has to touch) and the output block that is wanted.
struct ColsBlock {
  int in0, in_n;         // input rows
  int row0, row_n;       // output rows
  int col0, col_n;       // output columns
};

// ---------------------------------------------------------------- column transforms
// Planes [nplanes][N][W] of double-float, transformed along N (the columns);
// each CTA takes P pairs of adjacent columns of one plane (P * 32 bytes per
// row read), N/4 threads per pair, neighbouring threads on neighbouring pairs
// so that their 32-byte accesses join; then the centred post-modulation
// (-1)^(l + k + phase) * scale and complex128 out in place.  The planes'
// stride in shared memory puts the P pairs of one index on different banks.
constexpr int col_plane(int n, int P) {
  const int want = P >= 8 ? 1 : 8 / P % 8;  // stride mod 8 (16-byte units)
  int s = dfk::pair_plane(n);
  while (s % 8 != want) ++s;
  return s;
}

template <int LOGN, int P>
__global__ void __launch_bounds__((1 << LOGN) / 4 * P, dfk::DFFT_SM_THREADS / ((1 << LOGN) / 4 * P))
    k_dfft_cols_centred(double2 *d, int64_t nplanes, int W, ColsBlock B, int phase, float scale,
                        const float4 *__restrict__ tw, int inverse) {
  constexpr int N = 1 << LOGN;
  constexpr int Q = N / 4;
  constexpr int PL = col_plane(N, P);
  extern __shared__ __align__(16) unsigned char dsm_raw[];
  float4 *planes = (float4 *)dsm_raw;  // [re, im][P][PL]
  float4 *stw = planes + 2 * P * PL;   // [3N/4]
  const int p = threadIdx.x % P, t = threadIdx.x / P;
  float4 *re = planes + p * PL, *im = planes + (P + p) * PL;
  for (int k = threadIdx.x; k < 3 * Q; k += blockDim.x) stw[k] = tw[k];
  const bool inv = inverse != 0;
  const int g0 = B.col0 / (2 * P), groups = (B.col0 + B.col_n + 2 * P - 1) / (2 * P) - g0;
  const int64_t jobs = nplanes * groups;
  __syncthreads();
  for (int64_t job = blockIdx.x; job < jobs; job += gridDim.x) {
    const int64_t plane = job / groups;
    const int c = ((g0 + (int)(job - plane * groups)) * P + p) * 2;
    double2 *col = d + plane * N * W + c;
    cdf2 e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int l = t + k * Q;
      const float4 *src = (const float4 *)(col + (int64_t)l * W);
      const bool in = (unsigned)(l - B.in0) < (unsigned)B.in_n;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      e[k] = cdf2_pack(cdf_load(in ? src[0] : zero), cdf_load(in ? src[1] : zero));
    }
    dfk::pair_fft<LOGN>(e, re, im, stw, t, inv);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int l = t + ((k & 1) && !inv ? 4 - k : k) * Q;
      if ((unsigned)(l - B.row0) >= (unsigned)B.row_n) continue;
      const float sg = ((l + c + phase) & 1) ? -scale : scale;  // a power of two
      cdf a, b;
      cdf2_unpack(e[k], a, b);
      double2 *dst = col + (int64_t)l * W;
      dst[0] = cdf_to({{a.re.hi * sg, a.re.lo * sg}, {a.im.hi * sg, a.im.lo * sg}});
      dst[1] = cdf_to({{b.re.hi * -sg, b.re.lo * -sg}, {b.im.hi * -sg, b.im.lo * -sg}});
    }
  }
}

// ---------------------------------------------------------------- long rows
// n = N1 * 2048 (N1 = 2, 4) in three passes, the four-step factorisation
//   X[k1 + N1 k2] = sum_n2 w_n^(n2 k1) [sum_n1 x[n2 + 2048 n1] w_N1^(n1 k1)] w_2048^(n2 k2):
// k_dfft_long_pre forms the bracket times w_n^(n2 k1) in place (row position
// k1 * 2048 + n2), the 2048-point kernel transforms the N1 sub-rows, and
// k_dfft_long_T puts X back in natural order through shared memory.
constexpr int DF_LONG_N2 = 2048;

template <int N1>
__global__ void k_dfft_long_pre(float4 *d, int64_t batch, const float4 *__restrict__ tw,
                                int inverse) {
  constexpr int N2 = DF_LONG_N2, N = N1 * N2;
  const int64_t total = batch * N2;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = e / N2;
    const int n2 = (int)(e - b * N2);
    float4 *row = d + b * N;
    cdf x[N1], y[N1];
#pragma unroll
    for (int j = 0; j < N1; ++j) x[j] = cdf_load(row[n2 + N2 * j]);
    if (N1 == 2) {
      y[0] = cdf_add_f(x[0], x[1]);
      y[1] = cdf_sub_f(x[0], x[1]);
    } else {
      const cdf a0 = cdf_add_f(x[0], x[N1 > 2 ? 2 : 0]), a1 = cdf_sub_f(x[0], x[N1 > 2 ? 2 : 0]);
      const cdf b0 = cdf_add_f(x[1], x[N1 > 3 ? 3 : 1]);
      const cdf b1 = dfk::cdf_mul_j(cdf_sub_f(x[1], x[N1 > 3 ? 3 : 1]), inverse != 0);
      y[0] = cdf_add_f(a0, b0);
      y[1] = cdf_add_f(a1, b1);
      y[N1 > 2 ? 2 : 0] = cdf_sub_f(a0, b0);
      y[N1 > 3 ? 3 : 1] = cdf_sub_f(a1, b1);
    }
    row[n2] = cdf_store(y[0]);
#pragma unroll
    for (int k1 = 1; k1 < N1; ++k1)
      row[k1 * N2 + n2] = cdf_store(n2 == 0 ? y[k1] : cdf_mul_f(y[k1], cdf_load(tw[n2 * k1])));
  }
}

// X[k1 + N1 k2] = Z[k1][k2] for each row, in place; one CTA per row, the sub-
// rows padded by one element in shared memory
template <int N1>
__global__ void __launch_bounds__(1024) k_dfft_long_T(float4 *d, int64_t batch) {
  constexpr int N2 = DF_LONG_N2, N = N1 * N2, P = N2 + 1;
  extern __shared__ float dsm[];
  float4 *buf = (float4 *)dsm;  // [N1][P]
  for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
    float4 *row = d + b * N;
    for (int e = threadIdx.x; e < N; e += blockDim.x) buf[(e / N2) * P + (e % N2)] = row[e];
    __syncthreads();
    for (int k = threadIdx.x; k < N; k += blockDim.x) row[k] = buf[(k % N1) * P + k / N1];
    __syncthreads();
  }
}

// complex128 <-> double-float in place (the same 16 bytes per element)
__global__ void k_c128_to_df(double2 *d, int64_t count) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < count;
       e += (int64_t)gridDim.x * blockDim.x)
    ((float4 *)d)[e] = cdf_store(cdf_from(d[e]));
}
__global__ void k_df_to_c128(double2 *d, int64_t count) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < count;
       e += (int64_t)gridDim.x * blockDim.x)
    d[e] = cdf_to(cdf_load(((float4 *)d)[e]));
}

// ---------------------------------------------------------------- twiddles
}  // namespace

std::mutex g_tw_mu;
std::map<std::pair<int, int>, float4 *> g_tw;  // (device, n * sign) -> table

int dfft_twiddles(int n, int sign, const float4 **out) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_tw_mu);
  auto key = std::make_pair(dev, n * sign);
  auto it = g_tw.find(key);
  if (it != g_tw.end()) {
    *out = it->second;
    return CG_OK;
  }
  std::vector<float4> h(3 * n / 4);
  for (int k = 0; k < 3 * n / 4; ++k) {
    const double a = 2.0 * M_PI * (double)k / (double)n;
    const double c = std::cos(a), s = sign * std::sin(a);
    const float ch = (float)c, sh = (float)s;
    h[k] = make_float4(ch, (float)(c - (double)ch), sh, (float)(s - (double)sh));
  }
  float4 *d = nullptr;
  CG_CUDA(cudaMalloc(&d, h.size() * sizeof(float4)));
  CG_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(float4), cudaMemcpyHostToDevice));
  g_tw[key] = d;
  *out = d;
  return CG_OK;
}

namespace {

template <int LOGN, int P>
int launch_cols(double2 *d, int64_t nplanes, int W, const ColsBlock &B, int phase, float scale,
                const float4 *tw, int inverse, cudaStream_t st) {
  constexpr int N = 1 << LOGN;
  const size_t smem = (size_t)(2 * P * col_plane(N, P) + 3 * N / 4) * sizeof(float4);
  if (smem > 48 * 1024)
    CG_CUDA(cudaFuncSetAttribute(k_dfft_cols_centred<LOGN, P>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int groups = (B.col0 + B.col_n + 2 * P - 1) / (2 * P) - B.col0 / (2 * P);
  const int64_t jobs = nplanes * groups;
  const unsigned grid = (unsigned)std::min<int64_t>(jobs, (int64_t)num_sms() * 8);
  k_dfft_cols_centred<LOGN, P><<<grid, N / 4 * P, smem, st>>>(d, nplanes, W, B, phase, scale, tw,
                                                              inverse);
  CG_LAUNCH("double-float column FFT");
  return CG_OK;
}

}  // namespace

bool dfft_supported(int n) { return n >= 64 && n <= 2048 && (n & (n - 1)) == 0; }

// In-place batched FFT of `batch` contiguous complex128 rows of length n
// (a power of two, 64..2048); inverse: exp(+2 pi i), unnormalised.
int dfft_rows(double2 *data, int64_t batch, int n, int inverse, cudaStream_t st) {
  return dfft_rows_io(IoC128{data, n}, batch, n, inverse, st);
}

bool dfft_long_supported(int n) { return dfft_supported(n) || n == 4096 || n == 8192; }

namespace {
template <int N1>
int dfft_long(float4 *data, int64_t batch, int inverse, cudaStream_t st) {
  const int n = N1 * DF_LONG_N2;
  const float4 *tw;
  int rc = dfft_twiddles(n, inverse ? 1 : -1, &tw);
  if (rc) return rc;
  const int64_t total = batch * DF_LONG_N2;
  const unsigned g = (unsigned)std::min<int64_t>((total + 255) / 256, (int64_t)num_sms() * 16);
  k_dfft_long_pre<N1><<<g, 256, 0, st>>>(data, batch, tw, inverse);
  CG_LAUNCH("double-float long FFT (first pass)");
  if ((rc = dfft_rows_io(IoDF{data, DF_LONG_N2}, batch * N1, DF_LONG_N2, inverse, st)))
    return rc;
  const size_t smem = (size_t)N1 * (DF_LONG_N2 + 1) * sizeof(float4);
  CG_CUDA(cudaFuncSetAttribute(k_dfft_long_T<N1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
  const unsigned gt = (unsigned)std::min<int64_t>(batch, (int64_t)num_sms() * 4);
  k_dfft_long_T<N1><<<gt, 1024, smem, st>>>(data, batch);
  CG_LAUNCH("double-float long FFT (transpose)");
  return CG_OK;
}
}  // namespace

// The same on rows stored as double-float (float4 per element); lengths up to
// 8192 (4096 and 8192 by the four-step passes).
int dfft_rows_df(float4 *data, int64_t batch, int n, int inverse, cudaStream_t st) {
  if (batch <= 0) return CG_OK;
  if (n == 4096) return dfft_long<2>(data, batch, inverse, st);
  if (n == 8192) return dfft_long<4>(data, batch, inverse, st);
  return dfft_rows_io(IoDF{data, n}, batch, n, inverse, st);
}

// Centred 2-D FFT of `batch` complex128 planes [H][W] at data (numpy's
// fftshift(fft2(ifftshift(x))), or the normalised ifft2 for inverse), H and W
// powers of two 64..2048.  The fftshifts are the checkerboard modulations
// (-1)^(i+j) before and (-1)^(k+l+H/2+W/2) after the transform.  The input is
// the h x w planes at src (element strides plane, pitch) in the middle of
// zeros: rows of zeros are neither transformed nor written nor read.  Of the
// output only the middle oh x ow is written.  Four facets to 22 x 22 subgrids
// of 384^2 in 512^2 and back: 10.30 ms, against 12.07 ms with the padding, the
// copies and whole planes.
static int dfft2_window(double2 *data, const double2 *src, int64_t plane, int64_t pitch,
                        int64_t batch, int H, int W, int h, int w, int oh, int ow, int inverse,
                        cudaStream_t st) {
  CG_REQUIRE(dfft_supported(H) && dfft_supported(W),
             "double-float 2-D FFT sides are powers of two 64..2048");
  CG_REQUIRE(h >= 1 && w >= 1 && h <= H && w <= W && oh >= 1 && ow >= 1 && oh <= H && ow <= W,
             "double-float 2-D FFT: a block larger than the plane");
  CG_REQUIRE(batch * H < ((int64_t)1 << 31), "too many double-float 2-D FFT rows");
  if (batch <= 0) return CG_OK;
  const int r0 = H / 2 - h / 2, c0 = W / 2 - w / 2;
  int rc = dfft_rows_io(IoRowsCentred{src, (float4 *)data, plane, pitch, W, H, h, w, r0, c0},
                        batch * h, W, inverse, st);
  if (rc) return rc;
  const ColsBlock B = {r0, h, H / 2 - oh / 2, oh, W / 2 - ow / 2, ow};
  const float4 *tw;
  if ((rc = dfft_twiddles(H, inverse ? 1 : -1, &tw))) return rc;
  const int phase = (H / 2 + W / 2) & 1;
  const float scale = inverse ? 1.0f / ((float)H * (float)W) : 1.0f;  // a power of two
  switch (H) {  // pairs of columns per CTA: 256 threads up to 1024
    case 64: return launch_cols<6, dfk::pairs_for(6)>(data, batch, W, B, phase, scale, tw, inverse, st);
    case 128: return launch_cols<7, dfk::pairs_for(7)>(data, batch, W, B, phase, scale, tw, inverse, st);
    case 256: return launch_cols<8, dfk::pairs_for(8)>(data, batch, W, B, phase, scale, tw, inverse, st);
    case 512: return launch_cols<9, dfk::pairs_for(9)>(data, batch, W, B, phase, scale, tw, inverse, st);
    case 1024: return launch_cols<10, dfk::pairs_for(10)>(data, batch, W, B, phase, scale, tw, inverse, st);
    case 2048: return launch_cols<11, dfk::pairs_for(11)>(data, batch, W, B, phase, scale, tw, inverse, st);
  }
  return set_error(CG_ERR_ARG, "unsupported double-float FFT length %d", H);
}

// whole planes in place
int dfft2_centred(double2 *data, int64_t batch, int H, int W, int inverse, cudaStream_t st) {
  return dfft2_window(data, data, (int64_t)H * W, W, batch, H, W, H, W, H, W, inverse, st);
}

}  // namespace cg

extern "C" int cg_fft_rows_df(void *data_c128, int64_t batch, int n, int inverse,
                              cg_stream_t stream) {
  CG_REQUIRE(data_c128 && batch >= 0, "bad double-float FFT arguments");
  if (n == 4096 || n == 8192) {  // converted in place around the double-float passes
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t count = batch * n;
    if (count == 0) return CG_OK;
    const unsigned g =
        (unsigned)std::min<int64_t>((count + 255) / 256, (int64_t)cg::num_sms() * 16);
    cg::k_c128_to_df<<<g, 256, 0, st>>>((double2 *)data_c128, count);
    CG_LAUNCH("complex128 to double-float");
    const int rc = cg::dfft_rows_df((float4 *)data_c128, batch, n, inverse, st);
    if (rc) return rc;
    cg::k_df_to_c128<<<g, 256, 0, st>>>((double2 *)data_c128, count);
    CG_LAUNCH("double-float to complex128");
    return CG_OK;
  }
  return cg::dfft_rows((double2 *)data_c128, batch, n, inverse, (cudaStream_t)stream);
}

extern "C" int cg_fft2_centred_df(void *data_c128, int64_t batch, int H, int W, int inverse,
                                  cg_stream_t stream) {
  CG_REQUIRE(data_c128 && batch >= 0, "bad double-float 2-D FFT arguments");
  return cg::dfft2_centred((double2 *)data_c128, batch, H, W, inverse, (cudaStream_t)stream);
}

extern "C" int cg_fft2_window_df(void *data_c128, const void *src, int64_t src_plane,
                                 int64_t src_pitch, int64_t batch, int H, int W, int in_h,
                                 int in_w, int out_h, int out_w, int inverse,
                                 cg_stream_t stream) {
  CG_REQUIRE(data_c128 && batch >= 0, "bad double-float 2-D FFT arguments");
  CG_REQUIRE(src || (in_h == H && in_w == W), "a source block needs a source");
  if (!src) return cg::dfft2_window((double2 *)data_c128, (const double2 *)data_c128,
                                    (int64_t)H * W, W, batch, H, W, H, W, out_h, out_w, inverse,
                                    (cudaStream_t)stream);
  return cg::dfft2_window((double2 *)data_c128, (const double2 *)src, src_plane, src_pitch, batch,
                          H, W, in_h, in_w, out_h, out_w, inverse, (cudaStream_t)stream);
}
