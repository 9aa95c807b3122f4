// AW kernel generation by FFT (the complex64 table of aw_kernel_fn,
// crocodile/synthesis.py:701-734, for 16 x 16 AW kernels and w sub-kernels of
// support S <= 16).
//
// In FP64 (the complex64 form, k_aw_fftconv_f below, has shorter transforms):
// out[k, f] = convolve2d(akern_k, W[w_k, f], 'same') is the middle 16 x 16
// (offset o = (S - 1) / 2) of the full 31 x 31 linear convolution, which a
// 32 x 32 circular convolution of the zero-padded inputs reproduces exactly.
// So with FA_k = FFT32(akern_k) / 1024 and FW_wf = FFT32(W[w, f]) (batched
// cuFFT), out[k, f] = crop(IFFT32(FA_k * FW_wf)).  The direct form
// costs 256 x (taps <= 256) complex MACs per output sub-kernel; this one a
// 1024-point product and a pruned 32 x 32 inverse transform.
//
// k_aw_fftconv (complex128 tables): one CTA per AW key, FA_k in shared memory, each warp takes sub-kernels f
// in turn.  Lane = column k2: the warp loads FW_wf row by row
// (coalesced), multiplies by FA_k, runs a 32-point decimation-in-frequency
// inverse FFT over k1 in registers (twiddle indices compile-time, table in
// constant memory), keeps the 16 rows n1 of the crop, and transforms each of
// them across the lanes with butterflies over __shfl_xor (per-lane twiddles
// fixed per stage).  Output n2 lands on lane bitrev5(n2).
#include <cufft.h>

#include <cmath>

#include "cg_internal.cuh"
#include "fft32.h"

namespace cg {

int fft_plan(int batch, int H, int W, cufftType type, cufftHandle *out);

__constant__ float2 c_tw24[24];    // exp(+2 pi i t / 24) (complex64 tables)
__constant__ double2 c_tw32d[32];  // exp(+2 pi i t / 32) (complex128 tables)

namespace {

// the complex type of each precision, and its transforms' edge
template <typename R> struct Cx;
template <> struct Cx<float> {
  typedef float2 T;
  static constexpr int N = 24;
};
template <> struct Cx<double> {
  typedef double2 T;
  static constexpr int N = 32;
  static __device__ __forceinline__ T tw(int i) { return c_tw32d[i]; }
};

__host__ __device__ constexpr int bitrev5(int i) {
  return ((i & 1) << 4) | ((i & 2) << 2) | (i & 4) | ((i & 8) >> 2) | ((i & 16) >> 4);
}

template <int H, typename T>
__device__ __forceinline__ void dif_stage(T (&x)[32]) {
#pragma unroll
  for (int b = 0; b < 32; b += 2 * H) {
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const T a = x[b + j], c = x[b + j + H];
      x[b + j].x = a.x + c.x;
      x[b + j].y = a.y + c.y;
      T d;
      d.x = a.x - c.x;
      d.y = a.y - c.y;
      if (j == 0) {
        x[b + j + H] = d;
      } else {
        const T w = Cx<decltype(d.x)>::tw(j * (16 / H));
        x[b + j + H].x = d.x * w.x - d.y * w.y;
        x[b + j + H].y = d.x * w.y + d.y * w.x;
      }
    }
  }
}

// 32-point inverse DFT (exp(+2 pi i), unnormalised): natural order in,
// bit-reversed order out (x[i] holds output bitrev5(i))
template <typename T>
__device__ __forceinline__ void idft32_dif(T (&x)[32]) {
  dif_stage<16>(x);
  dif_stage<8>(x);
  dif_stage<4>(x);
  dif_stage<2>(x);
  dif_stage<1>(x);
}

// FA: akern [nk][16][16] zero-padded to [nk][N][N] and scaled by 1/N^2
template <typename T, int N>
__global__ void k_pad_akern(const T *__restrict__ akern, int nk, T *__restrict__ fa) {
  const int64_t total = (int64_t)nk * (N * N);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(e / (N * N)), m = (int)(e - (int64_t)k * (N * N)), r = m / N, c = m % N;
    T v;
    v.x = v.y = 0;
    if (r < 16 && c < 16) {
      v = akern[((int64_t)k * 16 + r) * 16 + c];
      v.x *= (decltype(v.x))(1.0 / (N * N));
      v.y *= (decltype(v.x))(1.0 / (N * N));
    }
    fa[e] = v;
  }
}

// FW: W [nWQ][S][S] (FP64) zero-padded to [nWQ][N][N] (rounded to FP32 for
// complex64 tables)
template <typename T, int N>
__global__ void k_pad_w(const double2 *__restrict__ W, int64_t nwq, int S, T *__restrict__ fw) {
  const int64_t total = nwq * (N * N);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = e / (N * N);
    const int m = (int)(e - g * (N * N)), r = m / N, c = m % N;
    T v;
    v.x = v.y = 0;
    if (r < S && c < S) {
      const double2 d = W[(g * S + r) * S + c];
      v.x = (decltype(v.x))d.x;
      v.y = (decltype(v.x))d.y;
    }
    fw[e] = v;
  }
}

template <typename T, int S>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 2 : 1) k_aw_fftconv(
    const T *__restrict__ fa, const T *__restrict__ fw, int nW, int QQ,
    const int32_t *__restrict__ wi, T *__restrict__ out, int32_t *status) {
  __shared__ T sfa[32][33];
  constexpr int o = (S - 1) / 2;
  const int k = blockIdx.x;
  const int w = wi[k];
  if (w < 0 || w >= nW) {
    if (threadIdx.x == 0) atomicAdd(&status[ST_INDEX], 1);
    return;
  }
  if ((status[ST_RANGE] | status[ST_INDEX]) != 0) return;
  for (int t = threadIdx.x; t < 1024; t += blockDim.x)
    sfa[t >> 5][t & 31] = fa[(int64_t)k * 1024 + t];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  typedef decltype(sfa[0][0].x) R;
  // this lane's twiddle in each across-lane stage (distance d = 16 .. 1)
  T tw[5];
#pragma unroll
  for (int st = 0; st < 5; ++st) {
    const int d = 16 >> st;
    tw[st] = Cx<R>::tw((lane & (d - 1)) * (16 / d));
  }
  const int n2 = bitrev5(lane);
  const bool keep = n2 >= o && n2 < o + 16;
  for (int f = warp; f < QQ; f += 8) {
    const T *src = fw + ((int64_t)w * QQ + f) * 1024;
    T x[32];
#pragma unroll
    for (int k1 = 0; k1 < 32; ++k1) {
      const T b = src[k1 * 32 + lane];
      const T a = sfa[k1][lane];
      x[k1].x = a.x * b.x - a.y * b.y;
      x[k1].y = a.x * b.y + a.y * b.x;
    }
    idft32_dif(x);  // over k1: x[i] = Y[bitrev5(i)][lane]
    T *dst = out + ((int64_t)k * QQ + f) * 256;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      T v = x[bitrev5(o + r)];  // row n1 = o + r
#pragma unroll
      for (int st = 0; st < 5; ++st) {
        const int d = 16 >> st;
        T p;
        p.x = __shfl_xor_sync(0xffffffffu, v.x, d);
        p.y = __shfl_xor_sync(0xffffffffu, v.y, d);
        if (lane & d) {  // upper element: (partner - v) * twiddle
          T q;
          q.x = p.x - v.x;
          q.y = p.y - v.y;
          v.x = q.x * tw[st].x - q.y * tw[st].y;
          v.y = q.x * tw[st].y + q.y * tw[st].x;
        } else {
          v.x = v.x + p.x;
          v.y = v.y + p.y;
        }
      }
      if (keep) dst[r * 16 + (n2 - o)] = v;
    }
  }
}

// The complex64 form: 24-point circular convolutions in place of 32-point ones.
// Of the 16 + S - 1 points of the full convolution only the 16 from o =
// (S - 1) / 2 are kept, so the wrapped-around rest may fall on the others: a
// period of 24 suffices (the last point, 14 + S, lands on S - 10 < o), and the
// spectra, which bound this kernel (L1, then L2: read once per sub-kernel), are
// 576 points instead of 1024.
//
// Column pass (lane < 24 = column k2): the inverse transform over k1 as three
// 8-point register transforms of the rows k1 = c mod 3 (fft32.h), Y[n] = sum_c
// w24^(c n) F_c[n mod 8], formed for the 16 kept rows only; they go to shared
// memory.  Row pass: lane 2r + h takes kept row r and the outputs n2 = 2m + h,
// the 12-point transforms of u[k] = (z[k] + (-1)^h z[k + 12]) w24^(k h): three
// 4-point ones of k = b mod 3, Out[m] = sum_b w12^(b m) G_b[m mod 4], for the
// nine m that either half keeps (the halves differ by one m when o is odd).  The
// 16 x 16 result leaves through shared memory, so that its stores are whole
// lines.
//
// 6000 keys of 256 sub-kernels, S 16: 1.38 ms against 2.21 with 32 points, 8-byte
// stores scattered over half sectors and 1,058 warp instructions per sub-kernel
// (852 now); error against 64 bits 3.8e-7 against 4.9e-7.
template <int S>
__global__ void __launch_bounds__(256, 3) k_aw_fftconv_f(
    const float2 *__restrict__ fa, const float2 *__restrict__ fw, int nW, int QQ,
    const int32_t *__restrict__ wi, float2 *__restrict__ out, int32_t *status) {
  using f32::cf;
  constexpr int N = 24, o = (S - 1) / 2, RP = N + 1;  // RP: pitch of the kept rows
  __shared__ float2 sfa[N][N];
  __shared__ float2 srow[8][16 * RP];  // per warp: the kept rows, then the result
  const int k = blockIdx.x;
  const int w = wi[k];
  if (w < 0 || w >= nW) {
    if (threadIdx.x == 0) atomicAdd(&status[ST_INDEX], 1);
    return;
  }
  if ((status[ST_RANGE] | status[ST_INDEX]) != 0) return;
  for (int t = threadIdx.x; t < N * N; t += blockDim.x)
    (&sfa[0][0])[t] = fa[(int64_t)k * (N * N) + t];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane >> 1, h = lane & 1, col = lane < N ? lane : N - 1;
  float2 *rows = srow[warp];
  auto mul = [](cf a, float2 b) {
    return cf{fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x)};
  };
  auto mac = [](cf s, cf a, float2 b) {  // s + a b
    return cf{fmaf(-a.y, b.y, fmaf(a.x, b.x, s.x)), fmaf(a.y, b.x, fmaf(a.x, b.y, s.y))};
  };
  for (int f = warp; f < QQ; f += 8) {
    const float2 *src = fw + ((int64_t)w * QQ + f) * (N * N) + col;
    {
      cf F[3][8];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const float2 x = __ldg(&src[(3 * a + c) * N]), y = sfa[3 * a + c][col];
          F[c][a] = mul(cf{y.x, y.y}, x);
        }
        f32::dft8(F[c], 1);  // inverse: exp(+2 pi i / 8); output q in slot out_slot(3, q)
      }
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        const int n = o + t, q = f32::out_slot(3, n & 7);
        const cf y = mac(mac(F[0][q], F[1][q], c_tw24[n]), F[2][q], c_tw24[2 * n % N]);
        if (lane < N) rows[t * RP + lane] = make_float2(y.x, y.y);
      }
    }
    __syncwarp();
    cf G[3][4];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int kk = 3 * a + b;
        const float2 z0 = rows[r * RP + kk], z1 = rows[r * RP + kk + 12];
        const cf sum = {z0.x + z1.x, z0.y + z1.y}, dif = {z0.x - z1.x, z0.y - z1.y};
        G[b][a] = h ? (kk ? mul(dif, c_tw24[kk]) : dif) : sum;
      }
      f32::dft4(G[b], 1);
    }
    __syncwarp();  // the rows have been read
    // out n2 = 2 m + h for m = m0 .. m0 + 8; this lane's eight from n2 >= o
    constexpr int m0 = o >> 1;
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      const int m = m0 + j;
      const cf v = mac(mac(G[0][m & 3], G[1][m & 3], c_tw24[2 * m % N]), G[2][m & 3],
                       c_tw24[4 * m % N]);
      const int n = 2 * m + h - o;
      if (n >= 0 && n < 16) rows[r * 17 + n] = make_float2(v.x, v.y);
    }
    __syncwarp();
    float2 *dst = out + ((int64_t)k * QQ + f) * 256;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int e = t * 32 + lane;
      dst[e] = rows[(e >> 4) * 17 + (e & 15)];
    }
    __syncwarp();  // rewritten by the next sub-kernel
  }
}

}  // namespace

bool aw_fft_supported(int SA, int S) { return SA == 16 && S >= 1 && S <= 16; }

// room for either precision (complex128 spectra)
size_t aw_fft_workspace_bytes(int nk, int nW, int Q) {
  return ((size_t)std::max(nk, 1) + (size_t)std::max(nW, 1) * Q * Q) * 1024 * sizeof(double2);
}

namespace {

// akern: [nk][16][16] A1 (*) A2 kernels in precision R, W: [nW][Q][Q][S][S] FP64;
// out: [nk][Q][Q][16][16] complex64 (R = float) or complex128 (R = double).
template <typename R>
int aw_fft_run(const typename Cx<R>::T *akern, int nk, const void *W, int nW, int Q, int S,
               const int32_t *wi, void *out, void *ws, size_t ws_bytes, int32_t *d_status,
               cudaStream_t st) {
  typedef typename Cx<R>::T T;
  CG_REQUIRE(aw_fft_supported(16, S), "FFT AW convolution needs 16 x 16 kernels, S <= 16");
  if (ws_bytes < aw_fft_workspace_bytes(nk, nW, Q))
    return set_error(CG_ERR_WORKSPACE, "AW FFT convolution workspace too small");
  constexpr int N = Cx<R>::N;
  T tw[N];
  for (int t = 0; t < N; ++t) {
    tw[t].x = (R)std::cos(2.0 * M_PI * t / N);
    tw[t].y = (R)std::sin(2.0 * M_PI * t / N);
  }
  if (sizeof(R) == 4)
    CG_CUDA(cudaMemcpyToSymbolAsync(c_tw24, tw, sizeof(tw), 0, cudaMemcpyHostToDevice, st));
  else
    CG_CUDA(cudaMemcpyToSymbolAsync(c_tw32d, tw, sizeof(tw), 0, cudaMemcpyHostToDevice, st));
  T *fa = (T *)ws;
  T *fw = fa + (size_t)nk * (N * N);
  const int64_t nwq = (int64_t)nW * Q * Q;
  const unsigned gb = (unsigned)std::min<int64_t>(((int64_t)nk * (N * N) + 255) / 256,
                                                  (int64_t)num_sms() * 16);
  k_pad_akern<T, N><<<gb, 256, 0, st>>>(akern, nk, fa);
  CG_LAUNCH("AW FFT pad A");
  const unsigned gw = (unsigned)std::min<int64_t>((nwq * (N * N) + 255) / 256,
                                                  (int64_t)num_sms() * 16);
  k_pad_w<T, N><<<gw, 256, 0, st>>>((const double2 *)W, nwq, S, fw);
  CG_LAUNCH("AW FFT pad W");
  cufftHandle plan;
  int rc;
  for (int pass = 0; pass < 2; ++pass) {
    const int batch = pass ? (int)nwq : nk;
    T *data = pass ? fw : fa;
    if ((rc = fft_plan(batch, N, N, sizeof(R) == 4 ? CUFFT_C2C : CUFFT_Z2Z, &plan))) return rc;
    if (cufftSetStream(plan, st) != CUFFT_SUCCESS)
      return set_error(CG_ERR_CUDA, "cufftSetStream failed");
    const cufftResult r =
        sizeof(R) == 4
            ? cufftExecC2C(plan, (cufftComplex *)data, (cufftComplex *)data, CUFFT_FORWARD)
            : cufftExecZ2Z(plan, (cufftDoubleComplex *)data, (cufftDoubleComplex *)data,
                           CUFFT_FORWARD);
    if (r != CUFFT_SUCCESS)
      return set_error(CG_ERR_CUDA, "cuFFT failed (AW FFT convolution)");
  }
  const int QQ = Q * Q;
#define CG_AW_FFT_CASE(SS)                                                                 \
  case SS:                                                                                 \
    if constexpr (sizeof(R) == 4)                                                          \
      k_aw_fftconv_f<SS><<<nk, 256, 0, st>>>(fa, fw, nW, QQ, wi, (float2 *)out, d_status);  \
    else                                                                                   \
      k_aw_fftconv<T, SS><<<nk, 256, 0, st>>>(fa, fw, nW, QQ, wi, (T *)out, d_status);     \
    break;
  switch (S) {
    CG_AW_FFT_CASE(1) CG_AW_FFT_CASE(2) CG_AW_FFT_CASE(3) CG_AW_FFT_CASE(4)
    CG_AW_FFT_CASE(5) CG_AW_FFT_CASE(6) CG_AW_FFT_CASE(7) CG_AW_FFT_CASE(8)
    CG_AW_FFT_CASE(9) CG_AW_FFT_CASE(10) CG_AW_FFT_CASE(11) CG_AW_FFT_CASE(12)
    CG_AW_FFT_CASE(13) CG_AW_FFT_CASE(14) CG_AW_FFT_CASE(15) CG_AW_FFT_CASE(16)
  }
#undef CG_AW_FFT_CASE
  CG_LAUNCH("AW FFT convolution");
  return CG_OK;
}

}  // namespace

int aw_fft_launch(const float2 *akern, int nk, const void *W, int nW, int Q, int S,
                  const int32_t *wi, void *out, int out_c64, void *ws, size_t ws_bytes,
                  int32_t *d_status, cudaStream_t st) {
  CG_REQUIRE(out_c64, "aw_fft_launch writes complex64 tables");
  return aw_fft_run<float>(akern, nk, W, nW, Q, S, wi, out, ws, ws_bytes, d_status, st);
}

// complex128 tables in FP64 throughout: FP64 spectra, products and transforms
int aw_fft_launch64(const double2 *akern, int nk, const void *W, int nW, int Q, int S,
                    const int32_t *wi, void *out, void *ws, size_t ws_bytes, int32_t *d_status,
                    cudaStream_t st) {
  return aw_fft_run<double>(akern, nk, W, nW, Q, S, wi, out, ws, ws_bytes, d_status, st);
}

}  // namespace cg
