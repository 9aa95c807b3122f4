// FP64 <-> double-float conversions by integer operations.
//
// GB300 executes FP64 arithmetic, including the F64 <-> F32 conversions, at
// a small fraction of its FP32 and integer rates, so a pipeline that keeps
// complex128 data as double-float pairs (hi + lo floats) spends most of its
// conversion time on the FP64 pipe.  These helpers compute the same results
// from the IEEE-754 bit patterns with 32/64-bit integer operations:
//
//   split(v) = (hi, lo) with hi = RN_float(v) (round to nearest, ties to
//              even, on the bit pattern: the 23 mantissa bits shifted down as
//              one word, plus one where the 29 dropped bits say so) and lo =
//              RN_float(v - hi) (v - hi is the dropped bits less the carry,
//              an integer times the ulp of v's binade; one int -> float
//              rounding);
//   join(hi, lo) = RN_double(hi + lo): hi's double pattern plus lo as an
//              integer in units of its last place (RN_int, ties to even: hi
//              is an even multiple of that unit, so ties fall as the 53-bit
//              sum's do).
//
// Both are bit-identical to the FP64 forms ((float)v, (float)(v - (double)hi)
// and (double)hi + (double)lo) wherever the fast path applies: |v| in
// [2^-74, 2^127) for split; for join |hi| in [2^-75, 2^127], |lo| at most half
// a unit of hi's last place, and not a power of two with lo of the other sign
// (the sum is then in the binade below, with half the unit).  Zeros are
// handled by bits; anything else takes the FP64 form, in a function of its
// own: inlined, the compiler evaluated it for every element beside the fast
// path and selected, and the FP64 pipe bounded the column transforms (45 % of
// its peak; with the 64-bit alignment and rounding that join did before, 187
// of a column element's 560 instructions).
//
// Plain C++ shared by the device code and a host test (no CUDA types).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define CG_DF_HD __host__ __device__ __forceinline__
#define CG_DF_SLOW static __host__ __device__ __noinline__
#else
#define CG_DF_HD inline
#define CG_DF_SLOW static inline
#endif

namespace cg {

CG_DF_HD uint64_t f64_bits(double v) {
  uint64_t u;
  memcpy(&u, &v, 8);
  return u;
}
CG_DF_HD double f64_from(uint64_t u) {
  double v;
  memcpy(&v, &u, 8);
  return v;
}
CG_DF_HD uint32_t f32_bits(float v) {
  uint32_t u;
  memcpy(&u, &v, 4);
  return u;
}
CG_DF_HD float f32_from(uint32_t u) {
  float v;
  memcpy(&v, &u, 4);
  return v;
}

// round to the nearest integer, ties to even (|v| < 2^31)
CG_DF_HD int32_t f32_to_int_rn(float v) {
#if defined(__CUDA_ARCH__)
  return __float2int_rn(v);
#else
  return (int32_t)lrintf(v);
#endif
}

CG_DF_SLOW uint64_t f64_split_slow(double v) {  // hi in the upper word, lo in the lower
  const float hi = (float)v, lo = (float)(v - (double)hi);
  return ((uint64_t)f32_bits(hi) << 32) | f32_bits(lo);
}

CG_DF_SLOW double f64_join_slow(float hi, float lo) { return (double)hi + (double)lo; }

// v -> (hi, lo)
CG_DF_HD void f64_split(double v, float &hi, float &lo) {
  const uint64_t b = f64_bits(v);
  const uint32_t w1 = (uint32_t)(b >> 32), w0 = (uint32_t)b;
  const uint32_t sgn = w1 & 0x80000000u;
  const uint32_t E = (w1 >> 20) & 0x7FFu;
  if (E - 949u > 200u) {  // outside [949, 1149]: zero, or beyond what the bit path covers
    if (((w1 << 1) | w0) == 0) {
      hi = f32_from(sgn);
      lo = 0.0f;
      return;
    }
    const uint64_t r = f64_split_slow(v);
    hi = f32_from((uint32_t)(r >> 32));
    lo = f32_from((uint32_t)r);
    return;
  }
  // exponent and mantissa truncated to a float's, then rounded to nearest even
  // (a carry out of the mantissa moves into the exponent)
  const uint32_t t = (((w1 << 3) | (w0 >> 29)) & 0x7FFFFFFFu);  // exponent mod 256 so far
  const uint32_t tr = t - (896u << 23);
  const uint32_t r = w0 & 0x1FFFFFFFu;
  const uint32_t up = (r + 0x0FFFFFFFu + (tr & 1u)) >> 29;
  hi = f32_from(((tr & 0x7FFFFFFFu) + up) | sgn);
  const int32_t d = (int32_t)(r - (up << 29));  // |d| <= 2^28: (|v| - |hi|) / ulp
  // ulp of v's binade, 2^(E - 1075), with v's sign; RN(d) scaled exactly, +0 if d = 0
  const float p = f32_from(((E - 948u) << 23) | sgn);
  lo = d == 0 ? 0.0f : (float)d * p;
}

// (hi, lo) -> RN(hi + lo)
CG_DF_HD double f64_join(float hi, float lo) {
  const uint32_t hb = f32_bits(hi), ha = hb & 0x7FFFFFFFu;
  const uint32_t eh = ha >> 23;
  // lo in units of hi's last double place, 2^(eh - 179)
  const float u = eh >= 52u && eh < 255u ? lo * f32_from((306u - eh) << 23) : 1e30f;
  // (a NaN fails the comparison)
  const bool fast = fabsf(u) <= 268435456.0f;
  const float v = hb >> 31 ? -u : u;  // along hi's sign
  if (!fast || ((ha & 0x7FFFFFu) == 0 && v < 0.0f)) {
    if ((ha | (f32_bits(lo) & 0x7FFFFFFFu)) == 0)  // +-0
      return f64_from((uint64_t)(hb & f32_bits(lo) & 0x80000000u) << 32);
    return f64_join_slow(hi, lo);
  }
  const uint64_t m = (((uint64_t)ha << 29) + ((uint64_t)896 << 52)) +
                     (uint64_t)(int64_t)f32_to_int_rn(v);
  return f64_from(m | ((uint64_t)(hb & 0x80000000u) << 32));
}

}  // namespace cg
