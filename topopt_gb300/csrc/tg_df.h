// tg_df.h -- "double-float": a value carried as an unevaluated sum hi + lo of
// two FP32 numbers (|lo| <= ulp(hi)/2), about 48 significant bits, computed on
// the FP32 pipe.  GB300 issues FP32 at roughly 58x its FP64 rate, so an FP64-
// accuracy residual in double-float arithmetic costs a fraction of the native
// FP64 one.
//
// The algorithms are the classical error-free transformations: Knuth's TwoSum
// and Dekker's Fast2Sum for addition, the FMA-based exact product for
// multiplication, with the renormalisations of the double-double arithmetic of
// Hida, Li and Bailey ("Algorithms for quad-double precision floating point
// arithmetic", 2001), here on FP32 pairs.  Every step is an explicitly rounded
// intrinsic so the compiler can neither fuse nor reorder it.
#pragma once
#include <cuda_runtime.h>

namespace tg {

struct df {
  float hi, lo;
  df() = default;
  __host__ __device__ __forceinline__ constexpr df(float h, float l) : hi(h), lo(l) {}
};

// The nearest double-float to a double: hi = rn(v), lo = rn(v - hi).
__host__ __device__ __forceinline__ df df_from(double v) {
  const float h = float(v);
  return df(h, float(v - double(h)));
}
#ifdef __CUDACC__
// The same on the device by integer operations.  The two conversions and the
// subtraction of df_from are four FP64-pipe instructions, 64 cycles each on a
// warp's scheduler, and they were most of the double-float residual's time;
// these fifteen run at the integer rate (256x128x128 residual with this and the
// shared transforms: 1,080 -> 500 us).  hi is the mantissa rounded to 24 bits
// (ties away from zero), lo the signed remainder of its low 29 bits, exactly
// scaled; magnitudes outside [2^-74, 2^127) -- where lo's scale or hi would leave
// FP32's normal range -- go through df_from, zeros apart.
__device__ __forceinline__ df df_split(double v) {
  const unsigned hb = unsigned(__double2hiint(v)), lb = unsigned(__double2loint(v));
  const unsigned e = (hb >> 20) & 0x7ffu;
  if (e - 949u <= 200u) {
    const unsigned rl = lb + 0x10000000u, rh = hb + (rl < lb ? 1u : 0u);
    const unsigned sign = hb & 0x80000000u;
    // Exponent rebiased by -896 and the 23 mantissa bits, modulo 2^31.
    const unsigned h = ((__funnelshift_l(rl, rh, 3) + 0x40000000u) & 0x7fffffffu) | sign;
    const int rem = int(lb << 3) >> 3;
    const unsigned sc = (((hb << 3) - (436u << 23)) & 0x7f800000u) | sign;  // 2^(e - 1075)
    return df(__uint_as_float(h), __fmul_rn(__int2float_rn(rem), __uint_as_float(sc)));
  }
  if (e == 0u) return df(0.0f, 0.0f);
  return df_from(v);
}
// An FP32 value as FP64: by integer operations where it is normal or zero, since the
// conversion is an FP64-pipe instruction like the multiply-add it feeds.
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) {
  const unsigned u = __float_as_uint(v), m = u & 0x7fffffffu, sign = u & 0x80000000u;
  if (m == 0u) return __hiloint2double(int(sign), 0);
  if (m - 0x00800000u >= 0x7f000000u) return double(v);  // denormal, infinite, NaN
  return __hiloint2double(int(sign | ((m >> 3) + (896u << 20))), int(u << 29));
}
#endif
__host__ __device__ __forceinline__ double df_to_double(df a) {
  return double(a.hi) + double(a.lo);
}

// Knuth's TwoSum: s + e == a + b exactly.
__device__ __forceinline__ df two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return df(s, e);
}
// Fast2Sum, valid when |a| >= |b| (or a == 0).
__device__ __forceinline__ df quick_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return df(s, __fsub_rn(b, __fsub_rn(s, a)));
}

// Addition: TwoSum of the high parts, the low parts and the exact error summed
// in FP32, one renormalisation (the "sloppy" double-double add).  Its error is
// bounded by about 2^-47 (|a| + |b|) -- relative to the operands, not to the
// sum, so a cancellation keeps the operands' absolute accuracy, which is what a
// residual b - A x needs -- at about half the operations of the variant whose
// error is relative to the sum.
__device__ __forceinline__ df operator+(df a, df b) {
  const df s = two_sum(a.hi, b.hi);
  return quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ df operator-(df a) { return df(-a.hi, -a.lo); }
__device__ __forceinline__ df operator-(df a, df b) { return a + (-b); }
__device__ __forceinline__ df operator*(df a, df b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);  // the exact rounding error of a.hi * b.hi
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  return quick_two_sum(p, e);
}
__device__ __forceinline__ df mad(df a, df b, df c) { return a * b + c; }
__device__ __forceinline__ bool df_nonzero(df a) { return a.hi != 0.0f || a.lo != 0.0f; }

}  // namespace tg
