// tg_sum3.h -- sums of products of FP32 values to beyond FP64's accuracy on the FP32
// pipe, which is 64 times wider than FP64's.  V is a float2 of two independent sums on
// the device (paired instructions), a float on the host.
#pragma once
#ifdef __CUDACC__
#include "tg_march.h"
#else
#include <cmath>
#endif
#include "tg_index.h"

namespace tg {

#ifdef __CUDACC__
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }
#else  // compiled without contraction
inline float vadd(float a, float b) { return a + b; }
inline float vsub(float a, float b) { return a - b; }
inline float vmul(float a, float b) { return a * b; }
inline float vmad(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float vneg(float a) { return -a; }
#endif

#ifdef __CUDACC__
#define TG_SUM3 __device__ __forceinline__
#else
#define TG_SUM3 inline
#endif

// An unevaluated sum h + m + l, the K-fold cascaded summation of Ogita, Rump and Oishi
// (2005) with K = 3: h the running FP32 sum, m the running sum of its
// rounding errors (and of the products'), both exact but for m's own errors, which l
// sums in FP32.  The terms' errors that are lost are l's roundings, about 2^-70 of the
// sum; converted to FP64 once, the total has the accuracy of the FP64 it is rounded to.
template <class V>
struct Sum3 {
  V h, m, l;
};

// s + e == a + b exactly (Knuth's TwoSum).
template <class V>
TG_SUM3 void exact_add(V& s, V& e, V a, V b) {
  s = vadd(a, b);
  const V t = vsub(s, a);
  e = vadd(vsub(a, vsub(s, t)), vsub(b, t));
}

// a += p + c.
template <class V>
TG_SUM3 void sum3_add(Sum3<V>& a, V p, V c) {
  V e1, e2, e3;
  exact_add(a.h, e1, a.h, p);
  exact_add(a.m, e2, a.m, e1);
  exact_add(a.m, e3, a.m, c);
  a.l = vadd(a.l, vadd(e2, e3));
}

// a += v v: the product is an FP32 value and its rounding error (one multiply-add),
// exactly.
template <class V>
TG_SUM3 void sum3_square(Sum3<V>& a, V v) {
  const V p = vmul(v, v);
  sum3_add(a, p, vmad(v, v, vneg(p)));
}

// a += d v v, exactly as four FP32 values: the product q of d and v and its error, each
// times v with its own error.
template <class V>
TG_SUM3 void sum3_weighted_square(Sum3<V>& a, V d, V v) {
  const V q = vmul(d, v), qe = vmad(d, v, vneg(q));
  const V p = vmul(q, v), pe = vmad(q, v, vneg(p));
  const V c = vmul(qe, v), ce = vmad(qe, v, vneg(c));
  V t, e;
  exact_add(t, e, pe, c);
  sum3_add(a, p, t);
  a.l = vadd(a.l, vadd(e, ce));
}

template <class V>
TG_SUM3 Sum3<V> sum3_join(const Sum3<V>& a, const Sum3<V>& b) {
  Sum3<V> s;
  V e1, e2, e3;
  exact_add(s.h, e1, a.h, b.h);
  exact_add(s.m, e2, a.m, b.m);
  exact_add(s.m, e3, s.m, e1);
  s.l = vadd(vadd(a.l, b.l), vadd(e2, e3));
  return s;
}

TG_HD double sum3_total(float h, float m, float l) { return double(h) + (double(m) + double(l)); }

}  // namespace tg
