// tg_march.h -- device pieces shared by the marching operator kernels
// (k_operator.cu, k_level1.cu): the modal arithmetic of the trilinear element on
// one or two packed element rows, and word copies to shared memory ahead of use.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "tg_df.h"
#include "tg_index.h"
#include "tg_internal.h"

namespace tg {

template <class T>
struct ModalT {
  T L0, L1, M0, M1, M02, LM2;  // per unit modulus; M02 = 2*M0, LM2 = L2 + 4*M2
};

// Storage (T) to compute (C) and back: the identity, except that a double is
// carried as a double-float (tg_df.h) by the residual-only instantiation.
template <class C>
__host__ __device__ __forceinline__ C cvt(double v) {
  return C(v);
}
template <>
__host__ __device__ __forceinline__ df cvt<df>(double v) {
  return df_from(v);
}
template <class C, class T>
__device__ __forceinline__ C load_c(T v) {
  return cvt<C>(v);
}
template <>
__device__ __forceinline__ df load_c<df, double>(double v) {
  return df_split(v);
}
template <>
__device__ __forceinline__ float load_c<float, float>(float v) {
  return v;
}
__device__ __forceinline__ double store_t(double v) { return v; }
__device__ __forceinline__ float store_t(float v) { return v; }
__device__ __forceinline__ double store_t(df v) { return df_to_double(v); }
__device__ __forceinline__ bool nonzero(float v) { return v != 0.0f; }
__device__ __forceinline__ bool nonzero(double v) { return v != 0.0; }
__device__ __forceinline__ bool nonzero(df v) { return df_nonzero(v); }
template <class C>
__host__ __device__ __forceinline__ C czero() {
  return cvt<C>(0.0);
}

template <class T>
ModalT<T> to_modal(const ModalConsts& c) {
  ModalT<T> m;
  m.L0 = cvt<T>(c.L[0]);
  m.L1 = cvt<T>(c.L[1]);
  m.M0 = cvt<T>(c.M[0]);
  m.M1 = cvt<T>(c.M[1]);
  m.M02 = cvt<T>(2.0 * c.M[0]);
  m.LM2 = cvt<T>(c.L[2] + 4.0 * c.M[2]);
  return m;
}

// a * b + c, spelled out so the modal arithmetic below maps to fused multiply-adds.
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }

// V: the type the element rows of a thread are carried in -- two rows packed in
// a float2 (Blackwell's paired FP32 instructions), or one row as float, double
// or double-float.
template <class V>
struct RowsOf;
template <>
struct RowsOf<float2> {
  using S = float;
  static constexpr int R = 2, kMaxWarps = 12;
};
template <>
struct RowsOf<float> {
  using S = float;
  static constexpr int R = 1, kMaxWarps = 12;
};
template <>
struct RowsOf<double> {
  using S = double;
  static constexpr int R = 1, kMaxWarps = 12;
};
template <>
struct RowsOf<df> {
  using S = df;
  static constexpr int R = 1, kMaxWarps = 12;
};

__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);  // a - b, one rounding
}
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vmad(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
template <class S>
__device__ __forceinline__ S vadd(S a, S b) { return a + b; }
template <class S>
__device__ __forceinline__ S vsub(S a, S b) { return a - b; }
template <class S>
__device__ __forceinline__ S vmul(S a, S b) { return a * b; }
template <class S>
__device__ __forceinline__ S vmad(S a, S b, S c) { return mad(a, b, c); }
template <class V, class S>
__device__ __forceinline__ V vset(S a) {
  if constexpr (RowsOf<V>::R == 2)
    return make_float2(a, a);
  else
    return a;
}

// The modes' stresses of unit-modulus constants times f, in place.  Index bits
// 1, 2, 4: the mode is linear in x, y, z.  Mode 0 (rigid translation) is not
// read, and has no stress.  M0 = 3 M1 merges the two gradient blocks that
// modes 3, 5 and 6 belong to: e.g. mode 3 of u_x gets M1 from T = {x} and 2 M1
// from T = {y}, and the three shears of those modes share one sum.
// This part: modes 1 to 6.
template <class V, class S>
__device__ __forceinline__ void modal_stress_12(const ModalT<S>& mc, V f, V (&ux)[8], V (&uy)[8],
                                                V (&uz)[8]) {
  const V m0 = vmul(vset<V>(mc.M0), f), m02 = vmul(vset<V>(mc.M02), f);
  const V l0 = vmul(vset<V>(mc.L0), f);
  {
    const V tr = vmul(l0, vadd(vadd(ux[1], uy[2]), uz[4]));
    ux[1] = vmad(m02, ux[1], tr);
    uy[2] = vmad(m02, uy[2], tr);
    uz[4] = vmad(m02, uz[4], tr);
    ux[2] = uy[1] = vmul(m0, vadd(uy[1], ux[2]));
    ux[4] = uz[1] = vmul(m0, vadd(uz[1], ux[4]));
    uy[4] = uz[2] = vmul(m0, vadd(uz[2], uy[4]));
  }
  const V l1 = vmul(vset<V>(mc.L1), f), m1 = vmul(vset<V>(mc.M1), f);
  {
    const V tx = vmul(l1, vadd(uy[3], uz[5]));
    const V ty = vmul(l1, vadd(ux[3], uz[6]));
    const V tz = vmul(l1, vadd(ux[5], uy[6]));
    ux[3] = vmad(m0, ux[3], ty);
    uy[3] = vmad(m0, uy[3], tx);
    ux[5] = vmad(m0, ux[5], tz);
    uz[5] = vmad(m0, uz[5], tx);
    uy[6] = vmad(m0, uy[6], tz);
    uz[6] = vmad(m0, uz[6], ty);
    const V sh = vmul(m1, vadd(vadd(uz[3], uy[5]), ux[6]));
    uz[3] = vmad(m1, uz[3], sh);
    uy[5] = vmad(m1, uy[5], sh);
    ux[6] = vmad(m1, ux[6], sh);
  }
}
template <class V, class S>
__device__ __forceinline__ void modal_stress(const ModalT<S>& mc, V f, V (&ux)[8], V (&uy)[8],
                                             V (&uz)[8]) {
  modal_stress_12<V, S>(mc, f, ux, uy, uz);
  const V lm2 = vmul(vset<V>(mc.LM2), f);
  ux[7] = vmul(lm2, ux[7]);
  uy[7] = vmul(lm2, uy[7]);
  uz[7] = vmul(lm2, uz[7]);
}

// xy-modes of a face from its node rows' own and right-neighbour values.
template <class V, class S>
__device__ __forceinline__ void face_modes(const S (&a)[RowsOf<V>::R + 1], const S (&b)[RowsOf<V>::R + 1],
                                           V (&F)[4]) {
  if constexpr (RowsOf<V>::R == 2) {
    const float2 a01 = make_float2(a[0], a[1]), b01 = make_float2(b[0], b[1]);
    const float2 s01 = vadd(b01, a01), d01 = vsub(b01, a01);
    const float2 s12 = make_float2(s01.y, b[2] + a[2]), d12 = make_float2(d01.y, b[2] - a[2]);
    F[0] = vadd(s12, s01);
    F[1] = vadd(d12, d01);
    F[2] = vsub(s12, s01);
    F[3] = vsub(d12, d01);
  } else {
    const S s0 = b[0] + a[0], d0 = b[0] - a[0], s1 = b[1] + a[1], d1 = b[1] - a[1];
    F[0] = s1 + s0;
    F[1] = d1 + d0;
    F[2] = s1 - s0;
    F[3] = d1 - d0;
  }
}

__device__ __forceinline__ float shfl_at(float v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ double shfl_at(double v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ df shfl_at(df v, int l) {
  return df(__shfl_sync(0xffffffffu, v.hi, l), __shfl_sync(0xffffffffu, v.lo, l));
}

constexpr int kDepth = 3;      // layers copied ahead
constexpr int kRowWords = 96;  // a copied row: 32 nodes x 3 components

__device__ __forceinline__ void copy_word(unsigned dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_word_or_zero(unsigned dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait_ahead() {  // all but the newest kDepth - 1 groups are in
  asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
}

}  // namespace tg
