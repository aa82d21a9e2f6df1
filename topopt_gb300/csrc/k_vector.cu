// k_vector.cu -- PCG vector updates and deterministic FP64 reductions.
//
// Reference counterpart: the dot products and AXPYs of mf_cg_solve and mf_mgpcg
// (core/src/fea/matfree.cpp:1006-1060, core/src/fea/multigrid.cpp:1287-1310).
// Every reduction runs on a fixed grid of kRedBlocks x 256 threads with a
// fixed-shape tree, so the same inputs give the same bits on every run; the PCG
// scalars (alpha, beta) are read from device memory, never round-tripped through
// the host.  These kernels are HBM-bound streaming passes.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "tg_internal.h"
#include "tg_launch.h"
#include "tg_reduce.h"

namespace tg {

namespace {
constexpr int kThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Deterministic block sum (fixed tree), result valid in thread 0.
__device__ __forceinline__ double block_sum256(double v) {
  __shared__ double red[kThreads / 32];
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double s = 0.0;
  if (wid == 0) {
    s = lane < kThreads / 32 ? red[lane] : 0.0;
    s = warp_sum(s);
  }
  __syncthreads();
  return s;
}

__device__ __forceinline__ double block_max256(double v) {
  __shared__ double red[kThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double s = 0.0;
  if (wid == 0) {
    s = lane < kThreads / 32 ? red[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = fmax(s, __shfl_down_sync(0xffffffffu, s, o));
  }
  __syncthreads();
  return s;
}

// FP32 vectors are summed in FP32 along each thread's grid-stride run (a few
// dozen terms) and in FP64 across threads and blocks: on GB300 an FP64 multiply
// per element would make these streaming kernels FP64-pipe-bound.
template <class T>
__global__ void k_dot(const T* __restrict__ a, const T* __restrict__ b, int64_t n, SumOut o) {
  T t = T(0);
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    t += a[i] * b[i];
  grid_sum(double(t), o, int(blockIdx.x), int(gridDim.x));
}

// One block: out = sum of n partials, fixed order.
__global__ void k_sum_partials(const double* __restrict__ part, int n, double* __restrict__ out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += kThreads) s += part[i];
  s = block_sum256(s);
  if (threadIdx.x == 0) *out = s;
}

__global__ void k_max_partials(const double* __restrict__ part, int n, double* __restrict__ out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += kThreads) s = fmax(s, part[i]);
  s = block_max256(s);
  if (threadIdx.x == 0) *out = s;
}

// A scalar of the step (an FP64 division) by one warp for the whole block: each warp
// that divides takes the SM's FP64 units ten or more times for 19 cycles, 3 us of a
// kernel with 32 warps on every SM.
template <class F>
__device__ __forceinline__ double block_scalar(const F& f) {
  __shared__ double s;
  if (threadIdx.x < 32) {
    const double v = f();
    if (threadIdx.x == 0) s = v;
  }
  __syncthreads();
  return s;
}

// x += alpha p; r -= alpha Ap with alpha = rz / pAp; sum of r.r (FP64).  With x0
// set, also x0 = omega invdiag .* r.  The FP64 PCG's update; the FP32 inner PCG
// runs it as two kernels below.
// NEXT: 0 as it is, 1 with x0, 2 with x0 and r.x0 (a template, since an FP64 product that
// nobody reads still takes its 19 cycles of the SM).
template <int NEXT>
__global__ void k_cg_update_xr(double* x, double* r,
                               const double* p, const double* ap,
                               const double* rz, const double* pap,
                               int64_t n, const double* invdiag, double omega,
                               double* x0, SumOut o, SumOut oz) {
  behind_previous();
  // A non-positive or non-finite pAp is a breakdown the host reports; leave the
  // iterate untouched so the last good x survives.
  const double a = block_scalar([&] {
    const double pp = *pap;
    return (pp > 0.0 && isfinite(pp)) ? *rz / pp : 0.0;
  });
  double t = 0.0, tz = 0.0;
  constexpr bool next = NEXT > 0;
  auto one = [&](double& xv, double pv, double& rv, double qv, double dv) {
    xv += a * pv;
    rv -= a * qv;
    t += rv * rv;
    const double zv = next ? omega * dv * rv : 0.0;
    if constexpr (NEXT == 2) tz += rv * zv;
    return zv;
  };
  // Pairs, two a round: all of a round's loads before its first store, since the
  // compiler may not move them past one.
  const int64_t n2 = n >> 1, step = int64_t(gridDim.x) * kThreads;
  double2 *x2 = reinterpret_cast<double2*>(x), *r2 = reinterpret_cast<double2*>(r),
          *z2 = reinterpret_cast<double2*>(x0);
  const double2 *p2 = reinterpret_cast<const double2*>(p),
                *q2 = reinterpret_cast<const double2*>(ap),
                *d2 = reinterpret_cast<const double2*>(invdiag);
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n2; i += 2 * step) {
    const int64_t j[2] = {i, i + step};
    double2 xv[2], pv[2], rv[2], qv[2], dv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (j[u] >= n2) continue;
      xv[u] = x2[j[u]];
      pv[u] = p2[j[u]];
      rv[u] = r2[j[u]];
      qv[u] = q2[j[u]];
      dv[u] = next ? d2[j[u]] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (j[u] >= n2) continue;
      double2 zv;
      zv.x = one(xv[u].x, pv[u].x, rv[u].x, qv[u].x, dv[u].x);
      zv.y = one(xv[u].y, pv[u].y, rv[u].y, qv[u].y, dv[u].y);
      x2[j[u]] = xv[u];
      r2[j[u]] = rv[u];
      if (next) z2[j[u]] = zv;
    }
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    double xv = x[n - 1], rv = r[n - 1];
    const double zv = one(xv, p[n - 1], rv, ap[n - 1], next ? invdiag[n - 1] : 0.0);
    x[n - 1] = xv;
    r[n - 1] = rv;
    if (next) x0[n - 1] = zv;
  }
  if constexpr (NEXT == 2) grid_sum(tz, oz, int(blockIdx.x), int(gridDim.x));
  grid_sum(t, o, int(blockIdx.x), int(gridDim.x));
}

// The FP32 inner PCG's update in two kernels (alpha as k_cg_update_xr forms it,
// 16-byte vector accesses): r -= alpha Ap with partial r.r, and x += alpha p,
// which the solver runs later, beside the next V-cycle's coarse levels
// (nothing in the loop reads x).
__device__ __forceinline__ float cg_alpha_f(const double* rz, const double* pap) {
  return float(block_scalar([&] {
    const double pp = *pap;
    return (pp > 0.0 && isfinite(pp)) ? *rz / pp : 0.0;
  }));
}
// With x0 set, also x0 = omega invdiag .* r (the next V-cycle's first smoothing
// sweep from zero, as k_jacobi_first computes it).
__global__ void k_cg_update_r_f(float* r, const float* ap,
                                const double* rz, const double* pap,
                                int64_t n, const float* invdiag, float omega,
                                float* x0, SumOut o) {
  behind_previous();
  const float af = cg_alpha_f(rz, pap);
  const int64_t n4 = n >> 2;
  float4* r4 = reinterpret_cast<float4*>(r);
  const float4* a4 = reinterpret_cast<const float4*>(ap);
  const float4* d4 = reinterpret_cast<const float4*>(invdiag);
  float4* x4 = reinterpret_cast<float4*>(x0);
  float tf = 0.0f;
  const int64_t step = int64_t(gridDim.x) * kThreads;
  // Two a round: all of a round's loads before its first store, since the compiler may
  // not move them past one.
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n4; i += 2 * step) {
    const int64_t j[2] = {i, i + step};
    float4 rv[2], qv[2], dv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (j[u] >= n4) continue;
      rv[u] = r4[j[u]];
      qv[u] = a4[j[u]];
      dv[u] = x0 != nullptr ? d4[j[u]] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (j[u] >= n4) continue;
      float4& v = rv[u];
      v.x -= af * qv[u].x; v.y -= af * qv[u].y; v.z -= af * qv[u].z; v.w -= af * qv[u].w;
      r4[j[u]] = v;
      tf += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
      if (x0 != nullptr)
        x4[j[u]] = make_float4(omega * dv[u].x * v.x, omega * dv[u].y * v.y,
                               omega * dv[u].z * v.z, omega * dv[u].w * v.w);
    }
  }
  float t = tf;
  for (int64_t i = (n4 << 2) + blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads) {
    const float ri = r[i] - af * ap[i];
    r[i] = ri;
    t += ri * ri;
    if (x0 != nullptr) x0[i] = omega * invdiag[i] * ri;
  }
  grid_sum(double(t), o, int(blockIdx.x), int(gridDim.x));
}
__global__ void k_cg_update_x_f(float* __restrict__ x, const float* __restrict__ p,
                                const double* __restrict__ rz, const double* __restrict__ pap,
                                int64_t n) {
  const float af = cg_alpha_f(rz, pap);
  const int64_t n4 = n >> 2;
  float4* x4 = reinterpret_cast<float4*>(x);
  const float4* p4 = reinterpret_cast<const float4*>(p);
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n4;
       i += int64_t(gridDim.x) * kThreads) {
    float4 xv = x4[i];
    const float4 pv = p4[i];
    xv.x += af * pv.x; xv.y += af * pv.y; xv.z += af * pv.z; xv.w += af * pv.w;
    x4[i] = xv;
  }
  for (int64_t i = (n4 << 2) + blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    x[i] += af * p[i];
}

// z = invdiag .* r (Jacobi preconditioner); sum of r.z.
__global__ void k_scale_mask(double* __restrict__ z, const double* __restrict__ r,
                             const double* __restrict__ invdiag, int64_t n, SumOut o) {
  double s = 0.0;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads) {
    const double zi = invdiag[i] * r[i];
    z[i] = zi;
    s += r[i] * zi;
  }
  grid_sum(s, o, int(blockIdx.x), int(gridDim.x));
}

// p = z + beta p, beta = rz_new / rz_old.
template <class T>
__global__ void k_cg_update_p(T* p, const T* z,
                              const double* rz_new, const double* rz_old,
                              int64_t n) {
  behind_previous();
  const T beta = T(block_scalar([&] { return *rz_new / *rz_old; }));
  // 16 bytes at a time, two a round, as in the updates above.
  using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  constexpr int kPer = int(sizeof(V) / sizeof(T));
  const int64_t nv = n / kPer, step = int64_t(gridDim.x) * kThreads;
  V* pw = reinterpret_cast<V*>(p);
  const V* zw = reinterpret_cast<const V*>(z);
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < nv; i += 2 * step) {
    const int64_t j[2] = {i, i + step};
    V pv[2], zv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (j[u] >= nv) continue;
      pv[u] = pw[j[u]];
      zv[u] = zw[j[u]];
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (j[u] >= nv) continue;
      T *a = reinterpret_cast<T*>(pv + u), *b = reinterpret_cast<T*>(zv + u);
#pragma unroll
      for (int k = 0; k < kPer; ++k) a[k] = b[k] + beta * a[k];
      pw[j[u]] = pv[u];
    }
  }
  for (int64_t i = nv * kPer + blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += step)
    p[i] = z[i] + beta * p[i];
}

__global__ void k_scale_d2f(float* __restrict__ d, const double* __restrict__ s,
                            const double* __restrict__ nrm2, int64_t n) {
  const double inv = *nrm2 > 0.0 ? 1.0 / sqrt(*nrm2) : 0.0;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    d[i] = float(s[i] * inv);
}

// y += sqrt(*nrm2) * x (undo the scaling while accumulating in double).
__global__ void k_axpy_scaled_f2d(double* __restrict__ y, const float* __restrict__ x,
                                  const double* __restrict__ nrm2, int64_t n) {
  const double sc = sqrt(*nrm2);
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    y[i] += sc * double(x[i]);
}

__global__ void k_scatter(double* __restrict__ v, const int64_t* __restrict__ at,
                          const double* __restrict__ val, int64_t n) {
  const int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x;
  if (i < n) v[at[i]] = val[i];
}

template <class T>
__global__ void k_fill(T* __restrict__ a, T v, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    a[i] = v;
}

__global__ void k_copy_d2f(float* __restrict__ d, const double* __restrict__ s, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    d[i] = float(s[i]);
}

__global__ void k_axpy_f2d(double* __restrict__ y, const float* __restrict__ x, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    y[i] += double(x[i]);
}

__global__ void k_sub_mask(double* __restrict__ r, const double* __restrict__ b,
                           const double* __restrict__ ax, const uint8_t* __restrict__ kept,
                           int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    r[i] = kept[i] ? b[i] - ax[i] : 0.0;
}

// u = kept ? x : alt (x is also allowed to be null -> 0 on kept DOFs).
__global__ void k_mask_select(double* __restrict__ u, const double* __restrict__ x,
                              const double* __restrict__ alt, const uint8_t* __restrict__ kept,
                              int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    u[i] = kept[i] ? (x ? x[i] : 0.0) : (alt ? alt[i] : 0.0);
}

__global__ void k_absdiff_max(const double* __restrict__ a, const double* __restrict__ b,
                              int64_t n, double* __restrict__ part) {
  double s = 0.0;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    s = fmax(s, fabs(a[i] - b[i]));
  s = block_max256(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// FMA throughput probe: 8 independent register-resident FMA chains per thread.
template <class T>
__global__ void k_fma_probe(T* __restrict__ out, int iters, T b, T c) {
  T a0 = T(threadIdx.x), a1 = a0 + T(1), a2 = a0 + T(2), a3 = a0 + T(3);
  T a4 = a0 + T(4), a5 = a0 + T(5), a6 = a0 + T(6), a7 = a0 + T(7);
  for (int i = 0; i < iters; ++i) {
    a0 = fma(a0, b, c); a1 = fma(a1, b, c); a2 = fma(a2, b, c); a3 = fma(a3, b, c);
    a4 = fma(a4, b, c); a5 = fma(a5, b, c); a6 = fma(a6, b, c); a7 = fma(a7, b, c);
  }
  const T s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == T(-1.2345)) out[blockIdx.x] = s;  // keeps the chains live
}

int stream_blocks(int64_t n) {
  const int64_t b = (n + kThreads - 1) / kThreads;
  return int(b < kRedBlocks ? (b > 0 ? b : 1) : kRedBlocks);
}
}  // namespace

double fma_probe_tflops(bool fp64) {
  const int blocks = 152 * 8, threads = 256;
  const int iters = fp64 ? 4096 : 262144;
  void* out = nullptr;
  TG_CUDA(cudaMalloc(&out, blocks * sizeof(double)));
  cudaEvent_t a, b;
  TG_CUDA(cudaEventCreate(&a));
  TG_CUDA(cudaEventCreate(&b));
  double best = 0.0;
  for (int rep = 0; rep < 3; ++rep) {
    TG_CUDA(cudaEventRecord(a));
    if (fp64)
      k_fma_probe<double><<<blocks, threads>>>(static_cast<double*>(out), iters, 0.999999, 1e-7);
    else
      k_fma_probe<float><<<blocks, threads>>>(static_cast<float*>(out), iters, 0.999999f, 1e-7f);
    TG_LAUNCH_CHECK();
    TG_CUDA(cudaEventRecord(b));
    TG_CUDA(cudaEventSynchronize(b));
    float ms = 0.0f;
    TG_CUDA(cudaEventElapsedTime(&ms, a, b));
    const double flops = 2.0 * 8.0 * double(iters) * blocks * threads;
    best = std::max(best, flops / (double(ms) * 1e-3) / 1e12);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(out);
  return best;
}

// An element a thread up to a CTA per SM -- a small vector's FP64 sums and updates are
// spread over the SMs' units (6,075 entries in 24 CTAs instead of 6: a 24x8x8 solve
// 8.07 -> 7.92 ms) -- then four and more a thread up to the full grid, which the last
// one's sum has to wait for.
int red_blocks(int64_t n) {
  const int64_t one = (n + kThreads - 1) / kThreads, four = (n + 4 * kThreads - 1) / (4 * kThreads);
  return int(std::min<int64_t>(
      kRedBlocks, std::max<int64_t>({int64_t(1), std::min<int64_t>(one, 152), four})));
}

void launch_dot(const double* a, const double* b, int64_t n, const SumOut& o, cudaStream_t s) {
  k_dot<double><<<red_blocks(n), kThreads, 0, s>>>(a, b, n, o);
  TG_LAUNCH_CHECK();
}

void launch_dot_f(const float* a, const float* b, int64_t n, const SumOut& o, cudaStream_t s) {
  // One term a thread as far as the grid goes (155,648): a thread's run is FP32.
  k_dot<float><<<stream_blocks(n), kThreads, 0, s>>>(a, b, n, o);
  TG_LAUNCH_CHECK();
}

void launch_sum_partials(const double* part, int n, double* out, cudaStream_t s) {
  k_sum_partials<<<1, kThreads, 0, s>>>(part, n, out);
  TG_LAUNCH_CHECK();
}

void launch_cg_update_xr(double* x, double* r, const double* p, const double* ap,
                         const double* rz, const double* pap, int64_t n, const SumOut& rr,
                         cudaStream_t s, const double* invdiag, double omega, double* x0,
                         const SumOut& r_x0) {
  auto kernel = x0 == nullptr          ? k_cg_update_xr<0>
                : r_x0.part == nullptr ? k_cg_update_xr<1>
                                       : k_cg_update_xr<2>;
  launch_behind(kernel, red_blocks(n), kThreads, 0, s, x, r, p, ap, rz, pap, n, invdiag, omega, x0,
                rr, r_x0);
  TG_LAUNCH_CHECK();
}

void launch_cg_update_r_f(float* r, const float* ap, const double* rz, const double* pap,
                          int64_t n, const SumOut& rr, cudaStream_t s, const float* invdiag,
                          float omega, float* x0) {
  launch_behind(k_cg_update_r_f, red_blocks(n), kThreads, 0, s, r, ap, rz, pap, n, invdiag, omega,
                x0, rr);
  TG_LAUNCH_CHECK();
}
void launch_cg_update_x_f(float* x, const float* p, const double* rz, const double* pap,
                          int64_t n, cudaStream_t s) {
  k_cg_update_x_f<<<red_blocks(n), kThreads, 0, s>>>(x, p, rz, pap, n);
  TG_LAUNCH_CHECK();
}

void launch_scale_mask(double* z, const double* r, const double* invdiag, int64_t n,
                       const SumOut& rz, cudaStream_t s) {
  k_scale_mask<<<red_blocks(n), kThreads, 0, s>>>(z, r, invdiag, n, rz);
  TG_LAUNCH_CHECK();
}

template <class T>
void launch_cg_update_p(T* p, const T* z, const double* rz_new, const double* rz_old, int64_t n,
                        cudaStream_t s) {
  launch_behind(k_cg_update_p<T>, red_blocks(n), kThreads, 0, s, p, z, rz_new, rz_old, n);
  TG_LAUNCH_CHECK();
}
template void launch_cg_update_p<double>(double*, const double*, const double*, const double*,
                                         int64_t, cudaStream_t);
template void launch_cg_update_p<float>(float*, const float*, const double*, const double*,
                                        int64_t, cudaStream_t);

void launch_scale_d2f(float* dst, const double* src, const double* nrm2, int64_t n,
                      cudaStream_t s) {
  k_scale_d2f<<<stream_blocks(n), kThreads, 0, s>>>(dst, src, nrm2, n);
  TG_LAUNCH_CHECK();
}

void launch_axpy_scaled_f2d(double* y, const float* x, const double* nrm2, int64_t n,
                            cudaStream_t s) {
  k_axpy_scaled_f2d<<<stream_blocks(n), kThreads, 0, s>>>(y, x, nrm2, n);
  TG_LAUNCH_CHECK();
}

template <class T>
void launch_fill(T* a, T v, int64_t n, cudaStream_t s) {
  k_fill<T><<<stream_blocks(n), kThreads, 0, s>>>(a, v, n);
  TG_LAUNCH_CHECK();
}
void launch_scatter(double* v, const int64_t* at, const double* val, int64_t n, cudaStream_t s) {
  k_scatter<<<unsigned((n + kThreads - 1) / kThreads), kThreads, 0, s>>>(v, at, val, n);
  TG_LAUNCH_CHECK();
}
template void launch_fill<double>(double*, double, int64_t, cudaStream_t);
template void launch_fill<float>(float*, float, int64_t, cudaStream_t);
template void launch_fill<uint8_t>(uint8_t*, uint8_t, int64_t, cudaStream_t);

void launch_copy_d2f(float* dst, const double* src, int64_t n, cudaStream_t s) {
  k_copy_d2f<<<stream_blocks(n), kThreads, 0, s>>>(dst, src, n);
  TG_LAUNCH_CHECK();
}

void launch_axpy_f2d(double* y, const float* x, int64_t n, cudaStream_t s) {
  k_axpy_f2d<<<stream_blocks(n), kThreads, 0, s>>>(y, x, n);
  TG_LAUNCH_CHECK();
}

void launch_sub_mask(double* r, const double* b, const double* ax, const uint8_t* kept, int64_t n,
                     cudaStream_t s) {
  k_sub_mask<<<stream_blocks(n), kThreads, 0, s>>>(r, b, ax, kept, n);
  TG_LAUNCH_CHECK();
}

void launch_mask_select(double* u, const double* x, const double* alt, const uint8_t* kept,
                        int64_t n, cudaStream_t s) {
  k_mask_select<<<stream_blocks(n), kThreads, 0, s>>>(u, x, alt, kept, n);
  TG_LAUNCH_CHECK();
}

void launch_absdiff_max(const double* a, const double* b, int64_t n, double* part, double* out,
                        cudaStream_t s) {
  k_absdiff_max<<<kRedBlocks, kThreads, 0, s>>>(a, b, n, part);
  TG_LAUNCH_CHECK();
  k_max_partials<<<1, kThreads, 0, s>>>(part, kRedBlocks, out);
  TG_LAUNCH_CHECK();
}

}  // namespace tg
