// k_level1.cu -- the level-1 Galerkin operator of the FP32 V-cycle, applied
// without an assembled matrix.
//
// Reference counterpart: the level-1 operator A1 = P0^T A0 P0 of the matrix-free
// hierarchy (core/src/fea/multigrid.cpp:1413-1446, galerkin_a1_from_prolong
// :1543-1899), applied by v_cycle's jacobi_sweep and residual (:780-817) as an
// Eigen SpMV.
//
// A coarse element's matrix is the sum over its eight children c of
// W_c^T (E_c Ke) W_c.  In the modal basis W_c is almost diagonal: on the child
// with corner signs s, the parent's coordinate is xi = (s + eta) / 2, so with
// a[S] = m[S] / 2^|S| the child's mode T is
//     m_c[T] = sum over S containing T of a[S] prod of s_i over S \ T,
// and the parent's stresses are the transpose of that applied to the children's.
// Over the eight children a component has 19 distinct child modes (a mode linear
// in k axes has 2^(3-k) variants), reached by 20 additions; the stress of a
// child is k_operator.cu's, with the child's modulus.  About 400 operations per
// coarse element, most of them on the two z-children packed in paired FP32
// instructions.  The eight dense 24x24 blocks G_c = W_c^T Ke W_c are 4,608
// multiply-adds; on the tensor cores (three TF32 products for FP32 accuracy) they
// were bound by each batch's chain stage -> MMA -> commit -> read back: 66 us on
// the 256x128x128 cantilever's level 1 and 43-53 us on small ones (24x8x8 to
// 128x64x64); this kernel with its pre-pass takes 40 us there, and 6-17 us on
// those.  The assembled stencil takes 105 us there and 16.5 at 128x64x64, but 4 to
// 10 up to 32,768 nodes, where the V-cycle uses it instead.
//
// Coarse elements that touch a Dirichlet DOF, an inactive coarse DOF or an odd
// axis's half element use their stored matrix: a pre-pass (one warp per element)
// leaves their stresses, already in the modal basis, in yspec.
//
// Scheduling is k_fine_march's with one element row per thread.
#include <cuda_runtime.h>

#include <algorithm>

#include "tg_internal.h"
#include "tg_launch.h"
#include "tg_march.h"
#include "tg_multigrid.h"

namespace tg {
namespace {

constexpr int kMaxWarps = 12;
constexpr int kOwn = 30;

// Words of one layer's copies of one warp: two rows of x, four fine rows of
// moduli (y child, z child), a row of the special elements' positions, and a row
// each of b and the inverse diagonal where the mode reads them.
template <int MODE>
__host__ __device__ constexpr int slot_words1() {
  return 2 * kRowWords + 4 * 64 + 32 + (MODE != kApply ? kRowWords : 0) +
         (MODE == kSmooth ? kRowWords : 0);
}

__device__ __forceinline__ float2 pair(float v) { return make_float2(v, v); }
__device__ __forceinline__ float zsum(float2 v) { return v.x + v.y; }
__device__ __forceinline__ float zdif(float2 v) { return v.y - v.x; }

// The parent's stresses from its modes u (index bits 1, 2, 4: linear in x, y, z)
// and its children's moduli: E[c] of the children c = x | y << 1, lower z child
// in .x, upper in .y.  In place; mode 0 is not read and gets no stress.
__device__ __forceinline__ void parent_stress(const ModalT<float>& mc, const float2 (&E)[4],
                                              float (&u)[3][8]) {
  // The child modes, by variant: {x} by the y sign, {y} by the x sign, {z} by both,
  // {xz} by the y sign, {yz} by the x sign; the z sign is the packed half.
  float2 mx[3][2], my[3][2], mz[3][4], mxy[3], mxz[3][2], myz[3][2];
  float a7[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float a1 = 0.5f * u[k][1], a2 = 0.5f * u[k][2], a4 = 0.5f * u[k][4];
    const float a3 = 0.25f * u[k][3], a5 = 0.25f * u[k][5], a6 = 0.25f * u[k][6];
    a7[k] = 0.125f * u[k][7];
    const float2 x0 = make_float2(a1 - a5, a1 + a5), y0 = make_float2(a2 - a6, a2 + a6);
    mxy[k] = make_float2(a3 - a7[k], a3 + a7[k]);
    mx[k][0] = vsub(x0, mxy[k]);
    mx[k][1] = vadd(x0, mxy[k]);
    my[k][0] = vsub(y0, mxy[k]);
    my[k][1] = vadd(y0, mxy[k]);
    const float2 p4 = pair(a4), p5 = pair(a5), p6 = pair(a6), p7 = pair(a7[k]);
    mxz[k][0] = vsub(p5, p7);
    mxz[k][1] = vadd(p5, p7);
    myz[k][0] = vsub(p6, p7);
    myz[k][1] = vadd(p6, p7);
    const float2 z0 = vsub(p4, p5), z1 = vadd(p4, p5);
    mz[k][0] = vsub(z0, myz[k][0]);
    mz[k][1] = vsub(z1, myz[k][1]);
    mz[k][2] = vadd(z0, myz[k][0]);
    mz[k][3] = vadd(z1, myz[k][1]);
  }
  // Children's stresses, summed by variant.
  float2 gx[3][2], gy[3][2], gz[3][4], gxy[3], gxz[3][2], gyz[3][2];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int cx = c & 1, cy = c >> 1;
    const float2 f = E[c];
    float2 v[3][8];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v[k][1] = mx[k][cy];
      v[k][2] = my[k][cx];
      v[k][3] = mxy[k];
      v[k][4] = mz[k][c];
      v[k][5] = mxz[k][cy];
      v[k][6] = myz[k][cx];
    }
    modal_stress_12<float2, float>(mc, f, v[0], v[1], v[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      gx[k][cy] = cx ? vadd(gx[k][cy], v[k][1]) : v[k][1];
      gy[k][cx] = cy ? vadd(gy[k][cx], v[k][2]) : v[k][2];
      gxy[k] = c ? vadd(gxy[k], v[k][3]) : v[k][3];
      gz[k][c] = v[k][4];
      gxz[k][cy] = cx ? vadd(gxz[k][cy], v[k][5]) : v[k][5];
      gyz[k][cx] = cy ? vadd(gyz[k][cx], v[k][6]) : v[k][6];
    }
  }
  const float lm2 = mc.LM2 * zsum(vadd(vadd(E[0], E[1]), vadd(E[2], E[3])));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float2 p1 = vadd(gx[k][1], gx[k][0]), p2 = vadd(gy[k][1], gy[k][0]);
    const float2 p3 =
        vadd(gxy[k], vadd(vsub(gx[k][1], gx[k][0]), vsub(gy[k][1], gy[k][0])));
    const float2 s01 = vadd(gz[k][1], gz[k][0]), d01 = vsub(gz[k][1], gz[k][0]);
    const float2 s23 = vadd(gz[k][3], gz[k][2]), d23 = vsub(gz[k][3], gz[k][2]);
    const float2 p4 = vadd(s23, s01);
    const float2 p5 = vadd(vadd(gxz[k][1], gxz[k][0]), vadd(d23, d01));
    const float2 p6 = vadd(vadd(gyz[k][1], gyz[k][0]), vsub(s23, s01));
    const float2 p7 = vadd(vadd(vsub(gxz[k][1], gxz[k][0]), vsub(gyz[k][1], gyz[k][0])),
                           vsub(d23, d01));
    u[k][1] = 0.5f * zsum(p1);
    u[k][2] = 0.5f * zsum(p2);
    u[k][4] = 0.5f * zsum(p4);
    u[k][3] = 0.25f * zsum(p3);
    u[k][5] = 0.25f * (zsum(p5) + zdif(p1));
    u[k][6] = 0.25f * (zsum(p6) + zdif(p2));
    u[k][7] = 0.125f * fmaf(lm2, a7[k], zsum(p7) + zdif(p3));
  }
}

template <int MODE>
__global__ void __launch_bounds__(32 * kMaxWarps, 1)
    k_level1_march(MgDims fd, MgDims cd, ModalT<float> mc, int KZ, int nss,
                   const float* ef, const uint8_t* __restrict__ an,
                   const int* __restrict__ spos, const float* yspec,
                   const float* x, const float* b,
                   const float* invdiag, float omega, float* __restrict__ y) {
  let_next_start();
  extern __shared__ __align__(16) unsigned char l1_smem[];
  float* const xs = reinterpret_cast<float*>(l1_smem);  // [2][W][6][32]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int rows = W - 1;
  constexpr int kSlot = slot_words1<MODE>();
  float* const mine = xs + 2 * W * 192 + w * (kDepth + 1) * kSlot;
  const unsigned mine_s = static_cast<unsigned>(__cvta_generic_to_shared(mine));
  // This lane's element column and strip; its element row ey, node rows ey, ey + 1.
  const int q = blockIdx.x * kOwn - 1 + lane;
  const int ss = q > 0 ? q / cd.nnx : 0, ex = q - ss * cd.nnx;
  const bool own_x = lane >= 1 && lane <= kOwn && ss < nss;
  const int rl = lane < 31 ? lane + 1 : lane, ll = lane > 0 ? lane - 1 : lane;
  const int ey = ss * rows - 1 + w;
  const bool ev = ex >= 0 && ss < nss && ex < cd.ex && ey >= 0 && ey < cd.ey;
  const bool own = own_x && w < W - 1 && ey + 1 < cd.nny;  // node row ey + 1 is this thread's
  const int plane = cd.nnx * cd.nny, eplane = cd.ex * cd.ey, fplane = fd.ex * fd.ey;
  const unsigned node = unsigned(cd.nnx * (ey + 1) + ex);  // within a layer, when own
  const int z0 = blockIdx.y * KZ;

  // Copies: word 32 j + lane of a node row belongs to lane (32 j + lane) / 3's
  // node, of a fine row to lane (32 j + lane) / 2's element.
  const int exc = min(max(ex, 0), cd.nnx - 1);
  unsigned wo[3][2], fo[2][2];
  int fok[2][2];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int word = 32 * j + lane, m = word / 3, k = word - 3 * m;
    const int exm = __shfl_sync(0xffffffffu, exc, m), ym = __shfl_sync(0xffffffffu, ey, m);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      wo[j][i] = 4u * unsigned(3 * (cd.nnx * min(max(ym + i, 0), cd.nny - 1) + exm) + k);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int word = 32 * j + lane, m = word / 2;
    const int fi = 2 * __shfl_sync(0xffffffffu, ex, m) + (word & 1);
    const int eym = __shfl_sync(0xffffffffu, ey, m);
    const bool evm = __shfl_sync(0xffffffffu, int(ev), m) != 0;
#pragma unroll
    for (int cy = 0; cy < 2; ++cy) {
      const int fj = 2 * eym + cy;
      const bool ok = evm && fi < fd.ex && fj < fd.ey;
      fo[j][cy] = ok ? 4u * unsigned(fj * fd.ex + fi) : 0u;
      fok[j][cy] = ok ? 4 : 0;
    }
  }
  const unsigned so = ev ? 4u * unsigned(ey * cd.ex + ex) : 0u;
  wait_for_previous();
  // Step s: node layer ez + 1 of x, everything else of layer ez.
  auto copy_step = [&](int s) {
    const int ez = z0 - 1 + s;
    if (s <= KZ && ez <= cd.nnz - 1) {
      const unsigned st = mine_s + (unsigned(s) % (kDepth + 1)) * (4u * kSlot) + 4u * lane;
      const float* xl = x + 3 * (plane * min(ez + 1, cd.nnz - 1));
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          copy_word(st + 4 * (i * kRowWords + 32 * j), at(xl, wo[j][i]));
      const bool vc = ez >= 0 && ez < cd.ez;
#pragma unroll
      for (int cz = 0; cz < 2; ++cz) {
        const int fk = 2 * ez + cz;
        const bool vf = vc && fk < fd.ez;
        const float* el = ef + int64_t(fplane) * (vf ? fk : 0);
#pragma unroll
        for (int cy = 0; cy < 2; ++cy)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            copy_word_or_zero(st + 4 * (2 * kRowWords + (2 * cz + cy) * 64 + 32 * j),
                              at(el, fo[j][cy]), vf ? fok[j][cy] : 0);
      }
      if (spos != nullptr)
        copy_word_or_zero(st + 4 * (2 * kRowWords + 256),
                          at(reinterpret_cast<const float*>(spos + eplane * (vc ? ez : 0)), so),
                          vc && ev ? 4 : 0);
      if (MODE != kApply && s >= 1) {
        const float *bl = b + 3 * plane * ez, *dl = invdiag + 3 * plane * ez;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const unsigned d = st + 4 * (2 * kRowWords + 288 + 32 * j);
          copy_word(d, at(bl, wo[j][1]));
          if (MODE == kSmooth) copy_word(d + 4 * kRowWords, at(dl, wo[j][1]));
        }
      }
    }
    copy_commit();
  };
  auto load_act = [&](int s) -> unsigned {
    const int ez = z0 - 1 + s;
    return s >= 1 && ez < cd.nnz && own ? unsigned(*at(an + plane * ez, node)) : 0u;
  };

  const int s0 = z0 == 0 ? 1 : 0;  // the first chunk has no element layer below it
  float Fc[3][4], pend[3][4], keep[3];
  {
    const float* xl = x + 3 * (plane * (z0 - 1 + s0));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float a[2], nb[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int yr = min(max(ey + i, 0), cd.nny - 1);
        a[i] = xl[3 * (cd.nnx * yr + exc) + k];
        nb[i] = shfl_at(a[i], rl);
      }
      face_modes<float, float>(a, nb, Fc[k]);
      keep[k] = a[1];
#pragma unroll
      for (int m = 0; m < 4; ++m) pend[k][m] = 0.0f;
    }
  }
#pragma unroll 1
  for (int d = 0; d < kDepth; ++d) copy_step(s0 + d);
  unsigned abn = load_act(s0);

#pragma unroll 1
  for (int s = s0; s <= KZ; ++s) {
    const int ez = z0 - 1 + s;
    if (ez > cd.nnz - 1) break;  // uniform: the last chunk ends with the grid
    const unsigned ab = abn;
    if (s < KZ) abn = load_act(s + 1);
    copy_wait_ahead();
    __syncwarp();  // every lane's words of this step are in, and the last step's are read
    copy_step(s + kDepth);
    const float* st = mine + (s % (kDepth + 1)) * kSlot;
    float Fn[3][4], knext[3], u[3][8];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float a[2], nb[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[i] = st[i * kRowWords + 3 * lane + k];
        nb[i] = st[i * kRowWords + 3 * rl + k];
      }
      face_modes<float, float>(a, nb, Fn[k]);
      knext[k] = a[1];
      u[k][0] = 0.0f;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (m > 0) u[k][m] = Fn[k][m] + Fc[k][m];
        u[k][m | 4] = Fn[k][m] - Fc[k][m];
      }
    }
    float2 E[4];
#pragma unroll
    for (int cy = 0; cy < 2; ++cy) {
      const float2 lo = *reinterpret_cast<const float2*>(st + 2 * kRowWords + cy * 64 + 2 * lane);
      const float2 hi =
          *reinterpret_cast<const float2*>(st + 2 * kRowWords + (2 + cy) * 64 + 2 * lane);
      E[2 * cy] = make_float2(lo.x, hi.x);
      E[2 * cy + 1] = make_float2(lo.y, hi.y);
    }
    parent_stress(mc, E, u);
    if (spos != nullptr && ev && ez >= 0 && ez < cd.ez) {
      const int sp = __float_as_int(st[2 * kRowWords + 256 + lane]);
      if (sp >= 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int m = 0; m < 8; ++m) u[k][m] = yspec[int64_t(sp) * 24 + 8 * k + m];
      }
    }
    float lo[3][2], up[3][2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float P[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        P[m] = pend[k][m] + (u[k][m] - u[k][m | 4]);
        pend[k][m] = u[k][m] + u[k][m | 4];
      }
      lo[k][0] = P[0] - P[2];
      lo[k][1] = P[1] - P[3];
      up[k][0] = P[0] + P[2];
      up[k][1] = P[1] + P[3];
    }
    float* const buf = xs + (s & 1) * (W * 192);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int m = 0; m < 2; ++m) buf[w * 192 + (2 * k + m) * 32 + lane] = lo[k][m];
    __syncthreads();
    if (w < W - 1) {
      float* const yl = y + 3 * (int64_t(plane) * ez + node);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float r0 = up[k][0] + buf[(w + 1) * 192 + (2 * k) * 32 + lane];
        const float r1 = up[k][1] + buf[(w + 1) * 192 + (2 * k + 1) * 32 + lane];
        const float right = r0 + r1;
        const float ax = (r0 - r1) + shfl_at(right, ll);
        if (!(s >= 1 && own)) continue;
        const float* qb = st + 2 * kRowWords + 288 + 3 * lane + k;
        float out;
        if constexpr (MODE == kApply)
          out = ax;
        else if constexpr (MODE == kResidual)
          out = qb[0] - ax;
        else
          out = keep[k] + omega * qb[kRowWords] * (qb[0] - ax);
        yl[k] = ((ab >> k) & 1u) ? out : 0.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      keep[k] = knext[k];
#pragma unroll
      for (int m = 0; m < 4; ++m) Fc[k][m] = Fn[k][m];
    }
  }
}

// The elements off the fast path: one warp per element, lane r < 24 (r = 3 corner
// + component) forms row r of (stored element matrix) x (element DOFs); then the
// modes of the result, 1/8 of the signed sums over the corners, by component.
__global__ void __launch_bounds__(256) k_level1_special(MgDims cd, int nspec,
                                                        const int* __restrict__ list,
                                                        const float* __restrict__ Kel,
                                                        const float* x,
                                                        float* __restrict__ yspec) {
  behind_previous();
  const int lane = threadIdx.x & 31;
  const int p = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (p >= nspec) return;
  const int64_t ce = list[p];
  const int I = int(ce % cd.ex), J = int((ce / cd.ex) % cd.ey), K = int(ce / (int64_t(cd.ex) * cd.ey));
  const int c = lane / 3, comp = lane % 3;
  float uk = 0.0f;
  if (lane < 24) {
    const int64_t node = (int64_t(K + (c >> 2)) * cd.nny + (J + ((c >> 1) & 1))) * cd.nnx +
                         (I + (c & 1));
    uk = x[3 * node + comp];
  }
  float a = 0.0f;
  const float* Kr = Kel + ce * 576 + int64_t(lane < 24 ? lane : 0) * 24;
#pragma unroll
  for (int k = 0; k < 24; ++k) a = fmaf(Kr[k], __shfl_sync(0xffffffffu, uk, k), a);
  float g = 0.0f;  // mode c of component comp
#pragma unroll
  for (int d = 0; d < 8; ++d) {
    const float v = __shfl_sync(0xffffffffu, a, min(3 * d + comp, 23));
    g += (__popc(c & ~d & 7) & 1) ? -v : v;
  }
  if (lane < 24) yspec[int64_t(p) * 24 + 8 * comp + c] = 0.125f * g;
}

// Cycles of a warp step, as march_cost (k_operator.cu) counts them; the tiles it
// picks are within 2 % of the fastest of 100 tried on each of seven grids.
constexpr double kBusy = 260.0, kChain = 3000.0, kStart = 3000.0;
constexpr int kSms = 152;

struct Tile {
  int W, kz;
};
dim3 tile_grid(const MgDims& cd, const Tile& t) {
  const int nss = (cd.nny + t.W - 2) / (t.W - 1);
  return dim3(unsigned((int64_t(cd.nnx) * nss + kOwn - 1) / kOwn),
              unsigned((cd.nnz + t.kz - 1) / t.kz));
}
Tile level1_tile(const MgDims& cd) {
  Tile best{4, 8};
  double best_cost = 1e300;
  for (int W : {2, 3, 4, 6, 8, 12})
    for (int target : {1, 2, 3, 4, 6, 8, 11, 16, 22, 32}) {
      const int chunks = (cd.nnz + target - 1) / target;
      const Tile t{W, (cd.nnz + chunks - 1) / chunks};
      const dim3 d = tile_grid(cd, t);
      const int64_t ctas = int64_t(d.x) * d.y;
      const int res = kMaxWarps / W;
      const int64_t per_sm = (ctas + kSms - 1) / kSms, rounds = (per_sm + res - 1) / res;
      const double cost = std::max(double(per_sm) * W * (t.kz + 1) * kBusy,
                                   double(rounds) * (t.kz + 1) * kChain) +
                          double(rounds) * kStart;
      if (cost < best_cost) {
        best_cost = cost;
        best = t;
      }
      if (target >= cd.nnz) break;
    }
  return best;
}

template <int MODE>
void launch(const Tile& t, const MgDims& fd, const MgDims& cd, const ModalConsts& c,
            const float* ef, const uint8_t* an, const int* spos, const float* yspec,
            const float* x, const float* b, const float* invdiag, float omega, float* y,
            cudaStream_t s) {
  const size_t per_warp = (2 * 192 + (kDepth + 1) * slot_words1<MODE>()) * sizeof(float);
  allow_shared<k_level1_march<MODE>>(int(kMaxWarps * per_warp));
  const int nss = (cd.nny + t.W - 2) / (t.W - 1);
  launch_behind(k_level1_march<MODE>, tile_grid(cd, t), 32 * t.W, t.W * per_warp, s, fd, cd,
                to_modal<float>(c), t.kz, nss, ef, an, spos, yspec, x, b, invdiag, omega, y);
  TG_LAUNCH_CHECK();
}

}  // namespace

void mg_level1_op(int mode, const MgDims& fd, const MgDims& cd, const ModalConsts& c,
                  const float* ef, const uint8_t* act_node, const int* spos, const int* slist,
                  int nspec, const float* Kel, const float* x, const float* b,
                  const float* invdiag, float omega, float* y, float* yspec, cudaStream_t s) {
  if (nspec > 0) {
    launch_behind(k_level1_special, (nspec + 7) / 8, 256, 0, s, cd, nspec, slist, Kel, x, yspec);
    TG_LAUNCH_CHECK();
  }
  const int* sp = nspec > 0 ? spos : nullptr;
  const Tile t = level1_tile(cd);
  if (mode == kApply)
    launch<kApply>(t, fd, cd, c, ef, act_node, sp, yspec, x, b, invdiag, omega, y, s);
  else if (mode == kResidual)
    launch<kResidual>(t, fd, cd, c, ef, act_node, sp, yspec, x, b, invdiag, omega, y, s);
  else
    launch<kSmooth>(t, fd, cd, c, ef, act_node, sp, yspec, x, b, invdiag, omega, y, s);
}

}  // namespace tg
