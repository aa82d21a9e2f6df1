// k_multigrid.cu -- geometric multigrid on the voxel hierarchy.
//
// Reference counterparts (core/src/fea/multigrid.cpp):
//   axis_weights           :494-505   trilinear vertex stencil 1 | 1/2,1/2
//   coarse active DOFs     :1387-1403 active iff the coincident fine DOF is
//   P0 and A1 = P0^T A0 P0 :1408-1446, galerkin_a1_from_prolong :1543-1899
//   levels 2.. (Galerkin)  :557-697 (build_hierarchy)
//   jacobi_sweep, v_cycle  :780-817, mf_jacobi_sweep / mf_v_cycle :1128-1160
//   coarsest direct solve  SimplicialLDLT :690-695 -> here a dense FP64 inverse, or
//     (above 2,048 DOFs) a Cholesky factor
//
// Coarse operators are Galerkin, formed element by element: a coarse element's
// 24x24 matrix is the sum over its (up to) eight children of W^T K_child W, with
// W the trilinear interpolation from the parent's 8 nodes to the child's 8
// nodes.  Because P restricted to an element is exactly that local W, the
// assembled sum equals P^T A P -- including the masks: rows and columns of
// inactive DOFs are zeroed on both sides, as the reference drops them from P.
// Odd axes are handled by ceil-halving the element extents; a coarse node whose
// coincident fine node lies beyond the grid is inactive, which reproduces the
// reference's index-space padding (multigrid.cpp:391-459).
//
// Coarse levels are applied as assembled 27-point node stencils.  The operator
// is symmetric, so only the self block and the 13 "forward" neighbour blocks
// (positive linear offset) are stored, as structure of arrays A[126][nnodes]
// (entry (j*3 + c1)*3 + c2 for block j): a thread per node reads its own rows
// coalesced and the backward blocks, transposed, from the neighbour's rows.
// Half the bytes of the full 243-entry stencil, the bound of the coarse apply.
#include <cuda_runtime.h>

#include "tg_df.h"
#include "tg_internal.h"
#include "tg_launch.h"
#include "tg_multigrid.h"

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <utility>

namespace tg {

namespace {
constexpr int kThreads = 256;

int nblk(int64_t n, int t = kThreads) {
  const int64_t b = (n + t - 1) / t;
  return int(b < 152 * 64 ? (b > 0 ? b : 1) : 152 * 64);
}

// Coordinates (a, b, c) of linear node index n of a level: 32-bit unsigned
// division whenever the index fits (every coarse level; a 64-bit division is a
// long dependent instruction sequence that small, latency-bound kernels pay on
// every item).
__device__ __forceinline__ void node_abc(const MgDims& d, int64_t n, int& a, int& b, int& c) {
  if (n <= int64_t(0xffffffffu)) {
    const unsigned un = unsigned(n), nx = unsigned(d.nnx), ny = unsigned(d.nny);
    const unsigned q = un / nx, r = q / ny;
    a = int(un - q * nx);
    b = int(q - r * ny);
    c = int(r);
  } else {
    a = int(n % d.nnx);
    b = int((n / d.nnx) % d.nny);
    c = int(n / (int64_t(d.nnx) * d.nny));
  }
}

// Local corner index -> offsets; corners in Walsh bit order (x | y<<1 | z<<2).
__device__ __forceinline__ int cx(int c) { return c & 1; }
__device__ __forceinline__ int cy(int c) { return (c >> 1) & 1; }
__device__ __forceinline__ int cz(int c) { return c >> 2; }

// v[3*corner + comp] <- sum_sc v[3*sc + comp] * prod_a M_a[sc_a][t_a] for every
// parent corner t: three 2x2 passes over the corner bits (x, y, z).
template <class T>
__device__ __forceinline__ void kron_map(const T (&mw)[3][4], T (&v)[24]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int bit = 1 << a;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i & bit) continue;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T lo = v[3 * i + c], hi = v[3 * (i | bit) + c];
        v[3 * i + c] = mw[a][0] * lo + mw[a][2] * hi;
        v[3 * (i | bit) + c] = mw[a][1] * lo + mw[a][3] * hi;
      }
    }
  }
}

// One block of eight warps per coarse element, a warp per child; lane c < 24 owns
// column c of the child's share (rows in corner-bit order, row = 3*corner +
// comp).  X = S W (lane r = row r of S), then Y = W^T X (lane c = column c), with
// the sparsity pattern of W uniform across the warp.  S is the child's matrix:
// level 1 -- f * Ke with inactive fine DOFs zeroed (or the precomputed
// G_c = W_c^T Ke W_c times f when all 24 are active); deeper levels -- the stored,
// already masked, child element matrix.  The shares are added in child order;
// rows/cols of inactive coarse DOFs are zeroed at the end.  (One warp walking its
// element's children took eight times as long a chain: 110 us in FP64 and 25 in
// FP32 on levels of any small size.)
// With list set, only the nlist coarse elements it names (level 1's others are
// k_galerkin1_fast's).
template <class T, bool LEVEL1>
__global__ void __launch_bounds__(256) k_galerkin(MgDims fd, MgDims cd, const T* __restrict__ ef,
                                                  const uint8_t* __restrict__ fact,
                                                  const uint8_t* __restrict__ cact,
                                                  const T* __restrict__ Ke,
                                                  const T* __restrict__ G,
                                                  const T* __restrict__ Kf, T* __restrict__ Kc,
                                                  const int* __restrict__ list, int64_t nlist) {
  constexpr int LD = 25;  // padded row stride: row and column walks are bank-conflict free
  __shared__ T sX[8][24 * LD];
  __shared__ bool s_have[8];
  __shared__ T s_f[8];  // a child's factor: its modulus where X holds G_c, else 1
  __shared__ unsigned s_cm;
  const int ch = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* X = sX[ch];
  for (int64_t q = blockIdx.x; q < nlist; q += gridDim.x) {
    const int64_t ce = list ? list[q] : q;
    const int I = int(ce % cd.ex), J = int((ce / cd.ex) % cd.ey),
              K = int(ce / (int64_t(cd.ex) * cd.ey));
    const int hm = cd.align ? ((2 * I + 1 == fd.ex) | ((2 * J + 1 == fd.ey) << 1) |
                               ((2 * K + 1 == fd.ez) << 2))
                            : 0;
    const int fi = 2 * I + cx(ch), fj = 2 * J + cy(ch), fk = 2 * K + cz(ch);
    bool have = fi < fd.ex && fj < fd.ey && fk < fd.ez;
    const int64_t fe = (int64_t(fk) * fd.ey + fj) * fd.ex + fi;
    const int cc = lane / 3, comp = lane % 3;
    T f = T(1);
    unsigned m = 0xffffffu;
    if (LEVEL1 && have) {
      f = ef[fe];
      have = f != T(0);
      unsigned bit = 0;
      if (lane < 24) {
        const int64_t node =
            (int64_t(fk + cz(cc)) * fd.nny + (fj + cy(cc))) * fd.nnx + (fi + cx(cc));
        bit = fact[3 * node + comp] ? 1u << lane : 0u;
      }
      m = __reduce_or_sync(0xffffffffu, bit);
    }
    if (have) {  // warp-uniform
      if (LEVEL1 && m == 0xffffffu && hm == 0) {
        if (lane < 24)
#pragma unroll
          for (int r = 0; r < 24; ++r) X[r * LD + lane] = G[ch * 576 + r * 24 + lane];
      } else {
        // W = W_x (x) W_y (x) W_z on the corner index (times I3 on components):
        // per axis a 2x2 map from the child's sub-corner bit to the parent's
        // corner bit -- [[1,0],[1/2,1/2]] for child bit 0, [[1/2,1/2],[0,1]] for
        // child bit 1, the identity on an aligned half element.  X = S W and
        // Y = W^T X are three 2x2 passes each instead of a dense 8x8 product.
        T mw[3][4];  // per axis: M[sc][t] as {m00, m01, m10, m11}; warp-uniform
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const bool half = (hm >> a) & 1, hi = (ch >> a) & 1;
          mw[a][0] = half ? T(1) : (hi ? T(0.5) : T(1));
          mw[a][1] = half ? T(0) : (hi ? T(0.5) : T(0));
          mw[a][2] = half ? T(0) : (hi ? T(0) : T(0.5));
          mw[a][3] = half ? T(1) : (hi ? T(1) : T(0.5));
        }
        // Row `lane` of S: staged through X, so that global reads are whole lines.
        for (int e = lane; e < 576; e += 32) {
          const int r = e / 24, c2 = e % 24;
          if (LEVEL1)
            X[r * LD + c2] = ((m >> r) & 1u) && ((m >> c2) & 1u) ? f * Ke[e] : T(0);
          else
            X[r * LD + c2] = Kf[fe * 576 + e];
        }
        __syncwarp();
        T v[24];
        if (lane < 24) {  // X = S W: lane = row
#pragma unroll
          for (int j = 0; j < 24; ++j) v[j] = X[lane * LD + j];
          kron_map(mw, v);
#pragma unroll
          for (int j = 0; j < 24; ++j) X[lane * LD + j] = v[j];
        }
        __syncwarp();
        if (lane < 24) {  // Y = W^T X: lane = column
#pragma unroll
          for (int j = 0; j < 24; ++j) v[j] = X[j * LD + lane];
          kron_map(mw, v);
#pragma unroll
          for (int j = 0; j < 24; ++j) X[j * LD + lane] = v[j];
        }
      }
    }
    if (lane == 0) {
      s_have[ch] = have;
      s_f[ch] = LEVEL1 && m == 0xffffffu && hm == 0 ? f : T(1);
    }
    if (ch == 0) {
      unsigned cm = 0;
      if (lane < 24) {
        const int64_t node =
            (int64_t(K + cz(cc)) * cd.nny + (J + cy(cc))) * cd.nnx + (I + cx(cc));
        if (cact[3 * node + comp]) cm = 1u << lane;
      }
      cm = __reduce_or_sync(0xffffffffu, cm);
      if (lane == 0) s_cm = cm;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 576; e += 256) {
      const int r = e / 24, c = e % 24;
      T acc = T(0);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (s_have[k]) acc = fma(s_f[k], sX[k][r * LD + c], acc);
      Kc[ce * 576 + e] = ((s_cm >> r) & 1u) && ((s_cm >> c) & 1u) ? acc : T(0);
    }
    __syncthreads();
  }
}

// Node stencil from the element matrices around each node: the self block and
// the forward blocks only.  Entry index q = (j*3 + c1)*3 + c2 with
// j = d - 13, d = (dz+1)*9 + (dy+1)*3 + (dx+1) >= 13.  One thread per node and
// block (blockIdx.y = j): a thread that formed a node's 14 blocks one after
// another took 20-50 us on the smallest levels.  With A null only the inverse
// diagonal is formed (one row of blocks, j = 0), from the same sums.
template <class T>
__global__ void k_assemble_stencil(MgDims d, const T* __restrict__ Kel,
                                   const uint8_t* __restrict__ act, T* __restrict__ A,
                                   T* __restrict__ invdiag) {
  const int64_t nn = int64_t(d.nnx) * d.nny * d.nnz;
  const int j = blockIdx.y, di = 13 + j;
  const int dx = di % 3 - 1, dy = (di / 3) % 3 - 1, dz = di / 9 - 1;
  for (int64_t n = blockIdx.x * int64_t(kThreads) + threadIdx.x; n < nn;
       n += int64_t(gridDim.x) * kThreads) {
    int a, b, c;
    node_abc(d, n, a, b, c);
    bool ra[3];
    for (int k = 0; k < 3; ++k) ra[k] = act[3 * n + k] != 0;
    T blk[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) blk[k] = T(0);
    // Elements containing both n and n+d: offsets ox in {-1,0} with the
    // node at corner (-ox) and the neighbour at corner (-ox + dx) in [0,1].
    for (int oz = -1; oz <= 0; ++oz) {
      const int lz = -oz, mz = lz + dz;
      if (mz < 0 || mz > 1) continue;
      for (int oy = -1; oy <= 0; ++oy) {
        const int ly = -oy, my = ly + dy;
        if (my < 0 || my > 1) continue;
        for (int ox = -1; ox <= 0; ++ox) {
          const int lx = -ox, mx = lx + dx;
          if (mx < 0 || mx > 1) continue;
          const int ei = a + ox, ej = b + oy, ek = c + oz;
          if (ei < 0 || ei >= d.ex || ej < 0 || ej >= d.ey || ek < 0 || ek >= d.ez) continue;
          const int64_t e = (int64_t(ek) * d.ey + ej) * d.ex + ei;
          const int ln = lx | (ly << 1) | (lz << 2), lm = mx | (my << 1) | (mz << 2);
          const T* Ke = Kel + e * 576;
#pragma unroll
          for (int c1 = 0; c1 < 3; ++c1)
#pragma unroll
            for (int c2 = 0; c2 < 3; ++c2) blk[c1 * 3 + c2] += Ke[(3 * ln + c1) * 24 + 3 * lm + c2];
        }
      }
    }
    if (A != nullptr)
#pragma unroll
      for (int c1 = 0; c1 < 3; ++c1)
#pragma unroll
        for (int c2 = 0; c2 < 3; ++c2)
          A[int64_t(j * 9 + c1 * 3 + c2) * nn + n] = ra[c1] ? blk[c1 * 3 + c2] : T(0);
    if (j == 0)
      for (int k = 0; k < 3; ++k) {
        const T dg = blk[k * 3 + k];
        invdiag[3 * n + k] = (ra[k] && dg > T(0)) ? T(1) / dg : T(0);
      }
  }
}

template <class T>
__global__ void k_to_float(const double* __restrict__ s, T* __restrict__ d, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    d[i] = T(s[i]);
}

// Stencil operator: y = A x / b - A x / x + w D^-1 (b - A x), masked by act.
// A thread per (node, output component r): row r of every 3x3 block.  Forward
// block j of node n couples n to n + off_j; the backward coupling of n to
// n - off_j is the forward block j of node n - off_j, transposed (its column r).
// Three threads per node keep the per-thread register count low and the number
// of independent coefficient loads in flight high: the kernel streams the
// stencil once from HBM (the backward re-reads hit L2) and is bound by how many
// of those loads are outstanding.  Out-of-grid neighbours are predicated (the
// stored forward block of a node whose neighbour lies outside the grid is zero,
// and the backward term is selected away).  Per output the terms are summed in
// the fixed order of stencil_row.
// Loads of vectors another CTA may have written earlier in the same launch (the
// fused coarse V-cycle) go through L2; elsewhere plain loads.
template <class T, bool COH>
__device__ __forceinline__ T vload(const T* p) {
  if constexpr (COH)
    return __ldcg(p);
  else
    return *p;
}

// Chebyshev direction update c0 * d_prev + c1 * res with one explicit rounding
// pattern (the product c1 * res rounded, then one fused multiply-add), so every
// kernel that takes the step produces the same bits.
__device__ __forceinline__ float cheb_dir(float c0, float dprev, float c1, float res) {
  return __fmaf_rn(c0, dprev, __fmul_rn(c1, res));
}
__device__ __forceinline__ double cheb_dir(double c0, double dprev, double c1, double res) {
  return __fma_rn(c0, dprev, __dmul_rn(c1, res));
}

// s plus one stencil block's row times x, in one rounding pattern in every kernel
// that evaluates it.  FP32: the block's sum first (a product, two fused
// multiply-adds), then one addition, so the blocks' sums do not wait for one
// another.  FP64, where each operation takes 64 cycles of the scheduler's unit
// whatever waits: three fused multiply-adds onto s, a quarter fewer.
__device__ __forceinline__ float add_block(float s, float a0, float x0, float a1, float x1,
                                           float a2, float x2, bool on) {
  const float u = __fmaf_rn(a2, x2, __fmaf_rn(a1, x1, __fmul_rn(a0, x0)));
  return __fadd_rn(s, on ? u : 0.0f);
}
__device__ __forceinline__ double add_block(double s, double a0, double x0, double a1, double x1,
                                            double a2, double x2, bool on) {
  const double t = __fma_rn(a2, x2, __fma_rn(a1, x1, __fma_rn(a0, x0, s)));
  return on ? t : s;
}

// The matrix entries of a part and the nodes that they meet (n itself beyond the grid);
// slot t is block j = 4 t + part (block 0, the self block, has no transposed partner).
template <class T>
struct StencilPart {
  T f[4][3], b[4][3];
  int m[4], p[4];
  bool fin[4], bin[4];
};
template <class T>
__device__ __forceinline__ void stencil_entries(const MgDims& d, const T* __restrict__ A, int a,
                                                int bb, int c, int r, int part,
                                                StencilPart<T>& w) {
  const int64_t nn = int64_t(d.nnx) * d.nny * d.nnz;
  const int sy = d.nnx, sz = d.nnx * d.nny, n = c * sz + bb * sy + a;
  const T* An = A + n + int64_t(3 * r) * nn;  // row r of the self block
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int j = 4 * t + part;
    if (j >= 14) continue;
    const int di = 13 + j;
    const int dx = di % 3 - 1, dy = (di / 3) % 3 - 1, dz = di / 9 - 1;
    const int off = dz * sz + dy * sy + dx;
    w.fin[t] = (a + dx) < d.nnx && (a + dx) >= 0 && (bb + dy) < d.nny && (bb + dy) >= 0 &&
               (c + dz) < d.nnz;
    w.bin[t] = j > 0 && (a - dx) >= 0 && (a - dx) < d.nnx && (bb - dy) >= 0 &&
               (bb - dy) < d.nny && (c - dz) >= 0;
    w.m[t] = w.fin[t] ? n + off : n;
    w.p[t] = w.bin[t] ? n - off : n;
    const T* Af = An + int64_t(j * 9) * nn;
    const T* Ab = A + int64_t(j * 9 + r) * nn + w.p[t];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      w.f[t][e] = Af[e * nn];
      w.b[t][e] = Ab[3 * e * nn];
    }
  }
}

// Part `part` (0..3) of row r of a node of a stored symmetric stencil times x.  The row
// is the self block (term 0) plus, for j = 1..13, forward block j (neighbour n + off_j)
// and the transposed forward block of neighbour n - off_j; part q accumulates the terms
// j = q, q + 4, ... in increasing j, and the row is ((p0 + p1) + p2) + p3.  Four parts
// let four threads share a row on the small levels, where a row's ~160 loads in one
// thread are a chain of dependent memory round trips -- and, in FP64, its 81
// multiply-adds a chain of 64 cycles each.
template <class T, bool COH>
__device__ __forceinline__ T stencil_part(const StencilPart<T>& w, int part, const T* x) {
  T s = T(0);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int j = 4 * t + part;
    if (j >= 14) continue;
    const T *xm = x + 3 * int64_t(w.m[t]), *xp = x + 3 * int64_t(w.p[t]);
    s = add_block(s, w.f[t][0], vload<T, COH>(xm), w.f[t][1], vload<T, COH>(xm + 1), w.f[t][2],
                  vload<T, COH>(xm + 2), w.fin[t]);
    if (j > 0)
      s = add_block(s, w.b[t][0], vload<T, COH>(xp), w.b[t][1], vload<T, COH>(xp + 1), w.b[t][2],
                    vload<T, COH>(xp + 2), w.bin[t]);
  }
  return s;
}

// Row r of node (a, bb, c) of the stencil times x: the four parts in order.
template <class T, bool COH>
__device__ __forceinline__ T stencil_row(const MgDims& d, const T* __restrict__ A, const T* x,
                                         int a, int bb, int c, int r) {
  T p[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    StencilPart<T> w;
    stencil_entries(d, A, a, bb, c, r, q, w);
    p[q] = stencil_part<T, COH>(w, q, x);
  }
  return ((p[0] + p[1]) + p[2]) + p[3];
}

// The per-DOF update of the stencil kernels from the row sum s, in one
// rounding pattern: kApply s, kResidual b - s, kSmooth x + (omega dinv)(b - s),
// kCheb the Chebyshev step (direction dprev of the previous step, coefficients
// of the level's table); inactive DOFs 0 (and a zero direction).
template <class T, int MODE>
__device__ __forceinline__ T stencil_update(bool active, T s, T xv, T bv, T dv, T omega,
                                            const float* cf, int step, T dprev, T& dnew) {
  dnew = T(0);
  if (!active) return T(0);
  if (MODE == kApply) return s;
  if (MODE == kResidual) return bv - s;
  if (MODE == kDinvA) return dv * s;
  if (MODE == kCheb) {
    // Chebyshev step (Saad, Iterative Methods, Alg. 12.1): d_k = rho_k rho_{k-1}
    // d_{k-1} + (2 rho_k / delta) D^-1 (b - A x_k), d_0 = D^-1 (b - A x_0) / theta,
    // x_{k+1} = x_k + d_k.
    const T res = dv * (bv - s);
    dnew = step == 0 ? T(cf[0]) * res : cheb_dir(T(cf[2 * step]), dprev, T(cf[2 * step + 1]), res);
    return xv + dnew;
  }
  if constexpr (sizeof(T) == 4)
    return __fmaf_rn(__fmul_rn(omega, dv), __fsub_rn(bv, s), xv);
  else
    return __fma_rn(__dmul_rn(omega, dv), __dsub_rn(bv, s), xv);
}

constexpr int kStencilThreads = 192;

template <class T, int MODE>
__global__ void __launch_bounds__(kStencilThreads) k_stencil_op(MgDims d, const T* __restrict__ A,
                                                    const uint8_t* __restrict__ act,
                                                    const T* x,
                                                    const T* b,
                                                    const T* __restrict__ invdiag, T omega,
                                                    T* __restrict__ y, ChebStep ch) {
  behind_previous();
  // 192 threads: two chunks of 32 consecutive nodes (in x-fastest order, across
  // row ends) x 3 components, one component per warp, so a warp's stencil and
  // vector reads are coalesced and no lane idles at the odd row lengths
  // (2^k + 1 nodes) of the coarse levels.
  const int64_t it = blockIdx.x * int64_t(kStencilThreads) + threadIdx.x;
  const int64_t n = (it / 96) * 32 + (it & 31);
  const int r = int((it / 32) % 3);
  if (n >= int64_t(d.nnx) * d.nny * d.nnz) return;
  int a, bb, c;
  node_abc(d, n, a, bb, c);
  const T s = stencil_row<T, false>(d, A, x, a, bb, c, r);
  const int64_t dof = 3 * n + r;
  T* dir = static_cast<T*>(ch.dir_);
  const bool ac = act[dof] != 0;
  T dnew;
  const T out = stencil_update<T, MODE>(
      ac, s, (MODE == kSmooth || MODE == kCheb) ? x[dof] : T(0),
      MODE != kApply && MODE != kDinvA ? b[dof] : T(0),
      (MODE == kSmooth || MODE == kCheb || MODE == kDinvA) ? invdiag[dof] : T(0), omega, ch.coef, ch.step,
      (MODE == kCheb && ch.step > 0 && ac) ? dir[dof] : T(0), dnew);
  if (MODE == kCheb) dir[dof] = dnew;
  y[dof] = out;
}

// The stencil kernels on small levels: four threads per (node, row), one
// part of the row each (stencil_part), combined in shared memory in the order
// stencil_row uses, so both kernels give the same bits.  384 threads: 32
// consecutive nodes x 3 rows x 4 parts.  A launch is a chain of round trips to the L2:
// the matrix entries are read before the wait for the previous kernel, so that behind
// it only the vectors' remain (24 launches of a 128x64x64 iteration: 224 -> 204 us
// with the other kernels of the chain launched that way too).
constexpr int kSplitThreads = 384;
// Up to here the four threads win.  FP32, bound by memory latency (a solve of many
// steps, launched behind one another): 2.4-3.6 us against 6.4-7.5 on 225 to 9,537 nodes,
// 14.4 against 15.0 ms for a solve whose level 1 has 26,400, 12.3 against 10.4 us on
// 30,625.  FP64, bound by its units: 7-10 us against 21 on 225 to 4,225 nodes, 19-26
// against 30 on 30,625.
template <class T>
constexpr int64_t split_max_nodes() {
  return sizeof(T) == 8 ? 100000 : 28672;
}

template <class T, int MODE>
__global__ void __launch_bounds__(kSplitThreads, 2) k_stencil_split(
    MgDims d, const T* __restrict__ A, const uint8_t* __restrict__ act,
    const T* x, const T* b, const T* __restrict__ invdiag,
    T omega, T* __restrict__ y, ChebStep ch) {
  __shared__ T parts[3][3][32];
  let_next_start();
  const int t = threadIdx.x, q = t / 96, r = (t / 32) % 3, lane = t & 31;
  const int64_t n = int64_t(blockIdx.x) * 32 + lane;
  const bool valid = n < int64_t(d.nnx) * d.nny * d.nnz;
  const int64_t dof = 3 * n + r;
  T* dir = static_cast<T*>(ch.dir_);
  bool ac = false;
  T xv = T(0), bv = T(0), dv = T(0), dprev = T(0);
  StencilPart<T> w;
  if (valid) {
    int a, bb, c;
    node_abc(d, n, a, bb, c);
    stencil_entries(d, A, a, bb, c, r, q, w);
    if (q == 0) {
      ac = act[dof] != 0;
      if (MODE == kSmooth || MODE == kCheb || MODE == kDinvA) dv = invdiag[dof];
    }
  }
  wait_for_previous();
  if (q == 0 && valid) {
    if (MODE == kSmooth || MODE == kCheb) xv = x[dof];
    if (MODE != kApply && MODE != kDinvA) bv = b[dof];
    if (MODE == kCheb && ch.step > 0) dprev = dir[dof];
  }
  const T p = valid ? stencil_part<T, false>(w, q, x) : T(0);
  if (q > 0) parts[q - 1][r][lane] = p;
  __syncthreads();
  if (q != 0 || !valid) return;
  const T s = ((p + parts[0][r][lane]) + parts[1][r][lane]) + parts[2][r][lane];
  T dnew;
  const T out = stencil_update<T, MODE>(ac, s, xv, bv, dv, omega, ch.coef, ch.step,
                                                ac ? dprev : T(0), dnew);
  if (MODE == kCheb) dir[dof] = dnew;
  y[dof] = out;
}

// Power iteration for lambda_max(D^-1 A) of one stencil level: v on the active
// DOFs from a fixed hash, then w = D^-1 A v, v = w; |w| / |v| of the last step ->
// lam.  Not normalised on the way: lambda is a few units, so ten steps stay far
// inside FP32's range, and a step is one launch instead of five (0.5 ms of a
// 256x128x128 hierarchy build's small dependent launches).
template <class T>
__global__ void k_pi_init(const uint8_t* __restrict__ act, int64_t n, T* __restrict__ v) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads) {
    uint32_t h = uint32_t(i) * 2654435761u;
    h ^= h >> 16;
    v[i] = act[i] ? T(0.5) + T(h & 0xffff) * T(1.0 / 65536.0) : T(0);
  }
}
__global__ void k_pi_lambda(const double* __restrict__ nrm2, double safety,
                            double* __restrict__ lam) {
  if (threadIdx.x == 0)
    lam[0] = safety * (nrm2[0] > 0.0 && nrm2[1] > 0.0 ? sqrt(nrm2[1] / nrm2[0]) : 1.0);
}

// Chebyshev coefficients on [lmax / ratio, lmax]: theta, delta the interval's
// centre and half-width, rho_0 = delta / theta, rho_k = 1 / (2 theta / delta -
// rho_{k-1}); thread k writes step k's pair.
__global__ void k_cheb_table(const double* __restrict__ lam, double ratio, int m,
                             float* __restrict__ coef) {
  const int k = threadIdx.x;
  if (k >= m) return;
  const double lmax = lam[0], lmin = lmax / ratio;
  const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin), sig = theta / delta;
  double rp = 1.0 / sig, rk = rp;
  for (int i = 1; i <= k; ++i) {
    rp = rk;
    rk = 1.0 / (2.0 * sig - rp);
  }
  if (k == 0) {
    coef[0] = float(1.0 / theta);
    coef[1] = 0.0f;
  } else {
    coef[2 * k] = float(rk * rp);
    coef[2 * k + 1] = float(2.0 * rk / delta);
  }
}

// x = omega * invdiag .* b (the first smoother sweep from a zero iterate).
template <class T>
__global__ void k_jacobi_first(const T* __restrict__ b, const T* __restrict__ invdiag, T omega,
                               int64_t n, T* __restrict__ x) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kThreads)
    x[i] = omega * invdiag[i] * b[i];
}

// Boundary-aligned coarsening (MgDims::align): on an odd fine axis the last
// fine node (index Ef) is the coincident node of coarse node (Ef + 1) / 2.
__device__ __forceinline__ bool tail_node(int i, int Ef, int align) {
  return align && (Ef & 1) && i == Ef;
}
// Weights of the fine nodes 2N - 1, 2N, 2N + 1 in coarse node N along one axis, 0
// beyond the grid.
template <class T>
__device__ __forceinline__ void axis_weights(int N, int Ef, int nf, int align, T (&w)[3]) {
#pragma unroll
  for (int d = -1; d <= 1; ++d) {
    const int i = 2 * N + d;
    T v = d == 0 ? T(1) : T(0.5);
    if (tail_node(i, Ef, align)) v = N == (Ef + 1) / 2 ? T(1) : T(0);
    w[d + 1] = i >= 0 && i < nf ? v : T(0);
  }
}

// Restriction R = P^T at component k of coarse node (a, b, c): the (up to 27) fine
// nodes 2N + delta, summed axis by axis -- 39 operations, where a weight product
// per fine node takes 108.  A fine node beyond the grid has weight 0 and is read
// at its clamped place.  Fine residuals are already 0 on inactive fine DOFs.
template <class T, bool COH>
__device__ __forceinline__ T restrict_dof(const MgDims& fd, const MgDims& cd, const T* rf, int a,
                                          int b, int c, int k) {
  T wx[3], wy[3], wz[3];
  axis_weights<T>(a, fd.ex, fd.nnx, cd.align, wx);
  axis_weights<T>(b, fd.ey, fd.nny, cd.align, wy);
  axis_weights<T>(c, fd.ez, fd.nnz, cd.align, wz);
  int ox[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) ox[d] = 3 * min(max(2 * a + d - 1, 0), fd.nnx - 1) + k;
  T sz = T(0);
#pragma unroll
  for (int dz = 0; dz < 3; ++dz) {
    const int z = min(max(2 * c + dz - 1, 0), fd.nnz - 1);
    T sy = T(0);
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
      const int y = min(max(2 * b + dy - 1, 0), fd.nny - 1);
      const T* row = rf + 3 * (int64_t(z) * fd.nny + y) * fd.nnx;
      const T sx = fma(wx[2], vload<T, COH>(row + ox[2]),
                       fma(wx[1], vload<T, COH>(row + ox[1]), wx[0] * vload<T, COH>(row + ox[0])));
      sy = fma(wy[dy], sx, sy);
    }
    sz = fma(wz[dz], sy, sz);
  }
  return sz;
}

// The prolonged correction at fine node (a, b, c): per axis one coarse node
// (an even fine node, or the aligned tail node) or two at weight 1/2.
template <class T, bool COH>
__device__ __forceinline__ void prolong_node(const MgDims& fd, const MgDims& cd, const T* ec,
                                             int a, int b, int c, T (&s)[3]) {
  const bool ta = tail_node(a, fd.ex, cd.align), tb = tail_node(b, fd.ey, cd.align),
             tc = tail_node(c, fd.ez, cd.align);
  const int na = (a & 1) && !ta ? 2 : 1, nb = (b & 1) && !tb ? 2 : 1, ncz = (c & 1) && !tc ? 2 : 1;
  const int ia0 = ta ? (a + 1) >> 1 : a >> 1, ia1 = (a + 1) >> 1;
  const int ib0 = tb ? (b + 1) >> 1 : b >> 1, ib1 = (b + 1) >> 1;
  const int ic0 = tc ? (c + 1) >> 1 : c >> 1, ic1 = (c + 1) >> 1;
  const T w = (na == 2 ? T(0.5) : T(1)) * (nb == 2 ? T(0.5) : T(1)) * (ncz == 2 ? T(0.5) : T(1));
  s[0] = s[1] = s[2] = T(0);
#pragma unroll
  for (int zz = 0; zz < 2; ++zz) {
    if (zz >= ncz) continue;
    const int k = zz ? ic1 : ic0;
#pragma unroll
    for (int yy = 0; yy < 2; ++yy) {
      if (yy >= nb) continue;
      const int j = yy ? ib1 : ib0;
#pragma unroll
      for (int xx = 0; xx < 2; ++xx) {
        if (xx >= na) continue;
        const int i = xx ? ia1 : ia0;
        if (i >= cd.nnx || j >= cd.nny || k >= cd.nnz) continue;
        const T* q = ec + 3 * ((int64_t(k) * cd.nny + j) * cd.nnx + i);
        s[0] += w * vload<T, COH>(q);
        s[1] += w * vload<T, COH>(q + 1);
        s[2] += w * vload<T, COH>(q + 2);
      }
    }
  }
}

// The restriction runs a thread per DOF, consecutive threads on consecutive DOFs
// of a coarse node layer (blockIdx.y): its reads are half-full lines instead of a
// node's 12 bytes of every 24, and in FP64 three threads share what one did at 64
// cycles an instruction (25x25x49 coarse nodes: 19.2 -> 10.5 us; FP32 on
// 65x33x33: 8.7 -> 6.8, 129x65x65 unchanged at 25).  The row of an entry comes
// from a multiplication by the row length's reciprocal (n < 2^31: exact).
struct RowDiv {
  unsigned len, mul, shift;
};
RowDiv row_div(int nnx) {
  RowDiv r{unsigned(3 * nnx), 0, 0};
  while ((1ull << r.shift) < r.len) ++r.shift;
  r.mul = unsigned(((1ull << 32) * ((1ull << r.shift) - r.len)) / r.len + 1);
  return r;
}
__device__ __forceinline__ unsigned row_of(const RowDiv& r, unsigned n) {
  return (__umulhi(r.mul, n) + n) >> r.shift;
}
constexpr int kRestrictThreads = 128;

// Right-hand side of the coarse level (inactive DOFs 0), and its first smoothing
// step from zero.
template <class T>
__global__ void __launch_bounds__(kRestrictThreads) k_restrict(MgDims fd, MgDims cd, RowDiv rd,
                                                               const T* rf,
                                                               const uint8_t* __restrict__ cact,
                                                               T* __restrict__ bc,
                                                               FirstStep<T> first) {
  let_next_start();
  const unsigned id = blockIdx.x * unsigned(kRestrictThreads) + threadIdx.x;
  const int c = blockIdx.y;
  if (id >= rd.len * unsigned(cd.nny)) return;
  const int b = int(row_of(rd, id)), e = int(id - unsigned(b) * rd.len), a = e / 3, k = e - 3 * a;
  const int64_t dof = int64_t(c) * rd.len * cd.nny + id;
  const bool ac = cact[dof] != 0;
  wait_for_previous();
  const T s = restrict_dof<T, false>(fd, cd, rf, a, b, c, k);
  const T bv = ac ? s : T(0);
  bc[dof] = bv;
  if (first.kind == 1) {
    first.x[dof] = first.omega * first.dinv[dof] * bv;
  } else if (first.kind == 2) {
    T dnew;
    first.x[dof] = stencil_update<T, kCheb>(ac, T(0), T(0), bv, first.dinv[dof], T(0), first.coef,
                                            0, T(0), dnew);
    first.chd[dof] = dnew;
  }
}

// Prolongation + correction: x_f += P e_c on active fine DOFs.  One thread per
// fine node on a 3D grid: a thread per DOF repeats the node's index arithmetic and
// took 79 us against 33 on 257x129x129 nodes.
__global__ void __launch_bounds__(256) k_prolong_add(MgDims fd, MgDims cd,
                                                     const double* ec,
                                                     const uint8_t* __restrict__ fact,
                                                     double* xf) {
  let_next_start();
  const int a = blockIdx.x * 32 + threadIdx.x, b = blockIdx.y * 8 + threadIdx.y, c = blockIdx.z;
  if (a >= fd.nnx || b >= fd.nny) return;
  const int64_t n = (int64_t(c) * fd.nny + b) * fd.nnx + a;
  // The iterate and the mask are read unconditionally, in parallel with the
  // coarse values: a read under the mask's branch would wait for the mask first.
  const bool f0 = fact[3 * n] != 0, f1 = fact[3 * n + 1] != 0, f2 = fact[3 * n + 2] != 0;
  wait_for_previous();
  const double x0 = xf[3 * n], x1 = xf[3 * n + 1], x2 = xf[3 * n + 2];
  double s[3];
  prolong_node<double, false>(fd, cd, ec, a, b, c, s);
  if (f0) xf[3 * n] = x0 + s[0];
  if (f1) xf[3 * n + 1] = x1 + s[1];
  if (f2) xf[3 * n + 2] = x2 + s[2];
}

// The same for FP32, a thread per two fine nodes, (a, b) of layers 2 cz and 2 cz + 1:
// the loads that one node leaves in flight are too few to reach the memory's rate
// (257x129x129 nodes: 33 us for 108 MB), and the two share the coarse layer between
// them.  Each node's sum is prolong_node's, in its order.  256x128x128 solves 36.3 ->
// 35.8 ms, 128x64x64 10.43 -> 10.26.  In FP64, where an absent neighbour's products
// cost what they cost, it is the slower one (60x36x28 33.2 -> 33.7 ms).
__global__ void __launch_bounds__(256) k_prolong_pair(MgDims fd, MgDims cd, const float* ec,
                                                     const uint8_t* __restrict__ fact, float* xf) {
  let_next_start();
  const int a = blockIdx.x * 32 + threadIdx.x, b = blockIdx.y * 8 + threadIdx.y, cz = blockIdx.z;
  if (a >= fd.nnx || b >= fd.nny) return;
  const bool ta = tail_node(a, fd.ex, cd.align), tb = tail_node(b, fd.ey, cd.align);
  const int na = (a & 1) && !ta ? 2 : 1, nb = (b & 1) && !tb ? 2 : 1;
  const int ia = ta ? (a + 1) >> 1 : a >> 1, ib = tb ? (b + 1) >> 1 : b >> 1;
  const int64_t layer = int64_t(fd.nnx) * fd.nny, n = (2 * cz) * layer + int64_t(b) * fd.nnx + a;
  const bool two = 2 * cz + 1 < fd.nnz;
  const bool tail = two && tail_node(2 * cz + 1, fd.ez, cd.align);  // at coarse layer cz + 1
  bool on[2][3];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int k = 0; k < 3; ++k) on[q][k] = (q == 0 || two) && fact[3 * (n + q * layer) + k] != 0;
  wait_for_previous();
  // The iterate is read unconditionally, with the coarse values: a read under the
  // mask's branch would wait for the mask first.
  float xv[2][3], e[2][2][2][3];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int k = 0; k < 3; ++k) xv[q][k] = q == 0 || two ? xf[3 * (n + q * layer) + k] : 0.0f;
#pragma unroll
  for (int zz = 0; zz < 2; ++zz)
#pragma unroll
    for (int yy = 0; yy < 2; ++yy)
#pragma unroll
      for (int xx = 0; xx < 2; ++xx) {
        const bool in = xx < na && yy < nb && (zz == 0 || two) && ia + xx < cd.nnx &&
                        ib + yy < cd.nny && cz + zz < cd.nnz;
        const float* p = ec + 3 * ((int64_t(cz + zz) * cd.nny + ib + yy) * cd.nnx + ia + xx);
#pragma unroll
        for (int k = 0; k < 3; ++k) e[zz][yy][xx][k] = in ? p[k] : 0.0f;
      }
  const float wxy = (na == 2 ? 0.5f : 1.0f) * (nb == 2 ? 0.5f : 1.0f);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (q == 1 && !two) continue;
    const bool both = q == 1 && !tail;
    const float w = wxy * (both ? 0.5f : 1.0f);
    float s[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int zz = 0; zz < 2; ++zz) {
      if (!both && zz != (q == 1 ? 1 : 0)) continue;
#pragma unroll
      for (int yy = 0; yy < 2; ++yy)
#pragma unroll
        for (int xx = 0; xx < 2; ++xx)
#pragma unroll
          for (int k = 0; k < 3; ++k) s[k] += w * e[zz][yy][xx][k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (on[q][k]) xf[3 * (n + q * layer) + k] = xv[q][k] + s[k];
  }
}

// ---------------------------------------------------------- coarsest solve
// Dense A (row-major, nc x nc) from the coarsest stencil over the compact
// numbering cidx (-1 = inactive): node n writes its self block and, for every
// forward block, the entry and its transpose -- each entry exactly once.
template <class T>
__global__ void k_dense_from_stencil(MgDims d, const T* __restrict__ A,
                                     const int* __restrict__ cidx, int nc,
                                     double* __restrict__ D) {
  const int64_t nn = int64_t(d.nnx) * d.nny * d.nnz;
  const int j = blockIdx.y, di = 13 + j;
  for (int64_t n = blockIdx.x * int64_t(kThreads) + threadIdx.x; n < nn;
       n += int64_t(gridDim.x) * kThreads) {
    int a, b, c;
    node_abc(d, n, a, b, c);
    const int i = a + di % 3 - 1, jj = b + (di / 3) % 3 - 1, k = c + di / 9 - 1;
    if (i < 0 || i >= d.nnx || jj < 0 || jj >= d.nny || k >= d.nnz) continue;
    const int64_t m = (int64_t(k) * d.nny + jj) * d.nnx + i;
    for (int c1 = 0; c1 < 3; ++c1) {
      const int row = cidx[3 * n + c1];
      if (row < 0) continue;
      for (int c2 = 0; c2 < 3; ++c2) {
        const int col = cidx[3 * m + c2];
        if (col < 0) continue;
        const double v = double(A[int64_t(j * 9 + c1 * 3 + c2) * nn + n]);
        D[int64_t(row) * nc + col] = v;
        if (j > 0) D[int64_t(col) * nc + row] = v;
      }
    }
  }
}

// Explicit inverse of the coarsest operator, for small coarsest levels (each
// V-cycle then needs one dense matvec): block Gauss-Jordan, 32 pivots at a time,
// from one buffer into another.  For pivot block K with P = M_KK^-1,
//   M_ij <- M_ij - M_iK (P M_Kj),  M_iK <- -M_iK P,  M_Kj <- P M_Kj,  M_KK <- P.
// The operator is symmetric positive definite, so its pivots are a Cholesky
// factorisation's and need no exchange; one that is not positive sets *fail.
// Two launches per block: the pivot block's inverse by one CTA, 32 dependent
// steps of about 900 cycles (one FP64 division each), then every 16x16 tile of
// the matrix.  A blocked Cholesky factor, its inverse by one warp per column and
// their product took 510 us for 135 unknowns and 2.3 ms for 325.
constexpr int kGjBlock = 32, kGjTile = 16;
__global__ void __launch_bounds__(1024) k_gj_pivot(const double* __restrict__ M, int nc, int k0,
                                                   double* __restrict__ P,
                                                   int* __restrict__ fail) {
  __shared__ double s[32][33];
  __shared__ double inv;
  // An earlier block met a pivot that is not positive: the inverse will not be used.
  const bool failed = *fail != 0;
  __syncthreads();  // before this block's own verdict
  if (failed) return;
  const int nb = min(kGjBlock, nc - k0);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const bool in = tx < nb && ty < nb;
  double v = in ? M[int64_t(k0 + ty) * nc + k0 + tx] : (tx == ty ? 1.0 : 0.0);
  auto reciprocal = [&] {  // of the pivot this thread holds
    if (!(v > 0.0)) *fail = 1;
    inv = v > 0.0 ? 1.0 / v : 1.0;
  };
  s[ty][tx] = v;
  if (threadIdx.x == 0) reciprocal();
  __syncthreads();
  for (int k = 0; k < nb; ++k) {
    // Row k of the new matrix, then everyone's update; the next pivot's
    // reciprocal as soon as its entry is known.
    const double p = inv, col = s[ty][k];
    double row = 0.0;
    if (ty == k) {
      row = tx == k ? p : s[k][tx] * p;
      s[k][tx] = row;
    }
    __syncthreads();
    if (ty == k)
      v = row;
    else
      v = tx == k ? -(col * p) : fma(-col, s[k][tx], v);
    __syncthreads();  // row k and column k read
    s[ty][tx] = v;
    if (ty == k + 1 && tx == k + 1 && k + 1 < nb) reciprocal();
    __syncthreads();
  }
  if (in) P[ty * kGjBlock + tx] = v;
}

// `tall` tiles of one column each, whose R = P M_Kj is formed once: two thirds of a
// single tile's multiply-adds.
__global__ void __launch_bounds__(256) k_gj_update(const double* __restrict__ M, int nc, int k0,
                                                   const double* __restrict__ P,
                                                   double* __restrict__ out, int tall,
                                                   const int* __restrict__ fail) {
  if (*fail != 0) return;
  __shared__ double sP[32][33], sC[kGjTile][33], sR[32][kGjTile + 1], sT[32][kGjTile + 1];
  const int nb = min(kGjBlock, nc - k0);
  const int j0 = blockIdx.x * kGjTile;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  for (int e = t; e < 32 * 32; e += 256) {
    const int r = e >> 5, c = e & 31;
    sP[r][c] = r < nb && c < nb ? P[r * kGjBlock + c] : 0.0;
  }
  for (int e = t; e < kGjTile * 32; e += 256) {
    const int rr = e >> 4, cc = e & 15;  // row block K of these columns
    sT[rr][cc] = rr < nb && j0 + cc < nc ? M[int64_t(k0 + rr) * nc + j0 + cc] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // R = P M_Kj
    const int r = ty + 16 * h;
    double v = 0.0;
#pragma unroll 8
    for (int k = 0; k < 32; ++k) v = fma(sP[r][k], sT[k][tx], v);
    sR[r][tx] = v;
  }
  const int j = j0 + tx;
  const bool jk = j >= k0 && j < k0 + nb;
  for (int q = 0; q < tall; ++q) {
    const int i0 = (blockIdx.y * tall + q) * kGjTile;
    if (i0 >= nc) break;  // uniform over the CTA
    __syncthreads();      // R formed, the last tile's C read
    for (int e = t; e < kGjTile * 32; e += 256) {
      const int r = e >> 5, c = e & 31;  // column block K of this tile's rows
      sC[r][c] = i0 + r < nc && c < nb ? M[int64_t(i0 + r) * nc + k0 + c] : 0.0;
    }
    __syncthreads();
    const int i = i0 + ty;
    if (i >= nc || j >= nc) continue;
    const bool ik = i >= k0 && i < k0 + nb;
    double v;
    if (ik && jk) {
      v = sP[i - k0][j - k0];
    } else if (ik) {
      v = sR[i - k0][tx];
    } else {
      v = jk ? 0.0 : M[int64_t(i) * nc + j];
#pragma unroll 8
      for (int k = 0; k < 32; ++k) v = fma(-sC[ty][k], jk ? sP[k][j - k0] : sR[k][tx], v);
    }
    out[int64_t(i) * nc + j] = v;
  }
}

// Blocked right-looking Cholesky, panel width 32.  Step 1: factor the diagonal
// block in shared memory (one CTA); a non-positive pivot sets *fail.
__global__ void k_chol_diag(double* __restrict__ D, int nc, int k0, int* __restrict__ fail) {
  __shared__ double s[32][33];
  const int nb = min(32, nc - k0);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 32 threads
  if (tx < nb && ty < nb) s[ty][tx] = D[int64_t(k0 + ty) * nc + k0 + tx];
  __syncthreads();
  for (int j = 0; j < nb; ++j) {
    if (tx == 0 && ty == 0) {
      const double p = s[j][j];
      if (!(p > 0.0)) *fail = 1;
      s[j][j] = p > 0.0 ? sqrt(p) : 1.0;
    }
    __syncthreads();
    if (ty == 0 && tx > j && tx < nb) s[tx][j] /= s[j][j];
    __syncthreads();
    if (ty > j && tx > j && ty < nb && tx <= ty) s[ty][tx] -= s[ty][j] * s[tx][j];
    __syncthreads();
  }
  if (tx < nb && ty < nb && tx <= ty) D[int64_t(k0 + ty) * nc + k0 + tx] = s[ty][tx];
}

// Step 2: rows below the diagonal block: L[i, k0:k0+nb] = A[i, .] L_kk^-T.
__global__ void k_chol_panel(double* __restrict__ D, int nc, int k0) {
  __shared__ double L[32][33];
  const int nb = min(32, nc - k0);
  for (int t = threadIdx.x; t < 32 * 32; t += blockDim.x) {
    const int r = t / 32, c = t % 32;
    L[r][c] = (r < nb && c < nb && c <= r) ? D[int64_t(k0 + r) * nc + k0 + c] : 0.0;
  }
  __syncthreads();
  const int i = k0 + nb + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  double row[32];
  for (int c = 0; c < nb; ++c) row[c] = D[int64_t(i) * nc + k0 + c];
  for (int c = 0; c < nb; ++c) {
    double v = row[c];
    for (int t = 0; t < c; ++t) v -= row[t] * L[c][t];
    row[c] = v / L[c][c];
  }
  for (int c = 0; c < nb; ++c) D[int64_t(i) * nc + k0 + c] = row[c];
}

// Step 3: trailing update of the lower triangle, 32x32 tiles.
__global__ void k_chol_update(double* __restrict__ D, int nc, int k0) {
  const int nb = min(32, nc - k0);
  const int r0 = k0 + nb + blockIdx.y * 32, c0 = k0 + nb + blockIdx.x * 32;
  if (c0 > r0 + 31) return;
  __shared__ double Li[32][33], Lj[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int yy = ty; yy < 32; yy += blockDim.x / 32) {
    Li[yy][tx] = (r0 + yy < nc && tx < nb) ? D[int64_t(r0 + yy) * nc + k0 + tx] : 0.0;
    Lj[yy][tx] = (c0 + yy < nc && tx < nb) ? D[int64_t(c0 + yy) * nc + k0 + tx] : 0.0;
  }
  __syncthreads();
  for (int yy = ty; yy < 32; yy += blockDim.x / 32) {
    const int i = r0 + yy, j = c0 + tx;
    if (i >= nc || j >= nc || j > i) continue;
    double s = 0.0;
    for (int t = 0; t < nb; ++t) s += Li[yy][t] * Lj[tx][t];
    D[int64_t(i) * nc + j] -= s;
  }
}

// x = Ainv b on the compact numbering, gathered from / scattered to the level
// vector (cidx and cdof null: Ainv is over the level's own numbering); one warp per
// row of Ainv.  Each lane's products are one chain of FP64 multiply-adds, 64 cycles
// a link on its scheduler, so a warp takes one row and the rows are spread over all
// SMs.
constexpr int kRowWarps = 4;
template <class T>
__global__ void __launch_bounds__(32 * kRowWarps) k_coarse_inv_apply(
    const double* __restrict__ Ainv, int nc, const int* __restrict__ cidx,
    const int* __restrict__ cdof, int64_t ndof, const T* b, T* __restrict__ x) {
  let_next_start();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  // The matrix is read kAhead entries a lane at a time, those of the warp's first row
  // before the previous kernel has ended.
  constexpr int kAhead = 12;
  double m[kAhead];
  auto fetch = [&](const double* row, int k0) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int k = k0 + 32 * i;
      m[i] = k < nc ? row[k] : 0.0;
    }
  };
  if (warp < nc) fetch(Ainv + int64_t(warp) * nc, lane);
  wait_for_previous();
  if (cidx != nullptr)
    for (int64_t dd = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; dd < ndof;
         dd += int64_t(gridDim.x) * blockDim.x)
      if (cidx[dd] < 0) x[dd] = T(0);
  for (int r = warp; r < nc; r += nwarps) {
    const double* row = Ainv + int64_t(r) * nc;
    double s = 0.0;
    for (int k0 = lane; k0 < nc; k0 += 32 * kAhead) {
      if (r != warp || k0 != lane) fetch(row, k0);
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int k = k0 + 32 * i;
        if (k < nc) s += m[i] * widen(b[cdof != nullptr ? cdof[k] : k]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) x[cdof != nullptr ? cdof[r] : r] = T(s);
  }
}

// Forward and backward substitution with the factor, one CTA; the coarsest
// right-hand side is gathered from / scattered to the stencil-level vector.
template <class T>
__global__ void k_chol_solve(const double* __restrict__ L, int nc, const int* __restrict__ cidx,
                             int64_t ndof, const T* __restrict__ b, T* __restrict__ x,
                             double* __restrict__ work) {
  for (int64_t d = threadIdx.x; d < ndof; d += blockDim.x) {
    const int ci = cidx[d];
    if (ci >= 0) work[ci] = double(b[d]);
  }
  __syncthreads();
  for (int j = 0; j < nc; ++j) {  // L y = b
    __shared__ double yj;
    if (threadIdx.x == 0) {
      yj = work[j] / L[int64_t(j) * nc + j];
      work[j] = yj;
    }
    __syncthreads();
    for (int i = j + 1 + threadIdx.x; i < nc; i += blockDim.x) work[i] -= L[int64_t(i) * nc + j] * yj;
    __syncthreads();
  }
  for (int j = nc - 1; j >= 0; --j) {  // L^T x = y
    __shared__ double xj;
    if (threadIdx.x == 0) {
      xj = work[j] / L[int64_t(j) * nc + j];
      work[j] = xj;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < j; i += blockDim.x) work[i] -= L[int64_t(j) * nc + i] * xj;
    __syncthreads();
  }
  for (int64_t d = threadIdx.x; d < ndof; d += blockDim.x) {
    const int ci = cidx[d];
    x[d] = ci >= 0 ? T(work[ci]) : T(0);
  }
}
}  // namespace

// Level 1's Galerkin matrices of the coarse elements on the fast path
// (spos[ce] < 0: no aligned half element, every coarse DOF active, every fine
// DOF of every existing child kept), where the matrix is sum_c f_c G_c.  The
// sum runs over the children inside the grid with a nonzero modulus, in child
// order, one fused multiply-add per term -- k_galerkin's arithmetic, so the
// entries are bit-identical.  A block of 576 threads, one per matrix entry,
// holds its entry of the 8 G_c in registers and walks a batch of elements: the
// 576 entries of an element are 576 consecutive floats written by consecutive
// threads.
constexpr int kGalFastBatch = 32;  // elements per block step
__global__ void __launch_bounds__(576) k_galerkin1_fast(MgDims fd, MgDims cd,
                                                        const float* __restrict__ ef,
                                                        const int* __restrict__ spos,
                                                        const float* __restrict__ G,
                                                        float* __restrict__ Kc) {
  __shared__ float sf[kGalFastBatch][8];
  __shared__ int sfast[kGalFastBatch];
  const int rc = threadIdx.x;  // this thread's matrix entry, 0 .. 575
  float g[8];                  // its 8 child blocks' entries, for every element
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) g[ch] = G[ch * 576 + rc];
  const int64_t nce = int64_t(cd.ex) * cd.ey * cd.ez;
  for (int64_t base = int64_t(blockIdx.x) * kGalFastBatch; base < nce;
       base += int64_t(gridDim.x) * kGalFastBatch) {
    __syncthreads();  // the previous step's sf / sfast consumed
    if (threadIdx.x < kGalFastBatch * 8) {
      const int el = threadIdx.x >> 3, ch = threadIdx.x & 7;
      const int64_t ce = base + el;
      float f = 0.0f;
      if (ce < nce) {
        const int I = int(ce % cd.ex), J = int((ce / cd.ex) % cd.ey),
                  K = int(ce / (int64_t(cd.ex) * cd.ey));
        const int fi = 2 * I + cx(ch), fj = 2 * J + cy(ch), fk = 2 * K + cz(ch);
        if (fi < fd.ex && fj < fd.ey && fk < fd.ez) f = ef[(int64_t(fk) * fd.ey + fj) * fd.ex + fi];
      }
      sf[el][ch] = f;
      if (ch == 0) sfast[el] = ce < nce && spos[ce] < 0;
    }
    __syncthreads();
    for (int el = 0; el < kGalFastBatch; ++el) {
      if (!sfast[el]) continue;  // uniform over the block
      float acc = 0.0f;
#pragma unroll
      for (int ch = 0; ch < 8; ++ch) {
        const float f = sf[el][ch];
        if (f != 0.0f) acc = __fmaf_rn(f, g[ch], acc);
      }
      Kc[(base + el) * 576 + rc] = acc;
    }
  }
}

template <class T>
void mg_galerkin_level1(const MgDims& fd, const MgDims& cd, const T* ef, const uint8_t* fact,
                        const uint8_t* cact, const T* Ke, const T* G, T* Kc, cudaStream_t s,
                        const int* spos, const int* slist, int nspec) {
  const int64_t nce = int64_t(cd.ex) * cd.ey * cd.ez;
  const int* list = nullptr;
  int64_t n = nce;
  if constexpr (sizeof(T) == 4) {
    if (spos != nullptr) {
      const int64_t steps = (nce + kGalFastBatch - 1) / kGalFastBatch;
      const int nb = int(std::min<int64_t>(steps, 152 * 6));
      k_galerkin1_fast<<<nb, 576, 0, s>>>(fd, cd, ef, spos, G, Kc);
      TG_LAUNCH_CHECK();
      list = slist;
      n = nspec;
    }
  }
  if (n == 0) return;
  k_galerkin<T, true><<<nblk(n, 1), 256, 0, s>>>(fd, cd, ef, fact, cact, Ke, G, nullptr, Kc, list,
                                                 n);
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_galerkin_coarse(const MgDims& fd, const MgDims& cd, const T* Kf, const uint8_t* cact,
                        T* Kc, cudaStream_t s) {
  const int64_t nce = int64_t(cd.ex) * cd.ey * cd.ez;
  k_galerkin<T, false><<<nblk(nce, 1), 256, 0, s>>>(fd, cd, nullptr, nullptr, cact, nullptr,
                                                    nullptr, Kf, Kc, nullptr, nce);
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_assemble_stencil(const MgDims& d, const T* Kel, const uint8_t* act, T* A, T* invdiag,
                         cudaStream_t s) {
  const int64_t nn = int64_t(d.nnx) * d.nny * d.nnz;
  k_assemble_stencil<T><<<dim3(unsigned(nblk(nn)), A != nullptr ? 14 : 1), kThreads, 0, s>>>(
      d, Kel, act, A, invdiag);
  TG_LAUNCH_CHECK();
}

void mg_to_float(const double* src, float* dst, int64_t n, cudaStream_t s) {
  k_to_float<float><<<nblk(n), kThreads, 0, s>>>(src, dst, n);
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_stencil_op(int mode, const MgDims& d, const T* A, const uint8_t* act, const T* x,
                   const T* b, const T* invdiag, T omega, T* y, cudaStream_t s,
                   ChebStep ch, bool settled) {
  const int64_t nn = int64_t(d.nnx) * d.nny * d.nnz;
  auto run = [&](auto kernel, unsigned blocks, int threads) {
    if (settled)
      launch_behind_if_spread<T>(kernel, blocks, threads, 0, s, d, A, act, x, b, invdiag, omega, y,
                                 ch);
    else
      kernel<<<blocks, threads, 0, s>>>(d, A, act, x, b, invdiag, omega, y, ch);
    TG_LAUNCH_CHECK();
  };
  auto pick = [&](auto m) {
    constexpr int MODE = decltype(m)::value;
    if (nn <= split_max_nodes<T>())
      run(k_stencil_split<T, MODE>, unsigned((nn + 31) / 32), kSplitThreads);
    else
      run(k_stencil_op<T, MODE>,
          unsigned(((nn + 31) / 32 * 96 + kStencilThreads - 1) / kStencilThreads),
          kStencilThreads);
  };
  switch (mode) {
    case kApply: pick(std::integral_constant<int, kApply>{}); break;
    case kResidual: pick(std::integral_constant<int, kResidual>{}); break;
    case kDinvA: pick(std::integral_constant<int, kDinvA>{}); break;
    case kCheb: pick(std::integral_constant<int, kCheb>{}); break;
    default: pick(std::integral_constant<int, kSmooth>{});
  }
}

void mg_cheb_table(const double* lam, double ratio, int m, float* coef, cudaStream_t s) {
  if (m < 1 || 2 * m > kChebCoefStride) raise(TG_EINVAL, "Chebyshev degree out of range");
  k_cheb_table<<<1, 32, 0, s>>>(lam, ratio, m, coef);
  TG_LAUNCH_CHECK();
}

void mg_lambda_max(const MgDims& d, const float* A, const uint8_t* act, const float* invdiag,
                   float* v, float* w, int iters, double safety, double* part, double* nrm2,
                   unsigned* count, double* lam, cudaStream_t s) {
  const int64_t n = 3 * int64_t(d.nnx) * d.nny * d.nnz;
  k_pi_init<float><<<nblk(n), kThreads, 0, s>>>(act, n, v);
  TG_LAUNCH_CHECK();
  for (int it = 0; it < iters; ++it) {
    if (it == iters - 1) launch_dot_f(v, v, n, SumOut{part, nrm2, count}, s);
    mg_stencil_op<float>(kDinvA, d, A, act, v, nullptr, invdiag, 0.0f, w, s);
    std::swap(v, w);
  }
  launch_dot_f(v, v, n, SumOut{part, nrm2 + 1, count}, s);
  k_pi_lambda<<<1, 32, 0, s>>>(nrm2, safety, lam);
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_jacobi_first(const T* b, const T* invdiag, T omega, int64_t n, T* x, cudaStream_t s) {
  k_jacobi_first<T><<<nblk(n), kThreads, 0, s>>>(b, invdiag, omega, n, x);
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_restrict(const MgDims& fd, const MgDims& cd, const T* rf, const uint8_t* cact, T* bc,
                 cudaStream_t s, FirstStep<T> first) {
  const dim3 grid((3 * cd.nnx * cd.nny + kRestrictThreads - 1) / kRestrictThreads, cd.nnz);
  launch_behind_if_spread<T>(k_restrict<T>, grid, kRestrictThreads, 0, s, fd, cd, row_div(cd.nnx),
                             rf, cact, bc, first);
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_prolong_add(const MgDims& fd, const MgDims& cd, const T* ec, const uint8_t* fact, T* xf,
                    cudaStream_t s, bool joined) {
  const unsigned gx = unsigned(fd.nnx + 31) / 32, gy = unsigned(fd.nny + 7) / 8;
  auto run = [&](auto kernel, dim3 grid) {
    if (joined)
      kernel<<<grid, dim3(32, 8), 0, s>>>(fd, cd, ec, fact, xf);
    else
      launch_behind_if_spread<T>(kernel, grid, dim3(32, 8), 0, s, fd, cd, ec, fact, xf);
  };
  if constexpr (sizeof(T) == 4)
    run(k_prolong_pair, dim3(gx, gy, unsigned(fd.nnz + 1) / 2));
  else
    run(k_prolong_add, dim3(gx, gy, unsigned(fd.nnz)));
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_dense_from_stencil(const MgDims& d, const T* A, const int* cidx, int nc, double* D,
                           cudaStream_t s) {
  const int64_t nn = int64_t(d.nnx) * d.nny * d.nnz;
  TG_CUDA(cudaMemsetAsync(D, 0, sizeof(double) * size_t(nc) * nc, s));
  k_dense_from_stencil<T><<<dim3(unsigned(nblk(nn)), 14), kThreads, 0, s>>>(d, A, cidx, nc, D);
  TG_LAUNCH_CHECK();
}

void mg_cholesky(double* D, int nc, int* fail, cudaStream_t s) {
  for (int k0 = 0; k0 < nc; k0 += 32) {
    k_chol_diag<<<1, 1024, 0, s>>>(D, nc, k0, fail);
    TG_LAUNCH_CHECK();
    const int rest = nc - k0 - 32;
    if (rest <= 0) break;
    k_chol_panel<<<(rest + 127) / 128, 128, 0, s>>>(D, nc, k0);
    TG_LAUNCH_CHECK();
    const int tiles = (rest + 31) / 32;
    k_chol_update<<<dim3(tiles, tiles), 256, 0, s>>>(D, nc, k0);
    TG_LAUNCH_CHECK();
  }
}

double* mg_dense_start(int nc, double* a, double* inv) {
  return ((nc + kGjBlock - 1) / kGjBlock) & 1 ? a : inv;
}

void mg_dense_inverse(int nc, double* a, double* inv, double* pivot, int* fail, cudaStream_t s) {
  double* src = mg_dense_start(nc, a, inv);
  double* dst = src == a ? inv : a;
  const unsigned tiles = unsigned((nc + kGjTile - 1) / kGjTile);
  const unsigned tall = std::max(1u, std::min(8u, tiles * tiles / (4 * 152)));  // 4 CTAs an SM
  for (int k0 = 0; k0 < nc; k0 += kGjBlock) {
    k_gj_pivot<<<1, 1024, 0, s>>>(src, nc, k0, pivot, fail);
    TG_LAUNCH_CHECK();
    k_gj_update<<<dim3(tiles, (tiles + tall - 1) / tall), 256, 0, s>>>(src, nc, k0, pivot, dst,
                                                                      int(tall), fail);
    TG_LAUNCH_CHECK();
    std::swap(src, dst);
  }
}

template <class T>
void mg_coarse_inv_apply(const double* Ainv, int nc, const int* cidx, const int* cdof,
                         int64_t ndof, const T* b, T* x, cudaStream_t s) {
  const int nb = std::max(1, std::min(152 * 4, (nc + kRowWarps - 1) / kRowWarps));
  launch_behind_if_spread<double>(k_coarse_inv_apply<T>, nb, 32 * kRowWarps, 0, s, Ainv, nc, cidx,
                                  cdof, ndof, b, x);
  TG_LAUNCH_CHECK();
}

template <class T>
void mg_chol_solve(const double* L, int nc, const int* cidx, int64_t ndof, const T* b, T* x,
                   double* work, cudaStream_t s) {
  k_chol_solve<T><<<1, 512, 0, s>>>(L, nc, cidx, ndof, b, x, work);
  TG_LAUNCH_CHECK();
}

// ------------------------------------------- the last smoothed level, dense
// One V-cycle of the last smoothed level (its smoothing steps, the transfers and the
// coarsest solve) is a linear map of the level's right-hand side.  Launch by launch
// it is five dependent kernels of a few hundred rows (damped Jacobi, one sweep a side)
// or eleven (Chebyshev of degree four), 3-4 us each, in every V-cycle; as a dense
// matrix it is one product (FP64 675 DOFs: 3.6 MB from the L2, an FP64 multiply-add an
// entry; per iteration 86 -> 80 us at 24x8x8 FP64, 73 -> 68 at 60x20x20 mixed, 244 ->
// 224 at 128x64x64 mixed, Chebyshev).  This kernel forms the matrix once per hierarchy: column j
// is the cycle applied to the unit vector e_j.  Columns are independent, so a CTA
// takes NC of them through the whole cycle with its vectors in shared memory, and each
// stencil entry that it reads (coalesced, from the L2) serves NC columns.  FP64
// hierarchies are formed in FP64, FP32 ones in double-float arithmetic: their matrix
// is kept in FP64, as the coarsest inverse is.
namespace {

__device__ __forceinline__ double cy_mad(double a, double x, double acc) {
  return __fma_rn(a, x, acc);
}
__device__ __forceinline__ df cy_mad(float a, df x, df acc) {
  const float p = __fmul_rn(a, x.hi);
  return acc + df(p, __fmaf_rn(a, x.lo, __fmaf_rn(a, x.hi, -p)));
}
__device__ __forceinline__ df cy_mad(df a, df x, df acc) { return acc + a * x; }
__device__ __forceinline__ double cy_sub(double a, double b) { return a - b; }
__device__ __forceinline__ df cy_sub(df a, df b) { return a - b; }
template <class C>
__device__ __forceinline__ C cy_const(float v);
template <>
__device__ __forceinline__ double cy_const<double>(float v) {
  return double(v);
}
template <>
__device__ __forceinline__ df cy_const<df>(float v) {
  return df(v, 0.0f);
}
__device__ __forceinline__ void cy_load(double v, double& c) { c = v; }
__device__ __forceinline__ void cy_load(double v, df& c) { c = df_split(v); }
__device__ __forceinline__ double cy_store(double v) { return v; }
__device__ __forceinline__ double cy_store(df v) { return df_to_double(v); }

// Row r of node (a, bb, c) of the stencil times NC columns x (n apart).
template <class T, class C, int NC>
__device__ __forceinline__ void stencil_columns(const MgDims& d, const T* __restrict__ A,
                                                const C* x, int n, int a, int bb, int c, int r,
                                                C (&s)[NC]) {
  const int nn = d.nnx * d.nny * d.nnz, sy = d.nnx, sz = d.nnx * d.nny;
  const int node = c * sz + bb * sy + a;
  const T* An = A + node + int64_t(3 * r) * nn;
  auto block = [&](const T* e, int64_t step, int m) {
    const T a0 = e[0], a1 = e[step], a2 = e[2 * step];
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const C* v = x + q * n + 3 * m;
      s[q] = cy_mad(a2, v[2], cy_mad(a1, v[1], cy_mad(a0, v[0], s[q])));
    }
  };
#pragma unroll
  for (int q = 0; q < NC; ++q) s[q] = cy_const<C>(0.0f);
  block(An, nn, node);
#pragma unroll 1
  for (int j = 1; j < 14; ++j) {
    const int di = 13 + j;
    const int dx = di % 3 - 1, dy = (di / 3) % 3 - 1, dz = di / 9 - 1;
    const int off = dz * sz + dy * sy + dx;
    if ((a + dx) < d.nnx && (a + dx) >= 0 && (bb + dy) < d.nny && (bb + dy) >= 0 &&
        (c + dz) < d.nnz)
      block(An + int64_t(j * 9) * nn, nn, node + off);
    if ((a - dx) >= 0 && (a - dx) < d.nnx && (bb - dy) >= 0 && (bb - dy) < d.nny && (c - dz) >= 0)
      block(A + int64_t(j * 9 + r) * nn + (node - off), 3 * int64_t(nn), node - off);
  }
}

constexpr int kCycleThreads = 768;

// Smoothing: Chebyshev of degree cheb_m (> 0; coef) or `sweeps` damped-Jacobi steps a
// side, as the V-cycle's.  M is row-major over the level's n DOFs.
template <class T, class C, int NC>
__global__ void __launch_bounds__(kCycleThreads, 1) k_cycle_columns(
    MgDims d, MgDims cd, const T* __restrict__ A, const uint8_t* __restrict__ act,
    const T* __restrict__ dinv, const float* __restrict__ coef, int cheb_m, int sweeps, T omega,
    const double* __restrict__ Ainv, int nc, const int* __restrict__ cidx,
    const int* __restrict__ cdof, double* __restrict__ M) {
  extern __shared__ double2 cycle_smem[];
  const int nodes = d.nnx * d.nny * d.nnz, n = 3 * nodes;
  C* x = reinterpret_cast<C*>(cycle_smem);
  C* y = x + NC * n;
  C* rc = y + NC * n;
  C* ec = rc + NC * nc;
  C* dir = ec + NC * nc;  // Chebyshev only
  const int j0 = blockIdx.x * NC, items = ((nodes + 31) / 32) * 96;
  const C zero = cy_const<C>(0.0f);
  // One item is a (node, row) pair, a component per warp.
  auto each_row = [&](auto&& f) {
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
      const int node = (it / 96) * 32 + (it & 31), r = (it / 32) % 3;
      if (node >= nodes) continue;
      const int a = node % d.nnx, b = (node / d.nnx) % d.nny, c = node / (d.nnx * d.nny);
      f(a, b, c, r, 3 * node + r);
    }
  };
  // dinv (e_j - s), the preconditioned residual of column q at DOF i.
  auto dres = [&](int i, int q, T dv, C s) {
    return cy_mad(dv, cy_sub(cy_const<C>(i == j0 + q ? 1.0f : 0.0f), s), zero);
  };
  auto step = [&](int k) {  // one smoothing step from x into y, then swapped
    each_row([&](int a, int b, int c, int r, int i) {
      C s[NC];
      stencil_columns<T, C, NC>(d, A, x, n, a, b, c, r, s);
      const bool ac = act[i] != 0;
      const T dv = dinv[i];
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        C out = zero;
        if (cheb_m > 0) {
          C dn = zero;
          if (ac) {
            const C res = dres(i, q, dv, s[q]);
            dn = k == 0 ? cy_mad(cy_const<C>(coef[0]), res, zero)
                        : cy_mad(cy_const<C>(coef[2 * k]), dir[q * n + i],
                                 cy_mad(cy_const<C>(coef[2 * k + 1]), res, zero));
            out = x[q * n + i] + dn;
          }
          dir[q * n + i] = dn;
        } else if (ac) {
          out = cy_mad(omega, dres(i, q, dv, s[q]), x[q * n + i]);
        }
        y[q * n + i] = out;
      }
    });
    __syncthreads();
    C* t = x;
    x = y;
    y = t;
  };
  // The first step, from zero: only DOF j of column j is not zero.
  for (int i = threadIdx.x; i < NC * n; i += blockDim.x) {
    const int q = i / n, dof = i - q * n;
    C v = zero;
    if (dof == j0 + q && act[dof]) {
      v = dres(dof, q, dinv[dof], zero);
      v = cheb_m > 0 ? cy_mad(cy_const<C>(coef[0]), v, zero) : cy_mad(omega, v, zero);
    }
    x[i] = v;
    if (cheb_m > 0) dir[i] = v;
  }
  __syncthreads();
  const int steps = cheb_m > 0 ? cheb_m : sweeps;
  for (int k = 1; k < steps; ++k) step(k);
  each_row([&](int a, int b, int c, int r, int i) {
    C s[NC];
    stencil_columns<T, C, NC>(d, A, x, n, a, b, c, r, s);
    const bool ac = act[i] != 0;
#pragma unroll
    for (int q = 0; q < NC; ++q)
      y[q * n + i] =
          ac ? cy_sub(cy_const<C>(i == j0 + q ? 1.0f : 0.0f), s[q]) : zero;
  });
  __syncthreads();
  for (int i = threadIdx.x; i < NC * nc; i += blockDim.x) {  // restriction
    const int q = i / nc, dof = cdof[i - q * nc], k = dof % 3, cn = dof / 3;
    const int a = cn % cd.nnx, b = (cn / cd.nnx) % cd.nny, c = cn / (cd.nnx * cd.nny);
    float wx[3], wy[3], wz[3];
    axis_weights<float>(a, d.ex, d.nnx, cd.align, wx);
    axis_weights<float>(b, d.ey, d.nny, cd.align, wy);
    axis_weights<float>(c, d.ez, d.nnz, cd.align, wz);
    C s = zero;
    for (int p = 0; p < 27; ++p) {
      const int dx = p % 3, dy = (p / 3) % 3, dz = p / 9;
      const float w = wx[dx] * wy[dy] * wz[dz];
      if (w == 0.0f) continue;  // beyond the grid
      const int m = ((2 * c + dz - 1) * d.nny + 2 * b + dy - 1) * d.nnx + 2 * a + dx - 1;
      s = cy_mad(cy_const<C>(w), y[q * n + 3 * m + k], s);
    }
    rc[i] = s;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < NC * nc; i += blockDim.x) {  // coarsest solve
    const int q = i / nc, k = i - q * nc;
    C s = zero;
    for (int m = 0; m < nc; ++m) {
      C v;
      cy_load(Ainv[int64_t(m) * nc + k], v);
      s = cy_mad(v, rc[q * nc + m], s);
    }
    ec[i] = s;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < NC * n; i += blockDim.x) {  // prolongation
    const int q = i / n, dof = i - q * n, k = dof % 3, node = dof / 3;
    if (!act[dof]) continue;
    const int a = node % d.nnx, b = (node / d.nnx) % d.nny, c = node / (d.nnx * d.nny);
    const bool ta = tail_node(a, d.ex, cd.align), tb = tail_node(b, d.ey, cd.align),
               tc = tail_node(c, d.ez, cd.align);
    const bool ha = (a & 1) && !ta, hb = (b & 1) && !tb, hc = (c & 1) && !tc;
    const float w = (ha ? 0.5f : 1.0f) * (hb ? 0.5f : 1.0f) * (hc ? 0.5f : 1.0f);
    C s = x[i];
    for (int p = 0; p < 8; ++p) {
      const int dx = p & 1, dy = (p >> 1) & 1, dz = p >> 2;
      if ((dx && !ha) || (dy && !hb) || (dz && !hc)) continue;
      const int ia = (ta ? (a + 1) >> 1 : a >> 1) + dx, ib = (tb ? (b + 1) >> 1 : b >> 1) + dy,
                ic = (tc ? (c + 1) >> 1 : c >> 1) + dz;
      if (ia >= cd.nnx || ib >= cd.nny || ic >= cd.nnz) continue;
      const int e = cidx[3 * ((ic * cd.nny + ib) * cd.nnx + ia) + k];
      if (e >= 0) s = cy_mad(cy_const<C>(w), ec[q * nc + e], s);
    }
    x[i] = s;
  }
  __syncthreads();
  for (int k = 0; k < steps; ++k) step(k);
  for (int i = threadIdx.x; i < NC * n; i += blockDim.x) {
    const int dof = i / NC, q = i - dof * NC;
    if (j0 + q < n) M[int64_t(dof) * n + j0 + q] = cy_store(x[q * n + dof]);
  }
}

constexpr size_t kCycleSmem = size_t(227) * 1024;
// Columns of a CTA: the fewest that put every column on an SM of its own at once.
int cycle_columns(int64_t ndof) { return ndof <= 3 * 152 ? 3 : ndof <= 5 * 152 ? 5 : 7; }
size_t cycle_bytes(int64_t ndof, int nc, bool cheb) {
  return 8 * size_t(cycle_columns(ndof)) * (size_t(ndof) * (cheb ? 3 : 2) + 2 * size_t(nc));
}

}  // namespace

bool mg_dense_cycle_fits(int64_t ndof, int nc, bool cheb) {
  return ndof <= kDenseCycleDof && cycle_bytes(ndof, nc, cheb) <= kCycleSmem;
}

template <class T>
void mg_dense_cycle(const MgDims& d, const MgDims& cd, const T* A, const uint8_t* act,
                    const T* dinv, const float* coef, int cheb_m, int sweeps, T omega,
                    const double* Ainv, int nc, const int* cidx, const int* cdof, double* M,
                    cudaStream_t s) {
  using C = typename std::conditional<sizeof(T) == 8, double, df>::type;
  const int64_t nodes = int64_t(d.nnx) * d.nny * d.nnz, ndof = 3 * nodes;
  const size_t sm = cycle_bytes(ndof, nc, cheb_m > 0);
  const int threads = int(std::min<int64_t>(kCycleThreads, (nodes + 31) / 32 * 96));
  auto run = [&](auto kernel, int cols) {
    // The same value from every thread: a level's own size could fall short of what
    // another job is about to launch with.
    TG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(kCycleSmem)));
    kernel<<<unsigned((ndof + cols - 1) / cols), threads, sm, s>>>(
        d, cd, A, act, dinv, coef, cheb_m, sweeps, omega, Ainv, nc, cidx, cdof, M);
    TG_LAUNCH_CHECK();
  };
  switch (cycle_columns(ndof)) {
    case 3: run(k_cycle_columns<T, C, 3>, 3); break;
    case 5: run(k_cycle_columns<T, C, 5>, 5); break;
    default: run(k_cycle_columns<T, C, 7>, 7);
  }
}

#define TG_INST(T)                                                                            \
  template void mg_dense_cycle<T>(const MgDims&, const MgDims&, const T*, const uint8_t*,     \
                                  const T*, const float*, int, int, T, const double*, int,    \
                                  const int*, const int*, double*, cudaStream_t);             \
  template void mg_stencil_op<T>(int, const MgDims&, const T*, const uint8_t*, const T*,      \
                                 const T*, const T*, T, T*, cudaStream_t, ChebStep, bool);    \
  template void mg_jacobi_first<T>(const T*, const T*, T, int64_t, T*, cudaStream_t);         \
  template void mg_restrict<T>(const MgDims&, const MgDims&, const T*, const uint8_t*, T*,    \
                               cudaStream_t, FirstStep<T>);                                   \
  template void mg_prolong_add<T>(const MgDims&, const MgDims&, const T*, const uint8_t*, T*, \
                                  cudaStream_t, bool);                                        \
  template void mg_chol_solve<T>(const double*, int, const int*, int64_t, const T*, T*,       \
                                 double*, cudaStream_t);                                      \
  template void mg_coarse_inv_apply<T>(const double*, int, const int*, const int*, int64_t,    \
                                       const T*, T*, cudaStream_t);                           \
  template void mg_galerkin_level1<T>(const MgDims&, const MgDims&, const T*, const uint8_t*,  \
                                      const uint8_t*, const T*, const T*, T*, cudaStream_t,   \
                                      const int*, const int*, int);                           \
  template void mg_galerkin_coarse<T>(const MgDims&, const MgDims&, const T*, const uint8_t*,  \
                                      T*, cudaStream_t);                                      \
  template void mg_assemble_stencil<T>(const MgDims&, const T*, const uint8_t*, T*, T*,       \
                                       cudaStream_t);                                         \
  template void mg_dense_from_stencil<T>(const MgDims&, const T*, const int*, int, double*,   \
                                         cudaStream_t);
TG_INST(double)
TG_INST(float)
#undef TG_INST



// ------------------------------------------------- fused coarse V-cycle
// The small levels of the FP32 V-cycle -- from the first level with at most
// kFusedMaxNodes nodes down to the coarsest -- in one launch of one thread-block
// cluster (off by default: a launch per step, 3-4 us each with the four-thread
// stencil kernel, measured faster than a phase of this kernel, ~9 us on 16
// SMs).  Launch by launch, each step on these levels is a kernel of a few
// thousand DOFs whose cost is its latency.  Here every step of the same
// V-cycle is a phase of one kernel -- a
// cluster-stride loop with the arithmetic and summation order of the separate
// kernels (stencil_row, restrict_dof, prolong_node, the coarsest inverse) --
// and phases are separated by the cluster's hardware barrier (release/acquire
// at cluster scope, no spin loop).  The restriction into a level and that
// level's first smoothing step (from a zero iterate, so it needs no operator)
// share a phase.  Vectors written in earlier phases are read through L2
// (another SM of the cluster may have written them).  The iterate ping-pongs
// between each level's two buffers exactly as the launch-by-launch V-cycle does.
namespace {

// Every thread of the cluster arrives; writes before the barrier (global and
// shared memory) are visible to every thread of the cluster after it.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\t"
      "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Work items of a per-DOF phase: chunks of 32 nodes x 3 components, one
// component per warp, so a warp's stencil reads are coalesced.
__device__ __forceinline__ void dof_item(int64_t it, const MgDims& d, int& a, int& b, int& c,
                                         int& r, int64_t& n) {
  const int64_t chunk = it / 96;
  r = int((it / 32) % 3);
  n = chunk * 32 + (it & 31);
  node_abc(d, n, a, b, c);
}

__global__ void __launch_bounds__(kFusedThreads, 1) k_coarse_vcycle(FusedCoarse fc) {
  const int64_t tid = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t nthreads = int64_t(gridDim.x) * blockDim.x;
  const int top = fc.nlev - 1;  // the coarsest
  int cur[kFusedMaxLevels] = {};  // 0: the iterate is in xp, 1: in xq
  auto X = [&](int i) { return cur[i] ? fc.L[i].xq : fc.L[i].xp; };
  auto O = [&](int i) { return cur[i] ? fc.L[i].xp : fc.L[i].xq; };
  auto nitems = [&](int i) { return ((int64_t(fc.L[i].d.nnx) * fc.L[i].d.nny * fc.L[i].d.nnz + 31) / 32) * 96; };

  // One smoothing step of level i from its current iterate (or from zero) into
  // the other buffer: Chebyshev step k, or damped Jacobi (whose first sweep from
  // zero writes the iterate's own buffer, as the separate launches do).
  auto smooth = [&](int i, int k, bool from_zero) {
    const FusedLevel& L = fc.L[i];
    const float* xin = X(i);
    const bool in_place = from_zero && fc.cheb_m == 0;
    float* xout = in_place ? X(i) : O(i);
    const int64_t ni = nitems(i), nn = int64_t(L.d.nnx) * L.d.nny * L.d.nnz;
    for (int64_t it = tid; it < ni; it += nthreads) {
      int a, b, c, r;
      int64_t n;
      dof_item(it, L.d, a, b, c, r, n);
      if (n >= nn) continue;
      const int64_t dof = 3 * n + r;
      const float s = from_zero ? 0.0f : stencil_row<float, true>(L.d, L.A, xin, a, b, c, r);
      const float xv = from_zero ? 0.0f : __ldcg(xin + dof);
      const bool ac = L.act[dof] != 0;
      float out, dnew;
      if (fc.cheb_m > 0) {
        out = stencil_update<float, kCheb>(ac, s, xv, __ldcg(L.b + dof), L.dinv[dof], 0.0f, L.coef,
                                           k, (k > 0 && ac) ? __ldcg(L.chd + dof) : 0.0f, dnew);
        L.chd[dof] = dnew;
      } else {
        out = stencil_update<float, kSmooth>(ac, s, xv, __ldcg(L.b + dof), L.dinv[dof], fc.omega,
                                             nullptr, 0, 0.0f, dnew);
      }
      xout[dof] = out;
    }
    if (!in_place) cur[i] ^= 1;
  };
  // r = b - A x of level i into its other buffer (the iterate stays).
  auto residual = [&](int i) {
    const FusedLevel& L = fc.L[i];
    const float* xin = X(i);
    float* rout = O(i);
    const int64_t ni = nitems(i), nn = int64_t(L.d.nnx) * L.d.nny * L.d.nnz;
    for (int64_t it = tid; it < ni; it += nthreads) {
      int a, b, c, r;
      int64_t n;
      dof_item(it, L.d, a, b, c, r, n);
      if (n >= nn) continue;
      const int64_t dof = 3 * n + r;
      const float s = stencil_row<float, true>(L.d, L.A, xin, a, b, c, r);
      rout[dof] = L.act[dof] ? __ldcg(L.b + dof) - s : 0.0f;
    }
  };
  // Level i's residual restricted into level i + 1's right-hand side, and --
  // for a smoothed level -- its first smoothing step from zero, per DOF.
  auto restrict_to = [&](int i) {
    const FusedLevel& F = fc.L[i];
    const FusedLevel& C = fc.L[i + 1];
    const float* rf = O(i);
    const bool smoothed = i + 1 < top;
    const int64_t nn = int64_t(C.d.nnx) * C.d.nny * C.d.nnz;
    float* xfirst = C.xq;  // Chebyshev step 0 writes the other buffer (x = 0 in xp)
    if (smoothed && fc.cheb_m == 0) xfirst = C.xp;  // Jacobi's first sweep writes the iterate
    for (int64_t n = tid; n < nn; n += nthreads) {
      int a, b, c;
      node_abc(C.d, n, a, b, c);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int64_t dof = 3 * n + k;
        const float s = restrict_dof<float, true>(F.d, C.d, rf, a, b, c, k);
        const float bv = C.act[dof] ? s : 0.0f;
        C.b[dof] = bv;
        if (!smoothed) continue;
        if (fc.cheb_m > 0) {
          const float dn = C.act[dof] ? C.coef[0] * (C.dinv[dof] * (bv - 0.0f)) : 0.0f;
          C.chd[dof] = dn;
          xfirst[dof] = C.act[dof] ? 0.0f + dn : 0.0f;
        } else {
          xfirst[dof] = fc.omega * C.dinv[dof] * bv;
        }
      }
    }
    if (smoothed && fc.cheb_m > 0) cur[i + 1] = 1;
  };
  auto prolong_from = [&](int i) {  // level i's iterate += P (level i + 1's iterate)
    const FusedLevel& F = fc.L[i];
    const FusedLevel& C = fc.L[i + 1];
    const float* ec = X(i + 1);
    float* xf = X(i);
    const int64_t nn = int64_t(F.d.nnx) * F.d.nny * F.d.nnz;
    for (int64_t n = tid; n < nn; n += nthreads) {
      int a, b, c;
      node_abc(F.d, n, a, b, c);
      float s[3];
      prolong_node<float, true>(F.d, C.d, ec, a, b, c, s);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (F.act[3 * n + k]) xf[3 * n + k] = __ldcg(xf + 3 * n + k) + s[k];
    }
  };
  // x = A^-1 b over the compact numbering, or the last smoothed level's dense cycle
  // over its own (cidx and cdof null), a warp per row.
  auto coarsest = [&]() {
    const FusedLevel& L = fc.L[top];
    const int64_t ndof = 3 * int64_t(L.d.nnx) * L.d.nny * L.d.nnz;
    for (int64_t dd = tid; dd < ndof; dd += nthreads)
      if (fc.cidx != nullptr && fc.cidx[dd] < 0) L.xp[dd] = 0.0f;
    const int lane = threadIdx.x & 31;
    const int64_t warp = tid >> 5, nwarps = nthreads >> 5;
    for (int64_t row = warp; row < fc.nc; row += nwarps) {
      double s = 0.0;
      for (int k = lane; k < fc.nc; k += 32)
        s += fc.Ainv[row * fc.nc + k] * double(__ldcg(L.b + (fc.cdof != nullptr ? fc.cdof[k] : k)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) L.xp[fc.cdof != nullptr ? fc.cdof[row] : row] = float(s);
    }
    cur[top] = 0;
  };

  // Down: level 0's first step from zero (its right-hand side came from level 1).
  smooth(0, 0, true);
  cluster_sync_all();
  for (int i = 0; i < top; ++i) {
    const int steps = fc.cheb_m > 0 ? fc.cheb_m : fc.sweeps;
    for (int k = 1; k < steps; ++k) {
      smooth(i, k, false);
      cluster_sync_all();
    }
    residual(i);
    cluster_sync_all();
    restrict_to(i);
    cluster_sync_all();
  }
  coarsest();
  for (int i = top - 1; i >= 0; --i) {
    cluster_sync_all();
    prolong_from(i);
    const int steps = fc.cheb_m > 0 ? fc.cheb_m : fc.sweeps;
    for (int k = 0; k < steps; ++k) {
      cluster_sync_all();
      smooth(i, k, false);
    }
  }
}

}  // namespace

// Cluster size of the fused launch: the largest of 16 (non-portable), 8, 4, 2
// CTAs that the device can co-schedule with this kernel's resources.
int fused_coarse_blocks() {
  static std::atomic<int> cached{0};
  const int c = cached.load();
  if (c > 0) return c;
  TG_CUDA(cudaFuncSetAttribute(k_coarse_vcycle, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  int best = 1;
  for (int cs : {16, 8, 4, 2}) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = unsigned(cs);
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(cs));
    cfg.blockDim = dim3(kFusedThreads);
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_coarse_vcycle, &cfg) == cudaSuccess && n >= 1) {
      best = cs;
      break;
    }
    cudaGetLastError();  // an unsupported size is not an error of the solve
  }
  cached.store(best);
  return best;
}

void mg_coarse_vcycle_fused(const FusedCoarse& fc, cudaStream_t s) {
  const int cs = fused_coarse_blocks();
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(cs);
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(unsigned(cs));
  cfg.blockDim = dim3(kFusedThreads);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  TG_CUDA(cudaLaunchKernelEx(&cfg, k_coarse_vcycle, fc));
  note_launch();
}

}  // namespace tg
