// k_operator.cu -- the matrix-free hex8 operator on the voxel grid.
//
// Reference counterpart: mf_apply_full / apply_one_element / axpy24
// (core/src/fea/matfree.cpp:535-553, :110-123, :75-96) and the reduced-system
// matvec apply_kgg_raw (matfree.cpp:595-608).  The reference multiplies every
// element's 24 DOFs by the dense 24x24 Ke (576 mul+add per element).  Here the
// same operator is evaluated in the Walsh-modal basis of the trilinear element:
//
//   u(xi) = sum_S m[S] prod_{i in S} xi_i,   S subset of {x,y,z}   (8 modes)
//
// The gradient coefficient of monomial T in du_j/dxi_i is m_j[T u {i}], and the
// monomials are orthogonal on the cube, so the 2x2x2-Gauss strain energy splits
// into independent blocks per T with weights 8/3^|T|.  K u is the gradient of
// that energy: a forward Walsh transform (24 add/sub per component), about 50
// flops of isotropic "stress" per element, and the inverse transform.  About 200
// floating-point operations replace 576 FMAs -- it matters because GB300 runs
// FP64 at roughly 1/64 of its FP32 rate.  The result equals Ke u to rounding
// (checked against the oracle's dense Ke in the tests).
//
// Scheduling: warps march in z over node columns (k_fine_march below), sharing
// the transforms between neighbouring elements; each node is finished exactly
// once, without atomics, in a fixed summation order -- the apply is
// deterministic run to run.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "tg_internal.h"
#include "tg_launch.h"
#include "tg_march.h"
#include "tg_reduce.h"

namespace tg {

ModalConsts ModalConsts::make(double nu, double h) {
  ModalConsts c;
  const double lam = nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
  const double mu = 1.0 / (2.0 * (1.0 + nu));
  double s = h / 16.0;
  for (int k = 0; k < 3; ++k) {
    c.L[k] = lam * s;
    c.M[k] = mu * s;
    s /= 3.0;
  }
  c.kdiag = 0.0;  // filled by the caller from the unit-modulus Ke (all 24 equal)
  return c;
}

struct GridDev {
  int nx, ny, nz, nnx, nny, nnz;
};

// Batched periodic applies (homogenization): system bi of the batch reads x, b,
// y at bi * sx and the cell fields (factors, kept bits) of cell bi / nrhs.  On the
// torus nodes and elements coincide (nnx == nx ...).
// Systems whose entry of `run` is not 1 are skipped: their y and partials stay.
struct BatchDev {
  int nrhs;         // systems per cell
  int64_t sx, se;   // strides: DOF vectors; a cell's element factors and kept bits
  const int* run;   // null: every system
  int flat;         // rows numbered in one sequence of nx + 2 columns (periodic_flat)
};

__device__ __forceinline__ int wrap_index(int a, int n) {
  a %= n;
  return a < 0 ? a + n : a;
}
// The same for -1 <= a <= n + 1 without a division (n = 1 wraps twice).
__device__ __forceinline__ int wrap_near(int a, int n) {
  a = a < 0 ? a + n : a;
  a = a >= n ? a - n : a;
  return a >= n ? a - n : a;
}

// ---------------------------------------------------------------------------
// The element operator in the modal basis, shared between neighbours.
//
// A trilinear element's modes are a tensor product, so the transform of an
// element is the z-difference and z-sum of the xy-modes of its two faces, and a
// face's xy-modes are y-sums and y-differences of the x-sums and x-differences
// of its two node rows.  Marching in z, a face is transformed once and serves
// the element above and the element below; with several element rows per thread
// a node row is x-transformed once for the rows on both sides.  The inverse runs
// the same way back: the top face of one element layer and the bottom face of
// the next are added as xy-modes, so y- and x-inverse, the exchange between
// lanes and the hand-over between warps happen once per node layer.  Per element
// and layer that is about 141 operations (x 12 forward, 6 back; y 12 and 12; z
// 21 and 30; 39 for the stress; 9 for combining), against 217 when every element
// transforms its own 24 values and combines 24 results, with half the shuffles.

// Tiling.  A CTA is W warps; lanes run along x, thread rows along y, the march
// along z.
//   x: the node columns of all the y strips are numbered in one sequence (strip
//      by strip), and a warp owns kOwn consecutive ones, so no lane idles at a
//      row's end; lane 0 is the halo column on the left, and with 30 owned
//      columns lane 31 only supplies its values (FP64 owns 31: lane 31 loads its
//      right neighbour itself, a load its arithmetic hides).
//      At a strip's end the next lane belongs to another strip: the element
//      column there lies past the grid, its factor is 0.
//      Periodic cells: a row is a group of nx lanes with no halo, 32 / nx rows
//      side by side in a warp (nx 8, 16, 32 fill it); where that leaves more lanes
//      idle than two halo columns per row do (nx 17-26, or above 32), rows of
//      nx + 2 columns are numbered in one sequence as above.
//   y: a warp evaluates R element rows; the node row between two warps is
//      finished by the lower one, the upper warp's share handed over as x-modes
//      through shared memory (one barrier per layer).  A CTA finishes W R - 1
//      node rows.
//   z: KZ node layers per CTA, and one more element layer below.
// Every node is finished once, by one thread, in an order that does not depend
// on the tiling: results are deterministic, and the same under every schedule.
//
// Two packed rows (FP32): what a step reads -- the next node layer's three rows,
// the element factors, the right-hand side and the inverse diagonal -- is copied
// to shared memory kDepth layers ahead (cp.async, each warp its own copy, so
// only the warp waits).  One layer ahead in registers left 38 % of the issue
// slots to DRAM latency (74 us on 256x128x128): 12 warps of 160 registers keep
// 14 KB per SM in flight, and the latency times the bandwidth needs three times
// that.  Copies are of consecutive words; rows and layers past the grid are read
// from its edge, since the elements there have factor 0.
//
// Measured per launch, one element at a time -> this kernel: FP32 apply on
// 256x128x128 71.8 -> 51.3 us (119 MB; issue-bound, 2.4 of 4 instructions per
// cycle), on 60x20x20 38 -> 5; FP64 apply on 256x128x128 2,340 -> 1,393 us (FP64
// units busy), on 60x36x28 258 -> 43, on 24x8x8 133 -> 14 (two layers of ~150
// FP64 instructions at 64 cycles).

// Words of one layer's copies of one warp: 3 rows of x, 2 rows of factors, and 2
// rows each of b and the inverse diagonal where the mode reads them.
template <int MODE>
__host__ __device__ constexpr int slot_words() {
  return 3 * kRowWords + 64 + (MODE != kApply ? 2 * kRowWords : 0) +
         (MODE == kSmooth ? 2 * kRowWords : 0);
}

template <class V, class T, int MODE, bool PER>
__global__ void __launch_bounds__(32 * RowsOf<V>::kMaxWarps, 1)
    k_fine_march(GridDev g, ModalT<typename RowsOf<V>::S> mc, int KZ, int nss,
                 const T* ef, const uint8_t* __restrict__ kn,
                 const T* x, const T* b, const T* invdiag,
                 T omega, T* __restrict__ y, SumOut dot, int guard,
                 BatchDev bd) {
  let_next_start();
  using S = typename RowsOf<V>::S;
  constexpr int R = RowsOf<V>::R;
  constexpr bool kXtra = !PER && std::is_same<S, double>::value;  // lane 31 loads its neighbour
  constexpr int kOwn = kXtra ? 31 : 30;
  extern __shared__ __align__(16) unsigned char march_smem[];
  S* const xs = reinterpret_cast<S*>(march_smem);  // [2][W][6][32]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int rows = W * R - 1;
  if constexpr (PER) {
    wait_for_previous();
    const int bi = blockIdx.z, cell = bi / bd.nrhs;
    if (bd.run != nullptr && bd.run[bi] != 1) return;  // uniform over the CTA
    x += bi * bd.sx;
    y += bi * bd.sx;
    if (b) b += bi * bd.sx;
    ef += cell * bd.se;
    if (kn) kn += cell * bd.se;
  }
  // This lane's element column ex, strip ss, and the lanes its x neighbours are in.
  int ex, ss, rl, ll;
  bool own_x;
  if constexpr (PER) {
    rl = lane < 31 ? lane + 1 : lane;
    ll = lane > 0 ? lane - 1 : lane;
    if (bd.flat) {
      const int len = g.nx + 2, q = blockIdx.x * kOwn - 1 + lane;
      ss = q > 0 ? q / len : 0;
      const int c = q - ss * len;  // 0: the left halo, 1 .. nx: owned, nx + 1: the right neighbour
      own_x = lane >= 1 && lane <= kOwn && ss < nss && c >= 1 && c <= g.nx;
      ex = wrap_index(c - 1, g.nx);
    } else {
      const int ng = 32 / g.nx, gi = lane / g.nx;
      ex = lane - gi * g.nx;
      ss = blockIdx.x * ng + gi;
      own_x = gi < ng && ss < nss;
      rl = own_x ? gi * g.nx + (ex + 1 == g.nx ? 0 : ex + 1) : lane;
      ll = own_x ? gi * g.nx + (ex == 0 ? g.nx - 1 : ex - 1) : lane;
      if (!own_x) ss = 0;
    }
  } else {
    const int q = blockIdx.x * kOwn - 1 + lane;
    ss = q > 0 ? q / g.nnx : 0;
    ex = q - ss * g.nnx;
    own_x = lane >= 1 && lane <= kOwn && ss < nss;
    rl = lane < 31 ? lane + 1 : lane;
    ll = lane > 0 ? lane - 1 : lane;
  }
  const int ey0 = ss * rows - 1 + w * R;  // element rows ey0 .. ey0+R-1, node rows ey0 .. ey0+R
  const bool vx = PER || (ex >= 0 && ss < nss);
  const int plane = g.nnx * g.nny, eplane = g.nx * g.ny;
  int no[R + 1];  // the nodes' indexes within a layer
  bool rv[R + 1], rown[R + 1];
#pragma unroll
  for (int i = 0; i <= R; ++i) {
    const int yr = ey0 + i;
    rv[i] = vx && (PER || (yr >= 0 && yr < g.nny));
    rown[i] = own_x && i >= 1 && (i < R || w < W - 1) && yr < g.nny;
    no[i] = g.nnx * (PER ? wrap_index(yr, g.nny) : yr) + ex;
  }
  int eo[R];
  bool ev[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int er = ey0 + j;
    ev[j] = vx && (PER || (ex < g.nx && er >= 0 && er < g.ny));
    eo[j] = (PER ? wrap_index(er, g.ny) : er) * g.nx + ex;
  }
  const int z0 = blockIdx.y * KZ;

  // Copied rows: word 32 j + lane of a row is component (32 j + lane) % 3 of the
  // lane (32 j + lane) / 3's node, whose strip and clamped (wrapped) row give the
  // word's offset within a layer.
  constexpr bool kPipe = R == 2;
  constexpr int kSlot = kPipe ? slot_words<MODE>() : 0;
  float* const mine = reinterpret_cast<float*>(xs + 2 * W * 192) + w * (kDepth + 1) * kSlot;
  const unsigned mine_s = static_cast<unsigned>(__cvta_generic_to_shared(mine));
  unsigned eb[R];  // bytes; and the bytes to copy: 4, or 0 for an absent element
  int eok[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    eb[j] = ev[j] ? 4u * unsigned(eo[j]) : 0u;
    eok[j] = ev[j] ? 4 : 0;
  }
  unsigned wo[kPipe ? 3 : 1][kPipe ? 3 : 1];  // bytes
  if constexpr (kPipe) {
    const int yc0 = PER ? 0 : ey0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int word = 32 * j + lane, m = word / 3, k = word - 3 * m;
      const int exm = __shfl_sync(0xffffffffu, PER ? ex : min(max(ex, 0), g.nnx - 1), m);
      const int ym = __shfl_sync(0xffffffffu, PER ? ss * rows - 1 + w * R : yc0, m);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int yr = PER ? wrap_index(ym + i, g.nny) : min(max(ym + i, 0), g.nny - 1);
        wo[j][i] = 4u * unsigned(3 * (g.nnx * yr + exm) + k);
      }
    }
  }
  if constexpr (!PER) wait_for_previous();
  // The copies of step s: node layer ez + 1, factors, b and diagonal of layer ez.
  auto copy_step = [&](int s) {
    if constexpr (kPipe) {
      const int ez = z0 - 1 + s;
      if (s <= KZ && ez <= g.nnz - 1) {
        const unsigned st = mine_s + (unsigned(s) % (kDepth + 1)) * (4u * kSlot) + 4u * lane;
        const float* xl =
            x + 3 * (plane * (PER ? wrap_near(ez + 1, g.nnz) : min(ez + 1, g.nnz - 1)));
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            copy_word(st + 4 * (i * kRowWords + 32 * j), at(xl, wo[j][i]));
        const bool vc = PER || (ez >= 0 && ez < g.nz);
        const float* el = ef + eplane * (PER ? wrap_near(ez, g.nz) : (vc ? ez : 0));
#pragma unroll
        for (int j = 0; j < 2; ++j)
          copy_word_or_zero(st + 4 * (3 * kRowWords + 32 * j), at(el, eb[j]), vc ? eok[j] : 0);
        if (MODE != kApply && s >= 1) {
          const float *bl = b + 3 * plane * ez, *dl = invdiag + 3 * plane * ez;
#pragma unroll
          for (int i = 1; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const unsigned d = st + 4 * (3 * kRowWords + 64 + (i - 1) * kRowWords + 32 * j);
              copy_word(d, at(bl, wo[j][i]));
              if (MODE == kSmooth) copy_word(d + 8 * kRowWords, at(dl, wo[j][i]));
            }
        }
      }
      copy_commit();
    }
  };

  auto load_layer = [&](int c, S (&r)[R + 1][3], S (&e)[R + 1][3]) {
    const bool vc = PER || (c >= 0 && c < g.nnz);
    const int o = plane * (PER ? wrap_near(c, g.nnz) : c);
#pragma unroll
    for (int i = 0; i <= R; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        r[i][k] = (vc && rv[i]) ? load_c<S>(x[3 * (o + no[i]) + k]) : czero<S>();
        if constexpr (kXtra)
          e[i][k] = (lane == 31 && vc && rv[i] && ex + 1 < g.nnx) ? load_c<S>(x[3 * (o + no[i]) + 3 + k])
                                                                   : czero<S>();
      }
  };
  auto load_f = [&](int c, S (&f)[R]) {
    const bool vc = PER || (c >= 0 && c < g.nz);
    const int o = eplane * (PER ? wrap_near(c, g.nz) : c);
#pragma unroll
    for (int j = 0; j < R; ++j) f[j] = (vc && ev[j]) ? load_c<S>(ef[o + eo[j]]) : czero<S>();
  };
  auto face = [&](const S (&r)[R + 1][3], const S (&e)[R + 1][3], V (&F)[3][4]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      S a[R + 1], nb[R + 1];
#pragma unroll
      for (int i = 0; i <= R; ++i) {
        a[i] = r[i][k];
        nb[i] = shfl_at(r[i][k], rl);
        if constexpr (kXtra) nb[i] = lane == 31 ? e[i][k] : nb[i];
      }
      face_modes<V, S>(a, nb, F[k]);
    }
  };

  // The first chunk of a bounded grid has no element layer below it.
  const int s0 = (!PER && z0 == 0) ? 1 : 0;
  S raw[R + 1][3], rext[R + 1][3], keep[R + 1][3];
  V Fc[3][4], pend[3][4];
  load_layer(z0 - 1 + s0, raw, rext);
  face(raw, rext, Fc);
#pragma unroll
  for (int i = 0; i <= R; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) keep[i][k] = raw[i][k];
  S fn[R];
  if constexpr (kPipe) {
#pragma unroll 1
    for (int q = 0; q < kDepth; ++q) copy_step(s0 + q);
  } else {
    load_layer(z0 + s0, raw, rext);
    load_f(z0 - 1 + s0, fn);
  }
  unsigned kbn[R + 1];  // kept bits of the owned rows, requested a step ahead
  auto load_kb = [&](int s, unsigned (&kb)[R + 1]) {
    const int ez = z0 - 1 + s;
#pragma unroll
    for (int i = 1; i <= R; ++i)
      kb[i] = kn == nullptr
                  ? 7u
                  : (s >= 1 && ez < g.nnz && rown[i] ? unsigned(*at(kn + plane * ez, unsigned(no[i]))) : 0u);
  };
  load_kb(s0, kbn);
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int m = 0; m < 4; ++m) pend[k][m] = vset<V>(czero<S>());
  S dsum = czero<S>();
  // Periodic FP32: a thread's share of p.Ap in runs of eight layers (16 nodes with two
  // rows), the runs added up as a double-float, since a march takes up to 64 layers.
  constexpr bool kRuns = PER && MODE == kApply && std::is_same<S, float>::value;
  df druns(0.0f, 0.0f);

  // Two steps per pass: this layer's faces become the last layer's without moves.
#pragma unroll(kPipe ? 2 : 1)
  for (int s = s0; s <= KZ; ++s) {
    const int ez = z0 - 1 + s;
    if (ez > g.nnz - 1) break;  // uniform: the last chunk ends with the grid
    const bool out_z = s >= 1;
    const int oz = plane * ez;
    unsigned kb[R + 1];
#pragma unroll
    for (int i = 1; i <= R; ++i) kb[i] = kbn[i];
    if (s < KZ) load_kb(s + 1, kbn);
    T bv[R + 1][3], dv[R + 1][3];
    V f;
    V Fn[3][4];
    S knext[R + 1][3];
    const float* st = nullptr;
    if constexpr (kPipe) {
      copy_wait_ahead();
      __syncwarp();  // every lane's words of this step are in, and the last step's are read
      copy_step(s + kDepth);
      st = mine + (s % (kDepth + 1)) * kSlot;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        S a[3], nb[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          a[i] = st[i * kRowWords + 3 * lane + k];
          nb[i] = st[i * kRowWords + 3 * rl + k];
        }
        face_modes<V, S>(a, nb, Fn[k]);
#pragma unroll
        for (int i = 1; i < 3; ++i) knext[i][k] = a[i];
      }
      f = make_float2(st[3 * kRowWords + lane], st[3 * kRowWords + 32 + lane]);
    } else {
      // Requested now, used at the end of the step: right-hand side and inverse
      // diagonal; and the layer after the next.
#pragma unroll
      for (int i = 1; i <= R; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const bool ok = out_z && rown[i];
          bv[i][k] = (MODE != kApply && ok) ? b[3 * (oz + no[i]) + k] : T(0);
          dv[i][k] = (MODE == kSmooth && ok) ? invdiag[3 * (oz + no[i]) + k] : T(0);
        }
      f = fn[0];
      face(raw, rext, Fn);
#pragma unroll
      for (int i = 1; i <= R; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) knext[i][k] = raw[i][k];
      if (s < KZ) {
        load_layer(ez + 2, raw, rext);
        load_f(ez + 1, fn);
      }
    }
    // z: element modes from the two faces (mode 0 is never used).
    V u[3][8];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      u[k][0] = vset<V>(czero<S>());
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (m > 0) u[k][m] = vadd(Fn[k][m], Fc[k][m]);
        u[k][m | 4] = vsub(Fn[k][m], Fc[k][m]);
      }
    }
    modal_stress<V, S>(mc, f, u[0], u[1], u[2]);
    if (guard) {
      // Values at a node of absent elements only must not reach its neighbours
      // whatever they are (0 times an infinity or NaN is not 0).
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int m = 1; m < 8; ++m) {
          if constexpr (R == 2) {
            u[k][m].x = f.x != 0.0f ? u[k][m].x : 0.0f;
            u[k][m].y = f.y != 0.0f ? u[k][m].y : 0.0f;
          } else {
            u[k][m] = nonzero(f) ? u[k][m] : czero<S>();
          }
        }
    }
    // Back in z: this layer's bottom face completes node layer ez, its top face
    // waits; then y.
    V lo[3][2], up[3][2];  // x-modes of the thread's element rows' lower and upper node rows
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      V P[4];
      P[0] = vsub(pend[k][0], u[k][4]);
      pend[k][0] = u[k][4];
#pragma unroll
      for (int m = 1; m < 4; ++m) {
        P[m] = vadd(pend[k][m], vsub(u[k][m], u[k][m | 4]));
        pend[k][m] = vadd(u[k][m], u[k][m | 4]);
      }
      lo[k][0] = vsub(P[0], P[2]);
      lo[k][1] = vsub(P[1], P[3]);
      up[k][0] = vadd(P[0], P[2]);
      up[k][1] = vadd(P[1], P[3]);
    }
    S* const buf = xs + (s & 1) * (W * 192);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        if constexpr (R == 2)
          buf[w * 192 + (2 * k + m) * 32 + lane] = lo[k][m].x;
        else
          buf[w * 192 + (2 * k + m) * 32 + lane] = lo[k][m];
      }
    // Writes node row i of layer ez from its x-modes r[k][2].
    auto finish = [&](int i, const S (&r)[3][2]) {
      S nd = czero<S>();
      T* const yl = at(y + 3 * int64_t(oz), node_bytes<T, kPipe>(no[i]));
      if constexpr (kPipe) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float* q = st + 3 * kRowWords + 64 + (i - 1) * kRowWords + 3 * lane + k;
          bv[i][k] = MODE != kApply ? q[0] : 0.0f;
          dv[i][k] = MODE == kSmooth ? q[2 * kRowWords] : 0.0f;
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const S right = r[k][0] + r[k][1];
        const S ax = (r[k][0] - r[k][1]) + shfl_at(right, ll);
        if (!(out_z && rown[i])) continue;
        const bool kk = ((kb[i] >> k) & 1u) != 0u;
        T out;
        if constexpr (MODE == kApply) {
          out = kk ? store_t(ax) : T(0);
          nd = nd + keep[i][k] * load_c<S>(out);
        } else if constexpr (MODE == kResidual) {
          out = kk ? T(bv[i][k] - store_t(ax)) : T(0);
        } else {
          out = kk ? T(store_t(keep[i][k]) + omega * dv[i][k] * (bv[i][k] - store_t(ax))) : T(0);
          nd = nd + load_c<S>(bv[i][k]) * load_c<S>(out);
        }
        yl[k] = out;
      }
      if constexpr (MODE != kResidual) dsum = dsum + nd;
    };
    if constexpr (R == 2) {
      S r1[3][2];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int m = 0; m < 2; ++m) r1[k][m] = up[k][m].x + lo[k][m].y;
      finish(1, r1);
    }
    __syncthreads();
    if (w < W - 1) {
      S r2[3][2];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const S hi = buf[(w + 1) * 192 + (2 * k + m) * 32 + lane];
          if constexpr (R == 2)
            r2[k][m] = up[k][m].y + hi;
          else
            r2[k][m] = up[k][m] + hi;
        }
      finish(R, r2);
    }
    if constexpr (kRuns) {
      if ((s & 7) == 0) {
        druns = druns + df(dsum, 0.0f);
        dsum = 0.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int m = 0; m < 4; ++m) Fc[k][m] = Fn[k][m];
#pragma unroll
    for (int i = 1; i <= R; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) keep[i][k] = knext[i][k];
  }
  if constexpr (MODE != kResidual) {
    double share;
    if constexpr (kRuns)
      share = df_to_double(druns + df(dsum, 0.0f));
    else
      share = double(store_t(dsum));
    if (dot.part != nullptr)
      grid_sum(share, dot,
               int((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x),
               int(gridDim.x * gridDim.y));
  }
}

// ------------------------------------------------------------------ schedules
constexpr int kSplitMaxRows = 5;  // element rows a CTA: 43 KB of shared memory
namespace {

// The FP64 operator with a warp per element row and component.  On a small grid the
// marching kernel's time is its chain: a warp instruction on FP64 takes 64 cycles of its
// scheduler whatever waits, a step has 150 of them, and a 24x8x8 grid has 66 rows of
// lanes for 608 schedulers.  The transforms of the three displacement components do not
// meet except in the modal stresses, so here three warps take one component each and
// exchange their modes in shared memory: 66 instructions a step and warp.  24x8x8 and
// 48x8x8: 14.5 -> 10.3 us, bound now by the six warps of a CTA on one SM's FP64 units.
// A row takes 198 instructions instead of 150, so the marching kernel keeps the grids
// that fill the SMs: its best tile takes 26.7 us against 28.8 on 60x20x20, 43.1 against
// 45.2 on 60x36x28, 110.7 against 137 on 96x48x48.
template <int MODE>
__global__ void __launch_bounds__(96 * kSplitMaxRows, 1)
    k_fine_split(GridDev g, ModalT<double> mc, int KZ, int nss, const double* ef,
                 const uint8_t* __restrict__ kn, const double* x, const double* b,
                 const double* invdiag, double omega, double* y, SumOut dot, int guard) {
  let_next_start();
  constexpr int kOwn = 31;
  extern __shared__ __align__(16) unsigned char march_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, w = wid / 3, k = wid - 3 * w;
  const int W = blockDim.x / 96, rows = W - 1;
  double* const xs = reinterpret_cast<double*>(march_smem);  // [2][W][3][2][32]
  double* const us = xs + 2 * W * 192 + w * (21 * 32) + lane;  // [3][7][32] of this row
  const int q = blockIdx.x * kOwn - 1 + lane;
  const int ss = q > 0 ? q / g.nnx : 0, ex = q - ss * g.nnx;
  const bool own_x = lane >= 1 && ss < nss;
  const int rl = lane < 31 ? lane + 1 : lane, ll = lane > 0 ? lane - 1 : lane;
  const int ey = ss * rows - 1 + w;  // element row ey, node rows ey and ey + 1
  const bool vx = ex >= 0 && ss < nss;
  const int plane = g.nnx * g.nny, eplane = g.nx * g.ny;
  const int no[2] = {g.nnx * ey + ex, g.nnx * (ey + 1) + ex};
  const bool rv[2] = {vx && ey >= 0 && ey < g.nny, vx && ey + 1 < g.nny};
  const bool own = own_x && w < W - 1 && ey + 1 < g.nny;
  const bool ev = vx && ex < g.nx && ey >= 0 && ey < g.ny;
  const int eo = ey * g.nx + ex, z0 = blockIdx.y * KZ;
  const bool far = lane == 31 && ex + 1 < g.nnx;  // its right neighbour has no lane
  wait_for_previous();

  auto load_layer = [&](int c, double (&r)[2], double (&e)[2]) {
    const bool vc = c >= 0 && c < g.nnz;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const bool ok = vc && rv[i];
      const double* xn = x + 3 * (plane * c + no[i]) + k;
      r[i] = ok ? xn[0] : 0.0;
      e[i] = ok && far ? xn[3] : 0.0;
    }
  };
  auto load_f = [&](int c) { return c >= 0 && c < g.nz && ev ? ef[eplane * c + eo] : 0.0; };
  auto face = [&](const double (&r)[2], const double (&e)[2], double (&F)[4]) {
    double nb[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      nb[i] = shfl_at(r[i], rl);
      nb[i] = lane == 31 ? e[i] : nb[i];
    }
    face_modes<double, double>(r, nb, F);
  };
  auto load_kb = [&](int s) -> unsigned {
    const int ez = z0 - 1 + s;
    return kn == nullptr ? 7u : (s >= 1 && ez < g.nnz && own ? unsigned(kn[plane * ez + no[1]]) : 0u);
  };

  const int s0 = z0 == 0 ? 1 : 0;
  double raw[2], rext[2], Fc[4], pend[4] = {0.0, 0.0, 0.0, 0.0};
  load_layer(z0 - 1 + s0, raw, rext);
  face(raw, rext, Fc);
  double keep = raw[1];
  load_layer(z0 + s0, raw, rext);
  double fn = load_f(z0 - 1 + s0);
  unsigned kbn = load_kb(s0);
  double dsum = 0.0;
#pragma unroll 1
  for (int s = s0; s <= KZ; ++s) {
    const int ez = z0 - 1 + s;
    if (ez > g.nnz - 1) break;  // uniform: the last chunk ends with the grid
    const bool out = s >= 1 && own;
    const unsigned kb = kbn;
    if (s < KZ) kbn = load_kb(s + 1);
    const int at1 = 3 * (plane * ez + no[1]) + k;
    const double bv = MODE != kApply && out ? b[at1] : 0.0;
    const double dv = MODE == kSmooth && out ? invdiag[at1] : 0.0;
    const double f = fn;
    double Fn[4];
    face(raw, rext, Fn);
    const double knext = raw[1];
    if (s < KZ) {
      load_layer(ez + 2, raw, rext);
      fn = load_f(ez + 1);
    }
    double u[8];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (m > 0) u[m] = Fn[m] + Fc[m];
      u[m | 4] = Fn[m] - Fc[m];
    }
#pragma unroll
    for (int m = 1; m < 8; ++m) us[(k * 7 + m - 1) * 32] = u[m];
    asm volatile("bar.sync %0, 96;" ::"r"(1 + w) : "memory");
    // modal_stress (tg_march.h) for component K alone: its axis' mode A, the others' B
    // and C.
    auto stress = [&](auto kc) {
      constexpr int K = decltype(kc)::value, KB = (K + 1) % 3, KC = (K + 2) % 3;
      constexpr int A = 1 << K, B = 1 << KB, C = 1 << KC;
      auto o = [&](int comp, int m) { return comp == K ? u[m] : us[(comp * 7 + m - 1) * 32]; };
      const double m0 = mc.M0 * f, m02 = mc.M02 * f, l0 = mc.L0 * f, l1 = mc.L1 * f,
                   m1 = mc.M1 * f, lm2 = mc.LM2 * f;
      const double tr = l0 * ((o(0, 1) + o(1, 2)) + o(2, 4));
      const double sh = m1 * ((o(2, 3) + o(1, 5)) + o(0, 6));
      const double tb = l1 * (u[A | B] + o(KC, B | C)), tc = l1 * (u[A | C] + o(KB, B | C));
      const double ub = m0 * (u[B] + o(KB, A)), uc = m0 * (u[C] + o(KC, A));
      u[A] = mad(m02, u[A], tr);
      u[B] = ub;
      u[C] = uc;
      u[A | B] = mad(m0, u[A | B], tb);
      u[A | C] = mad(m0, u[A | C], tc);
      u[B | C] = mad(m1, u[B | C], sh);
      u[7] = lm2 * u[7];
    };
    if (k == 0)
      stress(std::integral_constant<int, 0>{});
    else if (k == 1)
      stress(std::integral_constant<int, 1>{});
    else
      stress(std::integral_constant<int, 2>{});
    if (guard) {
#pragma unroll
      for (int m = 1; m < 8; ++m) u[m] = f != 0.0 ? u[m] : 0.0;
    }
    // Back in z and y, as in the marching kernel.
    double P[4];
    P[0] = pend[0] - u[4];
    pend[0] = u[4];
#pragma unroll
    for (int m = 1; m < 4; ++m) {
      P[m] = pend[m] + (u[m] - u[m | 4]);
      pend[m] = u[m] + u[m | 4];
    }
    double* const buf = xs + (s & 1) * (W * 192);
    buf[w * 192 + (2 * k) * 32 + lane] = P[0] - P[2];
    buf[w * 192 + (2 * k + 1) * 32 + lane] = P[1] - P[3];
    const double up0 = P[0] + P[2], up1 = P[1] + P[3];
    __syncthreads();  // the rows' exchange, and every row's modes are read
    if (w < W - 1) {
      const double r0 = up0 + buf[(w + 1) * 192 + (2 * k) * 32 + lane];
      const double r1 = up1 + buf[(w + 1) * 192 + (2 * k + 1) * 32 + lane];
      const double ax = (r0 - r1) + shfl_at(r0 + r1, ll);
      if (out) {
        const bool kk = ((kb >> k) & 1u) != 0u;
        double v;
        if constexpr (MODE == kApply) {
          v = kk ? ax : 0.0;
          dsum += keep * v;
        } else if constexpr (MODE == kResidual) {
          v = kk ? bv - ax : 0.0;
        } else {
          v = kk ? keep + omega * dv * (bv - ax) : 0.0;
          dsum += bv * v;
        }
        y[at1] = v;
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) Fc[m] = Fn[m];
    keep = knext;
  }
  if constexpr (MODE != kResidual) {
    if (dot.part != nullptr)
      grid_sum(dsum, dot, int(blockIdx.y * gridDim.x + blockIdx.x), int(gridDim.x * gridDim.y));
  }
}

}  // namespace

namespace {

struct MarchTile {
  int W, kz;  // warps per CTA, node layers per CTA
};

// SM cycles of one warp step (a layer of R element rows): kBusy while the SM's
// pipes are full, kChain for a warp that has them to itself, kStart to launch a
// CTA and load its first layers.  FP64: a warp instruction takes 64 cycles on its
// scheduler whatever its active lanes, 19 when four schedulers share the SM's
// units (measured), and a step has about 150.
template <class V>
struct StepCost;
template <>
struct StepCost<float2> {
  static constexpr double kBusy = 150.0, kChain = 900.0, kStart = 3000.0;
};
template <>
struct StepCost<float> {
  static constexpr double kBusy = 110.0, kChain = 800.0, kStart = 3000.0;
};
template <>
struct StepCost<double> {
  static constexpr double kBusy = 2900.0, kChain = 9600.0, kStart = 4000.0;
};
template <>
struct StepCost<df> {
  static constexpr double kBusy = 650.0, kChain = 6000.0, kStart = 4000.0;
};
constexpr int kSms = 152;

// Whether a periodic row of nx columns uses more of a warp's lanes in one sequence
// of nx + 2 columns (30 of 32 lanes own one) than in groups of nx lanes.
bool periodic_flat(int nx) {
  return nx > 32 || 30 * nx > (nx + 2) * nx * (32 / nx);
}

template <class V>
dim3 march_grid(int nnx, int nny, int nnz, int nsys, bool per, const MarchTile& t) {
  constexpr int R = RowsOf<V>::R;
  const int rows = t.W * R - 1, nss = (nny + rows - 1) / rows;
  int64_t gx;
  if (!per) {
    const int own = std::is_same<V, double>::value ? 31 : 30;
    gx = (int64_t(nnx) * nss + own - 1) / own;
  } else if (periodic_flat(nnx)) {
    gx = (int64_t(nnx + 2) * nss + 29) / 30;
  } else {
    gx = (nss + 32 / nnx - 1) / (32 / nnx);
  }
  return dim3(unsigned(gx), unsigned((nnz + t.kz - 1) / t.kz), unsigned(nsys));
}

// The tile with the least modelled time.  CTAs spread over the SMs and follow
// one another as they end, so the fullest SM runs ceil(CTAs / SMs) of them, as
// many together as its registers hold; a CTA's march takes kz + 1 steps.  Small
// grids get short marches over many SMs, large ones long marches with little
// halo and no nearly empty last round.
template <class V>
double march_cost(const MarchTile& t, const dim3& d) {
  using C = StepCost<V>;
  const int64_t ctas = int64_t(d.x) * d.y * d.z;
  const double res = std::max(1, RowsOf<V>::kMaxWarps / t.W);
  const double per_sm = double((ctas + kSms - 1) / kSms), rounds = std::ceil(per_sm / res);
  return std::max(per_sm * t.W * (t.kz + 1) * C::kBusy, rounds * (t.kz + 1) * C::kChain) +
         rounds * C::kStart;
}

template <class V>
MarchTile march_tile(int nnx, int nny, int nnz, int nsys, bool per) {
  MarchTile best{4, 8};
  double best_cost = 1e300;
  for (int W : {2, 3, 4, 5, 6, 8, 10, 12}) {
    if (W > RowsOf<V>::kMaxWarps) break;
    for (int target : {1, 2, 3, 4, 6, 8, 11, 16, 22, 32, 43, 64}) {
      const int chunks = (nnz + target - 1) / target;
      const MarchTile t{W, (nnz + chunks - 1) / chunks};
      const double c = march_cost<V>(t, march_grid<V>(nnx, nny, nnz, nsys, per, t));
      if (c < best_cost) {
        best_cost = c;
        best = t;
      }
      if (target >= nnz) break;
    }
  }
  return best;
}

// The FP64 operator's kernel and tile on a grid: whichever the model puts first.  A row
// of the split kernel is 1.3 times the FP64 work of the marching kernel's, and about
// half its chain.
struct Fp64Plan {
  bool split;
  MarchTile t;
};
Fp64Plan fp64_plan(int nnx, int nny, int nnz) {
  constexpr double kBusy = 3800.0, kChain = 5200.0, kStart = 4000.0;
  Fp64Plan best{false, march_tile<double>(nnx, nny, nnz, 1, false)};
  double cost = march_cost<double>(best.t, march_grid<double>(nnx, nny, nnz, 1, false, best.t));
  for (int W = 2; W <= kSplitMaxRows; ++W)
    for (int target : {1, 2, 3, 4, 6, 8, 11, 16}) {
      const int chunks = (nnz + target - 1) / target;
      const MarchTile t{W, (nnz + chunks - 1) / chunks};
      const dim3 d = march_grid<double>(nnx, nny, nnz, 1, false, t);
      const double per_sm = double((int64_t(d.x) * d.y + kSms - 1) / kSms);
      const double rounds = std::ceil(per_sm / std::max(1, 7 / W));
      const double c = std::max(per_sm * W * (t.kz + 1) * kBusy, rounds * (t.kz + 1) * kChain) +
                       rounds * kStart;
      if (c < cost) {
        cost = c;
        best = Fp64Plan{true, t};
      }
      if (target >= nnz) break;
    }
  return best;
}

template <int MODE>
void launch_split(const GridDev& gd, const MarchTile& t, const ModalConsts& c, const double* ef,
                  const uint8_t* kn, const double* x, const double* b, const double* invdiag,
                  double omega, double* y, const SumOut& dot, cudaStream_t s) {
  const dim3 grid = march_grid<double>(gd.nnx, gd.nny, gd.nnz, 1, false, t);
  const int nss = (gd.nny + t.W - 2) / (t.W - 1);
  const size_t smem = size_t(t.W) * (2 * 192 + 21 * 32) * sizeof(double);
  k_fine_split<MODE><<<grid, 96 * t.W, smem, s>>>(gd, to_modal<double>(c), t.kz, nss, ef, kn, x, b,
                                                 invdiag, omega, y, dot, kn == nullptr ? 1 : 0);
  TG_LAUNCH_CHECK();
}

template <class V, class T, int MODE, bool PER>
void launch_march(const GridDev& gd, const MarchTile& t, int nsys, const ModalConsts& c,
                  const T* ef, const uint8_t* kn, const T* x, const T* b, const T* invdiag,
                  T omega, T* y, const SumOut& dot, const BatchDev& bd, cudaStream_t s) {
  using S = typename RowsOf<V>::S;
  const dim3 grid = march_grid<V>(gd.nnx, gd.nny, gd.nnz, nsys, PER, t);
  const int rows = t.W * RowsOf<V>::R - 1, nss = (gd.nny + rows - 1) / rows;
  const size_t smem = size_t(2) * t.W * 192 * sizeof(S) +
                      (RowsOf<V>::R == 2 ? size_t(t.W) * (kDepth + 1) * slot_words<MODE>() * 4 : 0);
  if constexpr (RowsOf<V>::R == 2) {
    // More than the default 48 KB.
    allow_shared<k_fine_march<V, T, MODE, PER>>(
        RowsOf<V>::kMaxWarps * (2 * 192 + (kDepth + 1) * slot_words<MODE>()) * 4);
  }
  // Only the public apply takes values at nodes of absent elements; within the
  // solver (a kept mask) they are zeros.
  const int guard = kn == nullptr ? 1 : 0;
  auto kernel = k_fine_march<V, T, MODE, PER>;
  if constexpr (sizeof(T) == 4)
    launch_behind(kernel, grid, 32 * t.W, smem, s, gd, to_modal<S>(c), t.kz, nss, ef, kn, x, b,
                  invdiag, omega, y, dot, guard, bd);
  else  // the SMs' FP64 units (or double-float arithmetic) bound it: see tg_launch.h
    kernel<<<grid, 32 * t.W, smem, s>>>(gd, to_modal<S>(c), t.kz, nss, ef, kn, x, b, invdiag,
                                        omega, y, dot, guard, bd);
  TG_LAUNCH_CHECK();
}

template <class V, class T>
void launch_march_mode(int mode, const Grid& g, const MarchTile& t, const ModalConsts& c,
                       const T* ef, const uint8_t* kn, const T* x, const T* b, const T* invdiag,
                       T omega, T* y, const SumOut& dot, cudaStream_t s) {
  const GridDev gd{g.nx, g.ny, g.nz, g.nnx, g.nny, g.nnz};
  if (mode == kApply)
    launch_march<V, T, kApply, false>(gd, t, 1, c, ef, kn, x, b, invdiag, omega, y, dot,
                                      BatchDev{}, s);
  else if (mode == kResidual)
    launch_march<V, T, kResidual, false>(gd, t, 1, c, ef, kn, x, b, invdiag, omega, y, SumOut{},
                                         BatchDev{}, s);
  else
    launch_march<V, T, kSmooth, false>(gd, t, 1, c, ef, kn, x, b, invdiag, omega, y, dot,
                                       BatchDev{}, s);
}

// Warps per CTA of the FP32 tile shapes (two packed element rows per thread).
constexpr int kShapeWarps[] = {2, 3, 4, 5, 6, 8, 10, 12};
constexpr int kNumShapes = 8;
constexpr int kTunedMinKz = 8;  // shortest z-chunk of a stored or forced FP32 schedule

int blocks_of(const dim3& d) { return int(d.x * d.y); }
}  // namespace

int fine_op_blocks(const Grid& g, bool fp64) {
  if (fp64)
    return blocks_of(march_grid<double>(g.nnx, g.nny, g.nnz, 1, false,
                                        fp64_plan(g.nnx, g.nny, g.nnz).t));
  int n = std::max(blocks_of(march_grid<float2>(g.nnx, g.nny, g.nnz, 1, false,
                                                march_tile<float2>(g.nnx, g.nny, g.nnz, 1, false))),
                   blocks_of(march_grid<float>(g.nnx, g.nny, g.nnz, 1, false,
                                               march_tile<float>(g.nnx, g.nny, g.nnz, 1, false))));
  for (int W : kShapeWarps)
    n = std::max(n, blocks_of(march_grid<float2>(g.nnx, g.nny, g.nnz, 1, false,
                                                 MarchTile{W, kTunedMinKz})));
  return n;
}

FineSchedule default_fine_schedule(const Grid& g) {
  const MarchTile t = march_tile<float2>(g.nnx, g.nny, g.nnz, 1, false);
  FineSchedule s;
  s.kind = FineSchedule::kColumn;
  s.shape = int(std::find(kShapeWarps, kShapeWarps + kNumShapes, t.W) - kShapeWarps);
  s.kz = t.kz;
  return s;
}

int fine_schedule_shapes() { return kNumShapes; }

// The schedules worth measuring on g: of every tile shape with z-chunks of about 8 to
// 64 node layers, the sixteen that the cost model puts first (its error against
// measured times is a few percent; the sixteenth is beyond that).
std::vector<FineSchedule> fine_schedule_candidates(const Grid& g) {
  std::vector<std::pair<double, FineSchedule>> all;
  for (int sh = 0; sh < kNumShapes; ++sh) {
    int last = 0;
    for (int target : {64, 43, 33, 26, 22, 16, 13, 11, 8}) {
      const int chunks = std::max(1, (g.nnz + target - 1) / target);
      const MarchTile t{kShapeWarps[sh], std::max(kTunedMinKz, (g.nnz + chunks - 1) / chunks)};
      if (t.kz == last) continue;
      last = t.kz;
      FineSchedule s;
      s.shape = sh;
      s.kz = t.kz;
      all.emplace_back(march_cost<float2>(t, march_grid<float2>(g.nnx, g.nny, g.nnz, 1, false, t)),
                       s);
    }
  }
  std::stable_sort(all.begin(), all.end(),
                   [](const auto& a, const auto& b) { return a.first < b.first; });
  std::vector<FineSchedule> out;
  for (size_t i = 0; i < all.size() && i < 16; ++i) out.push_back(all[i].second);
  return out;
}

bool fine_schedule_valid(const FineSchedule& s) {
  if (s.kind == FineSchedule::kPencil) return true;
  return s.kind == FineSchedule::kColumn && s.shape >= 0 && s.shape < kNumShapes &&
         s.kz >= kTunedMinKz && s.kz <= 4096;
}

template <class T>
void launch_fine_op(int mode, const Grid& g, const ModalConsts& c, const T* ef, const uint8_t* kn,
                    const T* x, const T* b, const T* invdiag, T omega, T* y, const SumOut& dot,
                    cudaStream_t s) {
  if constexpr (std::is_same<T, float>::value) {
    launch_fine_op_sched(fine_schedule_for(g, mode), mode, g, c, ef, kn, x, b, invdiag, omega, y,
                         dot, s);
  } else {
    const Fp64Plan p = fp64_plan(g.nnx, g.nny, g.nnz);
    const GridDev gd{g.nx, g.ny, g.nz, g.nnx, g.nny, g.nnz};
    if (!p.split)
      launch_march_mode<double, double>(mode, g, p.t, c, ef, kn, x, b, invdiag, omega, y, dot, s);
    else if (mode == kApply)
      launch_split<kApply>(gd, p.t, c, ef, kn, x, b, invdiag, omega, y, dot, s);
    else if (mode == kResidual)
      launch_split<kResidual>(gd, p.t, c, ef, kn, x, b, invdiag, omega, y, SumOut{}, s);
    else
      launch_split<kSmooth>(gd, p.t, c, ef, kn, x, b, invdiag, omega, y, dot, s);
  }
}

// The FP32 operator under an explicit schedule (the autotuner times candidates
// through this without touching the process-wide table).
void launch_fine_op_sched(const FineSchedule& fs, int mode, const Grid& g, const ModalConsts& c,
                          const float* ef, const uint8_t* kn, const float* x, const float* b,
                          const float* invdiag, float omega, float* y, const SumOut& dot,
                          cudaStream_t s) {
  if (fs.kind == FineSchedule::kColumn)
    launch_march_mode<float2, float>(mode, g, MarchTile{kShapeWarps[fs.shape], fs.kz}, c, ef, kn,
                                     x, b, invdiag, omega, y, dot, s);
  else
    launch_march_mode<float, float>(mode, g, march_tile<float>(g.nnx, g.nny, g.nnz, 1, false), c,
                                    ef, kn, x, b, invdiag, omega, y, dot, s);
}

// The FP64 residual y = b - A x evaluated in double-float arithmetic (tg_df.h):
// FP64 inputs and output, about 48 significant bits inside, on the FP32 pipe.
void launch_fine_residual_df(const Grid& g, const ModalConsts& c, const double* ef,
                             const uint8_t* kn, const double* x, const double* b, double* y,
                             cudaStream_t s) {
  const GridDev gd{g.nx, g.ny, g.nz, g.nnx, g.nny, g.nnz};
  launch_march<df, double, kResidual, false>(gd, march_tile<df>(g.nnx, g.nny, g.nnz, 1, false), 1,
                                             c, ef, kn, x, b, nullptr, 0.0, y, SumOut{}, BatchDev{},
                                             s);
}

template void launch_fine_op<double>(int, const Grid&, const ModalConsts&, const double*,
                                     const uint8_t*, const double*, const double*,
                                     const double*, double, double*, const SumOut&, cudaStream_t);
template void launch_fine_op<float>(int, const Grid&, const ModalConsts&, const float*,
                                    const uint8_t*, const float*, const float*, const float*,
                                    float, float*, const SumOut&, cudaStream_t);

// Periodic batched apply: nsys systems on the nx*ny*nz torus; system bi uses
// x/b/y at bi*ndof and the factors and kept bits of cell bi / nrhs.  dot_part
// (kApply) receives one partial of x.y per CTA, the CTAs of a system
// contiguous: periodic_op_blocks<T>() per system.
namespace {
// One tile per cell size, whatever the batch, so that a system's partial sums
// and with them its iterates do not depend on who else runs: the tile of four
// cells' worth of strains, between a single cell's and a full GPU's.
constexpr int kTileSystems = 24;
template <class V>
MarchTile periodic_tile(int nx, int ny, int nz) {
  return march_tile<V>(nx, ny, nz, kTileSystems, true);
}
// f of a value of the type that the cell's rows are carried in: FP32 rows in pairs,
// whose offsets within a layer are 32 bits, unless the layer is too large for that (one
// of more than 357,913,941 nodes, a cell of a single one).
template <class T, class F>
auto periodic_rows(int nx, int ny, F&& f) {
  if constexpr (std::is_same<T, float>::value) {
    if (narrow_layer(int64_t(nx) * ny)) return f(float2{});
  }
  return f(T{});
}
}  // namespace
template <class T>
int periodic_op_blocks(int nx, int ny, int nz) {
  return periodic_rows<T>(nx, ny, [&](auto v) {
    using V = decltype(v);
    return blocks_of(march_grid<V>(nx, ny, nz, 1, true, periodic_tile<V>(nx, ny, nz)));
  });
}
template int periodic_op_blocks<double>(int, int, int);
template int periodic_op_blocks<float>(int, int, int);

template <class T>
void launch_periodic_op(int mode, int nx, int ny, int nz, const ModalConsts& c, const T* ef,
                        const uint8_t* kn, const T* x, const T* b, T* y, double* dot_part,
                        int nsys, int nrhs, const int* run, cudaStream_t s) {
  const GridDev gd{nx, ny, nz, nx, ny, nz};
  const int64_t nv = int64_t(nx) * ny * nz;
  const BatchDev bd{nrhs, 3 * nv, nv, run, periodic_flat(nx) ? 1 : 0};
  periodic_rows<T>(nx, ny, [&](auto v) {
    using V = decltype(v);
    const MarchTile t = periodic_tile<V>(nx, ny, nz);
    if (mode == kApply)
      launch_march<V, T, kApply, true>(gd, t, nsys, c, ef, kn, x, b, nullptr, T(0), y,
                                       SumOut{dot_part}, bd, s);
    else
      launch_march<V, T, kResidual, true>(gd, t, nsys, c, ef, kn, x, b, nullptr, T(0), y,
                                          SumOut{}, bd, s);
  });
}
template void launch_periodic_op<double>(int, int, int, int, const ModalConsts&, const double*,
                                         const uint8_t*, const double*, const double*, double*,
                                         double*, int, int, const int*, cudaStream_t);
template void launch_periodic_op<float>(int, int, int, int, const ModalConsts&, const float*,
                                        const uint8_t*, const float*, const float*, float*,
                                        double*, int, int, const int*, cudaStream_t);

// diag(A) at every DOF = kdiag * (sum of the adjacent element factors), summed
// in a fixed element order; invdiag = 1/diag on kept DOFs, 0 elsewhere
// (matfree.cpp:757-833 accumulates factor_e * Ke(r,r)).
__global__ void k_fine_invdiag(GridDev g, double kdiag, const double* __restrict__ ef,
                               const uint8_t* __restrict__ kept, double* __restrict__ invdiag) {
  const int64_t n = int64_t(g.nnx) * g.nny * g.nnz;
  for (int64_t node = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; node < n;
       node += int64_t(gridDim.x) * blockDim.x) {
    const int a = int(node % g.nnx);
    const int bb = int((node / g.nnx) % g.nny);
    const int c = int(node / (int64_t(g.nnx) * g.nny));
    double s = 0.0;
    for (int dz = -1; dz <= 0; ++dz)
      for (int dy = -1; dy <= 0; ++dy)
        for (int dx = -1; dx <= 0; ++dx) {
          const int i = a + dx, j = bb + dy, k = c + dz;
          if (i < 0 || i >= g.nx || j < 0 || j >= g.ny || k < 0 || k >= g.nz) continue;
          s += ef[(int64_t(k) * g.ny + j) * g.nx + i];
        }
    const double dg = kdiag * s;
    for (int comp = 0; comp < 3; ++comp) {
      const int64_t d = 3 * node + comp;
      invdiag[d] = (kept[d] && dg > 0.0) ? 1.0 / dg : 0.0;
    }
  }
}

void launch_fine_invdiag(const Grid& g, double kdiag, const double* ef, const uint8_t* kept,
                         double* invdiag, cudaStream_t s) {
  const GridDev gd{g.nx, g.ny, g.nz, g.nnx, g.nny, g.nnz};
  const int64_t blocks = std::min<int64_t>((g.nnodes + 255) / 256, 152 * 16);
  k_fine_invdiag<<<int(blocks), 256, 0, s>>>(gd, kdiag, ef, kept, invdiag);
  TG_LAUNCH_CHECK();
}

}  // namespace tg
