// tg_reduce.h -- device end of a sum over a grid of CTAs (SumOut, tg_internal.h).
#pragma once
#include <cuda_runtime.h>

#include "tg_internal.h"

namespace tg {

// Sum over the block, a fixed tree; valid in thread 0.
__device__ __forceinline__ double block_total(double v) {
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double s = 0.0;
  if (wid == 0) {
    const int nw = int(blockDim.x + 31) >> 5;
    s = lane < nw ? red[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  }
  return s;
}

// The loop decision of a graph-resident PCG, exactly the host loops': rr is the
// new r.r.  st[0] = iterations done, st[1] = budget, st[2] = breakdown.
__device__ __forceinline__ void loop_decision(const LoopCond& c, double rr) {
  if (c.pap != nullptr) {
    // MG-PCG: breakdown (p.Ap <= 0 or not finite) stops without counting the
    // iteration; else it counts, and the loop runs on while ||r|| > thr.
    const double pap = *c.pap;
    if (!(pap > 0.0) || !isfinite(pap)) {
      c.st[2] = 1;
      cudaGraphSetConditional(c.h, 0u);
      return;
    }
    const int k = c.st[0] + 1;
    c.st[0] = k;
    cudaGraphSetConditional(c.h, (!(sqrt(rr) <= *c.thr) && k < c.st[1]) ? 1u : 0u);
  } else {
    // Jacobi-PCG: thr is squared, and the converging iteration is not counted.
    const bool done = rr < *c.thr;
    const int k = c.st[0] + (done ? 0 : 1);
    c.st[0] = k;
    cudaGraphSetConditional(c.h, (!done && k < c.st[1]) ? 1u : 0u);
  }
}

// One CTA's share v of a sum: into o.part[bid], and the CTA that ends last adds all
// n shares up in a fixed order (so which one it is does not matter), instead of a
// launch of its own that only does that (about 2 us of a PCG iteration's launches,
// three times).  Called by every thread of the CTA.
__device__ __forceinline__ void grid_sum(double v, const SumOut& o, int bid, int n) {
  __shared__ bool last;
  const double s = block_total(v);
  if (o.count == nullptr) {
    if (threadIdx.x == 0) o.part[bid] = s;
    return;
  }
  if (threadIdx.x == 0) {
    o.part[bid] = s;
    __threadfence();
    last = atomicAdd(o.count, 1u) == unsigned(n - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) t += __ldcg(o.part + i);
  t = block_total(t);
  if (threadIdx.x == 0) {
    *o.count = 0u;
    *o.out = t;
    if (o.copy_to != nullptr) *o.copy_to = *o.copy_from;
    if (o.cond.st != nullptr) loop_decision(o.cond, t);
  }
}

}  // namespace tg
