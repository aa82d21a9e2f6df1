// tg_launch.h -- kernels launched behind the previous one of their stream.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <type_traits>

#include "tg_internal.h"

namespace tg {

// A multigrid iteration is a chain of some thirty dependent kernels of a few
// microseconds, and between two of them the chip drains, the launch of the next one
// is set up and its CTAs start.  A kernel launched by launch_behind may have its CTAs
// resident while the previous kernel of the stream still runs (programmatic dependent
// launch; the edge is kept when a stream is captured).  Every thread of such a kernel
// that touches memory first calls wait_for_previous(), which returns once the previous
// kernel has ended and its writes are visible; that kernel had itself waited for the
// one before it.  Before the wait a kernel may only read what no kernel still in
// flight can write: a hierarchy's matrices and masks, whose build the host has waited
// for.  Pointers to anything else are not __restrict__: that would let the compiler
// read through them before the wait.  let_next_start() lets the next kernel's CTAs in once all CTAs of this one
// have come that far.  A loop body of 30 empty kernels takes 1.05 to 1.25 us a kernel
// plainly launched, 0.9 to 1.1 this way.
__device__ __forceinline__ void let_next_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void behind_previous() {
  let_next_start();
  wait_for_previous();
}

template <class... P, class... A>
void launch_behind(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                   A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);  // checked by TG_LAUNCH_CHECK
}

// The same for a kernel on T that may be bound by the SMs' FP64 units: only while it
// and its like fit a CTA per SM side by side.  CTAs that come early go where the
// previous kernel left room, two on one SM and none on another, and FP64 work takes as
// long as the fullest SM's (the FP64 fine operator on 60x20x20, 106 CTAs: 26.7 us
// plainly, 41.9 this way; a 24x8x8 solve 10.5 ms with the fine operator plainly
// launched, 12.7 without).
constexpr unsigned kSpreadCtas = 152 / 2;
template <class T, class... P, class... A>
void launch_behind_if_spread(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t s, A&&... args) {
  if (sizeof(T) == 4 || grid.x * grid.y * grid.z <= kSpreadCtas)
    launch_behind(kernel, grid, block, smem, s, args...);
  else
    kernel<<<grid, block, smem, s>>>(static_cast<P>(args)...);
}

// Raises a kernel's dynamic shared-memory limit.  The limit belongs to the kernel on one
// device, so each device's first call sets it (any thread may be first: the value is the
// kernel's).  Set at every launch instead, eight designs in the serving loop, whose threads
// launch together, took 1.01 and 1.03 times as long; this way 0.99 to 1.00.
template <auto kKernel>
void allow_shared(int bytes) {
  static std::atomic<uint64_t> done[2]{};  // a bit per device
  int dev = 0;
  TG_CUDA(cudaGetDevice(&dev));
  const uint64_t bit = uint64_t(1) << (dev & 63);
  std::atomic<uint64_t>* const word = dev < 128 ? done + (dev >> 6) : nullptr;
  if (word != nullptr && (word->load(std::memory_order_acquire) & bit) != 0) return;
  TG_CUDA(cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  if (word != nullptr) word->fetch_or(bit, std::memory_order_release);
}

}  // namespace tg
