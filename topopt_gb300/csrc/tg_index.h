// tg_index.h -- addresses within a node layer.  Plain C++, so that the arithmetic can
// be checked on the host at sizes no test would allocate.
#pragma once
#include <cstdint>
#include <type_traits>

#ifndef TG_HD
#ifdef __CUDACC__
#define TG_HD __host__ __device__ __forceinline__
#else
#define TG_HD inline
#endif
#endif

namespace tg {

// base (the same for every lane) + a byte offset: one address operand where the
// offset is 32 bits.
template <class P, class O>
TG_HD P* at(P* base, O bytes) {
  using B = typename std::conditional<std::is_const<P>::value, const char, char>::type;
  return reinterpret_cast<P*>(reinterpret_cast<B*>(base) + bytes);
}

// Whether FP32 may address the nodes of a layer, 12 bytes each, by 32-bit byte offsets.
// Every layer of a bounded grid: DOF indices fit 32 bits, so one (of at least two) has
// at most 357,913,941 nodes.  A periodic cell's single layer may have twice as many.
TG_HD bool narrow_layer(int64_t nodes) { return 12 * nodes <= int64_t(1) << 32; }

// Bytes from a layer's first node to node `no` of a vector of T, three components a
// node, in 32 bits with kNarrow.  FP64's 24 bytes pass 2^32 from the 178,956,971st node
// on.
template <class T, bool kNarrow>
TG_HD auto node_bytes(int no) {
  using B = typename std::conditional<kNarrow, unsigned, int64_t>::type;
  return B(3 * sizeof(T)) * B(no);
}

}  // namespace tg
