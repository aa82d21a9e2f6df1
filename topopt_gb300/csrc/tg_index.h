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

// Bytes from a layer's first node to node `no` of a vector of T, three components a
// node: 32 bits with kNarrow, which FP32 on a bounded grid may use -- DOF indices fit 32
// bits, so a layer (of at least two) has at most 357,913,941 nodes of 12 bytes.  FP64's
// 24 bytes pass 2^32 from the 178,956,971st node on.
template <class T, bool kNarrow>
TG_HD auto node_bytes(int no) {
  using B = typename std::conditional<kNarrow, unsigned, int64_t>::type;
  return B(3 * sizeof(T)) * B(no);
}

}  // namespace tg
