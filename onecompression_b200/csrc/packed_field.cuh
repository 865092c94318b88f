// The packed AutoGPTQ words of one row, eight columns at a time (packed_linear.cu, pack.cu).
#pragma once
#include "common.cuh"

namespace {

__device__ __forceinline__ __half2 as_half2(unsigned v) { return *reinterpret_cast<__half2*>(&v); }

// The packed words that hold columns 8 * unit .. 8 * unit + 7 of one row, as one field of 8 * BITS bits
// (in two registers for 8 bits).  WORDS word rows are read, starting with word row first(unit).
template <int BITS> struct Field;
template <> struct Field<4> {
  static constexpr int WORDS = 1;
  static __device__ __forceinline__ int first(int unit) { return unit; }
  static __device__ __forceinline__ unsigned pair(const unsigned (&w)[2], int, int k) {   // columns k, k + 4
    return (w[0] >> (4 * k)) & 0x000f000fu;
  }
};
template <> struct Field<8> {
  static constexpr int WORDS = 2;
  static __device__ __forceinline__ int first(int unit) { return 2 * unit; }
  static __device__ __forceinline__ unsigned pair(const unsigned (&w)[2], int, int k) {
    return ((w[0] >> (8 * k)) & 0xffu) | (((w[1] >> (8 * k)) & 0xffu) << 16);
  }
};
template <> struct Field<2> {
  static constexpr int WORDS = 1;
  static __device__ __forceinline__ int first(int unit) { return unit >> 1; }
  static __device__ __forceinline__ unsigned pair(const unsigned (&w)[2], int unit, int k) {
    const unsigned v = w[0] >> (16 * (unit & 1));
    return ((v >> (2 * k)) & 3u) | (((v >> (2 * k + 8)) & 3u) << 16);
  }
};
template <> struct Field<3> {   // 32 columns in three words; unit u of them holds bits 24u .. 24u + 23
  static constexpr int WORDS = 2;
  static __device__ __forceinline__ int first(int unit) {
    const int u = unit & 3;
    return (unit >> 2) * 3 + (u == 0 ? 0 : u - 1);          // 0, 0, 1, 2
  }
  static __device__ __forceinline__ unsigned pair(const unsigned (&w)[2], int unit, int k) {
    const int u = unit & 3;
    // bits 24u .. counted from the first word read: 0, 24, 16, 8
    const unsigned v = __funnelshift_r(w[0], w[1], u == 0 ? 0 : 32 - 8 * u);
    return ((v >> (3 * k)) & 7u) | (((v >> (3 * k + 12)) & 7u) << 16);
  }
};

}  // namespace
