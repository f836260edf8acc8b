// lela_b200/csrc/elem_rep.cuh -- how Modular<T> stores a residue: Rep<T>::in
// reads a stored element as a residue 0 .. p - 1, Rep<T>::out stores one
// (see elem.cu); Packed is the narrowest type that holds T's residues in a
// shared-memory tile.
#pragma once
#include <cstdint>

namespace lela {

template <class T>
struct Rep;
template <>
struct Rep<uint32_t> {
  using Packed = uint32_t;
  static __device__ __forceinline__ uint32_t in(uint32_t x, uint32_t) { return x; }
  static __device__ __forceinline__ uint32_t out(uint32_t r, uint32_t) { return r; }
};
template <>
struct Rep<uint8_t> {
  using Packed = uint8_t;
  static __device__ __forceinline__ uint32_t in(uint8_t x, uint32_t) { return x; }
  static __device__ __forceinline__ uint8_t out(uint32_t r, uint32_t) { return (uint8_t)r; }
};
template <>
struct Rep<uint16_t> {
  using Packed = uint16_t;
  static __device__ __forceinline__ uint32_t in(uint16_t x, uint32_t) { return x; }
  static __device__ __forceinline__ uint16_t out(uint32_t r, uint32_t) { return (uint16_t)r; }
};
template <>
struct Rep<float> {
  using Packed = uint32_t;
  // x is an integer of magnitude below 2^24, so the conversions are exact
  static __device__ __forceinline__ uint32_t in(float x, uint32_t p) {
    const int v = (int)x;
    return v < 0 ? (uint32_t)(v + (int)p) : (uint32_t)v;
  }
  static __device__ __forceinline__ float out(uint32_t r, uint32_t p) {
    return 2ull * r > p ? (float)((int)r - (int)p) : (float)r;
  }
};
template <>
struct Rep<double> {
  using Packed = uint32_t;
  static __device__ __forceinline__ uint32_t in(double x, uint32_t p) {
    const long long v = (long long)x;
    return v < 0 ? (uint32_t)(v + (long long)p) : (uint32_t)v;
  }
  static __device__ __forceinline__ double out(uint32_t r, uint32_t p) {
    return 2ull * r > p ? (double)((long long)r - (long long)p) : (double)r;
  }
};

}  // namespace lela
