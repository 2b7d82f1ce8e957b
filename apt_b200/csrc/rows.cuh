// Feature rows as the sparse kernels see them: element conversion, loads and stores of a slice of
// a row, and the split of the lanes of a warp over the slices of a row.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace apt {

// ---- element <-> fp32 -----------------------------------------------------------
template <typename T> struct Elem;
template <> struct Elem<float> {
  static constexpr bool kIsBf16 = false;
  static __device__ __forceinline__ float to_f(float x) { return x; }
  static __device__ __forceinline__ float from_f(float x) { return x; }
};
template <> struct Elem<__nv_bfloat16> {
  static constexpr bool kIsBf16 = true;
  static __device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float x) { return __float2bfloat16_rn(x); }
};
template <> struct Elem<__half> {
  static constexpr bool kIsBf16 = false;
  static __device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half from_f(float x) { return __float2half_rn(x); }
};

// A slice of VE elements of a row, read and written with one access of 16, 8, 4 or 2 bytes.
template <typename T, int VE>
struct alignas(sizeof(T) * VE) Pack {
  T v[VE];
};

// The same slice as it came from memory, packed until its elements are used: a slice held as an array of
// 16-bit elements takes a register for each of them.
template <typename T, int VE>
struct Raw {
  static constexpr int B = sizeof(T) * VE;
  static_assert(B == 16 || B == 8 || B == 4 || B == 2, "slice of 16, 8, 4 or 2 bytes");
  unsigned int w[B < 4 ? 1 : B / 4];
  __device__ __forceinline__ float get(int t) const {
    if constexpr (sizeof(T) == 4) {
      return __uint_as_float(w[t]);
    } else {
      const unsigned int u = w[t >> 1];
      if constexpr (sizeof(T) == 2 && Elem<T>::kIsBf16) {
        return __uint_as_float((t & 1) ? u & 0xffff0000u : u << 16);   // bf16 is the upper half of an fp32
      } else {
        const __half2 h = *(const __half2*)&u;
        return (t & 1) ? __high2float(h) : __low2float(h);
      }
    }
  }
};

template <typename T, int VE>
__device__ __forceinline__ Raw<T, VE> load_raw(const T* p) {
  constexpr int B = sizeof(T) * VE;
  Raw<T, VE> r;
  if constexpr (B == 16) {
    const uint4 u = __ldg((const uint4*)p);
    r.w[0] = u.x, r.w[1] = u.y, r.w[2] = u.z, r.w[3] = u.w;
  }
  if constexpr (B == 8) {
    const uint2 u = __ldg((const uint2*)p);
    r.w[0] = u.x, r.w[1] = u.y;
  }
  if constexpr (B == 4) r.w[0] = __ldg((const unsigned int*)p);
  if constexpr (B == 2) r.w[0] = __ldg((const unsigned short*)p);
  return r;
}
template <typename T, int VE>
__device__ __forceinline__ Pack<T, VE> load_pack(const T* p) {
  constexpr int B = sizeof(T) * VE;
  Pack<T, VE> r;
  if constexpr (B == 16) *(uint4*)&r = __ldg((const uint4*)p);
  if constexpr (B == 8) *(uint2*)&r = __ldg((const uint2*)p);
  if constexpr (B == 4) *(unsigned int*)&r = __ldg((const unsigned int*)p);
  if constexpr (B == 2) *(unsigned short*)&r = __ldg((const unsigned short*)p);
  return r;
}
template <typename T, int VE>
__device__ __forceinline__ void store_pack(T* p, const Pack<T, VE>& r) {
  *(Pack<T, VE>*)p = r;
}

// ---- host side: widest access and lane split ---------------------------------------
// Elements of T in the widest access (at most 16 bytes) that `bits` (row size and base addresses,
// in bytes, or-ed together) is a multiple of.
inline int slice_elems(uint64_t bits, int esz) {
  int b = 16;
  while (b > esz && (bits & (uint64_t)(b - 1))) b >>= 1;
  return b / esz;
}
inline int pow2_ge(int64_t x, int cap = 32) {
  int g = 1;
  while (g < x && g < cap) g <<= 1;
  return g;
}
inline int pow2_le(int64_t x, int cap = 32) {
  int g = 1;
  while (2 * g <= x && 2 * g <= cap) g <<= 1;
  return g;
}

}  // namespace apt
