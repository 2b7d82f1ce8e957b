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

// Two fp32 values in one 64-bit register pair, as the packed fp32 instructions of sm_100 take them (each half rounds
// like the scalar instruction). They halve the adds of a gather that is bound by its instruction count.
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2_pack(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void f2_unpack(F2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
template <typename T, int VE>
__device__ __forceinline__ F2 pair_of(const Raw<T, VE>& v, int q) { return f2_pack(v.get(2 * q), v.get(2 * q + 1)); }

// fp32 sums of a slice.
template <int VE>
struct Acc {
  static constexpr int P = VE > 1 ? VE / 2 : 1;
  F2 p[P];      // VE 1: the sum is the first half
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int q = 0; q < P; ++q) p[q] = 0ull;
  }
  __device__ __forceinline__ float get(int t) const {
    float x, y;
    f2_unpack(p[t >> 1], x, y);
    return (t & 1) ? y : x;
  }
  template <typename T>
  __device__ __forceinline__ void add(const Raw<T, VE>& v) {
    if constexpr (VE == 1) {
      p[0] = f2_pack(get(0) + v.get(0), 0.f);
    } else {
#pragma unroll
      for (int q = 0; q < P; ++q) p[q] = f2_add(p[q], pair_of(v, q));
    }
  }
  __device__ __forceinline__ void add(const Acc& o) {
#pragma unroll
    for (int q = 0; q < P; ++q) p[q] = f2_add(p[q], o.p[q]);
  }
  // = v + u
  template <typename T>
  __device__ __forceinline__ void sum_of(const Raw<T, VE>& v, const Raw<T, VE>& u) {
    if constexpr (VE == 1) {
      p[0] = f2_pack(v.get(0) + u.get(0), 0.f);
    } else {
#pragma unroll
      for (int q = 0; q < P; ++q) p[q] = f2_add(pair_of(v, q), pair_of(u, q));
    }
  }
  // += w * v
  template <typename T>
  __device__ __forceinline__ void fma(const Raw<T, VE>& v, float w) {
    if constexpr (VE == 1) {
      p[0] = f2_pack(fmaf(w, v.get(0), get(0)), 0.f);
    } else {
      const F2 ww = f2_pack(w, w);
#pragma unroll
      for (int q = 0; q < P; ++q) p[q] = f2_fma(ww, pair_of(v, q), p[q]);
    }
  }
  // += v * u, element by element
  template <typename T>
  __device__ __forceinline__ void fma(const Raw<T, VE>& v, const Raw<T, VE>& u) {
    if constexpr (VE == 1) {
      p[0] = f2_pack(fmaf(v.get(0), u.get(0), get(0)), 0.f);
    } else {
#pragma unroll
      for (int q = 0; q < P; ++q) p[q] = f2_fma(pair_of(v, q), pair_of(u, q), p[q]);
    }
  }
  // += the value held by lane ^ o
  __device__ __forceinline__ void join(unsigned mask, int o) {
#pragma unroll
    for (int q = 0; q < P; ++q) p[q] = f2_add(p[q], __shfl_xor_sync(mask, p[q], o));
  }
  template <typename T>
  __device__ __forceinline__ Pack<T, VE> rounded() const {
    Pack<T, VE> o;
#pragma unroll
    for (int t = 0; t < VE; ++t) o.v[t] = Elem<T>::from_f(get(t));
    return o;
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

// A row is one 32 x 32 + 64 bit multiply-add away from the lane's column of row 0.
template <typename T>
__device__ __forceinline__ const T* at_row(const T* lane_base, uint32_t row, uint32_t row_bytes) {
  return (const T*)((const char*)lane_base + (uint64_t)row * row_bytes);
}

// ---- host side: resident blocks, widest access, lane split ---------------------------------------
// Elements of T in the widest access (at most 16 bytes) that `bits` (row size and base addresses,
// in bytes, or-ed together) is a multiple of.
inline int slice_elems(uint64_t bits, int esz) {
  int b = 16;
  while (b > esz && (bits & (uint64_t)(b - 1))) b >>= 1;
  return b / esz;
}
// Resident blocks of a kernel on an SM of the current device (asked once per kernel and device; `cache` has 64 entries).
template <typename K>
static int blocks_per_sm(K kernel, int block, int* cache, int* out) {
  int dev = 0;
  APT_CUDA(cudaGetDevice(&dev));
  const bool cacheable = dev >= 0 && dev < 64;
  int n = cacheable ? cache[dev] : 0;
  if (n == 0) {
    APT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, block, 0));
    if (n < 1) n = 1;
    if (cacheable) cache[dev] = n;
  }
  *out = n;
  return APT_OK;
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
