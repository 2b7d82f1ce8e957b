// Rows of any width copied to a pitch of whole 16-byte slices, zeros behind their ends.
//
// A row of 119 16-bit elements starts on a boundary of two bytes, and whoever reads such rows edge by edge reads them two bytes a
// lane. A sum reads each input row as often as it has edges, so one pass that lays the rows out anew (each read and written once) buys
// 16-byte slices for all of those reads.
//
// A warp takes a chunk of rows, which in the result are one run of slices (k_gather's way); a lane makes a slice of the two aligned
// 16-byte vectors that its bytes lie in, shifted in registers. Vectors that reach beyond the input are read by elements instead. Bound by HBM:
// 469 000 rows of 404 bytes 69 us (5.6 TB/s), 67 000 11.4, of 502 bytes 75 and 11.8. Which sums have it done: widen.cuh.
#include "widen.cuh"

namespace apt {

constexpr int kWidenSlices = 4;      // a lane has on their way

// Bytes [p, p + valid) in front of zeros; whole elements of 2 or 4 bytes.
__device__ __forceinline__ uint4 slice_by_elements(const char* p, int valid) {
  uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (2 * k < valid) w[k / 2] |= (uint32_t)*(const unsigned short*)(p + 2 * k) << (k & 1 ? 16 : 0);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// What a slice has of memory: the two vectors, or the slice itself.
struct SliceParts {
  uint4 lo, hi;
  int shift, valid;      // bytes; shift -1: `lo` is the slice
};
__device__ __forceinline__ SliceParts slice_load_any(const char* p, int valid, const char* begin, const char* end) {
  SliceParts r;
  r.shift = (int)((uintptr_t)p & 15);
  r.valid = valid;
  r.hi = make_uint4(0u, 0u, 0u, 0u);
  const char* const a = p - r.shift;
  const bool two = r.shift + valid > 16;
  if (a >= begin && a + (two ? 32 : 16) <= end) {
    r.lo = __ldg((const uint4*)a);
    if (two) r.hi = __ldg((const uint4*)(a + 16));
  } else {
    r.lo = slice_by_elements(p, valid);
    r.shift = -1;
  }
  return r;
}
__device__ __forceinline__ uint4 slice_of(const SliceParts& r) {
  if (r.shift < 0) return r.lo;
  uint32_t w[8] = {r.lo.x, r.lo.y, r.lo.z, r.lo.w, r.hi.x, r.hi.y, r.hi.z, r.hi.w};
  if (r.shift & 8) {
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = w[k + 2];
  }
  if (r.shift & 4) {
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = w[k + 1];
  }
  if (r.shift & 2) {
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = __funnelshift_r(w[k], w[k + 1], 16);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = r.valid >= 4 * k + 4 ? w[k] : r.valid > 4 * k ? w[k] & 0xffffu : 0u;
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void __launch_bounds__(256)
k_widen(const char* __restrict__ in, int64_t num_rows, int row_bytes, uint32_t slices, uint32_t inverse, int per, uint4* __restrict__ out) {
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  const char* const end = in + num_rows * row_bytes;
  for (int64_t first = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * per; first < num_rows; first += (int64_t)gridDim.x * 8 * per) {
    const uint32_t total = (uint32_t)min((int64_t)per, num_rows - first) * slices;
    const char* const src = in + first * row_bytes;
    uint4* const dst = out + first * slices;
    for (uint32_t i0 = lane; i0 < total; i0 += 32 * kWidenSlices) {
      SliceParts v[kWidenSlices];
#pragma unroll
      for (int u = 0; u < kWidenSlices; ++u) {
        const uint32_t i = i0 + 32 * u;
        if (i >= total) continue;
        const uint32_t r = __umulhi(2 * i + 1, inverse), at = (i - r * slices) * 16;
        v[u] = slice_load_any(src + (int64_t)r * row_bytes + at, min(16, row_bytes - (int)at), in, end);
      }
#pragma unroll
      for (int u = 0; u < kWidenSlices; ++u)
        if (i0 + 32 * u < total) dst[i0 + 32 * u] = slice_of(v[u]);
    }
  }
}

int widen_rows(const void* in, int64_t num_rows, int64_t row_bytes, void* out, cudaStream_t s) {
  const int64_t slices = ceil_div(row_bytes, 16);
  // about a round of slices for every lane of a chunk's warp, of 64 rows at most (rows of two slices and more); the row of slice i: exact while i < 2^18 and
  // slices < 2^12 (k_gather)
  const int per = (int)std::max<int64_t>(1, 32 * kWidenSlices / slices);
  const uint32_t inverse = (uint32_t)(((1ull << 31) + slices - 1) / slices);
  APT_FOLLOW(k_widen, wave_grid(ceil_div(num_rows, (int64_t)per * 8), 8), 256, 0, s, (const char*)in, num_rows, (int)row_bytes, (uint32_t)slices,
             inverse, per, (uint4*)out);
  return APT_OK;
}

}  // namespace apt
