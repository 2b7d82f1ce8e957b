// Input rows of any width laid out in whole 16-byte slices (widen.cu), and when a sum has that done.
#pragma once

#include <algorithm>

#include "rows.cuh"

namespace apt {

// When a sum has its input widened. The copy reads and writes every input row once (5.6 TB/s: 67 000 x 404 B 11 us, 469 000 x 404 B 69) and a call with
// one more buffer and launch takes the host 3 us longer; the gain is per edge, and in no order it lies with the rows of very many edges, whose items
// are walked by single warps at the pace of the narrow accesses, where k_spmm_stream cuts them anywhere. us of a call, rows as they are -> widened:
//   in no order, some rows with many of the edges (sources drawn at u^2 of the range, 10 edges a row)   1 000 000 edges from 125 000 rows bf16 x 17 .91 of the
//     time, x 61 .83, x 251 .45, x 198 .81; fp32 x 101 .76, x 137 .51; 99 000 from 12 000 bf16 x 61 .88, x 251 .55, fp32 x 101 .73, x 251 .56
//     where it does not pay   99 000 edges bf16 x 17 1.09, x 34 1.07, fp32 x 31 1.08 (400 000 .99; from 133 000 rows 1 000 000 1.09); rows beyond the 1024 bytes of
//     k_spmm_stream, fp32 x 602 from 8 edges a row 1.06, from 60 .94; accesses of 8 bytes, bf16 x 140 1.12, x 36 1.03; 70 000 edges, fp32 x 251 1.1
//   in no order, all rows alike   99 000 edges bf16 x 251 1.10, fp32 x 101 1.24, bf16 x 198 1.32; 400 000 bf16 x 251 .83 - .96, fp32 x 251 1.06 - 1.19; 1 000 000 bf16 x 251
//     .78, fp32 x 137 .82, x 251 .88, but bf16 x 101 .94 -
//     1.04, x 198 1.12, fp32 x 101 1.03, and from three edges a row fp32 x 251 1.13
//   grouped, 1 005 000 edges from 168 000 rows   bf16 x 17 40 -> 32, x 61 51 -> 41, x 251 139 -> 97; x 140 69 -> 83, fp32 x 101 76 -> 83; from 368 000
//     bf16 x 61 51 -> 54, x 101 79 -> 86; 240 000 edges from 44 000 bf16 x 61 22 -> 23, x 251 37 -> 35
constexpr int kWidenLeast = 34, kWidenMost = 4096;      // bytes of a row
constexpr int64_t kWidenEdges = 3 << 15, kWidenGrouped = 3 << 17, kWidenEven = 15 << 16;
// A mean row that is as good as some of very many edges: of 100 edges each bf16 x 198 .84 - .98 of the time, fp32 x 251 .63 - .92, bf16 x 250 .80 - .98, bf16 x 17 .92 - .97; of
// 150 .57, .40, .53, .82; of 60 bf16 x 198 1.01 - 1.33, bf16 x 250 1.11 - 1.25.
constexpr int64_t kHubMean = 128;
constexpr int kOrderEven = 3;          // kOrder without such rows

// A buffer that there is no memory for is done without, but only after PyTorch's allocator has given back all that it keeps: none larger than any that the lines
// here were measured with would be asked for (the widest rows of 1 000 000).
constexpr int64_t kWidenCopy = (int64_t)4 << 30;

// Elements of a row of `dim` in whole slices.
inline int64_t widened_dim(int64_t dim, size_t esz) { return (dim * (int64_t)esz + 15) / 16 * (16 / (int64_t)esz); }

inline bool widen_pays(int64_t dim, size_t esz, int64_t num_in_rows, int64_t num_edges, int mode) {
  const int64_t row = dim * (int64_t)esz, wide = widened_dim(dim, esz) * (int64_t)esz;
  const int slice = slice_elems((uint64_t)row, (int)esz) * (int)esz;
  if (slice == 16 || row < kWidenLeast || row > kWidenMost || num_in_rows <= 0 || num_in_rows > kWidenCopy / wide) return false;
  if (mode < 2) return slice == 2 && num_edges >= kWidenGrouped && num_edges / 4 >= num_in_rows;      // (grouped)
  if (mode == kOrderEven) return slice == (int)esz && row >= 480 && wide <= 1024 && num_edges >= (slice == 2 ? kWidenGrouped : kWidenEven) && num_edges / 8 >= num_in_rows;
  if (num_edges < kWidenEdges || num_edges / (wide > 1024 ? 16 : slice == (int)esz ? 3 : 4) < num_in_rows) return false;
  if (row <= 128 && (slice == 4 || row <= 64)) return slice <= 4 && num_edges >= 2 * kWidenEdges && (slice == 2 || (row >= 64 && num_edges / 6 >= num_in_rows));
  return slice == 2 || row >= (slice == 4 ? 384 : 768);
}

// The same for the attention layer, whose rows are widened head by head: in the forward the sources' (num_dst 0), in the backward both sides', for
// the dots as well as for the walk. us of forward and backward, rows as they are -> widened, 15 edges a destination:
//   900 000 edges, 150 000 sources   bf16 4 x 47 886 -> 383, 1 x 47 275 -> 175, 4 x 18 320 -> 263, 4 x 10 210 -> 192; fp32 4 x 47 1004 -> 460, 1 x 47 275 -> 222
//   900 000, 600 000 sources         bf16 4 x 47 1258 -> 610, 1 x 47 377 -> 304; fp32 4 x 47 1349 -> 781; there fp32 1 x 47 (walk and dots 272 -> 277) and
//     bf16 4 x 18 (305 -> 315) stay as they are, and the forwards of 4-byte accesses (fp32 4 x 47 223 -> 235)
//   150 000, 25 000 sources          bf16 4 x 47 205 -> 103, fp32 4 x 47 194 -> 112; 300 000, 50 000 fp32 1 x 47 120 -> 103. Below kWidenGatBytes the host's
//     90 us are what such a layer takes.
//   Accesses of 8 bytes, backward alone: bf16 4 x 12 87 -> 97, fp32 8 x 10 219 -> 217
//   Sources that few edges read: forward of 200 000 edges, 180 000 sources bf16 2 x 127 56 -> 67, 4 x 47 55 -> 61, 60 000 sources 2 x 127 .77 of the time; backward of
//     240 000, 72 000 sources fp32 1 x 47 76 -> 83, bf16 8 x 10 96 -> 100, of 900 000, 270 000 sources fp32 1 x 47 .87; forward of 200 000 edges,
//     18 000 sources fp32 1 x 47 21.7 -> 22.7, of 240 000, 22 000 sources .88
constexpr int64_t kWidenGatBytes = 32 << 20;      // that the edges read
constexpr int64_t kWidenGatMany = 1 << 19;
inline bool widen_gat_pays(int64_t head_dim, int heads, size_t esz, int64_t num_src, int64_t num_edges, bool backward) {
  const int64_t row = head_dim * (int64_t)esz;
  const int slice = slice_elems((uint64_t)row, (int)esz) * (int)esz;
  if (slice > 4 || row < 16 || row * heads > kWidenMost || num_src <= 0 || num_edges < kWidenEdges || num_edges * row * heads < kWidenGatBytes) return false;
  if (num_src > kWidenCopy / (widened_dim(head_dim, esz) * (int64_t)esz * heads)) return false;
  if (slice == 2) return num_edges / (backward ? 1 : 2) >= num_src;
  if (!backward) return row * heads >= 128 && num_edges / 4 >= num_src && num_edges * row * heads >= kWidenGatBytes / 4 * 5;
  return num_edges / (row * heads >= 384 ? 1 : num_edges >= kWidenGatMany ? 2 : 4) >= num_src;
}

// `out`: num_rows * ceil(row_bytes / 16) slices, 16-byte aligned. `in` is aligned to its elements of 2 or 4 bytes.
int widen_rows(const void* in, int64_t num_rows, int64_t row_bytes, void* out, cudaStream_t s);

// The first n elements of a slice, at any element's address: pairs of 16-bit ones where they are aligned. (k_spmm_rows, whose rows are several
// to a warp; bf16 x 101 114 us against 94 for 104 columns.)
template <typename T, int VE>
__device__ __forceinline__ void store_some(T* p, const Pack<T, VE>& r, int n) {
  if constexpr (sizeof(T) == 2) {
    const unsigned int* const w = (const unsigned int*)&r;
    if (((uintptr_t)p & 2) == 0) {
#pragma unroll
      for (int t = 0; t < VE; t += 2) {
        if (t + 1 < n) *(unsigned int*)(p + t) = w[t / 2];
        else if (t < n) p[t] = r.v[t];
      }
    } else {
      if (n > 0) p[0] = r.v[0];
#pragma unroll
      for (int t = 1; t < VE; t += 2) {
        if (t + 1 < VE && t + 1 < n) *(unsigned int*)(p + t) = __funnelshift_r(w[t / 2], w[(t + 1) / 2 < VE / 2 ? (t + 1) / 2 : 0], 16);
        else if (t < n) p[t] = r.v[t];
      }
    }
  } else {
#pragma unroll
    for (int t = 0; t < VE; ++t)
      if (t < n) p[t] = r.v[t];
  }
}

// A row of n elements that a warp has in shared memory, to any element's address: side by side lanes write side by side words. (k_spmm_stream, whose
// stores are in its loop many times over: lanes that write their slices themselves 244 us instead of 161 for bf16 x 251, four words a lane at a
// time 235, slices of 4 x 47 weighted ones put together in shared memory 450 instead of 145. As a run time branch beside aligned stores they had
// cost rows of 256 bf16 81 -> 110.)
// Weighted rows are in parts of `part` elements with `more` behind each; inverse: ceil(2^31 / part), else 0.
template <typename T>
__device__ __forceinline__ void store_row(T* out, const T* row, int n, int lane, uint32_t inverse, int more) {
  auto at = [&](int t) { return inverse ? t + (int)__umulhi(2u * t + 1u, inverse) * more : t; };
  if constexpr (sizeof(T) == 2) {
    const unsigned short* const h = (const unsigned short*)row;
    const int odd = (int)((uintptr_t)out >> 1 & 1), words = (n - odd) >> 1;
    unsigned int* const w = (unsigned int*)(out + odd);
#pragma unroll 1
    for (int t = lane; t < words; t += 32) w[t] = (unsigned int)h[at(odd + 2 * t)] | (unsigned int)h[at(odd + 2 * t + 1)] << 16;
    if (odd && lane == 0) out[0] = row[0];
    if ((n - odd & 1) && lane == 31) out[n - 1] = row[at(n - 1)];
  } else {
#pragma unroll 2
    for (int t = lane; t < n; t += 32) out[t] = row[at(t)];
  }
}

}  // namespace apt
