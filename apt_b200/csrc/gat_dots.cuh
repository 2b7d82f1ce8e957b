// The attention backward's dots <grad_out[dst], ft[src]> of every edge and head on the tensor cores, for 16-bit rows whose heads are 32, 64,
// 128 or 256 columns wide.
//
// A warp takes a stretch of the edges, 16 of them (M) against 8 destinations (N) a step: the edges' rows come to shared memory by cp.async, two
// groups on their way, the destinations' stay in registers while the edges, which are grouped, walk over them. Of the 16 x 8
// products of a head one in eight is an edge's own; what the others cost is 16 instructions a group of 256 columns (bf16 32) and their additions, where
// multiplying and reducing across lanes took 46 an edge. The k of a product may be in any order, so a lane's share of two steps is 16 bytes side by
// side in both operands: one load each.
//
// Sums are fp32 and no further from 64 bits than multiplied out (products()). 2-norm of the dots' error over theirs, multiplied out | here, normal values: bf16
// 1 x 32 2.94e-8 | 2.82e-8, 4 x 64 3.93e-8 | 3.84e-8, 2 x 128 4.80e-8 | 4.70e-8, 1 x 256 5.50e-8 | 5.46e-8; f16 4 x 32 5.59e-8 | 5.44e-8, 4 x 64 6.21e-8 | 6.14e-8, 2 x 128
// 6.77e-8 | 6.75e-8, 1 x 256 7.29e-8 | 7.23e-8. Accumulated in the tensor cores from step to step: bf16 1 x 32 3.9e-8, 4 x 64 6.5e-8, 1 x 256 2.3e-7, f16 1 x 256 3.4e-7.
//
// us of a backward pass, multiplied out -> here: bf16 4 x 64, 67 584 x 15 edges 190 -> 185, x 3 edges 87 -> 74, 30 000 x 10 86 -> 77; 4 x 32, 67 584 x 15 200 -> 160; 1 x 128
// 193 -> 148; 1 x 32 111 -> 98; f16 8 x 32 213 -> 200, 30 000 x 10 97 -> 85; 2 x 64, 67 584 x 15 199 -> 150. (Accumulated in the tensor cores bf16 4 x 64 170, 4 x 32 150: the
// products that make the cut good take 14 us of a million edges of 256 columns, the look for sums that are none, which these figures are without, 2 - 3.) So they take every shape they can be built for. Shared addresses worked out for every
// access and a predicate for every row, 27 instructions an edge, took the dots from 56 to 62.
#pragma once

#include "spmm_rows.cuh"

namespace apt {

constexpr int kDotsBlocks = 2, kDotsEdges = 16, kDotsTile = 8;
// Warps a block: as many as shared memory (rows of 512 bytes) or registers hold.
constexpr int dots_warps(int chunks) { return chunks == 8 ? 6 : chunks == 4 ? 10 : 14; }

template <typename T>
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1,
                                             float c0 = 0.f, float c1 = 0.f, float c2 = 0.f, float c3 = 0.f) {
  if constexpr (Elem<T>::kIsBf16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// The products of 32 columns, two steps of 16. The tensor cores cut sums off where fp32 additions round, so that nothing is added up in them beyond a step, and
// of 16-bit values whose own products are exact, which leaves the cut as the larger error, it is made good: what the same products leave of the sum.
template <typename T>
__device__ __forceinline__ void products(F2 (&sum)[2], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, uint32_t a4, uint32_t a5,
                                         uint32_t a6, uint32_t a7, uint32_t b2, uint32_t b3) {
  float p[4], q[4];
  mma_16x8x16<T>(p, a0, a1, a2, a3, b0, b1);
  mma_16x8x16<T>(q, a4, a5, a6, a7, b2, b3);
#pragma unroll
  for (int i = 0; i < 2; ++i) sum[i] = f2_add(f2_pack(p[2 * i], p[2 * i + 1]), f2_pack(q[2 * i], q[2 * i + 1]));
  if constexpr (Elem<T>::kIsBf16) {
    float p_rest[4], q_rest[4];
    mma_16x8x16<T>(p_rest, a0, a1, a2, a3, b0, b1, -p[0], -p[1], -p[2], -p[3]);
    mma_16x8x16<T>(q_rest, a4, a5, a6, a7, b2, b3, -q[0], -q[1], -q[2], -q[3]);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      sum[i] = f2_add(sum[i], f2_add(f2_pack(p_rest[2 * i], p_rest[2 * i + 1]), f2_pack(q_rest[2 * i], q_rest[2 * i + 1])));
  }
}

// An edge's dots that came to NaN, multiplied out: nothing is left of an infinite sum, and that taken from it is no number. us of a backward of 67 584 x 15 edges
// from 150 000 sources, without -> with: 4 x 64 196 -> 199, 1 x 256 185 -> 189, 1 x 128 138 -> 141, 1 x 32 86 -> 88, 8 x 32 235 -> 241. (What is left kept beside a
// head's sum and added where that is finite spilled: 8 x 32 256.)
template <typename T>
__device__ __noinline__ void dots_again(const T* __restrict__ x, const T* __restrict__ y, int heads, int head_dim, float* dots) {
  for (int h = 0; h < heads; ++h) {
    if (dots[h] == dots[h]) continue;
    float sum = 0.f;
    for (int c = h * head_dim; c < (h + 1) * head_dim; ++c) sum = fmaf(Elem<T>::to_f(x[c]), Elem<T>::to_f(y[c]), sum);
    dots[h] = sum;
  }
}

// NC chunks of 32 columns to a row, CPH of them to a head.
template <typename T, int NC, int CPH>
__global__ void __launch_bounds__(dots_warps(NC) * 32, kDotsBlocks)
k_gat_dots_mma(const int64_t* __restrict__ row, const int64_t* __restrict__ col, const T* __restrict__ ft, const T* __restrict__ grad, int64_t E,
               int64_t num_dst, int chunk, const Verdict none, float* __restrict__ dots, uint32_t num_src, int32_t* __restrict__ src_count,
               uint32_t* __restrict__ rank) {
  wait_for_previous();
  constexpr int H = NC / CPH, kRow = NC * 64, kVectors = NC * 4, kSide = 32 / kVectors;      // vectors of 16 bytes to a row, rows a copy instruction
  extern __shared__ __align__(128) unsigned char shared[];
  if (any_found(none)) return;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int warp = blockIdx.x * dots_warps(NC) + (threadIdx.x >> 5);
  unsigned char* const ring = shared + (threadIdx.x >> 5) * 2 * kDotsEdges * kRow;
  const int lo = (int)min((int64_t)warp * chunk, E), hi = (int)min((int64_t)(warp + 1) * chunk, E);
  if (lo >= hi) return;

  // 32 edges, a lane to each. Destinations stay below 2^31, whatever the ids are by now (they were looked at when the ranges were made, maybe a forward
  // pass ago): tiles then rise until a group is done, and no edge's is that of the lanes behind the last one.
  struct Batch {
    uint32_t src, dst, place;
  };
  auto load = [&](int base) {
    Batch b{0u, 0xffffffffu, kNoRank};
    const int e = base + lane;
    if (e < hi) {
      b.src = (uint32_t)row[e], b.dst = min((uint32_t)col[e], 0x7fffffffu);
      if (b.src < num_src) b.place = (uint32_t)atomicAdd(src_count + spread(b.src), 1);
    }
    return b;
  };
  // Vector v of row q of a stage. Neighbouring rows' halves of a line change places, so that eight lanes read eight different vectors: the
  // address of an even chunk and that of an odd one, beside which all others are constants.
  const int vec = lane % kVectors, side = lane / kVectors;
  const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring);
  const uint32_t put_even = ring_at + side * kRow + (NC > 1 ? vec ^ ((side & 1) << 2) : vec) * 16;
  const uint32_t put_odd = ring_at + side * kRow + (NC > 1 ? vec ^ ((~side & 1) << 2) : vec) * 16;
  const unsigned char* const get_even = ring + g * kRow + ((NC > 1 ? (g & 1) * 4 : 0) + t) * 16;
  const unsigned char* const get_odd = ring + g * kRow + (NC > 1 ? (~g & 1) * 4 + t : t) * 16;
  const char* const lane_ft = (const char*)ft + vec * 16;
  auto copy = [&](int stage, int q, uint32_t src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((kSide & 1 && q & 1 ? put_odd : put_even) + (stage * kDotsEdges + q) * kRow),
                 "l"(lane_ft + (uint64_t)src * kRow) : "memory");
  };
  auto issue = [&](uint32_t batch_src, int first, int count, int stage) {
    if (count >= kDotsEdges) {
#pragma unroll
      for (int q = 0; q < kDotsEdges; q += kSide) copy(stage, q, __shfl_sync(0xffffffffu, batch_src, first + q + side));
    } else {
#pragma unroll 1
      for (int q = 0; q < count; q += kSide) {      // (rows behind the last edge's: row 0)
        const uint32_t src = __shfl_sync(0xffffffffu, batch_src, first + q + side);
        copy(stage, q, src);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  Batch now = load(lo), next = load(lo + 32);
  issue(now.src, 0, hi - lo, 0);
  issue(now.src, kDotsEdges, hi - lo - kDotsEdges, 1);

  uint32_t tile = 0xfffffff0u;      // destinations in registers: tile ... tile + 7
  uint4 b[NC];
  const T* const lane_grad = grad + t * 8;
#pragma unroll 1
  for (int base = lo; base < hi; base += 32) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int pos = half * kDotsEdges, count = min(kDotsEdges, hi - base - pos);
      if (count <= 0) break;
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      const uint32_t d0 = __shfl_sync(0xffffffffu, now.dst, pos + g), d1 = __shfl_sync(0xffffffffu, now.dst, pos + g + 8);
      uint32_t first = __shfl_sync(0xffffffffu, now.dst, pos);
      const uint32_t last = __shfl_sync(0xffffffffu, now.dst, pos + count - 1);
#pragma unroll 1
      for (;;) {
        if (first - tile >= kDotsTile) {
          tile = first;
          const T* const own = lane_grad + min((uint64_t)tile + g, (uint64_t)num_dst - 1) * (NC * 32);
#pragma unroll
          for (int c = 0; c < NC; ++c) b[c] = __ldg((const uint4*)(own + c * 32));
        }
        F2 acc[H][2], part[4][2];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const unsigned char* const p = (c & 1 ? get_odd : get_even) + half * kDotsEdges * kRow + (c & ~1) * 64;
          const uint4 x = *(const uint4*)p, y = *(const uint4*)(p + 8 * kRow);
          F2 sum[2];
          products<T>(sum, x.x, y.x, x.y, y.y, b[c].x, b[c].y, x.z, y.z, x.w, y.w, b[c].z, b[c].w);
          // in pairs, pairs of pairs, ...
#pragma unroll
          for (int level = 0; level < 4; ++level) {
            const bool pair = (c % CPH + 1) % (2 << level) == 0 && (1 << level) < CPH;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (pair) sum[i] = f2_add(part[level][i], sum[i]);
              else part[level][i] = sum[i];
            }
            if (!pair) break;
          }
          if (c % CPH == CPH - 1) acc[c / CPH][0] = sum[0], acc[c / CPH][1] = sum[1];
        }
        // an edge's own product is with the lane that has its destination's column
        float* const out = dots + (int64_t)(base + pos + g) * H;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t s = (i ? d1 : d0) - tile;
          if ((s >> 1) == (uint32_t)t) {
            float v[H];
#pragma unroll
            for (int h = 0; h < H; ++h) {
              float even, odd;
              f2_unpack(acc[h][i], even, odd);
              v[h] = s & 1u ? odd : even;
            }
            if constexpr (H % 4 == 0) {
#pragma unroll
              for (int h = 0; h < H; h += 4) *(float4*)(out + 8 * i * H + h) = make_float4(v[h], v[h + 1], v[h + 2], v[h + 3]);
            } else if constexpr (H == 2) {
              *(float2*)(out + 8 * i * H) = make_float2(v[0], v[1]);
            } else {
              out[8 * i * H] = v[0];
            }
            if constexpr (Elem<T>::kIsBf16) {
              bool none = false;
#pragma unroll
              for (int h = 0; h < H; ++h) none |= v[h] != v[h];
              if (none) {
                const uint64_t src = min((uint32_t)row[base + pos + g + 8 * i], num_src - 1), dst = min((uint64_t)tile + s, (uint64_t)num_dst - 1);
                dots_again(ft + src * (NC * 32), grad + dst * (NC * 32), H, CPH * 32, out + 8 * i * H);
              }
            }
          }
        }
        if (last - tile < kDotsTile) break;
        // the first edge of the group whose destination lies behind these
        const unsigned behind = __ballot_sync(0xffffffffu, lane >= pos && lane < pos + count && now.dst >= tile + kDotsTile);
        if (!behind) break;      // (not of edges that rise)
        first = __shfl_sync(0xffffffffu, now.dst, __ffs(behind) - 1);
      }
      __syncwarp();      // read by all lanes: the next copies may overwrite it
      issue(next.src, pos, hi - base - 32 - pos, half);
    }
    if (base + lane < hi) rank[base + lane] = now.place;
    now = next;
    next = load(base + 64);
  }
}

// slice: bytes of the widest access to both sides' rows.
// Where most destinations have no edges, the eight rows of a tile are fetched for one or two that have, and a group of edges goes through several tiles.
// k_gat_dots, a warp to a destination, loses there all the same; k_spmm_stream, which takes wide rows of many edges, fetches those in use alone. us of a
// backward, k_spmm_stream -> here, 1 000 000 edges from 150 000 sources: f16 8 x 32, 66 666 destinations of 15 edges side by side 214 -> 200, 4 apart 309 -> 309, 8 apart
// 374 -> 396; bf16, whose products are made twice, side by side, 2 and 3 apart 1 x 256 192, 220, 226 -> 188, 216, 228, 2 x 128 201, 230, 236 -> 200, 227, 240, 4 x 64
// 198, 232, 247 -> 199, 231, 251, 8 x 32 233, 296, 345 -> 240, 305, 362; 100 000 of 10 1 x 256 197 -> 197, 2 x 128 205 -> 207, 4 x 64 208 -> 211, 8 x 32 257 -> 269. The lines, edges to a
// destination and columns of a bf16 head, are where none of them loses more than 3 %.
template <typename T>
inline bool dots_mma_fits(int heads, int64_t head_dim, int slice, int64_t num_edges, int64_t num_dst) {
  const int64_t dim = heads * head_dim;
  auto pow2 = [](int64_t x) { return x > 0 && (x & (x - 1)) == 0; };
  if (sizeof(T) != 2 || slice != 16 || num_edges > kStreamMaxEdges || head_dim < 32 || dim > 256 || !pow2(head_dim) || !pow2(heads)) return false;
  const bool many = Elem<T>::kIsBf16 ? head_dim >= 64 && num_edges / 5 >= num_dst : num_edges / 2 >= num_dst;
  return many || !stream_fits(kDots, slice, dim, sizeof(T), heads, num_edges, true);
}

template <typename T, int NC, int CPH>
static int launch_dots_mma(const int64_t* row, const int64_t* col, const T* ft, const T* grad, int64_t E, int64_t num_dst, const Verdict& none,
                           float* dots, uint32_t num_src, const SpmmWs& sort, cudaStream_t s) {
  constexpr int kWarps = dots_warps(NC), kShared = kWarps * 2 * kDotsEdges * NC * 64;
  static bool sized[64] = {};
  int dev = 0;
  APT_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !sized[dev]) {
    APT_CUDA(cudaFuncSetAttribute(k_gat_dots_mma<T, NC, CPH>, cudaFuncAttributeMaxDynamicSharedMemorySize, kShared));
    if (dev < 64) sized[dev] = true;
  }
  // stretches of whole groups, as many as there are warps; of 32 edges at least
  const int64_t warps = (int64_t)kNumSMs * kDotsBlocks * kWarps;
  const int64_t chunk = std::max<int64_t>(32, ceil_div(ceil_div(E, warps), kDotsEdges) * kDotsEdges);
  APT_FOLLOW((k_gat_dots_mma<T, NC, CPH>), (int)ceil_div(ceil_div(E, chunk), kWarps), kWarps * 32, kShared, s, row, col, ft, grad, E, num_dst,
             (int)chunk, none, dots, num_src, sort.cnt, sort.rank);
  return APT_OK;
}

template <typename T>
static int launch_dots_mma(int heads, int64_t head_dim, const int64_t* row, const int64_t* col, const T* ft, const T* grad, int64_t E, int64_t num_dst,
                           const Verdict& none, float* dots, uint32_t num_src, const SpmmWs& sort, cudaStream_t s) {
#define APT_DOTS(NC, CPH) \
  if (heads * head_dim == (NC) * 32 && head_dim == (CPH) * 32) return launch_dots_mma<T, NC, CPH>(row, col, ft, grad, E, num_dst, none, dots, num_src, sort, s)
  APT_DOTS(1, 1);
  APT_DOTS(2, 1);
  APT_DOTS(4, 1);
  APT_DOTS(8, 1);
  APT_DOTS(2, 2);
  APT_DOTS(4, 2);
  APT_DOTS(8, 2);
  APT_DOTS(4, 4);
  APT_DOTS(8, 4);
  APT_DOTS(8, 8);
#undef APT_DOTS
  set_error("apt_gat_backward: %d heads of %lld columns have no product kernel", heads, (long long)head_dim);
  return APT_ERR_BAD_ARG;
}

}  // namespace apt
