// Fused GAT edge pipeline over one sampled block whose edges are grouped by destination. For every destination d
// with its edges e (src_e -> d) and every head h
//   s_e = leaky_relu(el[src_e, h] + er[d, h]),  a_e = softmax of s over d's edges,
//   out[d, h, :] = sum_e a_e ft[src_e, h, :]
// (python/npc/model/gatconv.py:113-124), and in the backward, with g = grad_out[d, h, :],
//   dot_e = <g, ft[src_e, h, :]>,  t = sum_e a_e dot_e,
//   grad_s_e = a_e (dot_e - t) (el + er > 0 ? 1 : slope),  grad_er[d, h] = sum_e grad_s_e,
//   grad_ft[s, h, :] = sum over the edges out of s of a_e g,  grad_el[s, h] = sum of grad_s_e.
//
// The work per edge and head is a few scalars, the work per edge and column is a gather of rows; they want opposite
// kernels and are kept apart, with fp32 weights per edge and head between them (16 MB for a million edges of four
// heads, which stay in L2):
//
//   k_gat_ranges    where each destination's edges are (6.5 us with one edge a thread; a word that every kernel looks at had
//                   to be cleared in front, a launch more: attention of 30 000 x 15 edges, bf16 4 x 64, 41.5 -> 38.3 us forward)
//   k_gat_weights   scores and softmax, a few lanes per destination and up to four of its heads, two edges a lane; any number of
//                   edges and heads.
//   sums            the weighted sum is the SpMM's (kUMulW), any head width: k_spmm_stream for wide rows of many edges, else k_spmm_rows
//   k_gat_dots      backward: <g, ft> of every edge and head, one warp per destination (16-bit heads of 32 to 256 columns: k_gat_dots_mma,
//                   gat_dots.cuh; other wide rows of many edges: k_spmm_stream's kDots). The four partial dots of a lane are reduced together: each step halves the values
//                   a lane keeps, log2(lph) + 1 shuffles for four edges instead of 4 log2(lph).
//   k_gat_scores    backward: t, grad_s and grad_er, the same lanes; grad_el is added up in fp32 with one reduction per edge
//                   of up to four of its heads
//   sums            grad_ft: the weighted sum of the forward with the sides swapped. (grad_el as a second accumulator of the same
//                   walk cost k_spmm_rows a block an SM and the scores had to be written out for it: 150 us against 116.)
//   The counting sort by source that grad_ft needs rides along: the dots have every edge's source in a register and wait
//                   for rows most of the time, so they also count the edges (the add returns an edge's place in its
//                   row); k_dst_slots gives the rows their places; k_gat_scores writes the order. As launches of
//                   their own the first and the last pass took 23 + 16 us.
//   k_gat_source    grad_el in T
//   k_widen         heads that are no whole slices, laid out so first (widen.cuh)
//
// k_gat_alone and k_gat_alone_backward serve the two entry points that have no buffer for weights, k_gat_narrow forwards of
// narrow rows that nobody will ask for a backward.
//
// One kernel that did scores and rows in turn (a warp per destination) was bound by the registers of the one
// and the latency of the other: 133 - 149 us forward on 67 584 x 15 edges, bf16, 4 x 64, in three forms; the two
// kernels take 16 + 61 us. Backward of that block: 16 (saved after a forward) + 56 + 5 + 31 + 75 + 4 us (each kernel by itself, caches
// cold), where the edge kernel and two reverse SpMM calls with a sort each took 803 us.
#include <math.h>

#include <algorithm>

#include "gat_dots.cuh"
#include "spmm_rows.cuh"

namespace apt {

__device__ __forceinline__ float leaky(float x, float slope) { return x > 0.f ? x : x * slope; }

// A destination whose scores have no sum (all of them -inf, as a mask leaves them, or a NaN among them): up to this many edges
// its weights are zero, beyond it they are NaN. The bound lies where it has always been for callers: 32 edges for rows of
// more than 256 bytes in 16-byte slices and up to 8 heads, none for other shapes.
constexpr int kMaskedEdges = 32;
static int masked_edges(int num_heads, int64_t head_dim, size_t esz, uintptr_t rows) {
  const bool slices = ((uint64_t)(head_dim * esz) & 15) == 0 && (rows & 15) == 0;
  return slices && num_heads * head_dim * (int64_t)esz > 256 && num_heads <= 8 ? kMaskedEdges : 0;
}

// Sum over groups of n lanes (a power of two).
__device__ __forceinline__ float group_sum(float v, int n) {
  for (int o = n >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// First and last edge of every destination; a block's verdict is set when its edges are not grouped (nothing then belongs to
// anybody). Four edges a thread are in flight, on four blocks an SM at most.
__global__ void __launch_bounds__(256)
k_gat_ranges(const int64_t* __restrict__ col, int64_t E, int64_t num_dst, int2* __restrict__ range, uint32_t* __restrict__ verdict,
             int32_t* status) {
  wait_for_previous();
  constexpr int K = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  bool bad = false;
  for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e0 < E; e0 += K * stride) {
    int64_t at[K], before[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t e = e0 + k * stride;
      at[k] = e < E ? col[e] : 0;
      // (a negative one opens no gap in front of the table: its own edge is the bad one)
      before[k] = e < E && e > 0 ? max(col[e - 1], (int64_t)-1) : (int64_t)-1;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t e = e0 + k * stride, d = at[k], prev = before[k];
      if (e >= E) break;
      if (d < prev || d < 0 || d >= num_dst) {
        bad = true;
        continue;
      }
      if (d != prev) {
        if (prev >= 0) range[prev].y = (int)e;
        for (int64_t t = prev + 1; t < d; ++t) range[t] = make_int2(0, 0);
        range[d].x = (int)e;
      }
      if (e == E - 1) {
        range[d].y = (int)E;
        for (int64_t t = d + 1; t < num_dst; ++t) range[t] = make_int2(0, 0);
      }
    }
  }
  const int any = __syncthreads_or(bad);
  if (threadIdx.x != 0) return;
  verdict[blockIdx.x] = (uint32_t)any;
  if (any) atomicOr(status, APT_FLAG_NOT_GROUPED);
}

// W lanes to a destination, kGatEdges edges a lane, the edges of a round side by side: loads and stores of a value per edge are
// coalesced, a destination of up to W * kGatEdges edges is one round of latency, and the reductions to sums carry NH heads each.
// A thread per destination and head before: weights 19 -> 17.5 us, scores 43 -> 30 (67 584 x 15 edges, bf16, 4 heads); forward
// and backward of 30 000 destinations, bf16 4 x 64, 3 to 32 edges 114 - 290 -> 96 - 232 with the streams, fp32 1 x 32 x 25 170 -> 136.
constexpr int kGatEdges = 2;
template <int NH>
struct Heads {
  float v[NH];
};
template <int NH>
__device__ __forceinline__ Heads<NH> load_heads(const float* p) {      // aligned to all of them
  const Pack<float, NH> w = load_pack<float, NH>(p);
  Heads<NH> r;
#pragma unroll
  for (int h = 0; h < NH; ++h) r.v[h] = w.v[h];
  return r;
}
template <typename T, int NH>
__device__ __forceinline__ Heads<NH> load_scores(const T* p) {         // the same
  const Pack<T, NH> w = load_pack<T, NH>(p);
  Heads<NH> r;
#pragma unroll
  for (int h = 0; h < NH; ++h) r.v[h] = Elem<T>::to_f(w.v[h]);
  return r;
}
// What a group of lanes works on: destination i with its NH heads, or, where there are more heads (SIDE), the i-th block of NH of them,
// those of a destination one after another.
template <int NH, bool SIDE>
struct HeadBlocks {
  int64_t count;
  int per_row;
  __device__ __forceinline__ HeadBlocks(int64_t num_dst, int num_heads) : count(num_dst), per_row(1) {
    if (SIDE) per_row = num_heads / NH, count *= per_row;
  }
  __device__ __forceinline__ void at(int64_t i, int64_t& d, int& h0) const {
    d = i, h0 = 0;
    if (!SIDE) return;
    d = count >> 32 ? i / per_row : (int64_t)((uint32_t)i / (uint32_t)per_row);
    h0 = (int)(i - d * per_row) * NH;
  }
};
template <int W>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = 1; o < W; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Attention weights.
template <typename T, int W, int NH, bool SIDE>
__global__ void __launch_bounds__(256)
k_gat_weights(const int64_t* __restrict__ row, const T* __restrict__ el, const T* __restrict__ er, int num_heads, float slope,
              int64_t num_dst, const int2* __restrict__ range, const Verdict none, float* weight,
              T* __restrict__ attn, int masked) {
  wait_for_previous();
  constexpr int K = kGatEdges;
  if (any_found(none)) return;
  const int64_t stride = (int64_t)gridDim.x * (256 / W);
  const int part = threadIdx.x & (W - 1);
  // (all lanes of a warp stay: groups behind the last one have no edges)
  const HeadBlocks<NH, SIDE> blocks(num_dst, num_heads);
  for (int64_t i0 = ((int64_t)blockIdx.x * 256 + (threadIdx.x & ~31)) / W; i0 < blocks.count; i0 += stride) {
    const int64_t i = i0 + (threadIdx.x & 31) / W;
    const bool there = i < blocks.count;
    int64_t d;
    int h0;
    blocks.at(i, d, h0);
    const int2 r = there ? range[d] : make_int2(0, 0);
    const int deg = r.y - r.x;
    const bool few = deg <= K * W;
    uint32_t src[K];
#pragma unroll
    for (int k = 0; k < K; ++k) src[k] = few && part + k * W < deg ? (uint32_t)row[r.x + part + k * W] : 0u;
    Heads<NH> bias, s[K];
    float most[NH], sum[NH], inv[NH];
    bool zero[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      bias.v[h] = there ? Elem<T>::to_f(er[d * num_heads + h0 + h]) : 0.f;
      most[h] = -INFINITY;
      sum[h] = 0.f;
    }
    auto scores = [&](int64_t from) {
      Heads<NH> x = load_scores<T, NH>(el + from * num_heads + h0);
#pragma unroll
      for (int h = 0; h < NH; ++h) x.v[h] = leaky(x.v[h] + bias.v[h], slope);
      return x;
    };
    // (plain accesses: what a lane reads here it has written itself)
    auto keep = [&](int e, const Heads<NH>& x) {
      Pack<float, NH> w;
#pragma unroll
      for (int h = 0; h < NH; ++h) w.v[h] = x.v[h];
      store_pack<float, NH>(weight + (int64_t)e * num_heads + h0, w);
    };
    auto kept = [&](int e) {
      const Pack<float, NH> w = *(const Pack<float, NH>*)(weight + (int64_t)e * num_heads + h0);
      Heads<NH> x;
#pragma unroll
      for (int h = 0; h < NH; ++h) x.v[h] = w.v[h];
      return x;
    };
    if (few) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (part + k * W < deg) {
          s[k] = scores(src[k]);
#pragma unroll
          for (int h = 0; h < NH; ++h) most[h] = fmaxf(most[h], s[k].v[h]);
        }
    } else {
      // the scores wait where the weights will be: a source's is fetched once
#pragma unroll 2
      for (uint32_t j = part; j < (uint32_t)deg; j += W) {
        const Heads<NH> x = scores(row[r.x + j]);
#pragma unroll
        for (int h = 0; h < NH; ++h) most[h] = fmaxf(most[h], x.v[h]);
        keep(r.x + j, x);
      }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
      for (int o = 1; o < W; o <<= 1) most[h] = fmaxf(most[h], __shfl_xor_sync(0xffffffffu, most[h], o));
    if (few) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (part + k * W < deg)
#pragma unroll
          for (int h = 0; h < NH; ++h) {
            s[k].v[h] = expf(s[k].v[h] - most[h]);
            sum[h] += s[k].v[h];
          }
    } else {
#pragma unroll 2
      for (uint32_t j = part; j < (uint32_t)deg; j += W) {
        Heads<NH> x = kept(r.x + j);
#pragma unroll
        for (int h = 0; h < NH; ++h) {
          x.v[h] = expf(x.v[h] - most[h]);
          sum[h] += x.v[h];
        }
        keep(r.x + j, x);
      }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      sum[h] = lanes_sum<W>(sum[h]);
      inv[h] = sum[h] > 0.f ? 1.f / sum[h] : 0.f;
      zero[h] = !(sum[h] > 0.f) && deg <= masked;
    }
    auto put = [&](int e, const Heads<NH>& p) {
      const int64_t o = (int64_t)e * num_heads + h0;
      Pack<float, NH> w;
#pragma unroll
      for (int h = 0; h < NH; ++h) w.v[h] = zero[h] ? 0.f : p.v[h] * inv[h];
      store_pack<float, NH>(weight + o, w);
      if (attn)
#pragma unroll
        for (int h = 0; h < NH; ++h) attn[o + h] = Elem<T>::from_f(w.v[h]);
    };
    if (few) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (part + k * W < deg) put(r.x + part + k * W, s[k]);
    } else {
#pragma unroll 2
      for (uint32_t j = part; j < (uint32_t)deg; j += W) put(r.x + j, kept(r.x + j));
    }
  }
}

// Dots of the destination's gradient with its edges' rows. lph lanes to a head's slices, hpp heads side by side, ep
// edges side by side; heads and slices beyond that are walked in blocks.
template <typename T, int VE>
__global__ void __launch_bounds__(256, 3)
k_gat_dots(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ grad_out, int num_heads, int head_dim,
           int64_t num_dst_, const int2* __restrict__ range, const Verdict none, float* __restrict__ dots, int lph,
           int hpp, uint32_t num_src, int32_t* __restrict__ src_count, uint32_t* __restrict__ rank) {
  wait_for_previous();
  if (any_found(none)) return;
  const int lane = threadIdx.x & 31;
  const uint32_t G = gridDim.x * 8, num_dst = (uint32_t)num_dst_;
  const int lpe = lph * hpp, ep = 32 / lpe;
  const int epi = lane / lpe, rh = (lane & (lpe - 1)) / lph, p = lane & (lph - 1);
  const int nvh = head_dim / VE;
  const uint32_t row_bytes = (uint32_t)((int64_t)num_heads * head_dim * sizeof(T));
  uint32_t d = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (d >= num_dst) return;
  int2 r = range[d], nr = make_int2(0, 0);
  // lanes past the last edge hold its source too, so that a round may load past the end
  uint32_t src = r.x < r.y ? (uint32_t)row[r.x + min(lane, r.y - r.x - 1)] : 0u, nsrc = 0;
  if (d + G < num_dst) nr = range[d + G];
  for (; d < num_dst; d += G) {
    int2 nnr = make_int2(0, 0);
    if (nr.x < nr.y) nsrc = (uint32_t)row[nr.x + min(lane, nr.y - nr.x - 1)];
    if (d + 2 * G < num_dst) nnr = range[d + 2 * G];
    for (int h0 = 0; h0 < num_heads; h0 += hpp) {
      const int h = h0 + rh;
      const bool rows = h < num_heads;
      // lanes without a slice read one that exists and contribute nothing (no zero times what may be infinite)
      const int64_t col = (int64_t)(rows ? h : h0) * head_dim;
      const T* const grad = grad_out + (int64_t)d * num_heads * head_dim + col;
      F2 g[Acc<VE>::P];      // the gradient's slice, unpacked
      int at = 0;
      bool mine = false;
      auto block = [&](int c0) {
        at = min(c0 + p, nvh - 1) * VE;
        mine = c0 + p < nvh;
        const Raw<T, VE> raw = load_raw<T, VE>(grad + at);
#pragma unroll
        for (int q = 0; q < Acc<VE>::P; ++q) {
          if constexpr (VE > 1) g[q] = pair_of(raw, q); else g[q] = f2_pack(raw.get(0), 0.f);
        }
      };
      block(0);
#pragma unroll 1
      for (int rest = r.y - r.x; rest > 0; rest -= 32) {
        const int base = r.y - rest, cnt = min(32, rest);
        uint32_t my_src = src;
        if (base != r.x) my_src = (uint32_t)row[base + min(lane, rest - 1)];
        const bool ranked = h0 == 0 && lane < cnt;
        uint32_t place = kNoRank;
        if (ranked && my_src < num_src) place = (uint32_t)atomicAdd(src_count + spread(my_src), 1);
#pragma unroll 1
        for (int j0 = 0; j0 < cnt; j0 += ep * 4) {
          float dt[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
          for (int c0 = 0; c0 < nvh; c0 += lph) {
            if (nvh > lph) block(c0);
            const T* const lane_ft = ft + col + at;
            Raw<T, VE> v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              v[u] = load_raw<T, VE>(at_row(lane_ft, __shfl_sync(0xffffffffu, my_src, (j0 + u * ep + epi) & 31), row_bytes));
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              F2 pair = 0ull;
#pragma unroll
              for (int q = 0; q < Acc<VE>::P; ++q) {
                if constexpr (VE > 1) pair = f2_fma(g[q], pair_of(v[u], q), pair);
                else pair = f2_fma(g[q], f2_pack(v[u].get(0), 0.f), pair);
              }
              float lo, hi;
              f2_unpack(pair, lo, hi);
              dt[u] += mine ? lo + hi : 0.f;
            }
          }
          float* const out = dots + (int64_t)(base + j0 + epi) * num_heads + h;
          const int left = cnt - j0 - epi;       // edges of the chunk from this lane's first one on
          if (lph >= 4) {
            // this lane ends up with the dot of one of the four edges
            const bool hi = p & (lph >> 1), lo = p & (lph >> 2);
            const float b0 = (hi ? dt[2] : dt[0]) + __shfl_xor_sync(0xffffffffu, hi ? dt[0] : dt[2], lph >> 1);
            const float b1 = (hi ? dt[3] : dt[1]) + __shfl_xor_sync(0xffffffffu, hi ? dt[1] : dt[3], lph >> 1);
            const float v = group_sum((lo ? b1 : b0) + __shfl_xor_sync(0xffffffffu, lo ? b0 : b1, lph >> 2), lph >> 2);
            const int u = ((hi ? 2 : 0) + (lo ? 1 : 0)) * ep;
            if (rows && u < left && (p & ((lph >> 2) - 1)) == 0) out[(int64_t)u * num_heads] = v;
          } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (lph == 2) dt[u] += __shfl_xor_sync(0xffffffffu, dt[u], 1);
              if (rows && p == 0 && u * ep < left) out[(int64_t)u * ep * num_heads] = dt[u];
            }
          }
        }
        if (ranked) rank[base + lane] = place;
      }
    }
    r = nr, src = nsrc, nr = nnr;
  }
}

// sums[] += v, for NH heads at once.
template <int NH>
__device__ __forceinline__ void add_heads(float* p, const Heads<NH>& v) {
  if constexpr (NH == 4) atomicAdd((float4*)p, make_float4(v.v[0], v.v[1], v.v[2], v.v[3]));
  else if constexpr (NH == 2) atomicAdd((float2*)p, make_float2(v.v[0], v.v[1]));
  else atomicAdd(p, v.v[0]);
}

// Score gradients, added to sums[spread(source)][head], and the destination's edges to their places in the order by source.
template <typename T, int W, int NH, bool SIDE>
__global__ void __launch_bounds__(256)
k_gat_scores(const int64_t* __restrict__ row, const T* __restrict__ el, const T* __restrict__ er, int num_heads, float slope,
             int64_t num_src, int64_t num_dst, int64_t E, const int2* __restrict__ range, const Verdict none,
             float* __restrict__ weight, const float* __restrict__ dots, float* __restrict__ sums, const SpmmWs sort, OrderKind kind,
             T* __restrict__ grad_er) {
  wait_for_previous();
  constexpr int K = kGatEdges;
  const bool empty = any_found(none);
  if (empty)   // no edge belongs to anybody
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < E * num_heads; o += (int64_t)gridDim.x * blockDim.x) weight[o] = 0.f;
  const int64_t stride = (int64_t)gridDim.x * (256 / W);
  const int part = threadIdx.x & (W - 1);
  const HeadBlocks<NH, SIDE> blocks(num_dst, num_heads);
  for (int64_t i0 = ((int64_t)blockIdx.x * 256 + (threadIdx.x & ~31)) / W; i0 < blocks.count; i0 += stride) {
    const int64_t i = i0 + (threadIdx.x & 31) / W;
    const bool there = i < blocks.count;
    int64_t d;
    int h0;
    blocks.at(i, d, h0);
    const int2 r = there && !empty ? range[d] : make_int2(0, 0);
    const int deg = r.y - r.x;
    const bool few = deg <= K * W;
    // an edge to its place
    auto place_of = [&](int e) { return sort.rank[e]; };
    auto put = [&](int e, int64_t src, uint32_t place) {
      if (place == kNoRank) return;
      const uint32_t at = (uint32_t)sort.range[src].x + place;
      if (kind == kByBoth) ((uint4*)sort.order)[at] = make_uint4((uint32_t)d, (uint32_t)src, (uint32_t)e, 0u);
      else sort.order[at] = make_uint2((uint32_t)d, (uint32_t)e);
    };
    int64_t src[K];
    uint32_t place[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const bool mine = few && part + k * W < deg;
      src[k] = mine ? row[r.x + part + k * W] : 0;
      place[k] = mine && h0 == 0 ? place_of(r.x + part + k * W) : kNoRank;
    }
    Heads<NH> bias, w[K], dot[K], x[K];
    float t[NH], ger[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      bias.v[h] = there ? Elem<T>::to_f(er[d * num_heads + h0 + h]) : 0.f;
      t[h] = ger[h] = 0.f;
    }
    auto fetch = [&](int e, Heads<NH>& a, Heads<NH>& b) {
      a = load_heads<NH>(weight + (int64_t)e * num_heads + h0);
      b = load_heads<NH>(dots + (int64_t)e * num_heads + h0);
    };
    if (few) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (part + k * W < deg) {
          fetch(r.x + part + k * W, w[k], dot[k]);
          x[k] = load_scores<T, NH>(el + src[k] * num_heads + h0);
        }
      // (the lanes of the first heads have the places)
#pragma unroll
      for (int k = 0; k < K; ++k) put(r.x + part + k * W, src[k], place[k]);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (part + k * W < deg)
#pragma unroll
          for (int h = 0; h < NH; ++h) t[h] += w[k].v[h] * dot[k].v[h];
    } else {
#pragma unroll 2
      for (uint32_t j = part; j < (uint32_t)deg; j += W) {
        Heads<NH> a, b;
        fetch(r.x + j, a, b);
#pragma unroll
        for (int h = 0; h < NH; ++h) t[h] += a.v[h] * b.v[h];
      }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) t[h] = lanes_sum<W>(t[h]);
    auto grad = [&](int64_t from, const Heads<NH>& a, const Heads<NH>& b, const Heads<NH>& c) {
      Heads<NH> gs;
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        gs.v[h] = a.v[h] * (b.v[h] - t[h]) * (c.v[h] + bias.v[h] > 0.f ? 1.f : slope);
        ger[h] += gs.v[h];
      }
      if ((uint64_t)from < (uint64_t)num_src) add_heads<NH>(sums + (int64_t)spread((uint32_t)from) * num_heads + h0, gs);
    };
    if (few) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (part + k * W < deg) grad(src[k], w[k], dot[k], x[k]);
    } else {
      for (uint32_t j = part; j < (uint32_t)deg; j += W) {
        const int e = r.x + j;
        const int64_t from = row[e];
        fetch(e, w[0], dot[0]);
        x[0] = load_scores<T, NH>(el + from * num_heads + h0);
        if (h0 == 0) put(e, from, place_of(e));
        grad(from, w[0], dot[0], x[0]);
      }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      ger[h] = lanes_sum<W>(ger[h]);
      if (there && part == 0) grad_er[d * num_heads + h0 + h] = Elem<T>::from_f(ger[h]);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
k_gat_source(const float* __restrict__ sums, int64_t n, uint32_t num_heads, T* __restrict__ grad_el) {
  wait_for_previous();
  constexpr int K = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += K * stride) {
    float v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t i = i0 + k * stride;
      const uint32_t row = (uint32_t)(i / num_heads), h = (uint32_t)(i - (int64_t)row * num_heads);
      v[k] = i < n ? sums[(int64_t)spread(row) * num_heads + h] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (i0 + k * stride < n) grad_el[i0 + k * stride] = Elem<T>::from_f(v[k]);
  }
}

// ---- host side ----------------------------------------------------------------------
static size_t elem_size(int dtype) { return dtype == APT_F32 ? 4 : 2; }

// What the forward leaves for the backward: the ranges and the weights.
struct GatEdges {
  Verdict none;     // [kVerdicts] words
  int2* range;      // [num_dst]
  float* weight;    // [E][heads]
};
constexpr size_t kGatFront = (kVerdicts * 4 + 255) / 256 * 256;
// The blocks of k_gat_ranges.
static int gat_range_blocks(int64_t E) { return (int)std::min<int64_t>(kVerdicts, ceil_div(E, 1024)); }
static size_t gat_edges_layout(int64_t num_dst, int64_t E, int H, char* base, GatEdges* g) {
  const size_t o_range = kGatFront;
  const size_t o_weight = o_range + align_up((size_t)(num_dst > 0 ? num_dst : 1) * 8, 256);
  if (g) {
    g->none = Verdict{(const uint32_t*)base, gat_range_blocks(E)};
    g->range = (int2*)(base + o_range);
    g->weight = (float*)(base + o_weight);
  }
  return o_weight + align_up((size_t)(E > 0 ? E : 1) * H * 4, 256);
}

struct GatBwdWs {
  float* sums;      // [spread_rows(num_src)][heads], cleared with the front of the sort
  SpmmWs sort;
  float* dots;      // [E][heads]
  size_t zero_bytes;
};
static size_t gat_bwd_layout(int64_t num_src, int64_t E, int H, char* base, GatBwdWs* ws) {
  // slots of 16 bytes where k_spmm_stream may take the sums behind the sort, whatever the rows' width (kByBoth)
  const int slot = E >= kStreamMinOrdered && H <= kStreamHeadsWide ? 16 : 8;
  const size_t o_sort = align_up((size_t)spread_rows(num_src > 0 ? num_src : 1) * H * 4, 256);
  const size_t o_dots = o_sort + spmm_layout(num_src, E, base + o_sort, ws ? &ws->sort : nullptr, slot);
  if (ws) {
    ws->sums = (float*)base;
    ws->dots = (float*)(base + o_dots);
    ws->zero_bytes = o_sort + ws->sort.zero_bytes;
  }
  return o_dots + align_up((size_t)(E > 0 ? E : 1) * H * 4, 256);
}

struct GatProblem {
  const int64_t* row;
  const int64_t* col;
  int64_t E;
  const void *ft, *el, *er, *grad_out;
  int H;
  int64_t Dh;
  float slope;
  int64_t num_dst;
  int32_t* status;
};

static int gat_check(const char* who, int dtype, int64_t num_edges, int num_heads, int64_t head_dim, int64_t num_dst) {
  APT_CHECK_ARG(dtype >= APT_F32 && dtype <= APT_F16, "%s: dtype %d", who, dtype);
  APT_CHECK_ARG(num_edges >= 0 && num_heads >= 1 && head_dim >= 1 && num_dst >= 0, "%s: bad sizes", who);
  APT_CHECK_ARG(num_edges < (int64_t)0x7fffffff && num_dst < (int64_t)0x7fffffff && head_dim < (1 << 28), "%s: sizes beyond 31 bits", who);
  return APT_OK;
}

static int gat_ranges(const GatProblem& q, const GatEdges& g, cudaStream_t s) {
  ProfScope prof("spmm_ranges", s);
  APT_FOLLOW(k_gat_ranges, gat_range_blocks(q.E), 256, 0, s, q.col, q.E, q.num_dst, g.range, (uint32_t*)g.none.word, q.status);
  return APT_OK;
}

// Lanes to a destination: as many as hold a mean one's edges. Heads at a time: as many as there are, if el can be read so; where that leaves
// several blocks of them these are worked on side by side. One after another, which waits for as many rounds of latency, against
// that, us: forward of bf16 16 x 16, 30 000 destinations of 0 to 30 edges 105 -> 83, backward of fp32 5 x 4 152 -> 118, 3 x 16 142 -> 131;
// 67 584 x 15 edges 143 -> 149, 215 -> 183, 228 -> 221.
#define APT_GAT_SIDE(W, NH, H, RUN)  \
  do {                               \
    if ((H) == (NH)) RUN(W, NH, false); \
    else RUN(W, NH, true);           \
  } while (0)
#define APT_GAT_LANES(q, RUN)                                                             \
  do {                                                                                    \
    const int lanes__ = pow2_ge(ceil_div(ceil_div(q.E, q.num_dst), kGatEdges)), nh__ = gat_heads(q, sizeof(T)); \
    if (lanes__ <= 4) {                                                                   \
      if (nh__ == 4) APT_GAT_SIDE(4, 4, q.H, RUN);                                        \
      else if (nh__ == 2) APT_GAT_SIDE(4, 2, q.H, RUN);                                   \
      else APT_GAT_SIDE(4, 1, q.H, RUN);                                                  \
    } else if (lanes__ <= 8) {                                                            \
      if (nh__ == 4) APT_GAT_SIDE(8, 4, q.H, RUN);                                        \
      else if (nh__ == 2) APT_GAT_SIDE(8, 2, q.H, RUN);                                   \
      else APT_GAT_SIDE(8, 1, q.H, RUN);                                                  \
    } else if (lanes__ <= 16) {                                                           \
      if (nh__ == 4) APT_GAT_SIDE(16, 4, q.H, RUN);                                       \
      else if (nh__ == 2) APT_GAT_SIDE(16, 2, q.H, RUN);                                  \
      else APT_GAT_SIDE(16, 1, q.H, RUN);                                                 \
    } else {                                                                              \
      if (nh__ == 4) APT_GAT_SIDE(32, 4, q.H, RUN);                                       \
      else if (nh__ == 2) APT_GAT_SIDE(32, 2, q.H, RUN);                                  \
      else APT_GAT_SIDE(32, 1, q.H, RUN);                                                 \
    }                                                                                     \
  } while (0);
static int gat_heads(const GatProblem& q, size_t esz) {
  for (int nh = 4; nh > 1; nh >>= 1)
    if (q.H % nh == 0 && (uintptr_t)q.el % (nh * esz) == 0) return nh;
  return 1;
}

// Ranges and attention weights.
template <typename T>
static int gat_weights(const GatProblem& q, const GatEdges& g, void* attn, cudaStream_t s) {
  const int rc = gat_ranges(q, g, s);
  if (rc != APT_OK) return rc;
  ProfScope prof("gat_rows", s);
  const int masked = masked_edges(q.H, q.Dh, sizeof(T), (uintptr_t)q.ft);
#define APT_WEIGHTS(W, NH, SIDE)                                                                                                   \
  APT_FOLLOW((k_gat_weights<T, W, NH, SIDE>), wave_grid(ceil_div(q.num_dst * (SIDE ? q.H / NH : 1) * W, 256), 8), 256, 0, s, q.row, (const T*)q.el, (const T*)q.er, \
             q.H, q.slope, q.num_dst, g.range, g.none, g.weight, (T*)attn, masked)
  APT_GAT_LANES(q, APT_WEIGHTS)
#undef APT_WEIGHTS
  return APT_OK;
}

// Rows of heads that are no whole slices, widened head by head (widen.cuh); without a buffer, or where that does not pay, `dim` is 0.
struct GatWide {
  void *ft, *grad;
  int64_t dim;      // of a head
};
// num_dst 0: the sources only.
static size_t gat_wide_layout(int dtype, int64_t E, int64_t num_src, int64_t num_dst, int H, int64_t Dh, char* base, GatWide* w) {
  const size_t esz = elem_size(dtype);
  if (!widen_gat_pays(Dh, H, esz, num_src, E, num_dst > 0)) return 0;
  const int64_t dim = widened_dim(Dh, esz);
  const size_t o_grad = align_up((size_t)num_src * H * dim * esz, 256);
  if (w) *w = GatWide{base, base + o_grad, dim};
  return o_grad + (size_t)num_dst * H * dim * esz;
}

template <typename T>
static int gat_forward(const GatProblem& q, const GatEdges& g, const GatWide& wide, int64_t num_src, void* out, void* attn, cudaStream_t s) {
  int rc = gat_weights<T>(q, g, attn, s);
  if (rc == APT_OK && wide.dim) rc = widen_rows(q.ft, num_src * q.H, q.Dh * sizeof(T), wide.ft, s);
  if (rc != APT_OK) return rc;
  const int64_t dim = q.H * (wide.dim ? wide.dim : q.Dh);
  // a slice stays inside a head, so that one weight serves it
  const int ve = wide.dim ? 16 / sizeof(T) : slice_elems((uint64_t)(q.Dh * sizeof(T)) | (uintptr_t)q.ft | (uintptr_t)out, sizeof(T));
  SpmmWs ws{};
  ws.range = g.range;
  const RowArgs<T> a{q.row, (const T*)(wide.dim ? wide.ft : q.ft), (const T*)g.weight, q.H, dim, SegTable{nullptr, nullptr, nullptr, 1}, q.num_dst,
                     q.E, ws, (T*)out, kRanges, 0, row_split(dim, ve, q.E, q.num_dst, false), (int)dim, g.none, q.status, q.col, nullptr, nullptr, 0u,
                     wide.dim ? q.H * q.Dh : 0};
  ProfScope prof("gat_rows", s);
  return launch_spmm_rows<T>(kUMulW, a, s);
}

template <typename T, int VE>
static int launch_dots(const GatProblem& q, const GatEdges& g, int64_t num_src, float* dots, const SpmmWs& sort, cudaStream_t s) {
  static int occupancy[64] = {};
  int per_sm = 0;
  const int rc = blocks_per_sm(k_gat_dots<T, VE>, 256, occupancy, &per_sm);
  if (rc != APT_OK) return rc;
  const int lph = pow2_ge(q.Dh / VE), hpp = pow2_ge(q.H, 32 / lph);
  const int64_t want = ceil_div(q.num_dst, 8), wave = (int64_t)kNumSMs * per_sm;
  APT_FOLLOW((k_gat_dots<T, VE>), (int)(want < wave ? want : wave), 256, 0, s, q.row, (const T*)q.ft, (const T*)q.grad_out, q.H,
             (int)q.Dh, q.num_dst, g.range, g.none, dots, lph, hpp, (uint32_t)num_src, sort.cnt, sort.rank);
  return APT_OK;
}

// Dots of the edges, whose source rows are counted on the way.
template <typename T>
static int gat_dots(const GatProblem& q, const GatEdges& g, const GatBwdWs& ws, int64_t num_src, cudaStream_t s) {
  const int64_t dim = q.H * q.Dh;
  const int slice = slice_elems((uint64_t)(q.Dh * sizeof(T)) | (uintptr_t)q.ft | (uintptr_t)q.grad_out, sizeof(T)) * (int)sizeof(T);
  if constexpr (sizeof(T) == 2)
    if (dots_mma_fits<T>(q.H, q.Dh, slice, q.E, q.num_dst))
      return launch_dots_mma<T>(q.H, q.Dh, q.row, q.col, (const T*)q.ft, (const T*)q.grad_out, q.E, q.num_dst, g.none, ws.dots, (uint32_t)num_src, ws.sort, s);
  if (stream_fits(kDots, slice, dim, sizeof(T), q.H, q.E, true)) {
    SpmmWs counts = ws.sort;
    counts.range = g.range;
    const RowArgs<T> a{q.row, (const T*)q.ft, nullptr, q.H, dim, SegTable{nullptr, nullptr, nullptr, 1}, q.num_dst, q.E, counts,
                       nullptr, kRanges, 0, RowSplit{}, 0, g.none, q.status, q.col, (const T*)q.grad_out, ws.dots, (uint32_t)num_src};
    return launch_spmm_rows<T>(kDots, a, s);
  }
  switch (slice) {
    case 16: return launch_dots<T, 16 / sizeof(T)>(q, g, num_src, ws.dots, ws.sort, s);
    case 8: return launch_dots<T, 8 / sizeof(T)>(q, g, num_src, ws.dots, ws.sort, s);
    case 4: return launch_dots<T, 4 / sizeof(T)>(q, g, num_src, ws.dots, ws.sort, s);
    default: return launch_dots<T, 1>(q, g, num_src, ws.dots, ws.sort, s);
  }
}

// The weights are there already.
template <typename T>
static int gat_backward(const GatProblem& as_given, const GatEdges& g, const GatWide& wide, const GatBwdWs& ws, char* workspace, int64_t num_src,
                        void* grad_ft, void* grad_el, void* grad_er, cudaStream_t s) {
  GatProblem q = as_given;
  if (wide.dim) q.ft = wide.ft, q.grad_out = wide.grad, q.Dh = wide.dim;
  const int64_t dim = q.H * q.Dh;
  const int ve = wide.dim ? 16 / sizeof(T) : slice_elems((uint64_t)(q.Dh * sizeof(T)) | (uintptr_t)q.grad_out | (uintptr_t)grad_ft, sizeof(T));
  const RowSplit split = row_split(dim, ve, q.E, num_src, true);
  const OrderKind kind = order_kind(kUMulW, ve * (int)sizeof(T), dim, sizeof(T), q.H, q.E);
  APT_CUDA(cudaMemsetAsync(workspace, 0, ws.zero_bytes, s));
  int rc;
  if (wide.dim) {
    ProfScope prof("gat_widen", s);
    rc = widen_rows(as_given.ft, num_src * q.H, as_given.Dh * sizeof(T), wide.ft, s);
    if (rc == APT_OK) rc = widen_rows(as_given.grad_out, q.num_dst * q.H, as_given.Dh * sizeof(T), wide.grad, s);
    if (rc != APT_OK) return rc;
  }
  {
    ProfScope prof("gat_bwd_rows", s);
    rc = gat_dots<T>(q, g, ws, num_src, s);
    if (rc == APT_OK) rc = launch_slots(num_src, ws.sort, kOrder, kind, split.long_edges, (int)dim, s);
    if (rc != APT_OK) return rc;
#define APT_SCORES(W, NH, SIDE)                                                                                                    \
  APT_FOLLOW((k_gat_scores<T, W, NH, SIDE>), wave_grid(ceil_div(q.num_dst * (SIDE ? q.H / NH : 1) * W, 256), 8), 256, 0, s, q.row, (const T*)q.el, (const T*)q.er, \
             q.H, q.slope, num_src, q.num_dst, q.E, g.range, g.none, g.weight, ws.dots, ws.sums, ws.sort, kind, (T*)grad_er)
    APT_GAT_LANES(q, APT_SCORES)
#undef APT_SCORES
  }
  const RowArgs<T> a{nullptr, (const T*)q.grad_out, (const T*)g.weight, q.H, dim, SegTable{nullptr, nullptr, nullptr, 1}, num_src, q.E, ws.sort,
                     (T*)grad_ft, kOrder, 0, split, (int)dim, Verdict{}, q.status, nullptr, nullptr, nullptr, 0u, wide.dim ? q.H * as_given.Dh : 0};
  {
    ProfScope prof("spmm_rows", s);
    rc = launch_spmm_rows<T>(kUMulW, a, s);
  }
  if (rc != APT_OK) return rc;
  APT_FOLLOW(k_gat_source<T>, wave_grid(ceil_div(num_src * q.H, 1024), 8, 1), 256, 0, s, ws.sums, num_src * q.H, (uint32_t)q.H, (T*)grad_el);
  return APT_OK;
}

// ---- without a buffer for weights -----------------------------------------------------
// apt_gat_edge_softmax_sum and apt_gat_edge_backward have a few words a destination of workspace and allocate nothing: a warp
// to a destination keeps the weights of 32 edges and 4 heads in shared memory and works them out again for further edges
// and column blocks. They are for callers that do not hold E x heads fp32 values: 67 584 x 15 edges, bf16, 4 x 64, take 144 us
// forward and 203 for the edge part of the backward, with such a buffer 114 and 164. Three blocks an SM for the backward (four:
// 216, spills), four for the forward (three: 154); eight heads at a time 151 and 233.
constexpr int kAloneHeads = 4;

// The weights of one destination's edges, for the heads from h0 on, a lane to an edge. What outlives a step is in shared memory:
// as registers it took half the warps.
struct GatAloneWarp {
  float w[32][kAloneHeads];                                  // of the edges of the current chunk
  float bias[kAloneHeads], most[kAloneHeads], inv[kAloneHeads];      // needed again with more than 32 edges
};
template <typename T>
struct GatScores {
  GatAloneWarp& sh;
  const int64_t* row;
  const T* el;
  int H, h0, nh;
  float slope;
  int masked;
  bool few;
  unsigned positive;       // bit h: this lane's score before the leaky part

  __device__ __forceinline__ float score(int64_t src, int h, float bias) const { return Elem<T>::to_f(el[src * H + h0 + h]) + bias; }
  __device__ __forceinline__ void start(const T* er, int d, int2 r, int lane) {
    const uint32_t deg = r.y - r.x;
    few = deg <= 32;
    positive = 0u;
    const bool mine = few && lane < (int)deg;
    const int64_t src = mine ? row[r.x + lane] : 0;
    float bias[kAloneHeads], x[kAloneHeads];
#pragma unroll
    for (int h = 0; h < kAloneHeads; ++h) {
      if (h >= nh) break;
      bias[h] = Elem<T>::to_f(er[(int64_t)d * H + h0 + h]);
      x[h] = mine ? score(src, h, bias[h]) : -INFINITY;
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kAloneHeads; ++h) {
      if (h >= nh) break;
      float most = mine ? leaky(x[h], slope) : -INFINITY, sum = 0.f;
      if (!few)
        for (uint32_t k = lane; k < deg; k += 32) most = fmaxf(most, leaky(score(row[r.x + k], h, bias[h]), slope));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
      if (mine) sum = expf(leaky(x[h], slope) - most);
      if (!few)
        for (uint32_t k = lane; k < deg; k += 32) sum += expf(leaky(score(row[r.x + k], h, bias[h]), slope) - most);
      const float own = sum;
      sum = group_sum(sum, 32);
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
      if (mine) sh.w[lane][h] = !(sum > 0.f) && (int)deg <= masked ? 0.f : own * inv;
      if (mine && x[h] > 0.f) positive |= 1u << h;
      if (!few && lane == 0) sh.bias[h] = bias[h], sh.most[h] = most, sh.inv[h] = inv;
    }
    __syncwarp();
  }
  // The weights of a chunk of edges.
  __device__ __forceinline__ void chunk(int64_t src, bool mine, int lane) {
    if (few) return;
    __syncwarp();
    positive = 0u;
#pragma unroll
    for (int h = 0; h < kAloneHeads; ++h) {
      if (h >= nh || !mine) break;
      const float x = score(src, h, sh.bias[h]);
      sh.w[lane][h] = expf(leaky(x, slope) - sh.most[h]) * sh.inv[h];
      if (x > 0.f) positive |= 1u << h;
    }
    __syncwarp();
  }
};

template <typename T, int VE>
__global__ void __launch_bounds__(256, 4)
k_gat_alone(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el, const T* __restrict__ er, int num_heads,
            int head_dim, float slope, int64_t num_dst, const int2* __restrict__ range, const Verdict none,
            T* __restrict__ out, T* __restrict__ attn, int lpe, int masked) {
  wait_for_previous();
  constexpr int U = 4;
  __shared__ GatAloneWarp shared[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & (lpe - 1), epi = lane / lpe, ep = 32 / lpe;
  const int nvh = head_dim / VE;
  const int64_t dim = (int64_t)num_heads * head_dim;
  const uint32_t row_bytes = (uint32_t)(dim * sizeof(T));
  const bool empty = any_found(none);
  for (int64_t d = (int64_t)blockIdx.x * 8 + warp; d < num_dst; d += (int64_t)gridDim.x * 8) {
    const int2 r = empty ? make_int2(0, 0) : range[d];
    const int deg = r.y - r.x;
    for (int h0 = 0; h0 < num_heads; h0 += kAloneHeads) {
      GatScores<T> sc{shared[warp], row, el, num_heads, h0, min(kAloneHeads, num_heads - h0), slope, masked};
      if (deg > 0) sc.start(er, (int)d, r, lane);
      const int slices = sc.nh * nvh;
      for (int c0 = 0; c0 < slices; c0 += lpe) {
        const int c = c0 + sub, h = c < slices ? c / nvh : 0;
        const int64_t col = (int64_t)h0 * head_dim + (int64_t)c * VE;
        const T* const lane_ft = ft + col;
        Acc<VE> acc;
        acc.zero();
        for (int rest = deg; rest > 0; rest -= 32) {
          const int base = r.y - rest, cnt = min(32, rest);
          const uint32_t src = lane < cnt ? (uint32_t)row[base + lane] : 0u;
          if (c0 == 0 || deg > 32) {
            sc.chunk(src, lane < cnt, lane);
            if (attn && c0 == 0 && lane < cnt)
              for (int k = 0; k < sc.nh; ++k) attn[(int64_t)(base + lane) * num_heads + h0 + k] = Elem<T>::from_f(sc.sh.w[lane][k]);
          }
          for (int j0 = epi; j0 - epi < cnt; j0 += ep * U) {
            Raw<T, VE> v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const uint32_t from = __shfl_sync(0xffffffffu, src, (j0 + u * ep) & 31);
              if (j0 + u * ep < cnt && c < slices) v[u] = load_raw<T, VE>(at_row(lane_ft, from, row_bytes));
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (j0 + u * ep < cnt && c < slices) acc.fma(v[u], sc.sh.w[j0 + u * ep][h]);
          }
        }
        for (int o = lpe; o < 32; o <<= 1) acc.join(0xffffffffu, o);
        if (epi == 0 && c < slices) store_pack<T, VE>(out + d * dim + col, acc.template rounded<T>());
      }
      __syncwarp();
    }
  }
}

// Narrow rows (up to APT_GAT_NARROW_BYTES in 16-byte slices), forward: a lane to a slice, as many lanes to a destination, and every lane works
// its head's scores out itself. There are few lanes to share them, and what it saves is the weights' way through memory and a
// launch. 30 000 destinations of 3 / 10 / 25 edges, with the weights apart -> here, us: fp32 x 32 16 / 33 / 47 -> 12 / 18 / 33,
// bf16 8 x 8 22 / 37 / 59 -> 12 / 20 / 37, fp32 4 x 16 23 / 36 / 57 -> 16 / 27 / 49. Wider rows and other slices gain by the weights
// apart, against one such kernel: bf16 4 x 64 35 / 45 / 67 -> 27 / 37 / 72, fp16 2 x 10 27 / 41 / 79 -> 18 / 27 / 45.
// (For fp32 the compiler takes 40 registers when left alone and has fewer loads in flight; five blocks an SM keep it at 48: 8 x 8, 30 000
// destinations of 0 to 30 edges 51 -> 45 us, 1 x 32 36.4 -> 31.7, one of 20 000 edges 10.0 -> 7.5 ms. 16-bit types have 47 registers either way, but
// lose by the bound: bf16 1 x 16 20.4 -> 23.9, 12 x 8 50.6 -> 54.2.)
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 5 : 0)
k_gat_narrow(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el, const T* __restrict__ er, int num_heads,
             int head_dim, float slope, int64_t num_dst, const int2* __restrict__ range, const Verdict none,
             T* __restrict__ out, T* __restrict__ attn, int lpe) {
  wait_for_previous();
  constexpr int VE = 16 / sizeof(T);
  const bool empty = any_found(none);
  const int c = threadIdx.x & (lpe - 1), dim = num_heads * head_dim;
  if (c * VE >= dim) return;
  const int h = c * VE / head_dim;
  const uint32_t row_bytes = (uint32_t)(dim * sizeof(T));
  const bool writes_attn = attn && c * VE % head_dim == 0;
  const T* const lane_ft = ft + c * VE;
  const T* const lane_el = el + h;
  const int per_block = 256 / lpe;
  for (int64_t d = (int64_t)blockIdx.x * per_block + threadIdx.x / lpe; d < num_dst; d += (int64_t)gridDim.x * per_block) {
    const int2 r = empty ? make_int2(0, 0) : range[d];
    const float bias = Elem<T>::to_f(er[d * num_heads + h]);
    auto score = [&](int64_t src) { return leaky(Elem<T>::to_f(lane_el[src * num_heads]) + bias, slope); };
    float most = -INFINITY, sum = 0.f;
#pragma unroll 4
    for (int e = r.x; e < r.y; ++e) most = fmaxf(most, score(row[e]));
#pragma unroll 4
    for (int e = r.x; e < r.y; ++e) sum += expf(score(row[e]) - most);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    Acc<VE> acc;
    acc.zero();
#pragma unroll 4
    for (int e = r.x; e < r.y; ++e) {
      const int64_t src = row[e];
      const Raw<T, VE> v = load_raw<T, VE>(at_row(lane_ft, (uint32_t)src, row_bytes));
      const float w = expf(score(src) - most) * inv;
      if (writes_attn) attn[(int64_t)e * num_heads + h] = Elem<T>::from_f(w);
      acc.fma(v, w);
    }
    store_pack<T, VE>(out + d * dim + c * VE, acc.template rounded<T>());
  }
}

template <typename T, int VE>
__global__ void __launch_bounds__(256, 3)
k_gat_alone_backward(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el, const T* __restrict__ er,
                     const T* __restrict__ grad_out, int num_heads, int head_dim, float slope, int64_t num_dst, int64_t E,
                     const int2* __restrict__ range, const Verdict none, T* __restrict__ attn,
                     T* __restrict__ grad_score, T* __restrict__ grad_er, int lph, int hpp, int masked) {
  wait_for_previous();
  constexpr int U = 4;
  __shared__ GatAloneWarp shared[8];
  __shared__ float dot_sh[8][32][kAloneHeads];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = lane & (lph - 1), rh = (lane & (lph * hpp - 1)) / lph, epi = lane / (lph * hpp), ep = 32 / (lph * hpp);
  const int nvh = head_dim / VE;
  const int64_t dim = (int64_t)num_heads * head_dim;
  const uint32_t row_bytes = (uint32_t)(dim * sizeof(T));
  const bool empty = any_found(none);
  if (empty)   // no edge belongs to anybody
    for (int64_t o = (int64_t)blockIdx.x * 256 + threadIdx.x; o < E * num_heads; o += (int64_t)gridDim.x * 256)
      attn[o] = grad_score[o] = Elem<T>::from_f(0.f);
  for (int64_t d = (int64_t)blockIdx.x * 8 + warp; d < num_dst; d += (int64_t)gridDim.x * 8) {
    const int2 r = empty ? make_int2(0, 0) : range[d];
    const int deg = r.y - r.x;
    for (int h0 = 0; h0 < num_heads; h0 += kAloneHeads) {
      GatScores<T> sc{shared[warp], row, el, num_heads, h0, min(kAloneHeads, num_heads - h0), slope, masked};
      if (deg > 0) sc.start(er, (int)d, r, lane);
      float t[kAloneHeads], ger[kAloneHeads];
#pragma unroll
      for (int k = 0; k < kAloneHeads; ++k) t[k] = ger[k] = 0.f;
      // up to 32 edges: t first, then the results, from the same dots; more: two walks
      const int passes = deg > 32 ? 2 : 1;
      for (int pass = 0; pass < passes; ++pass) {
        for (int rest = deg; rest > 0; rest -= 32) {
          const int base = r.y - rest, cnt = min(32, rest);
          const uint32_t src = lane < cnt ? (uint32_t)row[base + lane] : 0u;
          __syncwarp();
          for (int hb = 0; hb < sc.nh; hb += hpp) {
            const int h = hb + rh;
            const T *const g_head = grad_out + d * dim + (int64_t)(h0 + h) * head_dim, *const ft_head = ft + (int64_t)(h0 + h) * head_dim;
            for (int j0 = epi; j0 - epi < cnt; j0 += ep * U) {
              uint32_t from[U];
              float dot[U];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                from[u] = __shfl_sync(0xffffffffu, src, (j0 + u * ep) & 31);
                dot[u] = 0.f;
              }
              if (h < sc.nh)
                for (int c = p; c < nvh; c += lph) {
                  const Raw<T, VE> g = load_raw<T, VE>(g_head + c * VE);
                  Raw<T, VE> v[U];
#pragma unroll
                  for (int u = 0; u < U; ++u)
                    if (j0 + u * ep < cnt) v[u] = load_raw<T, VE>(at_row(ft_head + c * VE, from[u], row_bytes));
#pragma unroll
                  for (int u = 0; u < U; ++u) {
                    if (j0 + u * ep >= cnt) break;
#pragma unroll
                    for (int q = 0; q < VE; ++q) dot[u] = fmaf(g.get(q), v[u].get(q), dot[u]);
                  }
                }
              if (lph >= 4) {      // each step halves the edges a lane sums for (k_gat_dots)
                const bool hi = p & (lph >> 1), lo = p & (lph >> 2);
                const float b0 = (hi ? dot[2] : dot[0]) + __shfl_xor_sync(0xffffffffu, hi ? dot[0] : dot[2], lph >> 1);
                const float b1 = (hi ? dot[3] : dot[1]) + __shfl_xor_sync(0xffffffffu, hi ? dot[1] : dot[3], lph >> 1);
                const float v = group_sum((lo ? b1 : b0) + __shfl_xor_sync(0xffffffffu, lo ? b0 : b1, lph >> 2), lph >> 2);
                const int j = j0 + ((hi ? 2 : 0) + (lo ? 1 : 0)) * ep;
                if ((p & ((lph >> 2) - 1)) == 0 && j < cnt && h < sc.nh) dot_sh[warp][j][h] = v;
              } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                  dot[u] = group_sum(dot[u], lph);
                  if (p == 0 && j0 + u * ep < cnt && h < sc.nh) dot_sh[warp][j0 + u * ep][h] = dot[u];
                }
              }
            }
          }
          sc.chunk(src, lane < cnt, lane);
          __syncwarp();
#pragma unroll
          for (int k = 0; k < kAloneHeads; ++k) {
            if (k >= sc.nh) break;
            const float w = lane < cnt ? sc.sh.w[lane][k] : 0.f, dot = lane < cnt ? dot_sh[warp][lane][k] : 0.f;
            if (pass == 0) t[k] += group_sum(lane < cnt ? w * dot : 0.f, 32);
            if (pass < passes - 1) continue;
            const float gs = w * (dot - t[k]) * (sc.positive >> k & 1u ? 1.f : slope);
            if (lane < cnt) {
              attn[(int64_t)(base + lane) * num_heads + h0 + k] = Elem<T>::from_f(w);
              grad_score[(int64_t)(base + lane) * num_heads + h0 + k] = Elem<T>::from_f(gs);
            }
            ger[k] += group_sum(lane < cnt ? gs : 0.f, 32);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kAloneHeads; ++k)
        if (k < sc.nh && lane == 0) grad_er[d * num_heads + h0 + k] = Elem<T>::from_f(ger[k]);
    }
  }
}

template <typename T, int VE>
static int launch_alone(const GatProblem& q, const GatEdges& g, void* out, void* attn, void* grad_score, void* grad_er, cudaStream_t s) {
  const int nvh = (int)(q.Dh / VE), grid = wave_grid(ceil_div(q.num_dst, 8), 8);
  const int masked = masked_edges(q.H, q.Dh, sizeof(T), (uintptr_t)q.ft);
  if (grad_er) {
    const int lph = pow2_ge(nvh), hpp = pow2_ge(std::min(q.H, kAloneHeads), 32 / lph);
    APT_FOLLOW((k_gat_alone_backward<T, VE>), grid, 256, 0, s, q.row, (const T*)q.ft, (const T*)q.el, (const T*)q.er,
               (const T*)q.grad_out, q.H, (int)q.Dh, q.slope, q.num_dst, q.E, g.range, g.none, (T*)attn, (T*)grad_score, (T*)grad_er,
               lph, hpp, masked);
  } else if (VE * sizeof(T) == 16 && q.H * q.Dh * (int64_t)sizeof(T) <= APT_GAT_NARROW_BYTES) {
    const int lpe = pow2_ge(q.H * nvh);
    APT_FOLLOW((k_gat_narrow<T>), wave_grid(ceil_div(q.num_dst, 256 / lpe), 8), 256, 0, s, q.row, (const T*)q.ft, (const T*)q.el,
               (const T*)q.er, q.H, (int)q.Dh, q.slope, q.num_dst, g.range, g.none, (T*)out, (T*)attn, lpe);
  } else {
    APT_FOLLOW((k_gat_alone<T, VE>), grid, 256, 0, s, q.row, (const T*)q.ft, (const T*)q.el, (const T*)q.er, q.H, (int)q.Dh, q.slope,
               q.num_dst, g.range, g.none, (T*)out, (T*)attn, pow2_ge((int64_t)std::min(q.H, kAloneHeads) * nvh), masked);
  }
  return APT_OK;
}

// The ranges are in the front of a workspace of apt_spmm_workspace_bytes(num_dst, 0) bytes. Backward with grad_er, else forward.
template <typename T>
static int gat_alone(const GatProblem& q, void* workspace, void* out, void* attn, void* grad_score, void* grad_er, cudaStream_t s) {
  const GatEdges g{Verdict{(const uint32_t*)workspace, gat_range_blocks(q.E)}, (int2*)((char*)workspace + kGatFront), nullptr};
  const int rc = gat_ranges(q, g, s);
  if (rc != APT_OK) return rc;
  ProfScope prof(grad_er ? "gat_bwd_rows" : "gat_rows", s);
  const uintptr_t other = (uintptr_t)(grad_er ? q.grad_out : out);
  switch (slice_elems((uint64_t)(q.Dh * sizeof(T)) | (uintptr_t)q.ft | other, sizeof(T)) * (int)sizeof(T)) {
    case 16: return launch_alone<T, 16 / sizeof(T)>(q, g, out, attn, grad_score, grad_er, s);
    case 8: return launch_alone<T, 8 / sizeof(T)>(q, g, out, attn, grad_score, grad_er, s);
    case 4: return launch_alone<T, 4 / sizeof(T)>(q, g, out, attn, grad_score, grad_er, s);
    default: return launch_alone<T, 1>(q, g, out, attn, grad_score, grad_er, s);
  }
}

static int gat_alone(const char* who, int dtype, const GatProblem& q, void* workspace, size_t workspace_bytes, void* out, void* attn,
                     void* grad_score, void* grad_er, cudaStream_t s) {
  APT_CHECK_ARG(((uintptr_t)workspace & 255) == 0, "%s: workspace must be 256-byte aligned", who);
  const size_t need = spmm_layout(q.num_dst, 0, nullptr, nullptr);
  if (workspace_bytes < need) {
    set_error("%s: workspace %zu < %zu bytes", who, workspace_bytes, need);
    return APT_ERR_CAPACITY;
  }
  switch (dtype) {
    case APT_F32: return gat_alone<float>(q, workspace, out, attn, grad_score, grad_er, s);
    case APT_BF16: return gat_alone<__nv_bfloat16>(q, workspace, out, attn, grad_score, grad_er, s);
    default: return gat_alone<__half>(q, workspace, out, attn, grad_score, grad_er, s);
  }
}

}  // namespace apt

extern "C" size_t apt_gat_edges_bytes(int64_t num_dst, int64_t num_edges, int num_heads) {
  if (num_dst < 0 || num_edges < 0 || num_heads < 1) return 0;
  return apt::gat_edges_layout(num_dst, num_edges, num_heads, nullptr, nullptr);
}

extern "C" size_t apt_gat_widened_bytes(int dtype, int64_t num_edges, int64_t num_src, int64_t num_dst, int num_heads, int64_t head_dim) {
  using namespace apt;
  if (dtype < APT_F32 || dtype > APT_F16 || num_edges < 0 || num_src < 0 || num_dst < 0 || num_heads < 1 || head_dim < 1) return 0;
  return gat_wide_layout(dtype, num_edges, num_src, num_dst, num_heads, head_dim, nullptr, nullptr);
}

// The buffer of widened rows as the caller gives it, or none.
static int gat_wide(const char* who, int dtype, int64_t E, int64_t num_src, int64_t num_dst, int H, int64_t Dh, void* widened, size_t bytes,
                    apt::GatWide* w) {
  using namespace apt;
  *w = GatWide{};
  if (!widened) return APT_OK;
  APT_CHECK_ARG(((uintptr_t)widened & 255) == 0, "%s: the buffer of widened rows must be 256-byte aligned", who);
  const size_t need = gat_wide_layout(dtype, E, num_src, num_dst, H, Dh, (char*)widened, w);
  if (bytes < need) {
    set_error("%s: %zu < %zu bytes for widened rows", who, bytes, need);
    return APT_ERR_CAPACITY;
  }
  return APT_OK;
}

extern "C" int apt_gat_forward(int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t num_edges, const void* ft,
                               const void* el, const void* er, int num_heads, int64_t head_dim, float negative_slope,
                               int64_t num_dst, void* out, void* out_attn, void* edges, size_t edges_bytes,
                               int32_t* status_word, void* stream) {
  return apt_gat_forward_widened(dtype, coo_row, coo_col, num_edges, ft, el, er, num_heads, head_dim, negative_slope, 0, num_dst, out, out_attn,
                                 edges, edges_bytes, nullptr, 0, status_word, stream);
}

extern "C" int apt_gat_forward_widened(int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t num_edges, const void* ft,
                                       const void* el, const void* er, int num_heads, int64_t head_dim, float negative_slope,
                                       int64_t num_src, int64_t num_dst, void* out, void* out_attn, void* edges, size_t edges_bytes,
                                       void* widened, size_t widened_bytes, int32_t* status_word, void* stream) {
  using namespace apt;
  int rc = gat_check("apt_gat_forward", dtype, num_edges, num_heads, head_dim, num_dst);
  if (rc != APT_OK || num_dst == 0) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  APT_CHECK_ARG(out && status_word, "apt_gat_forward: null output");
  if (num_edges == 0) {
    APT_CUDA(cudaMemsetAsync(out, 0, (size_t)num_dst * num_heads * head_dim * elem_size(dtype), s));
    return APT_OK;
  }
  APT_CHECK_ARG(coo_row && coo_col && ft && el && er && edges, "apt_gat_forward: null pointer");
  APT_CHECK_ARG(((uintptr_t)edges & 255) == 0, "apt_gat_forward: the edge buffer must be 256-byte aligned");
  GatEdges g;
  const size_t need = gat_edges_layout(num_dst, num_edges, num_heads, (char*)edges, &g);
  if (edges_bytes < need) {
    set_error("apt_gat_forward: edge buffer %zu < %zu bytes", edges_bytes, need);
    return APT_ERR_CAPACITY;
  }
  GatWide wide;
  rc = gat_wide("apt_gat_forward", dtype, num_edges, num_src, 0, num_heads, head_dim, widened, widened_bytes, &wide);
  if (rc != APT_OK) return rc;
  const GatProblem q{coo_row, coo_col, num_edges, ft, el, er, nullptr, num_heads, head_dim, negative_slope, num_dst, status_word};
  switch (dtype) {
    case APT_F32: return gat_forward<float>(q, g, wide, num_src, out, out_attn, s);
    case APT_BF16: return gat_forward<__nv_bfloat16>(q, g, wide, num_src, out, out_attn, s);
    default: return gat_forward<__half>(q, g, wide, num_src, out, out_attn, s);
  }
}

extern "C" size_t apt_gat_backward_workspace_bytes(int64_t num_src, int64_t num_edges, int num_heads) {
  if (num_src < 0 || num_edges < 0 || num_heads < 1) return 0;
  return apt::gat_bwd_layout(num_src, num_edges, num_heads, nullptr, nullptr);
}

extern "C" int apt_gat_backward(int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t num_edges,
                                const void* ft, const void* el, const void* er, const void* grad_out, int num_heads,
                                int64_t head_dim, float negative_slope, int64_t num_src, int64_t num_dst, void* grad_ft,
                                void* grad_el, void* grad_er, void* edges, size_t edges_bytes, int edges_valid,
                                void* workspace, size_t workspace_bytes, int32_t* status_word, void* stream) {
  return apt_gat_backward_widened(dtype, coo_row, coo_col, num_edges, ft, el, er, grad_out, num_heads, head_dim, negative_slope, num_src,
                                  num_dst, grad_ft, grad_el, grad_er, edges, edges_bytes, edges_valid, workspace, workspace_bytes, nullptr, 0,
                                  status_word, stream);
}

extern "C" int apt_gat_backward_widened(int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t num_edges,
                                        const void* ft, const void* el, const void* er, const void* grad_out, int num_heads,
                                        int64_t head_dim, float negative_slope, int64_t num_src, int64_t num_dst, void* grad_ft,
                                        void* grad_el, void* grad_er, void* edges, size_t edges_bytes, int edges_valid,
                                        void* workspace, size_t workspace_bytes, void* widened, size_t widened_bytes,
                                        int32_t* status_word, void* stream) {
  using namespace apt;
  int rc = gat_check("apt_gat_backward", dtype, num_edges, num_heads, head_dim, num_dst);
  if (rc != APT_OK) return rc;
  APT_CHECK_ARG(num_src >= 0 && num_src < (int64_t)0x7fffffff, "apt_gat_backward: bad num_src");
  cudaStream_t s = (cudaStream_t)stream;
  const size_t esz = elem_size(dtype);
  const int64_t dim = (int64_t)num_heads * head_dim;
  APT_CHECK_ARG((num_src == 0 || (grad_ft && grad_el)) && (num_dst == 0 || grad_er) && status_word, "apt_gat_backward: null output");
  if (num_edges == 0 || num_src == 0 || num_dst == 0) {
    if (num_src > 0) {
      APT_CUDA(cudaMemsetAsync(grad_ft, 0, (size_t)num_src * dim * esz, s));
      APT_CUDA(cudaMemsetAsync(grad_el, 0, (size_t)num_src * num_heads * esz, s));
    }
    if (num_dst > 0) APT_CUDA(cudaMemsetAsync(grad_er, 0, (size_t)num_dst * num_heads * esz, s));
    return APT_OK;
  }
  APT_CHECK_ARG(coo_row && coo_col && ft && el && er && grad_out && edges && workspace, "apt_gat_backward: null pointer");
  APT_CHECK_ARG((((uintptr_t)workspace | (uintptr_t)edges) & 255) == 0, "apt_gat_backward: buffers must be 256-byte aligned");
  GatEdges g;
  GatBwdWs ws;
  const size_t need_e = gat_edges_layout(num_dst, num_edges, num_heads, (char*)edges, &g);
  const size_t need_w = gat_bwd_layout(num_src, num_edges, num_heads, (char*)workspace, &ws);
  if (edges_bytes < need_e || workspace_bytes < need_w) {
    set_error("apt_gat_backward: buffers of %zu and %zu bytes, %zu and %zu needed", edges_bytes, workspace_bytes, need_e, need_w);
    return APT_ERR_CAPACITY;
  }
  GatWide wide;
  rc = gat_wide("apt_gat_backward", dtype, num_edges, num_src, num_dst, num_heads, head_dim, widened, widened_bytes, &wide);
  if (rc != APT_OK) return rc;
  const GatProblem q{coo_row, coo_col, num_edges, ft, el, er, grad_out, num_heads, head_dim, negative_slope, num_dst, status_word};
#define APT_RUN(T)                                                                                          \
  do {                                                                                                      \
    if (!edges_valid && (rc = gat_weights<T>(q, g, nullptr, s)) != APT_OK) return rc;                       \
    return gat_backward<T>(q, g, wide, ws, (char*)workspace, num_src, grad_ft, grad_el, grad_er, s);              \
  } while (0)
  switch (dtype) {
    case APT_F32: APT_RUN(float);
    case APT_BF16: APT_RUN(__nv_bfloat16);
    default: APT_RUN(__half);
  }
#undef APT_RUN
}

extern "C" int apt_gat_edge_softmax_sum(int dtype, const int64_t* coo_row, const int64_t* coo_col,
                                        int64_t num_edges, const void* ft, const void* el, const void* er,
                                        int num_heads, int64_t head_dim, float negative_slope,
                                        int64_t num_dst, void* out, void* out_attn, void* workspace,
                                        size_t workspace_bytes, int32_t* status_word, void* stream) {
  using namespace apt;
  const int rc = gat_check("apt_gat_edge_softmax_sum", dtype, num_edges, num_heads, head_dim, num_dst);
  if (rc != APT_OK || num_dst == 0) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  APT_CHECK_ARG(out && status_word, "apt_gat_edge_softmax_sum: null output");
  if (num_edges == 0) {
    APT_CUDA(cudaMemsetAsync(out, 0, (size_t)num_dst * num_heads * head_dim * elem_size(dtype), s));
    return APT_OK;
  }
  APT_CHECK_ARG(coo_row && coo_col && ft && el && er && workspace, "apt_gat_edge_softmax_sum: null pointer");
  const GatProblem q{coo_row, coo_col, num_edges, ft, el, er, nullptr, num_heads, head_dim, negative_slope, num_dst, status_word};
  return gat_alone("apt_gat_edge_softmax_sum", dtype, q, workspace, workspace_bytes, out, out_attn, nullptr, nullptr, s);
}

extern "C" int apt_gat_edge_backward(int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t num_edges,
                                     const void* ft, const void* el, const void* er, const void* grad_out,
                                     int num_heads, int64_t head_dim, float negative_slope, int64_t num_dst,
                                     void* out_attn, void* out_grad_score, void* out_grad_er, void* workspace,
                                     size_t workspace_bytes, int32_t* status_word, void* stream) {
  using namespace apt;
  const int rc = gat_check("apt_gat_edge_backward", dtype, num_edges, num_heads, head_dim, num_dst);
  if (rc != APT_OK || num_dst == 0) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  APT_CHECK_ARG(out_grad_er && status_word, "apt_gat_edge_backward: null output");
  if (num_edges == 0) {
    APT_CUDA(cudaMemsetAsync(out_grad_er, 0, (size_t)num_dst * num_heads * elem_size(dtype), s));
    return APT_OK;
  }
  APT_CHECK_ARG(coo_row && coo_col && ft && el && er && grad_out && out_attn && out_grad_score && workspace,
                "apt_gat_edge_backward: null pointer");
  const GatProblem q{coo_row, coo_col, num_edges, ft, el, er, grad_out, num_heads, head_dim, negative_slope, num_dst, status_word};
  return gat_alone("apt_gat_edge_backward", dtype, q, workspace, workspace_bytes, nullptr, out_attn, out_grad_score, out_grad_er, s);
}
