// Fused GAT edge pipeline over one sampled block: forward and the edge part of the backward.
#include <math.h>

#include "spmm_rows.cuh"

namespace apt {

struct GatWs {
  int32_t* range;   // [num_dst + 1] first edge of every destination
  int32_t* flags;   // [1] 1 when the edges are not grouped by destination
};

static bool gat_layout(int64_t num_dst, char* base, size_t bytes, GatWs* ws) {
  SpmmWs w;
  if (bytes < spmm_layout(num_dst, 0, base, &w)) return false;
  ws->range = (int32_t*)w.range;
  ws->flags = w.num_items;
  return true;
}

__global__ void __launch_bounds__(256)
k_edge_ranges_single(const int64_t* __restrict__ col, int64_t E, int64_t num_out_rows, GatWs ws) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  bool bad = false;
  for (; e < E; e += stride) {
    const int64_t d = col[e];
    const int64_t prev = e > 0 ? col[e - 1] : (int64_t)-1;
    if (d < prev || d < 0 || d >= num_out_rows) {
      bad = true;
      continue;
    }
    for (int64_t t = prev + 1; t <= d; ++t) ws.range[t] = (int32_t)e;
    if (e == E - 1)
      for (int64_t t = d + 1; t <= num_out_rows; ++t) ws.range[t] = (int32_t)E;
  }
  if (bad) atomicOr(ws.flags, 1);
}

// ---- fused GAT edge pipeline ---------------------------------------------------------
// For every destination row d with its edges e (src_e -> d) and every head h:
//   s_e = leaky_relu(el[src_e, h] + er[d, h]);  a_e = softmax over the edges of d;
//   out[d, h, :] = sum_e a_e * ft[src_e, h, :]
// which is u_add_v -> leaky_relu -> edge_softmax -> u_mul_e + sum in one pass
// over a grouped block (python/npc/model/gatconv.py:113-124). One lane group per
// destination row as in k_spmm_rows; scores are recomputed per lane (a block has
// at most a few dozen edges per row), sums stay in fp32 registers.
template <typename T, int VE>
__global__ void __launch_bounds__(256)
k_gat_rows(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el,
           const T* __restrict__ er, int num_heads, int64_t head_dim, float slope,
           int64_t num_dst, GatWs ws, T* __restrict__ out, T* __restrict__ attn,
           int group, int32_t* status) {
  const bool unsorted = *ws.flags != 0;
  if (unsorted && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(status, APT_FLAG_NOT_GROUPED);
  const int sub = threadIdx.x % group;
  const int64_t rows_per_block = blockDim.x / group;
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  const int64_t nvec = feat_dim / VE;
  int64_t d = (int64_t)blockIdx.x * rows_per_block + threadIdx.x / group;
  const int64_t stride = (int64_t)gridDim.x * rows_per_block;
  for (; d < num_dst; d += stride) {
    const int64_t e0 = unsorted ? 0 : ws.range[d];
    const int64_t e1 = unsorted ? 0 : ws.range[d + 1];
    for (int64_t c = sub; c < nvec; c += group) {
      const int h = (int)((c * VE) / head_dim);
      const float r = Elem<T>::to_f(er[d * num_heads + h]);
      float m = -INFINITY;
      for (int64_t e = e0; e < e1; ++e) {
        float s = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
        s = s > 0.f ? s : s * slope;
        m = fmaxf(m, s);
      }
      float denom = 0.f;
      for (int64_t e = e0; e < e1; ++e) {
        float s = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
        s = s > 0.f ? s : s * slope;
        denom += expf(s - m);
      }
      const float inv = denom > 0.f ? 1.f / denom : 0.f;
      float acc[VE];
#pragma unroll
      for (int t = 0; t < VE; ++t) acc[t] = 0.f;
      const bool writes_attn = attn != nullptr && (c * VE) % head_dim == 0;
      for (int64_t e = e0; e < e1; ++e) {
        const int64_t src = row[e];
        float s = Elem<T>::to_f(el[src * num_heads + h]) + r;
        s = s > 0.f ? s : s * slope;
        const float a = expf(s - m) * inv;
        if (writes_attn) attn[e * num_heads + h] = Elem<T>::from_f(a);
        const Pack<T, VE> p = load_pack<T, VE>(ft + src * feat_dim + c * VE);
#pragma unroll
        for (int t = 0; t < VE; ++t) acc[t] += a * Elem<T>::to_f(p.v[t]);
      }
      Pack<T, VE> o;
#pragma unroll
      for (int t = 0; t < VE; ++t) o.v[t] = Elem<T>::from_f(acc[t]);
      store_pack<T, VE>(out + d * feat_dim + c * VE, o);
    }
  }
}

// Fast path of the same operator for wide rows (one warp per destination row), up to
// kGatHeads heads and up to 32 edges per row (fixed-fanout blocks): lane j computes the scores
// of edge j for all heads once (one exp per edge and head instead of two per edge and lane),
// the softmax statistics are warp reductions, the attention values and source ids wait in
// shared memory, and the weighted sum then walks the edges with one shared-memory read each.
// Rows with more than 32 edges take the recomputing walk of k_gat_rows.
constexpr int kGatHeads = 8;

template <typename T, int VE>
__global__ void __launch_bounds__(256)
k_gat_rows_warp(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el,
                const T* __restrict__ er, int num_heads, int64_t head_dim, float slope,
                int64_t num_dst, GatWs ws, T* __restrict__ out, T* __restrict__ attn, int32_t* status) {
  __shared__ float a_sh[8][32][kGatHeads];
  __shared__ int64_t src_sh[8][32];
  const bool unsorted = *ws.flags != 0;
  if (unsorted && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(status, APT_FLAG_NOT_GROUPED);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  const int64_t nvec = feat_dim / VE;
  int64_t d = (int64_t)blockIdx.x * 8 + warp;
  const int64_t stride = (int64_t)gridDim.x * 8;
  for (; d < num_dst; d += stride) {
    const int64_t e0 = unsorted ? 0 : ws.range[d];
    const int64_t e1 = unsorted ? 0 : ws.range[d + 1];
    const int deg = (int)(e1 - e0);
    if (deg <= 32) {
      const bool has = lane < deg;
      const int64_t src = has ? row[e0 + lane] : 0;
      src_sh[warp][lane] = src;
#pragma unroll
      for (int h = 0; h < kGatHeads; ++h) {
        if (h < num_heads) {
          float sc = -INFINITY;
          if (has) {
            sc = Elem<T>::to_f(el[src * num_heads + h]) + Elem<T>::to_f(er[d * num_heads + h]);
            sc = sc > 0.f ? sc : sc * slope;
          }
          float m = sc;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
          const float p = has ? expf(sc - m) : 0.f;
          float sum = p;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
          const float a = sum > 0.f ? p / sum : 0.f;
          a_sh[warp][lane][h] = a;
          if (has && attn) attn[(e0 + lane) * num_heads + h] = Elem<T>::from_f(a);
        }
      }
      __syncwarp();
      for (int64_t c = lane; c < nvec; c += 32) {
        const int h = (int)((c * VE) / head_dim);
        float acc[VE];
#pragma unroll
        for (int t = 0; t < VE; ++t) acc[t] = 0.f;
#pragma unroll 4
        for (int j = 0; j < deg; ++j) {
          const float a = a_sh[warp][j][h];
          const Pack<T, VE> p = load_pack<T, VE>(ft + src_sh[warp][j] * feat_dim + c * VE);
#pragma unroll
          for (int t = 0; t < VE; ++t) acc[t] += a * Elem<T>::to_f(p.v[t]);
        }
        Pack<T, VE> o;
#pragma unroll
        for (int t = 0; t < VE; ++t) o.v[t] = Elem<T>::from_f(acc[t]);
        store_pack<T, VE>(out + d * feat_dim + c * VE, o);
      }
      __syncwarp();
      continue;
    }
    for (int64_t c = lane; c < nvec; c += 32) {
      const int h = (int)((c * VE) / head_dim);
      const float r = Elem<T>::to_f(er[d * num_heads + h]);
      float m = -INFINITY;
      for (int64_t e = e0; e < e1; ++e) {
        float sc = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
        sc = sc > 0.f ? sc : sc * slope;
        m = fmaxf(m, sc);
      }
      float denom = 0.f;
      for (int64_t e = e0; e < e1; ++e) {
        float sc = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
        sc = sc > 0.f ? sc : sc * slope;
        denom += expf(sc - m);
      }
      const float inv = denom > 0.f ? 1.f / denom : 0.f;
      float acc[VE];
#pragma unroll
      for (int t = 0; t < VE; ++t) acc[t] = 0.f;
      const bool writes_attn = attn != nullptr && (c * VE) % head_dim == 0;
      for (int64_t e = e0; e < e1; ++e) {
        const int64_t src = row[e];
        float sc = Elem<T>::to_f(el[src * num_heads + h]) + r;
        sc = sc > 0.f ? sc : sc * slope;
        const float a = expf(sc - m) * inv;
        if (writes_attn) attn[e * num_heads + h] = Elem<T>::from_f(a);
        const Pack<T, VE> p = load_pack<T, VE>(ft + src * feat_dim + c * VE);
#pragma unroll
        for (int t = 0; t < VE; ++t) acc[t] += a * Elem<T>::to_f(p.v[t]);
      }
      Pack<T, VE> o;
#pragma unroll
      for (int t = 0; t < VE; ++t) o.v[t] = Elem<T>::from_f(acc[t]);
      store_pack<T, VE>(out + d * feat_dim + c * VE, o);
    }
  }
}

template <typename T>
static int launch_gat(bool vec, const int64_t* row, const void* ft, const void* el, const void* er,
                      int num_heads, int64_t head_dim, float slope, int64_t num_dst, GatWs ws, void* out,
                      void* attn, int32_t* status, cudaStream_t s) {
  constexpr int VE = 16 / sizeof(T);
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  ProfScope prof("gat_rows", s);
  if (vec && feat_dim / VE > 16 && num_heads <= kGatHeads) {
    const int grid = wave_grid(ceil_div(num_dst, 8), 8);
    APT_LAUNCH((k_gat_rows_warp<T, VE>), grid, 256, 0, s, row, (const T*)ft, (const T*)el, (const T*)er, num_heads,
               head_dim, slope, num_dst, ws, (T*)out, (T*)attn, status);
  } else if (vec) {
    const int group = pow2_ge(feat_dim / VE);
    const int grid = wave_grid(ceil_div(num_dst, 256 / group), 8);
    APT_LAUNCH((k_gat_rows<T, VE>), grid, 256, 0, s, row, (const T*)ft, (const T*)el, (const T*)er, num_heads,
               head_dim, slope, num_dst, ws, (T*)out, (T*)attn, group, status);
  } else {
    const int group = pow2_ge(feat_dim);
    const int grid = wave_grid(ceil_div(num_dst, 256 / group), 8);
    APT_LAUNCH((k_gat_rows<T, 1>), grid, 256, 0, s, row, (const T*)ft, (const T*)el, (const T*)er, num_heads,
               head_dim, slope, num_dst, ws, (T*)out, (T*)attn, group, status);
  }
  return APT_OK;
}

// ---- backward of the fused GAT edge pipeline: the edge part ---------------------------
// Per destination row d and head h (s_e, a_e as in k_gat_rows, g = grad_out[d, h, :]):
//   dot_e = <g, ft[src_e, h, :]>;  t = sum_e a_e dot_e;
//   grad_s_e = a_e (dot_e - t) * (s_e > 0 ? 1 : slope);  grad_er[d, h] = sum_e grad_s_e
// attn[e, h] = a_e and grad_score[e, h] = grad_s_e go out per edge; the sums over the
// source side (grad_ft = sum a_e g, grad_el = sum grad_s_e) are SpMM calls in the
// reverse direction. The lanes of one head (lanes_per_head of them, a power of two
// inside the lane group) each hold a slice of g and of the ft row and meet in a
// butterfly of shuffles for the dot product.
template <typename T, int VE>
__global__ void __launch_bounds__(256)
k_gat_bwd_rows(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el,
               const T* __restrict__ er, const T* __restrict__ grad_out, int num_heads, int64_t head_dim,
               float slope, int64_t num_dst, GatWs ws, T* __restrict__ attn, T* __restrict__ grad_score,
               T* __restrict__ grad_er, int group, int lanes_per_head, int32_t* status,
               int64_t skip_up_to /* rows with at most this many edges belong to k_gat_bwd_warp */) {
  const bool unsorted = *ws.flags != 0;
  if (unsorted && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(status, APT_FLAG_NOT_GROUPED);
  const int lane = threadIdx.x & 31;
  const int sub = lane % group;
  const unsigned gmask = group == 32 ? 0xffffffffu : (((1u << group) - 1u) << (lane - sub));
  const int64_t rows_per_block = blockDim.x / group;
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  const int64_t nvec = feat_dim / VE;
  int64_t d = (int64_t)blockIdx.x * rows_per_block + threadIdx.x / group;
  const int64_t stride = (int64_t)gridDim.x * rows_per_block;
  for (; d < num_dst; d += stride) {
    const int64_t e0 = unsorted ? 0 : ws.range[d];
    const int64_t e1 = unsorted ? 0 : ws.range[d + 1];
    if (e1 - e0 <= skip_up_to) continue;
    for (int64_t c0 = 0; c0 < nvec; c0 += group) {
      const int64_t c = c0 + sub;
      const bool live = c < nvec;
      const int h = live ? (int)((c * VE) / head_dim) : 0;
      const bool leader = live && (c * VE) % head_dim == 0;
      const float r = Elem<T>::to_f(er[d * num_heads + h]);
      float m = -INFINITY;
      for (int64_t e = e0; e < e1; ++e) {
        float s = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
        s = s > 0.f ? s : s * slope;
        m = fmaxf(m, s);
      }
      float denom = 0.f;
      for (int64_t e = e0; e < e1; ++e) {
        float s = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
        s = s > 0.f ? s : s * slope;
        denom += expf(s - m);
      }
      const float inv = denom > 0.f ? 1.f / denom : 0.f;
      float g[VE];
#pragma unroll
      for (int t = 0; t < VE; ++t) g[t] = 0.f;
      if (live) {
        const Pack<T, VE> p = load_pack<T, VE>(grad_out + d * feat_dim + c * VE);
#pragma unroll
        for (int t = 0; t < VE; ++t) g[t] = Elem<T>::to_f(p.v[t]);
      }
      // first walk: t = sum_e a_e dot_e; second walk: the per-edge results
      float tsum = 0.f, ger = 0.f;
      for (int pass = 0; pass < 2; ++pass) {
        for (int64_t e = e0; e < e1; ++e) {
          const int64_t src = row[e];
          const float raw = Elem<T>::to_f(el[src * num_heads + h]) + r;
          const float s = raw > 0.f ? raw : raw * slope;
          const float a = expf(s - m) * inv;
          float dot = 0.f;
          if (live) {
            const Pack<T, VE> p = load_pack<T, VE>(ft + src * feat_dim + c * VE);
#pragma unroll
            for (int t = 0; t < VE; ++t) dot += g[t] * Elem<T>::to_f(p.v[t]);
          }
          for (int o = lanes_per_head >> 1; o > 0; o >>= 1) dot += __shfl_xor_sync(gmask, dot, o, group);
          if (pass == 0) {
            tsum += a * dot;
          } else {
            const float gs = a * (dot - tsum) * (raw > 0.f ? 1.f : slope);
            ger += gs;
            if (leader) {
              attn[e * num_heads + h] = Elem<T>::from_f(a);
              grad_score[e * num_heads + h] = Elem<T>::from_f(gs);
            }
          }
        }
      }
      if (leader) grad_er[d * num_heads + h] = Elem<T>::from_f(ger);
    }
  }
}

// Wide rows with at most 32 edges (fixed-fanout blocks), one warp per destination: lane j
// scores edge j for all heads once, the lanes then walk the edges ONCE over ft (each lane its
// slice of grad_out and of the row, the lanes of a head meeting in a shuffle butterfly) and
// leave <grad_out, ft> per edge and head in shared memory, and lane j finishes edge j.
template <typename T, int VE>
__global__ void __launch_bounds__(256)
k_gat_bwd_warp(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el,
               const T* __restrict__ er, const T* __restrict__ grad_out, int num_heads, int64_t head_dim,
               float slope, int64_t num_dst, GatWs ws, T* __restrict__ attn, T* __restrict__ grad_score,
               T* __restrict__ grad_er, int lanes_per_head, int32_t* status) {
  __shared__ float a_sh[8][32][kGatHeads], fac_sh[8][32][kGatHeads], dot_sh[8][32][kGatHeads];
  __shared__ int64_t src_sh[8][32];
  const bool unsorted = *ws.flags != 0;
  if (unsorted && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(status, APT_FLAG_NOT_GROUPED);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  const int64_t nvec = feat_dim / VE;
  int64_t d = (int64_t)blockIdx.x * 8 + warp;
  const int64_t stride = (int64_t)gridDim.x * 8;
  for (; d < num_dst; d += stride) {
    const int64_t e0 = unsorted ? 0 : ws.range[d];
    const int64_t e1 = unsorted ? 0 : ws.range[d + 1];
    const int deg = (int)(e1 - e0);
    if (deg > 32) continue;            // left to k_gat_bwd_rows
    const bool has = lane < deg;
    const int64_t src = has ? row[e0 + lane] : 0;
    src_sh[warp][lane] = src;
#pragma unroll
    for (int h = 0; h < kGatHeads; ++h) {
      if (h < num_heads) {
        float raw = 0.f, sc = -INFINITY;
        if (has) {
          raw = Elem<T>::to_f(el[src * num_heads + h]) + Elem<T>::to_f(er[d * num_heads + h]);
          sc = raw > 0.f ? raw : raw * slope;
        }
        float m = sc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float p = has ? expf(sc - m) : 0.f;
        float sum = p;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        a_sh[warp][lane][h] = sum > 0.f ? p / sum : 0.f;
        fac_sh[warp][lane][h] = raw > 0.f ? 1.f : slope;
      }
    }
    __syncwarp();
    for (int64_t c0 = 0; c0 < nvec; c0 += 32) {
      const int64_t c = c0 + lane;
      const bool live = c < nvec;
      const int h = live ? (int)((c * VE) / head_dim) : 0;
      const bool leader = live && (c * VE) % head_dim == 0;
      float g[VE];
#pragma unroll
      for (int t = 0; t < VE; ++t) g[t] = 0.f;
      if (live) {
        const Pack<T, VE> p = load_pack<T, VE>(grad_out + d * feat_dim + c * VE);
#pragma unroll
        for (int t = 0; t < VE; ++t) g[t] = Elem<T>::to_f(p.v[t]);
      }
      for (int j = 0; j < deg; ++j) {
        float dot = 0.f;
        if (live) {
          const Pack<T, VE> p = load_pack<T, VE>(ft + src_sh[warp][j] * feat_dim + c * VE);
#pragma unroll
          for (int t = 0; t < VE; ++t) dot += g[t] * Elem<T>::to_f(p.v[t]);
        }
        for (int o = lanes_per_head >> 1; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (leader) dot_sh[warp][j][h] = dot;
      }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kGatHeads; ++h) {
      if (h < num_heads) {
        const float a = has ? a_sh[warp][lane][h] : 0.f;
        const float dot = has ? dot_sh[warp][lane][h] : 0.f;
        float t = a * dot;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        const float gs = has ? a * (dot - t) * fac_sh[warp][lane][h] : 0.f;
        if (has) {
          attn[(e0 + lane) * num_heads + h] = Elem<T>::from_f(a);
          grad_score[(e0 + lane) * num_heads + h] = Elem<T>::from_f(gs);
        }
        float ger = gs;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ger += __shfl_xor_sync(0xffffffffu, ger, o);
        if (lane == 0) grad_er[d * num_heads + h] = Elem<T>::from_f(ger);
      }
    }
    __syncwarp();
  }
}

// Any head width: one thread per (destination, head), everything in turn.
template <typename T>
__global__ void __launch_bounds__(256)
k_gat_bwd_generic(const int64_t* __restrict__ row, const T* __restrict__ ft, const T* __restrict__ el,
                  const T* __restrict__ er, const T* __restrict__ grad_out, int num_heads, int64_t head_dim,
                  float slope, int64_t num_dst, GatWs ws, T* __restrict__ attn, T* __restrict__ grad_score,
                  T* __restrict__ grad_er, int32_t* status) {
  const bool unsorted = *ws.flags != 0;
  if (unsorted && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(status, APT_FLAG_NOT_GROUPED);
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  const int64_t total = num_dst * num_heads;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int64_t d = i / num_heads;
    const int h = (int)(i - d * num_heads);
    const int64_t e0 = unsorted ? 0 : ws.range[d];
    const int64_t e1 = unsorted ? 0 : ws.range[d + 1];
    const float r = Elem<T>::to_f(er[d * num_heads + h]);
    float m = -INFINITY;
    for (int64_t e = e0; e < e1; ++e) {
      float s = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
      s = s > 0.f ? s : s * slope;
      m = fmaxf(m, s);
    }
    float denom = 0.f;
    for (int64_t e = e0; e < e1; ++e) {
      float s = Elem<T>::to_f(el[row[e] * num_heads + h]) + r;
      s = s > 0.f ? s : s * slope;
      denom += expf(s - m);
    }
    const float inv = denom > 0.f ? 1.f / denom : 0.f;
    const T* g = grad_out + d * feat_dim + (int64_t)h * head_dim;
    float tsum = 0.f, ger = 0.f;
    for (int pass = 0; pass < 2; ++pass) {
      for (int64_t e = e0; e < e1; ++e) {
        const int64_t src = row[e];
        const float raw = Elem<T>::to_f(el[src * num_heads + h]) + r;
        const float s = raw > 0.f ? raw : raw * slope;
        const float a = expf(s - m) * inv;
        const T* f = ft + src * feat_dim + (int64_t)h * head_dim;
        float dot = 0.f;
        for (int64_t k = 0; k < head_dim; ++k) dot += Elem<T>::to_f(g[k]) * Elem<T>::to_f(f[k]);
        if (pass == 0) {
          tsum += a * dot;
        } else {
          const float gs = a * (dot - tsum) * (raw > 0.f ? 1.f : slope);
          ger += gs;
          attn[e * num_heads + h] = Elem<T>::from_f(a);
          grad_score[e * num_heads + h] = Elem<T>::from_f(gs);
        }
      }
    }
    grad_er[d * num_heads + h] = Elem<T>::from_f(ger);
  }
}

template <typename T>
static int launch_gat_bwd(bool vec, const int64_t* row, const void* ft, const void* el, const void* er,
                          const void* grad_out, int num_heads, int64_t head_dim, float slope, int64_t num_dst,
                          GatWs ws, void* attn, void* grad_score, void* grad_er, int32_t* status, cudaStream_t s) {
  constexpr int VE = 16 / sizeof(T);
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  ProfScope prof("gat_bwd_rows", s);
  const int64_t lph = head_dim / VE;                   // lanes per head when rows are read as 16-byte vectors
  const bool pow2 = lph >= 1 && lph <= 32 && (lph & (lph - 1)) == 0;
  if (vec && pow2) {
    const int group = pow2_ge(feat_dim / VE);
    if (group % lph == 0) {
      int64_t skip = -1;
      if (group == 32 && num_heads <= kGatHeads) {
        // rows of up to 32 edges: one warp per row; the kernel after it takes the longer rows
        const int grid_w = wave_grid(ceil_div(num_dst, 8), 8);
        APT_LAUNCH((k_gat_bwd_warp<T, VE>), grid_w, 256, 0, s, row, (const T*)ft, (const T*)el, (const T*)er,
                   (const T*)grad_out, num_heads, head_dim, slope, num_dst, ws, (T*)attn, (T*)grad_score,
                   (T*)grad_er, (int)lph, status);
        skip = 32;
      }
      const int grid = wave_grid(ceil_div(num_dst, 256 / group), 8);
      APT_LAUNCH((k_gat_bwd_rows<T, VE>), grid, 256, 0, s, row, (const T*)ft, (const T*)el, (const T*)er,
                 (const T*)grad_out, num_heads, head_dim, slope, num_dst, ws, (T*)attn, (T*)grad_score, (T*)grad_er,
                 group, (int)lph, status, skip);
      return APT_OK;
    }
  }
  const int grid = wave_grid(ceil_div(num_dst * num_heads, 256), 8);
  APT_LAUNCH((k_gat_bwd_generic<T>), grid, 256, 0, s, row, (const T*)ft, (const T*)el, (const T*)er,
             (const T*)grad_out, num_heads, head_dim, slope, num_dst, ws, (T*)attn, (T*)grad_score, (T*)grad_er, status);
  return APT_OK;
}

}  // namespace apt

extern "C" int apt_gat_edge_softmax_sum(int dtype, const int64_t* coo_row, const int64_t* coo_col,
                                        int64_t num_edges, const void* ft, const void* el, const void* er,
                                        int num_heads, int64_t head_dim, float negative_slope,
                                        int64_t num_dst, void* out, void* out_attn, void* workspace,
                                        size_t workspace_bytes, int32_t* status_word, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(dtype >= APT_F32 && dtype <= APT_F16, "apt_gat_edge_softmax_sum: dtype %d", dtype);
  APT_CHECK_ARG(num_edges >= 0 && num_heads >= 1 && head_dim >= 1 && num_dst >= 0,
                "apt_gat_edge_softmax_sum: bad sizes");
  if (num_dst == 0) return APT_OK;
  const size_t esz = (size_t)(dtype == APT_F32 ? 4 : 2);
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  cudaStream_t s = (cudaStream_t)stream;
  APT_CHECK_ARG(out && status_word, "apt_gat_edge_softmax_sum: null output");
  if (num_edges == 0) {
    APT_CUDA(cudaMemsetAsync(out, 0, (size_t)num_dst * feat_dim * esz, s));
    return APT_OK;
  }
  APT_CHECK_ARG(coo_row && coo_col && ft && el && er && workspace, "apt_gat_edge_softmax_sum: null pointer");
  APT_CHECK_ARG(((uintptr_t)workspace & 255) == 0, "apt_gat_edge_softmax_sum: workspace must be 256-byte aligned");
  GatWs ws;
  if (!gat_layout(num_dst, (char*)workspace, workspace_bytes, &ws)) {
    set_error("apt_gat_edge_softmax_sum: workspace of %zu bytes is too small", workspace_bytes);
    return APT_ERR_CAPACITY;
  }
  APT_CUDA(cudaMemsetAsync(ws.flags, 0, 4, s));
  {
    ProfScope prof("spmm_ranges", s);
    const int grid = wave_grid(ceil_div(num_edges, 256), 8);
    APT_LAUNCH(k_edge_ranges_single, grid, 256, 0, s, coo_col, num_edges, num_dst, ws);
  }
  const int ve = 16 / (int)esz;
  const bool vec = (((uint64_t)(feat_dim * esz) | (uintptr_t)ft | (uintptr_t)out) & 15) == 0 && head_dim % ve == 0;
  switch (dtype) {
    case APT_F32:
      return launch_gat<float>(vec, coo_row, ft, el, er, num_heads, head_dim, negative_slope, num_dst, ws, out,
                               out_attn, status_word, s);
    case APT_BF16:
      return launch_gat<__nv_bfloat16>(vec, coo_row, ft, el, er, num_heads, head_dim, negative_slope, num_dst, ws,
                                       out, out_attn, status_word, s);
    default:
      return launch_gat<__half>(vec, coo_row, ft, el, er, num_heads, head_dim, negative_slope, num_dst, ws, out,
                                out_attn, status_word, s);
  }
}

extern "C" int apt_gat_edge_backward(int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t num_edges,
                                     const void* ft, const void* el, const void* er, const void* grad_out,
                                     int num_heads, int64_t head_dim, float negative_slope, int64_t num_dst,
                                     void* out_attn, void* out_grad_score, void* out_grad_er, void* workspace,
                                     size_t workspace_bytes, int32_t* status_word, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(dtype >= APT_F32 && dtype <= APT_F16, "apt_gat_edge_backward: dtype %d", dtype);
  APT_CHECK_ARG(num_edges >= 0 && num_heads >= 1 && head_dim >= 1 && num_dst >= 0, "apt_gat_edge_backward: bad sizes");
  if (num_dst == 0) return APT_OK;
  const size_t esz = (size_t)(dtype == APT_F32 ? 4 : 2);
  const int64_t feat_dim = (int64_t)num_heads * head_dim;
  cudaStream_t s = (cudaStream_t)stream;
  APT_CHECK_ARG(out_grad_er && status_word, "apt_gat_edge_backward: null output");
  if (num_edges == 0) {
    APT_CUDA(cudaMemsetAsync(out_grad_er, 0, (size_t)num_dst * num_heads * esz, s));
    return APT_OK;
  }
  APT_CHECK_ARG(coo_row && coo_col && ft && el && er && grad_out && out_attn && out_grad_score && workspace,
                "apt_gat_edge_backward: null pointer");
  APT_CHECK_ARG(((uintptr_t)workspace & 255) == 0, "apt_gat_edge_backward: workspace must be 256-byte aligned");
  GatWs ws;
  if (!gat_layout(num_dst, (char*)workspace, workspace_bytes, &ws)) {
    set_error("apt_gat_edge_backward: workspace of %zu bytes is too small", workspace_bytes);
    return APT_ERR_CAPACITY;
  }
  APT_CUDA(cudaMemsetAsync(ws.flags, 0, 4, s));
  // edges that name no valid destination keep zeros
  APT_CUDA(cudaMemsetAsync(out_attn, 0, (size_t)num_edges * num_heads * esz, s));
  APT_CUDA(cudaMemsetAsync(out_grad_score, 0, (size_t)num_edges * num_heads * esz, s));
  {
    ProfScope prof("spmm_ranges", s);
    const int grid = wave_grid(ceil_div(num_edges, 256), 8);
    APT_LAUNCH(k_edge_ranges_single, grid, 256, 0, s, coo_col, num_edges, num_dst, ws);
  }
  const int ve = 16 / (int)esz;
  const bool vec = (((uint64_t)(feat_dim * esz) | (uintptr_t)ft | (uintptr_t)grad_out) & 15) == 0 && head_dim % ve == 0;
  switch (dtype) {
    case APT_F32:
      return launch_gat_bwd<float>(vec, coo_row, ft, el, er, grad_out, num_heads, head_dim, negative_slope, num_dst,
                                   ws, out_attn, out_grad_score, out_grad_er, status_word, s);
    case APT_BF16:
      return launch_gat_bwd<__nv_bfloat16>(vec, coo_row, ft, el, er, grad_out, num_heads, head_dim, negative_slope,
                                           num_dst, ws, out_attn, out_grad_score, out_grad_er, status_word, s);
    default:
      return launch_gat_bwd<__half>(vec, coo_row, ft, el, er, grad_out, num_heads, head_dim, negative_slope,
                                    num_dst, ws, out_attn, out_grad_score, out_grad_er, status_word, s);
  }
}
