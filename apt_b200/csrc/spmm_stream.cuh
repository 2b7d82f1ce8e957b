// The kernel for wide rows of many edges: sums (kCopyU, kUMulW) and the attention backward's dots (kDots). A warp walks a
// stretch of the edges as one stream; input rows travel to shared memory asynchronously.
//
// What bounds it: rows mostly come out of L2, which hands a random gather of 512-byte or 1 KiB rows to the SMs at 12 - 13 TB/s
// however they are fetched (cp.async, cp.async.bulk, tile::gather4: 39 - 43 and 82 - 87 us for a million rows). k_spmm_rows stays
// below that because registers bound the bytes it has in flight. Here it takes 128 to 192 KB an SM on their way (two groups of
// rows a warp) and few instructions an edge; what is left is a third to a half of the issue slots (22 an edge for fp32 x 128,
// 38 with weights in bf16).
//
//   stretch     every warp has the same number of slots. Edges that come grouped are cut at row ends; behind the counting sort
//               they are cut anywhere, sums of a row of several stretches are left in scratch and the warp that comes last adds
//               them up in order, above 32 stretches in two steps: long rows need no items of their own.
//   copies      rows of up to 512 bytes by 16-byte cp.async, an instruction a row; wider ones by one cp.async.bulk each, from a lane
//               each (that instruction is issued lane by lane, 13 instructions a row, and two cp.async with their addresses are
//               as many: fp32 x 256 142 against 146 us in reverse, x 132 134 against 142, dots of 4 x 64 faster too).
//   row ends    a bit per slot, looked at four slots at a time: a quarter without one is straight-line code.
//   weights     (kUMulW) of 32 edges at a time by cp.async, two batches ahead.
//   kDots       the output row's own slices in registers, those of the row behind it fetched ahead. The atomics that count the
//               edges of every input row, for the sort behind, ride on the fetch of the edges.
//
// us of the whole call, k_spmm_rows or a bulk-copy kernel for rows above 512 bytes (rows dealt to the warps one by one) -> here,
// 67 584 x 15 edges:
//   sums         fp32 x 256 forward 98 -> 101, reverse 190 -> 129; x 128 71 -> 52, 134 -> 97; bf16 x 256 79 -> 59, 143 -> 111
//   attention    forward, both directions: bf16 4 x 64 104 -> 75, 375 -> 261; fp32 4 x 64 158 -> 116, 556 -> 380; 4 x 32 100 -> 67, 357 -> 236
// Against it: the start of a stream is three dependent fetches, which few edges a warp do not make up for. Hence the lines of stream_fits.
// 16-bit rows of two slices a lane spill 92 bytes with weights and 20 in kDots at ten warps (bf16 2 x 256, 67 584 x 15 edges,
// both directions 676 -> 456 all the same).
// Hub rows: 100 000 edges in no order, half of them in one row, fp32 x 128: 135 -> 77, 400 000 330 -> 192 (218 and 400 with one warp to add up
// all parts of a row).
// Both gradients of the attention in one walk (a source's features in registers, dots and sums of its edges) saved a walk and lost
// it again: 70 instructions an edge, 147 us, which the two walks take as well; with the dots on mma.sync 181.
#pragma once

#include "spmm_rows.cuh"

namespace apt {

constexpr uint32_t kNoRow = 0xffffffffu;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// By all lanes of a warp, which agree on the answer.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int polls) {
  for (int k = 0; k < polls; ++k)
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  return false;
}
// `bytes` and both addresses are multiples of 16.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void copy_16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// 32 slots of a warp's stretch, a lane to each.
struct SlotBatch {
  uint32_t src;        // input row
  uint32_t row;        // output row; kNoRow behind the last slot
  uint32_t e;          // edge; kDots: its place among those of its input row
};

template <typename T, int OP, int VPL, bool WIDENED>
__global__ void __launch_bounds__(stream_warps(VPL == 1) * 32, kStreamBlocks)
k_spmm_stream(const __grid_constant__ RowArgs<T> a, const __grid_constant__ StreamPlan plan, int polls, volatile int32_t* pending) {
  wait_for_previous();
  constexpr int VE = 16 / sizeof(T), GE = stream_group(VPL == 1), P = Acc<VE>::P, kSlot = 512 * VPL;
  constexpr bool kWeights = OP == kUMulW, kIsDots = OP == kDots, kBulk = VPL == 2;
  extern __shared__ __align__(128) unsigned char shared[];
  __shared__ uint64_t bars[stream_warps(VPL == 1)][2];
  __shared__ int64_t coo[kMaxSegments + 1], ioff[kMaxSegments + 1], ooff[kMaxSegments + 1];
  int mode = a.mode, fixed = a.fixed;
  if (mode == kDevice) {
    const int64_t w = *a.ws.result;
    mode = probe_mode(w);
    fixed = mode == kFixed ? (int)(a.num_edges / a.num_rows) : 0;
  }
  for (int t = threadIdx.x; t <= a.st.nseg; t += blockDim.x) {
    // no table: one segment whose rows start at 0
    coo[t] = a.st.coo_off ? a.st.coo_off[t] : 0;
    ioff[t] = a.st.in_off ? a.st.in_off[t] : 0;
    ooff[t] = a.st.out_off ? a.st.out_off[t] : 0;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t* const bar = bars[w];
  if (lane < 2) mbar_init(bar + lane, kBulk ? 1 : 32);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();

  const uint32_t num_rows = (uint32_t)a.num_rows;
  const int heads = OP != kCopyU ? (int)a.edata_dim : 1;
  const int warps = gridDim.x * plan.warps, warp = blockIdx.x * plan.warps + w;
  const uint32_t row_bytes = plan.row_bytes;
  unsigned char* const ring = shared + w * plan.warp_bytes;
  float* const weights = (float*)(ring + 2 * GE * kSlot);      // [2][32][heads]; WIDENED: the row that is written behind them

  // the lane's slices of 16 bytes, 32 apart; in kDots a head's slices have a power of two of lanes (plan.lph)
  int col[VPL], head[VPL];
  bool valid[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int v = lane + 32 * i;
    if constexpr (kIsDots) {
      const int nvh = (int)(a.feat_dim / heads) / VE, h = v / plan.lph, p = v & (plan.lph - 1);
      valid[i] = h < heads && p < nvh;
      head[i] = 0;
      col[i] = valid[i] ? (h * nvh + p) * VE : 0;
    } else {
      const int nvec = (int)(a.feat_dim / VE);
      valid[i] = v < nvec;
      col[i] = min(v, nvec - 1) * VE;
      head[i] = kWeights ? col[i] / (int)(a.feat_dim / heads) : 0;
    }
  }

  // this warp's slots, [lo, hi) of `total`; a stretch ends inside a group only where the last row ends
  const bool none = any_found(a.none);
  const int total = mode == kOrder ? *a.ws.num_slots : none ? 0 : (int)a.num_edges;
  const int chunk = max(GE, (int)(((int64_t)total + warps - 1) / warps + GE - 1) & ~(GE - 1));
  auto out_row = [&](int k) -> uint32_t { return (uint32_t)(ooff[a.st.nseg > 1 ? seg_of(coo, a.st.nseg, k) : 0] + a.col[k]); };
  auto border = [&](int64_t at) -> int {
    const int k = (int)min(at, (int64_t)total);
    if (mode == kOrder || k == 0 || k == total) return k;
    if (mode == kFixed) return (int)(((int64_t)k + fixed - 1) / fixed * fixed);
    const uint32_t before = out_row(k - 1);          // rows are not split
    return out_row(k) == before ? a.ws.range[before].y : k;
  };
  const int lo = border((int64_t)warp * chunk), hi = border((int64_t)(warp + 1) * chunk);

  auto load = [&](int base) -> SlotBatch {
    SlotBatch r{0u, kNoRow, 0u};
    const int k = base + lane;
    if (k > hi || k >= total) return r;
    if (mode == kOrder) {
      if constexpr (kWeights) {
        const uint4 o = ((const uint4*)a.ws.order)[k];
        r.src = o.x, r.row = o.y, r.e = o.z;
      } else {
        const uint2 o = a.ws.order[k];
        r.src = o.x, r.row = o.y;
      }
    } else {
      r.e = (uint32_t)k;
      r.row = mode == kFixed ? (uint32_t)k / (uint32_t)fixed : out_row(k);
      if (k < hi) r.src = (uint32_t)(ioff[a.st.nseg > 1 ? seg_of(coo, a.st.nseg, k) : 0] + a.row[k]);
    }
    if constexpr (kIsDots) r.e = k < hi && r.src < a.num_in ? (uint32_t)atomicAdd(a.ws.cnt + spread(r.src), 1) : kNoRank;
    return r;
  };
  // what was under way when the batch was loaded has arrived
  auto settle = [&](const SlotBatch& b, int base) {
    if constexpr (kIsDots)
      if (base + lane < hi) a.ws.rank[base + lane] = b.e;
  };
  // the weights of a batch, on their way to half `half` of the buffer
  auto fetch_weights = [&](const SlotBatch& b, int base, int half) {
    if (base + lane < hi) {
      float* const dst = weights + (half * 32 + lane) * heads;
      const float* const src = (const float*)a.edata + (uint64_t)b.e * heads;
      if ((heads & 3) == 0) {
        for (int h = 0; h < heads; h += 4) copy_16(dst + h, src + h);
      } else {
        for (int h = 0; h < heads; ++h) copy_4(dst + h, src + h);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  Acc<VE> acc[VPL];
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < VPL; ++i) acc[i].zero();
  };
  clear();
  const int part = WIDENED ? (int)a.width / heads : 0, part_more = WIDENED ? (int)a.feat_dim / heads - part : 0;
  const uint32_t part_inverse = WIDENED && kWeights ? (uint32_t)(((1ull << 31) + part - 1) / part) : 0u;
  auto write = [&](uint32_t d) {
    if constexpr (WIDENED) {
      T* const row = (T*)(weights + (kWeights ? 64 * heads : 0));
      __syncwarp();
#pragma unroll
      for (int i = 0; i < VPL; ++i)
        if (valid[i]) store_pack<T, VE>(row + col[i], acc[i].template rounded<T>());
      __syncwarp();
      store_row(a.out + (uint64_t)d * a.width, row, (int)a.width, lane, kWeights ? part_inverse : 0u, part_more);
      return;
    }
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (valid[i]) store_pack<T, VE>(a.out + (uint64_t)d * a.feat_dim + col[i], acc[i].template rounded<T>());
  };
  // sums of a row that other warps have edges of, until the last of them adds them up
  auto part_of = [&](int slot) { return a.ws.part + (int64_t)slot * a.part_stride; };
  auto leave = [&](int slot) {
    float* const p = part_of(slot);
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (valid[i])
#pragma unroll
        for (int t = 0; t < VE; t += 4)
          __stcg((float4*)(p + col[i] + t), make_float4(acc[i].get(t), acc[i].get(t + 1), acc[i].get(t + 2), acc[i].get(t + 3)));
  };

  SlotBatch now = load(lo), next = load(lo + 32), after{0u, kNoRow, 0u};
  if constexpr (kWeights) {
    if (lo < hi) {
      fetch_weights(now, lo, 0);
      fetch_weights(next, lo + 32, 1);
      after = load(lo + 64);
    }
  }
  // the rows of a group, whose `left` slots start at lane `first` of a batch, to one half of the ring
  auto issue = [&](uint32_t batch_src, int first, int left, int stage) {
    if constexpr (kBulk) {
      const int count = min(GE, left);
      const uint32_t row = __shfl_sync(0xffffffffu, batch_src, first + (lane & (GE - 1)));
      if (lane == 0) mbar_expect(bar + stage, (uint32_t)count * row_bytes);
      if (lane < count) bulk_copy(ring + (stage * GE + lane) * kSlot, (const char*)a.in + (uint64_t)row * row_bytes, row_bytes, bar + stage);
    } else {
#pragma unroll
      for (int q = 0; q < GE; ++q) {      // (slots behind the last one read row 0)
        const uint32_t row = __shfl_sync(0xffffffffu, batch_src, first + q);
        if (valid[0]) copy_16(ring + (stage * GE + q) * kSlot + lane * 16, (const char*)(a.in + col[0]) + (uint64_t)row * row_bytes);
      }
      // every lane's arrival waits for its own copies
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar + stage)) : "memory");
    }
  };
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (lo + k * GE < hi) issue(now.src, k * GE, hi - lo - k * GE, k);

  if (!kIsDots && mode != kFixed) {
    // rows without edges, while the first copies are on their way
    for (uint32_t first = warp * 32; first < num_rows; first += warps * 32) {
      bool empty = false;
      if (first + lane < num_rows) {
        const int2 r = none ? make_int2(0, 0) : a.ws.range[first + lane];
        empty = r.x == r.y;
      }
      for (unsigned m = __ballot_sync(0xffffffffu, empty); m; m &= m - 1) write(first + __ffs(m) - 1);
    }
  }
  if (lo >= hi) return;

  const uint32_t first_row = __shfl_sync(0xffffffffu, now.row, 0);
  bool open = mode == kOrder && a.ws.range[first_row].x < lo;     // the first row's first edges are another warp's
  const bool opened = open;
  // kDots: the output row's own slices, and those of the row that is likely to be the next
  F2 f[VPL][P];
  Raw<T, VE> ahead[VPL];
  uint32_t ahead_row = kNoRow;
  auto look_ahead = [&](uint32_t d) {
    ahead_row = min(d, num_rows - 1);
#pragma unroll
    for (int i = 0; i < VPL; ++i) ahead[i] = load_raw<T, VE>(a.own + (uint64_t)ahead_row * a.feat_dim + col[i]);
  };
  auto turn_to = [&](uint32_t d) {
    if (ahead_row != d) look_ahead(d);
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int t = 0; t < P; ++t) f[i][t] = pair_of(ahead[i], t);
    look_ahead(d + 1);
  };
  if constexpr (kIsDots) turn_to(first_row);
  // the row in hand is done, `following` is the next one
  auto finish = [&](uint32_t d, uint32_t following) {
    if constexpr (kIsDots) {
      if (following != kNoRow) turn_to(following);
    } else {
      if (open) leave(2 * warp);
      else write(d);
      open = false;
      clear();
    }
  };
  // kDots: of four edges' dots this lane adds up one, and may be the one to write it
  const int lph = kIsDots ? min(plan.lph, 32) : 32, sub = lane & (lph - 1);
  const int my_edge = (sub & (lph >> 1) ? 2 : 0) + (sub & (lph >> 2) ? 1 : 0);
  float* const lane_dots = a.dots + lane / lph;
  bool writes[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) writes[i] = (sub & ((lph >> 2) - 1)) == 0 && lane / lph + i * (32 / lph) < heads && (i == 0 || plan.lph < 64);

  settle(now, lo);
  int failed = -1;      // slot of the batch from which on rows did not come
  int half = 0, base = lo;
  uint32_t behind = kNoRow;      // the row of the next slot
  auto ends = [&]() {            // slots that end their row
    behind = __shfl_down_sync(0xffffffffu, now.row, 1);
    const uint32_t opens = __shfl_sync(0xffffffffu, next.row, 0);
    if (lane == 31) behind = opens;
    return __ballot_sync(0xffffffffu, base + lane < hi && now.row != behind);
  };
#pragma unroll 1
  for (;; base += 32) {
    const unsigned last = ends();
    if constexpr (kWeights) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
    }
    const float* const wt = weights + half * 32 * heads;
    const int count = min(32, hi - base);
#pragma unroll 2
    for (int pos = 0; pos < 32; pos += GE) {
      if (pos >= count) break;
      const int stage = pos / GE & 1;
      if (!mbar_wait(bar + stage, pos / GE >> 1 & 1, polls)) {
        failed = pos;
        break;
      }
      const unsigned char* const g = ring + stage * GE * kSlot;
#pragma unroll
      for (int quad = 0; quad < GE; quad += 4) {
        const int at = pos + quad;
        const unsigned marks = last >> at & 15u;
        Raw<T, VE> v[4][VPL];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int i = 0; i < VPL; ++i) *(uint4*)&v[q][i] = *(const uint4*)(g + (quad + q) * kSlot + (kBulk ? col[i] * (int)sizeof(T) : lane * 16));
        if (quad + 4 == GE) {
          __syncwarp();           // read by all lanes: the next copies may overwrite it
          const int to = pos + 2 * GE;
          if (base + to < hi) issue(to < 32 ? now.src : next.src, to & 31, hi - base - to, stage);
        }
        float dt[4][VPL];
        auto add = [&](int q) {
#pragma unroll
          for (int i = 0; i < VPL; ++i) {
            if constexpr (kIsDots) {
              F2 pair = 0ull;
#pragma unroll
              for (int t = 0; t < P; ++t) pair = f2_fma(f[i][t], pair_of(v[q][i], t), pair);
              float x, y;
              f2_unpack(pair, x, y);
              dt[q][i] = valid[i] ? x + y : 0.f;      // (not zero times what may be infinite)
            } else if constexpr (kWeights) {
              acc[i].fma(v[q][i], wt[(at + q) * heads + head[i]]);
            } else {
              acc[i].add(v[q][i]);
            }
          }
        };
        if (marks == 0u) {
          if constexpr (OP == kCopyU) {
            // in pairs: a long row is no further from 64 bits than in the items of k_spmm_rows
#pragma unroll
            for (int i = 0; i < VPL; ++i) {
              Acc<VE> front, back;
              front.sum_of(v[0][i], v[1][i]);
              back.sum_of(v[2][i], v[3][i]);
              front.add(back);
              acc[i].add(front);
            }
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) add(q);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            add(q);
            if (marks >> q & 1u) finish(__shfl_sync(0xffffffffu, now.row, at + q), kIsDots ? __shfl_sync(0xffffffffu, behind, at + q) : 0u);
          }
        }
        if constexpr (kIsDots) {
          // a lane ends up with the dot of one of the four edges (k_gat_dots)
          const int k = at + my_edge;
          if (VPL == 2 && plan.lph == 64) {
#pragma unroll
            for (int q = 0; q < 4; ++q) dt[q][0] += dt[q][VPL - 1];
          }
#pragma unroll
          for (int i = 0; i < VPL; ++i) {
            const float b0 = (my_edge & 2 ? dt[2][i] : dt[0][i]) + __shfl_xor_sync(0xffffffffu, my_edge & 2 ? dt[0][i] : dt[2][i], lph >> 1);
            const float b1 = (my_edge & 2 ? dt[3][i] : dt[1][i]) + __shfl_xor_sync(0xffffffffu, my_edge & 2 ? dt[1][i] : dt[3][i], lph >> 1);
            float s = (my_edge & 1 ? b1 : b0) + __shfl_xor_sync(0xffffffffu, my_edge & 1 ? b0 : b1, lph >> 2);
            if (lph > 4) s += __shfl_xor_sync(0xffffffffu, s, lph >> 3);
            if (lph > 8) s += __shfl_xor_sync(0xffffffffu, s, lph >> 4);
            if (lph > 16) s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (k < count && writes[i]) lane_dots[(int64_t)(base + k) * heads + i * (32 / lph)] = s;
          }
        }
      }
    }
    if (failed >= 0 || base + 32 >= hi) break;
    now = next;
    settle(now, base + 32);
    if constexpr (kWeights) {
      next = after;
      __syncwarp();
      fetch_weights(next, base + 64, half);
      after = load(base + 96);
      half ^= 1;
    } else {
      next = load(base + 64);
    }
  }
  if (failed >= 0) {
    // waited in vain: zeros from here on, and a flag. The block may go once the copies on their way are done. (They have this long; the
    // block goes all the same.)
#pragma unroll 1
    for (int pos = failed; pos < failed + 2 * GE && base + pos < hi; pos += GE) mbar_wait(bar + (pos / GE & 1), pos / GE >> 1 & 1, kStreamWaitPolls);
    if (lane == 0) {
      if (a.status) atomicOr(a.status, APT_FLAG_COPY_TIMEOUT);
      else *pending = APT_FLAG_COPY_TIMEOUT;
    }
    clear();
#pragma unroll 1
    for (;; base += 32, failed = 0) {
      const unsigned last = ends();
      if constexpr (kIsDots) {
        if (lane >= failed && base + lane < hi)
          for (int h = 0; h < heads; ++h) a.dots[(int64_t)(base + lane) * heads + h] = 0.f;
      } else {
        for (unsigned m = last & (~0u << failed); m; m &= m - 1) finish(__shfl_sync(0xffffffffu, now.row, __ffs(m) - 1), 0u);
      }
      if (base + 32 >= hi) break;
      now = next;
      settle(now, base + 32);
      next = kWeights ? after : load(base + 64);
      if constexpr (kWeights) after = load(base + 96);
    }
  }
  if (kIsDots || mode != kOrder) return;
  // rows shared with other warps: their sums are left behind, and who comes last adds them up in the order of the slots
  const uint32_t last_row = __shfl_sync(0xffffffffu, now.row, hi - 1 - base);
  const bool goes_on = a.ws.range[last_row].y > hi;
  if (goes_on) leave(open ? 2 * warp : 2 * warp + 1);
  __threadfence();
  __syncwarp();
  // whether this warp is the last of `of` that come by `counter`; what the others left can then be read
  auto comes_last = [&](int counter, int of) {
    int done = 0;
    if (lane == 0 && of > 1) done = atomicAdd(a.ws.part_done + counter, 1);
    if (__shfl_sync(0xffffffffu, done, 0) != of - 1) return false;
    __threadfence();
    return true;
  };
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    // the first row; the last one, unless it is the first and began before this stretch
    if (k == 0 ? !opened : !goes_on || open) continue;
    const uint32_t d = k == 0 ? first_row : last_row;
    const int2 r = a.ws.range[d];
    const int first = r.x / chunk, parts = (r.y - 1) / chunk - first + 1;
    auto slot = [&](int q) { return 2 * (first + q) + (q == 0 ? 1 : 0); };
    auto sum = [&](int from, int count, int step) {
      clear();
#pragma unroll 2
      for (int q = 0; q < count; ++q) {
        const float* const p = part_of(slot(from + q * step));
#pragma unroll
        for (int i = 0; i < VPL; ++i)
#pragma unroll
          for (int t = 0; t < VE; t += 4) {
            const float4 x = __ldcg((const float4*)(p + col[i] + t));
            acc[i].p[t / 2] = f2_add(acc[i].p[t / 2], f2_pack(x.x, x.y));
            acc[i].p[t / 2 + 1] = f2_add(acc[i].p[t / 2 + 1], f2_pack(x.z, x.w));
          }
      }
    };
    // The last of every kStreamParts stretches adds up theirs, the last of these the row. Counters: the group's first stretch, and the
    // row's second one, in neither of which another row begins (a group of one needs none).
    const int group = (warp - first) / kStreamParts * kStreamParts, size = min(kStreamParts, parts - group);
    if (!comes_last(first + group, size)) continue;
    sum(group, size, 1);
    if (parts > kStreamParts) {
      leave(slot(group));
      __threadfence();
      __syncwarp();
      if (!comes_last(first + 1, (parts + kStreamParts - 1) / kStreamParts)) continue;
      sum(0, (parts + kStreamParts - 1) / kStreamParts, kStreamParts);
    }
    write(d);
  }
}

// Wide rows of many edges: see the top of the file.
template <typename T, int OP, int VPL, bool WIDENED>
static int launch_stream(const RowArgs<T>& a, cudaStream_t s) {
  const StreamPlan plan = stream_plan(OP, a.feat_dim, sizeof(T), (int)a.edata_dim, WIDENED);
  static bool sized[64] = {};
  int dev = 0;
  APT_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !sized[dev]) {
    APT_CUDA(cudaFuncSetAttribute(k_spmm_stream<T, OP, VPL, WIDENED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamShared));
    if (dev < 64) sized[dev] = true;
  }
  int32_t* pending = nullptr;
  if (!a.status) {
    const int rc = pending_word(&pending);
    if (rc != APT_OK) return rc;
  }
  const int blocks = stream_blocks(a.feat_dim, a.num_edges, a.ws.part_floats, plan.warps, a.mode == kFixed || a.mode == kRanges);
  APT_FOLLOW((k_spmm_stream<T, OP, VPL, WIDENED>), blocks, plan.warps * 32, plan.shared, s, a, plan,
             bulk_wait_polls(), (volatile int32_t*)pending);
  return APT_OK;
}

template <typename T, int OP>
static int launch_stream(const RowArgs<T>& a, cudaStream_t s) {
  const bool one_slice = stream_one_slice(OP, a.feat_dim, sizeof(T), (int)a.edata_dim);
  if constexpr (OP == kCopyU || OP == kUMulW)
    if (a.width) return one_slice ? launch_stream<T, OP, 1, true>(a, s) : launch_stream<T, OP, 2, true>(a, s);
  return one_slice ? launch_stream<T, OP, 1, false>(a, s) : launch_stream<T, OP, 2, false>(a, s);
}

}  // namespace apt
