// The row sums for wide rows: input rows travel to shared memory as bulk copies.
//
// k_spmm_rows (spmm_rows.cuh) reads its rows into registers, and what a thread can hold bounds the bytes in flight once a
// lane has two slices to a row. Here one lane a row issues a copy of the whole row (cp.async.bulk, completion on an
// mbarrier); a warp keeps two groups of rows on their way in a ring of its own and sums a group from shared memory when it
// is there: 192 KB of rows an SM in flight.
//
// A warp walks its output rows as one stream of edges: 32 rows a chunk, a lane to each, whose lengths are summed up; a lane
// to each of the next 32 edges finds its row by bisection and fetches the edge's source, so copies run on across
// the ends of rows. Rows are dealt to the warps in turn (the long ones of a block's reverse direction are
// neighbours). Items of long rows (kOrder) go through the same stream before the rows. Weights (kUMulW) follow their rows by
// cp.async onto the same mbarrier.
//
// In us, k_spmm_rows -> here:                        forward        reverse
//   67 584 x 15 edges, fp32 x 256                    112 -> 87      148 -> 122     (1.04 GB: 12 TB/s out of L2 forward)
//   53 000 x 15, fp32 x 192 / x 132                  77 -> 56, 67 -> 57    103 -> 86, 95 -> 86
//   53 000 x 15, bf16 x 512 / x 264                  122 -> 84, 102 -> 83  161 -> 121, 126 -> 117
//   16 000 x 15, fp32 x 256                          30 -> 26       66 -> 46
//   67 584 x 15, weights, fp32 x 4 x 64              133 -> 129     215 -> 156
// and against it: 9 000 x 15, fp32 x 256 13 -> 17 forward (the stream's start costs three dependent rounds), rows of
// one slice a lane 44 -> 56 (fp32 x 128; an SM issues a copy every 13 ns whatever its size). Hence the rule of launch_bulk:
// rows of more than 32 slices, 196 608 edges, and with weights only where edges are ordered.
#pragma once

#include "spmm_rows.cuh"

namespace apt {

constexpr int kBulkWarps = 12, kBulkStages = 2;
// Rows to a group and blocks to an SM: 192 KB of rows either way. Plain sums keep 24 warps of groups of four within
// 80 registers; weights need more.
constexpr int bulk_group(int op) { return op == kCopyU ? 4 : 8; }
constexpr int bulk_blocks(int op) { return op == kCopyU ? 2 : 1; }
constexpr int kBulkMinSlices = 33, kBulkMinEdges = 3 << 16;
constexpr int kBulkHeads = 16;               // weights an edge can bring along
constexpr int kBulkVpl = 2;                  // 16-byte slices a lane
constexpr int kBulkSlot = 512 * kBulkVpl;

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

// The groups of rows (and of their edges' weights) on their way to one warp.
template <int GE>
struct BulkRing {
  unsigned char* slots;     // [kBulkStages][GE][kBulkSlot]
  float* weights;           // [kBulkStages][GE * heads]
  uint64_t* bars;           // [kBulkStages]
  uint32_t row_bytes;
  int heads;
  const char* rows;
  const float* edata;
  int issued = 0, taken = 0;     // groups

  // The next group: rows `src` and edges `e` of the lanes from `first` on; by all lanes.
  template <bool WEIGHTS>
  __device__ __forceinline__ void issue(uint32_t src, uint32_t e, int first, int count, int lane) {
    const int s = issued++ % kBulkStages;
    const uint32_t row = __shfl_sync(0xffffffffu, src, first + (lane & (GE - 1)));
    if (lane == 0) mbar_expect(bars + s, (uint32_t)count * row_bytes);
    if (lane < count) bulk_copy(slots + (s * GE + lane) * kBulkSlot, rows + (uint64_t)row * row_bytes, row_bytes, bars + s);
    if constexpr (WEIGHTS) {
      for (int t = lane; t - lane < count * heads; t += 32) {
        const int q = t / heads;
        const uint32_t edge = __shfl_sync(0xffffffffu, e, (first + q) & 31);
        if (t < count * heads)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(weights + s * GE * kBulkHeads + t)),
                       "l"(edata + (uint64_t)edge * heads + (t - q * heads))
                       : "memory");
      }
      // every lane's arrival waits for its own copies
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bars + s)) : "memory");
    }
  }
  __device__ __forceinline__ const unsigned char* group() const { return slots + taken % kBulkStages * GE * kBulkSlot; }
  __device__ __forceinline__ const float* group_weights() const { return weights + taken % kBulkStages * GE * kBulkHeads; }
  __device__ __forceinline__ bool wait(int polls) const {
    return mbar_wait(bars + taken % kBulkStages, (uint32_t)(taken / kBulkStages) & 1u, polls);
  }
  // Copies that nobody will read: the block may go once they are done. (They have this long; the block goes all the same.)
  __device__ __forceinline__ void drain() {
    for (; taken < issued; ++taken) wait(kBulkWaitPolls);
  }
};

// 32 of a warp's edges, a lane to each.
struct EdgeBatch {
  uint32_t src, e;
  int unit;            // lane that holds the edge's row
  unsigned last;       // edges that end their row
};

template <typename T, int OP>
__global__ void __launch_bounds__(kBulkWarps * 32, bulk_blocks(OP))
k_spmm_bulk(const __grid_constant__ RowArgs<T> a, int polls, volatile int32_t* pending) {
  wait_for_previous();
  constexpr int VE = 16 / sizeof(T), GE = bulk_group(OP), VPL = kBulkVpl;
  constexpr bool kWeights = OP == kUMulW;
  extern __shared__ __align__(128) unsigned char rings[];
  __shared__ uint64_t bars[kBulkWarps][kBulkStages];
  __shared__ int64_t coo[kMaxSegments + 1], ioff[kMaxSegments + 1];
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
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane < kBulkStages) mbar_init(&bars[w][lane], kWeights ? 33 : 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  const int nvec = (int)(a.feat_dim / VE), num_rows = (int)a.num_rows;
  const bool none = a.none && *a.none != 0;
  const int warps = gridDim.x * kBulkWarps, warp = blockIdx.x * kBulkWarps + w;
  const int num_items = mode == kOrder ? min(*a.ws.num_items, (int)a.ws.max_items) : 0;
  BulkRing<GE> ring{rings + w * kBulkStages * GE * kBulkSlot,
                (float*)(rings + kBulkWarps * kBulkStages * GE * kBulkSlot) + w * kBulkStages * GE * kBulkHeads,
                bars[w], (uint32_t)(a.feat_dim * sizeof(T)), (int)a.edata_dim, (const char*)a.in, (const float*)a.edata};

  int col[VPL], head[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    col[i] = min(lane + 32 * i, nvec - 1) * VE;
    head[i] = kWeights ? col[i] / (int)(a.feat_dim / a.edata_dim) : 0;
  }
  Acc<VE> acc[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) acc[i].zero();

  auto write = [&](int d) {
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (lane + 32 * i < nvec) store_pack<T, VE>(a.out + (int64_t)d * a.feat_dim + col[i], acc[i].template rounded<T>());
  };
  // An item of a row of several: its sums go to scratch, and the item that finishes last adds them up in item order.
  auto write_part = [&](int d, int part, int first_slot) {
    float* const p = a.ws.part + (int64_t)part * a.part_stride;
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (lane + 32 * i < nvec)
#pragma unroll
        for (int t = 0; t < VE; ++t) __stcg(p + col[i] + t, acc[i].get(t));
    const int2 r = a.ws.range[d];
    const int size = item_edges(r.y - r.x), parts = (r.y - r.x + size - 1) / size;
    const int first = part - (first_slot - r.x) / size;
    __threadfence();
    __syncwarp();
    int last = 0;
    if (lane == 0) last = atomicAdd(a.ws.part_done + first, 1) == parts - 1;
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      acc[i].zero();
#pragma unroll 1
      for (int q = 0; q < parts; ++q) {
        const float* const s = a.ws.part + (int64_t)(first + q) * a.part_stride + col[i];
#pragma unroll
        for (int t = 0; t < VE; t += 2) acc[i].p[t / 2] = f2_add(acc[i].p[t / 2], f2_pack(__ldcg(s + t), __ldcg(s + t + 1)));
      }
    }
    write(d);
  };

  // One chunk: this lane's unit is `len` edges from `b` on, for row d (part: see write_part). False: a copy never came.
  auto run = [&](int b, int len, int d, int part) -> bool {
    int upto = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    const int n = __shfl_sync(0xffffffffu, upto, 31);
    auto fetch = [&](int base) {
      EdgeBatch r{0u, 0u, 0, 0u};
      const int i = base + lane;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(0xffffffffu, upto, r.unit + o - 1) <= i) r.unit += o;
      const int end = __shfl_sync(0xffffffffu, upto, r.unit), slots = __shfl_sync(0xffffffffu, b + len, r.unit);
      if (i < n) {
        const int k = slots - (end - i);
        if (mode == kOrder) {
          const uint2 o = a.ws.order[k];
          r.src = o.x;
          r.e = o.y;
        } else {
          r.e = (uint32_t)k;
          r.src = (uint32_t)(ioff[a.st.nseg > 1 ? seg_of(coo, a.st.nseg, k) : 0] + a.row[k]);
        }
      }
      r.last = __ballot_sync(0xffffffffu, i < n && i + 1 == end);
      return r;
    };
    EdgeBatch now = fetch(0), next = now;
    auto issue = [&](const EdgeBatch& from, int k, int left) {
      ring.template issue<kWeights>(from.src, from.e, k * GE, min(GE, left), lane);
    };
#pragma unroll
    for (int k = 0; k < kBulkStages; ++k)
      if (k * GE < n) issue(now, k, n - k * GE);
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
      if (base + 32 < n) next = fetch(base + 32);
#pragma unroll 1
      for (int k = 0; k < 32 / GE; ++k) {
        const int at = base + k * GE, cnt = min(GE, n - at);
        if (cnt <= 0) break;
        if (!ring.wait(polls)) return false;
        Raw<T, VE> v[GE][VPL];
        float wt[GE][VPL];
        const unsigned char* const g = ring.group() + lane * 16;
        const float* const gw = ring.group_weights();
#pragma unroll
        for (int q = 0; q < GE; ++q)
#pragma unroll
          for (int i = 0; i < VPL; ++i) {
            *(uint4*)&v[q][i] = *(const uint4*)(g + q * kBulkSlot + i * 512);
            if constexpr (kWeights) wt[q][i] = gw[q * ring.heads + head[i]];
          }
        ++ring.taken;
        __syncwarp();           // read by all lanes: the next copies may overwrite it
        const int more = n - at - kBulkStages * GE;
        if (more > 0) issue(k + kBulkStages < 32 / GE ? now : next, (k + kBulkStages) & (32 / GE - 1), more);
#pragma unroll
        for (int q = 0; q < GE; ++q) {
          if (q >= cnt) break;
#pragma unroll
          for (int i = 0; i < VPL; ++i) {
            if constexpr (kWeights) acc[i].fma(v[q][i], wt[q][i]);
            else acc[i].add(v[q][i]);
          }
          if (now.last >> (k * GE + q) & 1u) {
            const int unit = __shfl_sync(0xffffffffu, now.unit, k * GE + q);
            const int row = __shfl_sync(0xffffffffu, d, unit), p = __shfl_sync(0xffffffffu, part, unit);
            if (p < 0) write(row);
            else write_part(row, p, __shfl_sync(0xffffffffu, b, unit));
#pragma unroll
            for (int i = 0; i < VPL; ++i) acc[i].zero();
          }
        }
      }
      now = next;
    }
    return true;
  };

  // Items are dealt from the last warp on, since the first rows, often the longest, are the first warps', while an item is
  // a large part of a warp's edges: 16 000 x 15 edges, fp32 x 256, reverse 56 -> 46 us; with weights 160 -> 156. Plain sums
  // of a million edges keep the other order (125 against 128 us).
  const bool from_last = kWeights || a.num_edges < (int64_t)2 * kItemEdges * warps;
  bool ok = true;
#pragma unroll 1
  for (int64_t first = from_last ? warps - 1 - warp : warp; first < num_items && ok; first += (int64_t)32 * warps) {
    const int64_t it = first + (int64_t)lane * warps;
    const int4 m = it < num_items ? a.ws.items[it] : make_int4(0, 0, 0, -1);
    ok = run(m.y, m.z - m.y, m.x, m.w);
  }
#pragma unroll 1
  for (int64_t first = warp; first < num_rows && ok; first += (int64_t)32 * warps) {
    const int64_t d = first + (int64_t)lane * warps;
    int b = 0, len = 0;
    bool empty = false;
    if (d < num_rows) {
      if (mode == kFixed) {
        b = (int)d * fixed;
        len = fixed;
      } else {
        const int2 r = none ? make_int2(0, 0) : a.ws.range[d];
        b = r.x;
        len = r.y - r.x;
      }
      empty = len == 0;
      if (mode == kOrder && len > a.split.long_edges) len = 0;     // in items
    }
    for (unsigned m = __ballot_sync(0xffffffffu, empty); m; m &= m - 1) write(__shfl_sync(0xffffffffu, (int)d, __ffs(m) - 1));
    ok = run(b, len, (int)d, -1);
  }
  if (ok) return;
  // waited in vain: zeros for all of this warp's rows, and a flag
  ring.drain();
#pragma unroll
  for (int i = 0; i < VPL; ++i) acc[i].zero();
#pragma unroll 1
  for (int64_t it = from_last ? warps - 1 - warp : warp; it < num_items; it += warps) write(a.ws.items[it].x);
#pragma unroll 1
  for (int64_t d = warp; d < num_rows; d += warps)
    if (mode != kOrder || a.ws.range[d].y - a.ws.range[d].x <= a.split.long_edges) write((int)d);
  if (lane != 0) return;
  if (a.status) atomicOr(a.status, APT_FLAG_COPY_TIMEOUT);
  else *pending = APT_FLAG_COPY_TIMEOUT;
}

// Wide rows of many edges: see the top of the file.
template <typename T, int OP>
static int launch_bulk(const RowArgs<T>& a, cudaStream_t s, bool* taken) {
  const int64_t nvec = a.feat_dim / a.split.ve;
  *taken = a.split.ve * (int)sizeof(T) == 16 && nvec >= kBulkMinSlices && nvec <= 32 * kBulkVpl && a.num_edges >= kBulkMinEdges &&
           (OP != kUMulW || (a.mode == kOrder && a.edata_dim <= kBulkHeads));
  if (!*taken) return APT_OK;
  constexpr int smem = kBulkWarps * kBulkStages * bulk_group(OP) * (kBulkSlot + (OP == kUMulW ? kBulkHeads * 4 : 0));
  static bool sized[64] = {};
  int dev = 0;
  APT_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !sized[dev]) {
    APT_CUDA(cudaFuncSetAttribute(k_spmm_bulk<T, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (dev < 64) sized[dev] = true;
  }
  int32_t* pending = nullptr;
  if (!a.status) {
    const int rc = pending_word(&pending);
    if (rc != APT_OK) return rc;
  }
  const int64_t want = ceil_div(a.num_rows, kBulkWarps), wave = (int64_t)kNumSMs * bulk_blocks(OP);
  APT_FOLLOW((k_spmm_bulk<T, OP>), (int)(want < wave ? want : wave), kBulkWarps * 32, smem, s, a, bulk_wait_polls(),
             (volatile int32_t*)pending);
  return APT_OK;
}

}  // namespace apt
