// Segment-batched COO SpMM (sum reduce) and SDDMM over sampled blocks: entry points, the probe that
// looks a block over and the counting sort that groups its edges by output row. The sums themselves
// are in spmm_rows.cuh.
//
// A block is looked over by one kernel (k_spmm_probe): are its edges grouped by output row, does
// every row have the same number of edges, does any row have very many. apt_spmm_probe hands the answer
// to the host together with the number of output rows, which the host has to read anyway before it can
// allocate the result: the kernel stores both in mapped host memory, where the host polls for them. The
// call behind it (apt_spmm_sum_known) then launches what the block needs and nothing else: one kernel
// for a sampled block. apt_spmm_sum, for callers that may not wait, leaves the answer on the device and
// enqueues every preparing kernel; those the block does not need return at once.
#include <math.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <mutex>

#include "spmm_rows.cuh"

namespace apt {

size_t spmm_layout(int64_t num_rows, int64_t num_edges, char* base, SpmmWs* ws, int slot_bytes) {
  const int64_t rows = num_rows > 0 ? num_rows : 1, edges = num_edges > 0 ? num_edges : 1;
  // a row handed to whole warps has more than kLongRowNarrow edges and becomes at most edges / kItemEdges + 1 items;
  // rows of several items have more than kItemEdges
  const int64_t max_items = num_edges / kItemEdges + num_edges / kLongRowNarrow + 1;
  const int64_t max_parts = 2 * (num_edges / kItemEdges) + 1;
  const int64_t part_floats = part_room(num_edges);
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at += align_up(bytes, 256);
    return o;
  };
  const size_t o_words = take(64);
  const size_t o_cnt = take((size_t)spread_rows(rows) * 4);
  const size_t o_done = take((size_t)max_parts * 4);
  const size_t zero = at;
  const size_t o_range = take((size_t)(rows + 1) * 8);
  const size_t o_rank = take((size_t)edges * 4);
  const size_t o_order = take((size_t)edges * slot_bytes);
  const size_t o_items = take((size_t)max_items * 16);
  const size_t o_part = take((size_t)part_floats * 4);
  if (ws) {
    ws->result = (int64_t*)(base + o_words);
    ws->probe = (unsigned long long*)(base + o_words + 8);
    ws->num_items = (int32_t*)(base + o_words + 16);
    ws->num_slots = (int32_t*)(base + o_words + 20);
    ws->num_parts = (int32_t*)(base + o_words + 24);
    ws->cnt = (int32_t*)(base + o_cnt);
    ws->part_done = (int32_t*)(base + o_done);
    ws->zero_bytes = zero;
    ws->range = (int2*)(base + o_range);
    ws->rank = (uint32_t*)(base + o_rank);
    ws->order = (uint2*)(base + o_order);
    ws->items = (int4*)(base + o_items);
    ws->part = (float*)(base + o_part);
    ws->max_items = max_items;
    ws->max_parts = max_parts;
    ws->part_floats = part_floats;
  }
  return at;
}

// ---- the probe -------------------------------------------------------------------------
constexpr uint32_t kNotGrouped = 1u, kNotFixed = 2u, kHasLong = 4u;

__device__ __forceinline__ int64_t out_row(const int64_t* coo, const int64_t* ooff, int nseg, const int64_t* col, int64_t e) {
  return ooff[nseg > 1 ? seg_of(coo, nseg, e) : 0] + col[e];
}

// One 64-bit word collects the blocks' answers: blocks done, how many of them saw each of the three (10 bits each), and pairs of one row (24). The add that
// counts a block also returns what the others saw, so the last block has the answer without a fence or a second
// read (fence, counter and read in turn: 5.6 -> 4.5 us for 10 240 edges). The word, `agg` or the slot's own, is zero before
// and after; `result` may be mapped host memory.
constexpr int kProbeSlots = 64;
constexpr unsigned long long kVoteMask = 1023, kMostPairs = 16383;      // pairs a block adds at most
static_assert(kNumSMs * 4 < (int)kVoteMask && (unsigned long long)kNumSMs * 4 * kMostPairs < 1ull << 24, "votes of a wave of four blocks an SM");
__device__ unsigned long long g_probe_votes[kProbeSlots];
__device__ __forceinline__ unsigned long long probe_votes(uint32_t bits, uint32_t pairs) {
  return 1ull | (bits & kNotGrouped ? 1ull << 10 : 0ull) | (bits & kNotFixed ? 1ull << 20 : 0ull) | (bits & kHasLong ? 1ull << 30 : 0ull) |
         min((unsigned long long)pairs, kMostPairs) << 40;
}

// Rows with many of the edges (`count_pairs`): of edges in no order, how many of the pairs that a warp's first 32 edges make are of one row. All rows
// alike, that is one pair in as many as there are rows; kHubs times as many, and rows of far more edges than
// the mean take part (the source of a draw at u^1.5 of the range 1.4 times, at u^2 3.2, at u^3 25 and more). 100 000 edges make 390 000 pairs, 600 000 and more
// 2.3 million. It takes a call 0.3 to 1.1 us. (Two rounds of every warp, a million edges: 12.4 us for this kernel instead of 8, the match takes its unit
// a while.)
constexpr int kHubs = 2;

// num_rows: the output rows there are (the caller's result may have more, or fewer, than the offsets end at); -1: as the offsets say.
// K edges a thread at a time: four, eight where more than one wave of four would be needed (1.01 M edges 8.1 -> 7 us).
template <int K>
__global__ void __launch_bounds__(256)
k_spmm_probe(const int64_t* __restrict__ col, int64_t E, SegTable st, int64_t num_rows, unsigned long long* agg, int slot,
             volatile int64_t* result, int64_t sequence, int count_pairs) {
  wait_for_previous();
  if (!agg) agg = g_probe_votes + slot;
  __shared__ int64_t coo[kMaxSegments + 1], ooff[kMaxSegments + 1];
  __shared__ uint32_t s_bits, s_pairs;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t e0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, c[K];
  auto fetch = [&]() {
#pragma unroll
    for (int k = 0; k < K; ++k) c[k] = e0 + k * stride < E ? col[e0 + k * stride] : 0;
  };
  fetch();     // on its way while the offsets are
  for (int t = threadIdx.x; t <= st.nseg; t += blockDim.x) {
    coo[t] = st.coo_off[t];
    ooff[t] = st.out_off[t];
  }
  if (threadIdx.x == 0) s_bits = s_pairs = 0u;
  __syncthreads();
  if (count_pairs) {
    const bool there = e0 < E;
    const unsigned all = __ballot_sync(0xffffffffu, there);
    // (edges that do not fall are likely to be grouped, which asks for no pairs)
    const int64_t before = __shfl_up_sync(0xffffffffu, c[0], 1);
    if (__any_sync(0xffffffffu, there && (threadIdx.x & 31) && c[0] < before)) {
      const uint32_t pairs = __reduce_add_sync(0xffffffffu, there ? __popc(__match_any_sync(all, (unsigned)c[0])) - 1 : 0);      // each of them twice
      if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(&s_pairs, pairs / 2);
    }
  }
  const int64_t rows = num_rows >= 0 ? num_rows : ooff[st.nseg];
  // the one fanout that fits the sizes
  const uint32_t f = rows > 0 && E % rows == 0 ? (uint32_t)(E / rows) : 0u;
  uint32_t bits = f ? 0u : kNotFixed;
  // edges that are not grouped need the counting sort whatever the others are
  while (e0 < E && !(bits & kNotGrouped)) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t e = e0 + k * stride;
      if (e >= E || (bits & kNotGrouped)) break;
      const int64_t d = ooff[st.nseg > 1 ? seg_of(coo, st.nseg, e) : 0] + c[k];
      if (f && d == (int64_t)((uint32_t)e / f)) continue;
      bits |= kNotFixed;
      const int64_t prev = e > 0 ? out_row(coo, ooff, st.nseg, col, e - 1) : (int64_t)-1;
      if (d < prev || d < 0 || d >= rows) bits |= kNotGrouped;
      // the next edge may match the fanout and then does not look back itself
      if (e + 1 < E && out_row(coo, ooff, st.nseg, col, e + 1) < d) bits |= kNotGrouped;
      // a run of kLongRun edges covers two neighbouring multiples of half that length
      if (e % (kLongRun / 2) == 0 && e >= kLongRun / 2 && out_row(coo, ooff, st.nseg, col, e - kLongRun / 2) == d)
        bits |= kHasLong;
    }
    e0 += K * stride;
    if (e0 < E) fetch();
  }
  bits = __reduce_or_sync(0xffffffffu, bits);
  if ((threadIdx.x & 31) == 0 && bits) atomicOr(&s_bits, bits);
  __syncthreads();
  if (threadIdx.x != 0) return;
  unsigned long long all = probe_votes(s_bits, s_pairs);
  if (gridDim.x > 1) {
    all += atomicAdd(agg, all);
    if ((all & kVoteMask) != gridDim.x) return;
    atomicExch(agg, 0ull);
  }
  const bool fixed = !(all >> 20 & kVoteMask), grouped = !(all >> 10 & kVoteMask), has_long = (all >> 30 & kVoteMask) != 0;
  const bool fits = rows >= 0 && rows < 0x7fffffff;
  // 32 edges make 496 pairs; a warp's are of one segment, whose rows are taken to be as many as the others'
  const int64_t looked_at = min(E, (int64_t)gridDim.x * 256);
  const bool hubs = count_pairs && fits && (int64_t)(all >> 40) * 2 * rows >= looked_at * 31 * kHubs * st.nseg;
  *result = probe_pack(fits ? rows : 0, !fits ? 3 : fixed ? kFixed : !grouped || has_long ? kOrder : kRanges, hubs, sequence);
}

static int launch_probe(const int64_t* col, int64_t E, SegTable st, int64_t num_rows, unsigned long long* agg, int slot,
                        int64_t* result, int64_t sequence, bool count_pairs, cudaStream_t s) {
  // a thousand edges a block and one wave at most: small blocks of edges are looked over by one thread block
  const int grid = wave_grid(ceil_div(E, 1024), 4, 1);
  ProfScope prof("spmm_ranges", s);
  if (E > (int64_t)grid * 256 * 4)
    APT_FOLLOW(k_spmm_probe<8>, grid, 256, 0, s, col, E, st, num_rows, agg, slot, (volatile int64_t*)result, sequence, (int)count_pairs);
  else
    APT_FOLLOW(k_spmm_probe<4>, grid, 256, 0, s, col, E, st, num_rows, agg, slot, (volatile int64_t*)result, sequence, (int)count_pairs);
  return APT_OK;
}

// Where probes leave their answers for the host: a fixed number of slots, each taken by one call and given
// back before it returns, so that calls of several threads and streams do not meet.
struct ProbeSlots {
  std::mutex mu;
  std::condition_variable cv;
  int64_t* host = nullptr;            // mapped: 8 words a slot
  uint64_t taken = 0;
  int64_t sequence = 0;
};
static ProbeSlots g_probe;

static int take_slot(int* slot, int64_t* sequence) {
  std::unique_lock<std::mutex> lk(g_probe.mu);
  if (!g_probe.host) {
    void* p = nullptr;
    RelaxedCapture relaxed;
    APT_CUDA(cudaHostAlloc(&p, kProbeSlots * 64, cudaHostAllocMapped | cudaHostAllocPortable));
    g_probe.host = (int64_t*)p;
    for (int k = 0; k < kProbeSlots * 8; ++k) g_probe.host[k] = 0;
  }
  g_probe.cv.wait(lk, [] { return g_probe.taken != ~0ull; });
  *slot = __builtin_ctzll(~g_probe.taken);
  g_probe.taken |= 1ull << *slot;
  *sequence = ++g_probe.sequence & kProbeSequences;
  return APT_OK;
}

static void give_slot(int slot) {
  {
    std::lock_guard<std::mutex> lk(g_probe.mu);
    g_probe.taken &= ~(1ull << slot);
  }
  g_probe.cv.notify_one();
}

// Where kernels without a status word of their caller leave flags: mapped memory, made by the first call that may need it.
static std::atomic<int32_t*> g_pending{nullptr};

int pending_word(int32_t** word) {
  static std::mutex mu;
  *word = g_pending.load(std::memory_order_acquire);
  if (*word) return APT_OK;
  std::lock_guard<std::mutex> lk(mu);
  if (!g_pending.load()) {
    void* p = nullptr;
    RelaxedCapture relaxed;
    APT_CUDA(cudaHostAlloc(&p, 64, cudaHostAllocMapped | cudaHostAllocPortable));
    *(int32_t*)p = 0;
    g_pending.store((int32_t*)p, std::memory_order_release);
  }
  *word = g_pending.load();
  return APT_OK;
}

static int32_t take_pending() {
  int32_t* const word = g_pending.load(std::memory_order_acquire);
  return word && *(volatile int32_t*)word ? __atomic_exchange_n(word, 0, __ATOMIC_ACQ_REL) : 0;
}

// Sums that came out wrong are reported by the next call that sums, whatever its size.
static int check_pending(const char* who) {
  if (!take_pending()) return APT_OK;
  set_error("%s: in an earlier call input rows did not reach shared memory in time; some of its sums are zero", who);
  return APT_ERR_TIMEOUT;
}

static std::atomic<int> g_bulk_wait_polls{kStreamWaitPolls};
void set_bulk_wait_polls(int polls) { g_bulk_wait_polls = polls; }
int bulk_wait_polls() { return g_bulk_wait_polls; }

// Polls a mapped word until it carries `sequence`. The stream is asked now and then, so that an error on it ends the wait.
static int wait_for(const volatile int64_t* word, int64_t sequence, cudaStream_t s) {
  for (int64_t spin = 1;; ++spin) {
    if (probe_sequence(*word) == sequence) break;
    if ((spin & 0x3fff) == 0) {
      RelaxedCapture relaxed;
      const cudaError_t e = cudaStreamQuery(s);
      if (e == cudaErrorNotReady) continue;
      APT_CUDA(e);
      if (probe_sequence(*word) == sequence) break;
      set_error("apt_spmm_probe: the stream is idle and the probe has not answered");
      return APT_ERR_TIMEOUT;
    }
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
  }
  return APT_OK;
}

// ---- where a row's edges are ---------------------------------------------------------------
__device__ __forceinline__ int resolve_mode(int mode, const SpmmWs& ws) {
  return mode == kDevice ? probe_mode(*ws.result) : mode;
}

// Grouped edges: the edge that opens a row closes the one before and leaves the rows in between empty.
__global__ void __launch_bounds__(256)
k_edge_ranges(const int64_t* __restrict__ col, int64_t E, SegTable st, int64_t num_rows, SpmmWs ws, int mode) {
  wait_for_previous();
  if (resolve_mode(mode, ws) != kRanges) return;
  __shared__ int64_t coo[kMaxSegments + 1], ooff[kMaxSegments + 1];
  for (int t = threadIdx.x; t <= st.nseg; t += blockDim.x) {
    coo[t] = st.coo_off[t];
    ooff[t] = st.out_off[t];
  }
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) {
    const int64_t d = out_row(coo, ooff, st.nseg, col, e);
    // the probe has seen that no edge is out of order or of no row; where it has not been asked, nothing is written outside the table
    const int64_t prev = e > 0 ? max(out_row(coo, ooff, st.nseg, col, e - 1), (int64_t)-1) : (int64_t)-1;
    if (d < prev || d < 0 || d >= num_rows) continue;
    if (d != prev) {
      if (prev >= 0) ws.range[prev].y = (int)e;
      for (int64_t t = prev + 1; t < d; ++t) ws.range[t] = make_int2(0, 0);
      ws.range[d].x = (int)e;
    }
    if (e == E - 1) {
      ws.range[d].y = (int)E;
      for (int64_t t = d + 1; t < num_rows; ++t) ws.range[t] = make_int2(0, 0);
    }
  }
}

// Counting sort by output row. The add that counts an edge also returns its place inside its row, so the pass
// that writes the order needs no second round of atomics (1.01 M edges: 25 + 28 us with one in both passes).
__global__ void __launch_bounds__(256)
k_dst_rank(const int64_t* __restrict__ col, int64_t E, SegTable st, int64_t num_rows, SpmmWs ws, int mode) {
  wait_for_previous();
  if (resolve_mode(mode, ws) != kOrder) return;
  __shared__ int64_t coo[kMaxSegments + 1], ooff[kMaxSegments + 1];
  for (int t = threadIdx.x; t <= st.nseg; t += blockDim.x) {
    coo[t] = st.coo_off ? st.coo_off[t] : 0;
    ooff[t] = st.out_off ? st.out_off[t] : 0;
  }
  __syncthreads();
  constexpr int K = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e0 < E; e0 += K * stride) {
    int64_t d[K];
    uint32_t r[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t e = e0 + k * stride;
      d[k] = e < E ? out_row(coo, ooff, st.nseg, col, e) : (int64_t)-1;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) r[k] = d[k] >= 0 && d[k] < num_rows ? (uint32_t)atomicAdd(ws.cnt + spread((uint32_t)d[k]), 1) : kNoRank;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (e0 + k * stride < E) ws.rank[e0 + k * stride] = r[k];
  }
}

// The items of a row of n edges from slot `at` on.
__device__ __forceinline__ void leave_items(const SpmmWs& ws, int d, int at, int n, int part_stride) {
  int size = item_edges(n), parts = (n + size - 1) / size, part = -1;
  if (parts > 1) {
    part = atomicAdd(ws.num_parts, parts);
    if (part + parts > ws.max_parts || (int64_t)(part + parts) * part_stride > ws.part_floats) {
      part = -1;         // no room for partial sums: one item
      parts = 1;
      size = n;
    }
  }
  const int base = atomicAdd(ws.num_items, parts);
  for (int p = 0; p < parts; ++p) ws.items[base + p] = make_int4(d, at + p * size, at + min((p + 1) * size, n), part < 0 ? -1 : part + p);
}

// Rows to slots. The rows' shares of order[] need not follow one another, so a block takes the room for its
// rows with one add and no block waits for another. Long rows leave their items.
constexpr int kScanRows = 4;
__global__ void __launch_bounds__(256)
k_dst_slots(int64_t num_rows, SpmmWs ws, int mode, OrderKind kind, int long_edges, int part_stride) {
  wait_for_previous();
  if (resolve_mode(mode, ws) != kOrder) return;
  __shared__ int scratch[33];
  __shared__ int s_base;
  const int64_t first = ((int64_t)blockIdx.x * 256 + threadIdx.x) * kScanRows;
  int v[kScanRows], mine = 0;
#pragma unroll
  for (int k = 0; k < kScanRows; ++k) {
    v[k] = first + k < num_rows ? ws.cnt[spread((uint32_t)(first + k))] : 0;
    mine += v[k];
  }
  int total;
  const int ex = block_exclusive_scan(mine, scratch, &total);
  if (threadIdx.x == 0) s_base = atomicAdd(ws.num_slots, total);
  __syncthreads();
  int at = s_base + ex;
#pragma unroll
  for (int k = 0; k < kScanRows; ++k) {
    const int64_t d = first + k;
    if (d >= num_rows) break;
    ws.range[d] = make_int2(at, at + v[k]);
    if (kind == kByEdge && v[k] > long_edges) leave_items(ws, (int)d, at, v[k], part_stride);
    at += v[k];
  }
}

__global__ void __launch_bounds__(256)
k_dst_fill(const int64_t* __restrict__ row, const int64_t* __restrict__ col, int64_t E, SegTable st, SpmmWs ws, int mode, OrderKind kind) {
  wait_for_previous();
  if (resolve_mode(mode, ws) != kOrder) return;
  __shared__ int64_t coo[kMaxSegments + 1], ooff[kMaxSegments + 1], ioff[kMaxSegments + 1];
  for (int t = threadIdx.x; t <= st.nseg; t += blockDim.x) {
    coo[t] = st.coo_off ? st.coo_off[t] : 0;
    ooff[t] = st.out_off ? st.out_off[t] : 0;
    ioff[t] = st.in_off ? st.in_off[t] : 0;
  }
  __syncthreads();
  constexpr int K = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e0 < E; e0 += K * stride) {
    uint32_t r[K];
    uint2 o[K];
    int64_t d[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t e = e0 + k * stride;
      r[k] = e < E ? ws.rank[e] : kNoRank;
      if (r[k] == kNoRank) continue;
      const int seg = st.nseg > 1 ? seg_of(coo, st.nseg, e) : 0;
      d[k] = ooff[seg] + col[e];
      o[k] = make_uint2((uint32_t)(ioff[seg] + row[e]), (uint32_t)(kind == kByRow ? d[k] : e));
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (r[k] != kNoRank) r[k] += (uint32_t)ws.range[d[k]].x;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (r[k] != kNoRank) ws.order[r[k]] = o[k];
  }
}

// The whole sort of a small block of edges in one launch: a thread block to a range of rows goes through all edges, keeps those of its rows,
// a warp at a time, in lists and counts them in shared memory, and writes their places; the edges of rows before its own, which it counts
// on the way, tell where they begin. Two launches less than the passes above and no atomics on memory, for reading the edges once per block. us of a
// forward and a reverse sum: 900 edges 47 -> 42, 2 000 48 -> 43, 8 000 49 -> 45.5, 16 000 in eight segments 53 -> 48.5, in one 52 -> 50.5; with lists for
// 41 000 edges 55 -> 59 (each block then goes through edges for 17 us). The line lies at what a warp's list holds.
constexpr int kSmallSortThreads = 1024, kSmallSortRows = 8192, kSmallSortBlocks = 64;
constexpr int kSmallSortList = 512;      // of a warp: as many edges as it goes through
constexpr int64_t kSmallSortEdges = kSmallSortThreads / 32 * kSmallSortList;
constexpr size_t kSmallSortShared = kSmallSortRows * 4 + kSmallSortEdges * 8;

__global__ void __launch_bounds__(kSmallSortThreads)
k_dst_small(const int64_t* __restrict__ row, const int64_t* __restrict__ col, int E, SegTable st, int64_t num_rows, int per_block, SpmmWs ws,
            int long_edges, int part_stride) {
  wait_for_previous();
  constexpr int K = 8, U = 4;
  extern __shared__ __align__(16) unsigned char small_sort[];
  int* const cnt = (int*)small_sort;
  __shared__ int64_t coo[kMaxSegments + 1], ooff[kMaxSegments + 1], ioff[kMaxSegments + 1];
  __shared__ int scratch[33], s_below;
  for (int t = threadIdx.x; t <= st.nseg; t += kSmallSortThreads) {
    coo[t] = st.coo_off[t];
    ooff[t] = st.out_off[t];
    ioff[t] = st.in_off ? st.in_off[t] : 0;
  }
  const int lo = blockIdx.x * per_block, rows = (int)min((int64_t)per_block, num_rows - lo), lane = threadIdx.x & 31;
  uint2* const list = (uint2*)(small_sort + kSmallSortRows * 4) + (threadIdx.x >> 5) * kSmallSortList;      // (edge, row << 16 | place in its row)
  for (int t = threadIdx.x; t < rows; t += kSmallSortThreads) cnt[t] = 0;
  if (threadIdx.x == 0) s_below = 0;
  __syncthreads();
  int below = 0, seg = 0, kept = 0;
  for (int e0 = threadIdx.x & ~31; e0 < E; e0 += K * kSmallSortThreads) {      // (whole warps)
    int64_t c[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = e0 + lane + k * kSmallSortThreads;
      c[k] = e < E ? __ldg(col + e) : 0;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int e = e0 + lane + k * kSmallSortThreads;
      while (seg + 1 < st.nseg && coo[seg + 1] <= e) ++seg;      // (edges rise)
      const int64_t g = ooff[seg] + c[k];
      const bool is = e < E && (uint64_t)g < (uint64_t)num_rows;
      const int d = (int)g - lo;
      below += is && d < 0;
      const bool mine = is && (uint32_t)d < (uint32_t)rows;
      const unsigned all = __ballot_sync(0xffffffffu, mine);
      if (mine) list[kept + __popc(all & ((1u << lane) - 1u))] = make_uint2((uint32_t)e, (uint32_t)d << 16 | (uint32_t)atomicAdd(cnt + d, 1));
      kept += __popc(all);
    }
  }
  below = __reduce_add_sync(0xffffffffu, below);
  if (lane == 0) atomicAdd(&s_below, below);
  __syncthreads();
  // counts to places
  const int each = (rows + kSmallSortThreads - 1) / kSmallSortThreads, first = threadIdx.x * each, last = min(rows, first + each);
  int sum = 0, total;
  for (int t = first; t < last; ++t) sum += cnt[t];
  int at = s_below + block_exclusive_scan(sum, scratch, &total);
  for (int t = first; t < last; ++t) {
    const int n = cnt[t];
    cnt[t] = at;
    ws.range[lo + t] = make_int2(at, at + n);
    if (n > long_edges) leave_items(ws, lo + t, at, n, part_stride);
    at += n;
  }
  __syncthreads();
  for (int t0 = lane; t0 < kept; t0 += 32 * U) {
    uint2 x[U];
    int64_t from[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (t0 + u * 32 >= kept) continue;
      x[u] = list[t0 + u * 32];
      from[u] = row[x[u].x];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (t0 + u * 32 >= kept) continue;
      const int64_t in = ioff[st.nseg > 1 ? seg_of(coo, st.nseg, x[u].x) : 0] + from[u];
      ws.order[cnt[x[u].y >> 16] + (int)(x[u].y & 0xffffu)] = make_uint2((uint32_t)in, x[u].x);
    }
  }
}

static bool small_sort_fits(int64_t num_edges, int64_t num_rows, OrderKind kind) {
  return kind == kByEdge && num_edges <= kSmallSortEdges && num_rows <= (int64_t)kSmallSortBlocks * kSmallSortRows;
}
static int launch_small_sort(const int64_t* row, const int64_t* col, int64_t num_edges, SegTable st, int64_t num_rows, const SpmmWs& ws,
                             int long_edges, int part_stride, cudaStream_t s) {
  static bool sized[64] = {};
  int dev = 0;
  APT_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !sized[dev]) {
    APT_CUDA(cudaFuncSetAttribute(k_dst_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSortShared));
    if (dev < 64) sized[dev] = true;
  }
  ProfScope prof("spmm_group", s);
  const int64_t per = std::max<int64_t>(64, ceil_div(num_rows, kSmallSortBlocks));
  APT_FOLLOW(k_dst_small, (int)ceil_div(num_rows, per), kSmallSortThreads, kSmallSortShared, s, row, col, (int)num_edges, st, num_rows, (int)per, ws,
             long_edges, part_stride);
  return APT_OK;
}

int launch_slots(int64_t num_rows, const SpmmWs& ws, int mode, OrderKind kind, int long_edges, int part_stride, cudaStream_t s) {
  APT_FOLLOW(k_dst_slots, (int)ceil_div(num_rows, 256 * kScanRows), 256, 0, s, num_rows, ws, mode, kind, long_edges, part_stride);
  return APT_OK;
}

static int launch_group(const int64_t* row, const int64_t* col, int64_t num_edges, SegTable st, int64_t num_rows, const SpmmWs& ws, int mode,
                        OrderKind kind, int long_edges, int part_stride, cudaStream_t s) {
  ProfScope prof("spmm_group", s);
  const int ge = wave_grid(ceil_div(num_edges, 256 * 4), 8, 1);
  APT_FOLLOW(k_dst_rank, ge, 256, 0, s, col, num_edges, st, num_rows, ws, mode);
  const int rc = launch_slots(num_rows, ws, mode, kind, long_edges, part_stride, s);
  if (rc != APT_OK) return rc;
  APT_FOLLOW(k_dst_fill, ge, 256, 0, s, row, col, num_edges, st, ws, mode, kind);
  return APT_OK;
}

// ---- SDDMM -------------------------------------------------------------------------
// A warp takes a chunk of edges, a lane to each to find its two rows, whose addresses go to shared memory. In the result the chunk is one run of
// slices, which the warp makes from end to end, U of 32 lanes each in flight (k_gather's way). A group of lanes to an edge, which left the lanes
// beside 47 columns idle and kept its slices unpacked -> here, us: products of 900 000 edges x 256 bf16 355 -> 123 (0.46 GB written), x 32 41 -> 19, 187 000 x 47
// bf16 27 -> 12, 150 000 x 64 fp32 16 -> 9.7, 61 000 x 64 fp32 7.8 -> 5.5; sums of scores of 61 000 x 4 fp32 3.7 -> 2.9.
constexpr int kSddmmSlices = 4, kSddmmBytes = 4096, kSddmmEdges = 128;
// ONE: a slice to an edge, whose lane then finds its rows for itself.
template <typename T, int VE, int OP, bool ONE>
__global__ void __launch_bounds__(256)
k_sddmm(const int64_t* __restrict__ row, const int64_t* __restrict__ col, int64_t E,
        const T* __restrict__ lhs, const T* __restrict__ rhs, int64_t feat_dim,
        SegTable st, const int64_t* __restrict__ rhs_off, T* __restrict__ out, uint32_t slices, uint32_t inverse, int per_chunk) {
  wait_for_previous();
  constexpr int U = kSddmmSlices;
  __shared__ int64_t coo[kMaxSegments + 1], loff[kMaxSegments + 1], roff[kMaxSegments + 1];
  __shared__ const T* sides[8][kSddmmEdges][2];
  for (int t = threadIdx.x; t <= st.nseg; t += blockDim.x) {
    coo[t] = st.coo_off[t];
    loff[t] = st.in_off[t];
    roff[t] = rhs_off[t];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const T*(*const side)[2] = sides[threadIdx.x >> 5];
  const int64_t step = (int64_t)gridDim.x * 8 * per_chunk;
  for (int64_t e0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * per_chunk; e0 < E; e0 += step) {
    const int edges = (int)min((int64_t)per_chunk, E - e0);
    if (!ONE) __syncwarp();      // (the chunk before has been read)
#pragma unroll
    for (int q = 0; q < kSddmmEdges && !ONE; q += 32) {
      if (q + lane >= edges) break;
      const int64_t e = e0 + q + lane;
      const int k = st.nseg > 1 ? seg_of(coo, st.nseg, e) : 0;
      side[q + lane][0] = lhs + (loff[k] + row[e]) * feat_dim;
      side[q + lane][1] = rhs + (roff[k] + col[e]) * feat_dim;
    }
    if (!ONE) __syncwarp();
    const uint32_t total = (uint32_t)edges * slices;
    T* const dst = out + e0 * feat_dim + lane * VE;
    for (uint32_t i0 = 0; i0 < total; i0 += 32 * U) {
      Raw<T, VE> a[U], b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t i = i0 + u * 32 + lane;
        if (i >= total) continue;
        if constexpr (ONE) {
          const int64_t e = e0 + i;
          const int k = st.nseg > 1 ? seg_of(coo, st.nseg, e) : 0;
          a[u] = load_raw<T, VE>(lhs + (loff[k] + row[e]) * VE);
          b[u] = load_raw<T, VE>(rhs + (roff[k] + col[e]) * VE);
        } else {
          const uint32_t e = __umulhi(2 * i + 1, inverse), c = (i - e * slices) * VE;
          a[u] = load_raw<T, VE>(side[e][0] + c);
          b[u] = load_raw<T, VE>(side[e][1] + c);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (i0 + u * 32 + lane >= total) continue;
        Pack<T, VE> o;
#pragma unroll
        for (int t = 0; t < VE; ++t) {
          const float x = a[u].get(t), y = b[u].get(t);
          o.v[t] = Elem<T>::from_f(OP == 0 ? x + y : x * y);
        }
        store_pack<T, VE>(dst + (i0 + u * 32) * VE, o);
      }
    }
  }
}

template <typename T, int VE>
static int launch_sddmm(int op, const int64_t* row, const int64_t* col, int64_t E,
                        const T* lhs, const T* rhs, int64_t feat_dim, SegTable st,
                        const int64_t* rhs_off, T* out, cudaStream_t s) {
  ProfScope prof("sddmm", s);
  // one edge of wide rows, else as many as fill the lanes or, while every warp of the chip has them, take kSddmmBytes
  const int64_t slices = feat_dim / VE, bytes = feat_dim * (int64_t)sizeof(T);
  int per = 1;
  while (per < kSddmmEdges && ((per < 32 && per * slices < 32) || ((int64_t)per * kNumSMs * 64 < E && (per < 32 ? 2 * per * bytes <= kSddmmBytes : per * slices < 32 * kSddmmSlices))))
    per <<= 1;
  // the edge of slice i: exact while i < 2^18 and slices < 2^12 (k_gather); edges that share a chunk have 2048 slices or fewer together
  const uint32_t inverse = per > 1 ? (uint32_t)(((1ull << 31) + slices - 1) / slices) : 0u;
  const int grid = wave_grid(ceil_div(E, (int64_t)per * 8), 8);
#define APT_SDDMM(OP, ONE) APT_FOLLOW((k_sddmm<T, VE, OP, ONE>), grid, 256, 0, s, row, col, E, lhs, rhs, feat_dim, st, rhs_off, out, (uint32_t)slices, inverse, per)
  if (op == 0) {
    if (slices == 1) APT_SDDMM(0, true); else APT_SDDMM(0, false);
  } else {
    if (slices == 1) APT_SDDMM(1, true); else APT_SDDMM(1, false);
  }
#undef APT_SDDMM
  return APT_OK;
}

template <typename T>
static int dispatch_sddmm(int op, int ve, const int64_t* row, const int64_t* col, int64_t E,
                          const void* lhs, const void* rhs, int64_t feat_dim, SegTable st,
                          const int64_t* rhs_off, void* out, cudaStream_t s) {
  switch (ve * (int)sizeof(T)) {
    case 16: return launch_sddmm<T, 16 / sizeof(T)>(op, row, col, E, (const T*)lhs, (const T*)rhs, feat_dim, st, rhs_off, (T*)out, s);
    case 8: return launch_sddmm<T, 8 / sizeof(T)>(op, row, col, E, (const T*)lhs, (const T*)rhs, feat_dim, st, rhs_off, (T*)out, s);
    case 4: return launch_sddmm<T, 4 / sizeof(T)>(op, row, col, E, (const T*)lhs, (const T*)rhs, feat_dim, st, rhs_off, (T*)out, s);
    default: return launch_sddmm<T, 1>(op, row, col, E, (const T*)lhs, (const T*)rhs, feat_dim, st, rhs_off, (T*)out, s);
  }
}

static size_t elem_size(int dtype) { return dtype == APT_F32 ? 4 : 2; }

template <typename T>
static int run_rows(int op, const RowSplit& split, const int64_t* row, const int64_t* col, int64_t E, const void* in, const void* edata,
                    int64_t edata_dim, int64_t feat_dim, SegTable st, int64_t num_rows, const SpmmWs& ws, int mode, int fixed,
                    void* out, int64_t width, cudaStream_t s) {
  const RowArgs<T> a{row, (const T*)in, (const T*)edata, edata_dim, feat_dim, st, num_rows, E, ws, (T*)out,
                     mode, fixed, split, (int)feat_dim, Verdict{}, nullptr, col, nullptr, nullptr, 0u, width};
  ProfScope prof("spmm_rows", s);
  return launch_spmm_rows<T>(op, a, s);
}

// Everything behind the argument checks; mode kDevice: nothing is known about the block yet. `width`: RowArgs (no slice of the result is
// aligned then, and the input is).
static int spmm_run(int op, int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t E, const void* input,
                    const void* edata, int64_t edata_dim, int64_t feat_dim, SegTable st, int64_t num_rows, void* out,
                    void* workspace, size_t workspace_bytes, int mode, int fixed, int64_t width, cudaStream_t s) {
  const size_t esz = elem_size(dtype);
  SpmmWs ws{};
  if (mode != kFixed) {
    APT_CHECK_ARG(workspace && ((uintptr_t)workspace & 255) == 0, "apt_spmm_sum: workspace must be 256-byte aligned");
    const size_t need = spmm_layout(num_rows, E, (char*)workspace, &ws);
    if (workspace_bytes < need) {
      set_error("apt_spmm_sum: workspace %zu < %zu bytes", workspace_bytes, need);
      return APT_ERR_CAPACITY;
    }
  }
  // edge values are read in slices only when there is one per column
  uint64_t bits = (uint64_t)(feat_dim * esz) | (width ? 0 : (uintptr_t)out);
  if (op != kCopyE) bits |= (uintptr_t)input;
  if (op != kCopyU && edata_dim == feat_dim) bits |= (uintptr_t)edata;
  const RowSplit split = row_split(feat_dim, slice_elems(bits, (int)esz), E, num_rows, mode == kOrder || mode == kDevice);
  if (mode == kDevice || mode == kOrder) APT_CUDA(cudaMemsetAsync(workspace, 0, ws.zero_bytes, s));
  if (mode == kDevice) {
    const int rc = launch_probe(coo_col, E, st, num_rows, ws.probe, 0, ws.result, 1, false, s);
    if (rc != APT_OK) return rc;
  }
  if (mode == kDevice || mode == kRanges) {
    ProfScope prof("spmm_ranges", s);
    APT_FOLLOW(k_edge_ranges, wave_grid(ceil_div(E, 256), 8), 256, 0, s, coo_col, E, st, num_rows, ws, mode);
  }
  if (mode == kDevice || mode == kOrder) {
    const OrderKind kind = order_kind(op, split.ve * (int)esz, feat_dim, esz, 1, E);
    const int rc = mode == kOrder && small_sort_fits(E, num_rows, kind)
                       ? launch_small_sort(coo_row, coo_col, E, st, num_rows, ws, split.long_edges, (int)feat_dim, s)
                       : launch_group(coo_row, coo_col, E, st, num_rows, ws, mode, kind, split.long_edges, (int)feat_dim, s);
    if (rc != APT_OK) return rc;
  }
  switch (dtype) {
    case APT_F32: return run_rows<float>(op, split, coo_row, coo_col, E, input, edata, edata_dim, feat_dim, st, num_rows, ws, mode, fixed, out, width, s);
    case APT_BF16: return run_rows<__nv_bfloat16>(op, split, coo_row, coo_col, E, input, edata, edata_dim, feat_dim, st, num_rows, ws, mode, fixed, out, width, s);
    default: return run_rows<__half>(op, split, coo_row, coo_col, E, input, edata, edata_dim, feat_dim, st, num_rows, ws, mode, fixed, out, width, s);
  }
}

static int spmm_check(const char* who, int op, int dtype, int64_t num_edges, int64_t* edata_dim, int64_t feat_dim,
                      int num_segments, int64_t num_out_rows) {
  APT_CHECK_ARG(op >= 0 && op <= 3, "%s: op %d", who, op);
  APT_CHECK_ARG(dtype >= APT_F32 && dtype <= APT_F16, "%s: dtype %d", who, dtype);
  APT_CHECK_ARG(num_edges >= 0 && feat_dim > 0 && num_out_rows >= 0, "%s: bad sizes", who);
  APT_CHECK_ARG(num_segments >= 1 && num_segments <= kMaxSegments, "%s: %d segments outside [1,%d]", who, num_segments,
                kMaxSegments);
  if (op == kCopyU) *edata_dim = feat_dim;
  APT_CHECK_ARG(*edata_dim > 0 && feat_dim % *edata_dim == 0 && (op != kCopyE || *edata_dim == feat_dim),
                "%s: edata_dim %lld does not divide feat_dim %lld", who, (long long)*edata_dim, (long long)feat_dim);
  APT_CHECK_ARG(num_edges < (int64_t)0x7fffffff && num_out_rows < (int64_t)0x7fffffff, "%s: too many edges or rows", who);
  return APT_OK;
}

}  // namespace apt

extern "C" int32_t apt_pending_flags(void) { return apt::take_pending(); }

extern "C" size_t apt_spmm_workspace_bytes(int64_t num_out_rows, int64_t num_edges) {
  if (num_out_rows < 0 || num_edges < 0) return 0;
  return apt::spmm_layout(num_out_rows, num_edges, nullptr, nullptr);
}

extern "C" int apt_spmm_probe(const int64_t* coo_col, int64_t num_edges, const int64_t* coo_offset,
                              const int64_t* output_offset, int num_segments, int64_t* out_rows_mode_fixed,
                              void* stream) {
  int64_t answer[4];
  const int rc = apt_spmm_probe_rows(coo_col, num_edges, coo_offset, output_offset, num_segments, 0, out_rows_mode_fixed ? answer : nullptr, stream);
  if (rc == APT_OK)
    for (int k = 0; k < 3; ++k) out_rows_mode_fixed[k] = answer[k];
  return rc;
}

extern "C" int apt_spmm_probe_rows(const int64_t* coo_col, int64_t num_edges, const int64_t* coo_offset,
                                   const int64_t* output_offset, int num_segments, int want_hubs, int64_t* out_rows_mode_fixed_hubs,
                                   void* stream) {
  using namespace apt;
  int64_t* const out_rows_mode_fixed = out_rows_mode_fixed_hubs;
  APT_CHECK_ARG(num_segments >= 1 && num_segments <= kMaxSegments, "apt_spmm_probe: %d segments outside [1,%d]",
                num_segments, kMaxSegments);
  APT_CHECK_ARG(num_edges >= 0 && num_edges < (int64_t)0x7fffffff, "apt_spmm_probe: bad num_edges");
  APT_CHECK_ARG((num_edges == 0 || coo_col) && coo_offset && output_offset && out_rows_mode_fixed,
                "apt_spmm_probe: null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  APT_CUDA(cudaStreamIsCapturing(s, &capturing));
  APT_CHECK_ARG(capturing == cudaStreamCaptureStatusNone,
                "apt_spmm_probe: the number of output rows is read on the host, which a stream capture does not allow");
  int rc = check_pending("apt_spmm_probe");
  if (rc != APT_OK) return rc;
  int slot = -1;
  int64_t sequence = 0;
  rc = take_slot(&slot, &sequence);
  if (rc != APT_OK) return rc;
  int64_t* host = g_probe.host + slot * 8;
  SegTable st{coo_offset, nullptr, output_offset, num_segments};
  rc = launch_probe(coo_col, num_edges, st, -1, nullptr, slot, host, sequence, want_hubs != 0, s);
  if (rc == APT_OK) rc = wait_for(host, sequence, s);
  if (rc == APT_OK) {
    const int64_t w = *(volatile int64_t*)host, rows = probe_rows(w);
    out_rows_mode_fixed[0] = rows;
    out_rows_mode_fixed[1] = probe_mode(w);
    out_rows_mode_fixed[2] = probe_mode(w) == kFixed && rows > 0 ? num_edges / rows : 0;
    out_rows_mode_fixed[3] = probe_mode(w) == kOrder && (probe_hubs(w) || (want_hubs && num_edges / kHubMean >= rows));
    if (probe_mode(w) == 3) {
      set_error("apt_spmm_probe: the number of output rows is negative or above 2^31");
      rc = APT_ERR_BAD_ARG;
    }
  }
  give_slot(slot);
  return rc;
}

extern "C" int apt_spmm_sum_known(int op, int dtype, const int64_t* coo_row, const int64_t* coo_col,
                                  int64_t num_edges, const void* input, const void* edata,
                                  int64_t edata_dim, int64_t feat_dim, const int64_t* coo_offset,
                                  const int64_t* input_offset, const int64_t* output_offset,
                                  int num_segments, int64_t num_out_rows, int mode, int fixed, void* out,
                                  void* workspace, size_t workspace_bytes, void* stream) {
  using namespace apt;
  int rc = spmm_check("apt_spmm_sum", op, dtype, num_edges, &edata_dim, feat_dim, num_segments, num_out_rows);
  if (rc == APT_OK && mode == kDevice) rc = check_pending("apt_spmm_sum");
  if (rc != APT_OK) return rc;
  APT_CHECK_ARG(mode >= kDevice && mode <= kOrder, "apt_spmm_sum: mode %d", mode);
  APT_CHECK_ARG(mode != kFixed || (fixed >= 0 && (int64_t)fixed * num_out_rows == num_edges),
                "apt_spmm_sum: %lld rows of %d edges are not %lld edges", (long long)num_out_rows, fixed,
                (long long)num_edges);
  cudaStream_t s = (cudaStream_t)stream;
  if (num_out_rows == 0) return APT_OK;
  APT_CHECK_ARG(out, "apt_spmm_sum: null output");
  if (num_edges == 0) {
    APT_CUDA(cudaMemsetAsync(out, 0, (size_t)num_out_rows * feat_dim * elem_size(dtype), s));
    return APT_OK;
  }
  APT_CHECK_ARG(coo_row && coo_col && coo_offset && output_offset && (op == kCopyE || (input && input_offset)) &&
                    (op == kCopyU || edata),
                "apt_spmm_sum: null pointer");
  const SegTable st{coo_offset, input_offset, output_offset, num_segments};
  return spmm_run(op, dtype, coo_row, coo_col, num_edges, input, edata, edata_dim, feat_dim, st, num_out_rows, out,
                  workspace, workspace_bytes, mode, fixed, 0, s);
}

extern "C" size_t apt_spmm_widened_bytes(int dtype, int64_t num_edges, int64_t num_input_rows, int64_t feat_dim, int mode) {
  using namespace apt;
  if (dtype < APT_F32 || dtype > APT_F16 || num_edges < 0 || feat_dim <= 0 || mode < kFixed || mode > kOrderEven) return 0;
  const size_t esz = elem_size(dtype);
  return widen_pays(feat_dim, esz, num_input_rows, num_edges, mode) ? (size_t)num_input_rows * widened_dim(feat_dim, esz) * esz : 0;
}

extern "C" int apt_spmm_copy_u_widened(int dtype, const int64_t* coo_row, const int64_t* coo_col, int64_t num_edges, const void* input,
                                       int64_t num_input_rows, int64_t feat_dim, const int64_t* coo_offset,
                                       const int64_t* input_offset, const int64_t* output_offset, int num_segments,
                                       int64_t num_out_rows, int mode, int fixed, void* out, void* widened, size_t widened_bytes,
                                       void* workspace, size_t workspace_bytes, void* stream) {
  using namespace apt;
  const size_t need = apt_spmm_widened_bytes(dtype, num_edges, num_input_rows, feat_dim, mode);
  if (mode == kOrderEven) mode = kOrder;
  if (need == 0 || num_out_rows <= 0 || !input)
    return apt_spmm_sum_known(kCopyU, dtype, coo_row, coo_col, num_edges, input, nullptr, feat_dim, feat_dim, coo_offset, input_offset,
                              output_offset, num_segments, num_out_rows, mode, fixed, out, workspace, workspace_bytes, stream);
  int64_t edata_dim = 0;
  int rc = spmm_check("apt_spmm_copy_u_widened", kCopyU, dtype, num_edges, &edata_dim, feat_dim, num_segments, num_out_rows);
  if (rc != APT_OK) return rc;
  APT_CHECK_ARG(mode != kFixed || (fixed >= 0 && (int64_t)fixed * num_out_rows == num_edges),
                "apt_spmm_copy_u_widened: %lld rows of %d edges are not %lld edges", (long long)num_out_rows, fixed, (long long)num_edges);
  APT_CHECK_ARG(coo_row && coo_col && coo_offset && input_offset && output_offset && out && widened, "apt_spmm_copy_u_widened: null pointer");
  APT_CHECK_ARG(((uintptr_t)widened & 15) == 0, "apt_spmm_copy_u_widened: the buffer of widened rows must be 16-byte aligned");
  if (widened_bytes < need) {
    set_error("apt_spmm_copy_u_widened: %zu < %zu bytes for widened rows", widened_bytes, need);
    return APT_ERR_CAPACITY;
  }
  const size_t esz = elem_size(dtype);
  cudaStream_t s = (cudaStream_t)stream;
  rc = widen_rows(input, num_input_rows, feat_dim * (int64_t)esz, widened, s);
  if (rc != APT_OK) return rc;
  const SegTable st{coo_offset, input_offset, output_offset, num_segments};
  const int64_t dim = widened_dim(feat_dim, esz);
  return spmm_run(kCopyU, dtype, coo_row, coo_col, num_edges, widened, nullptr, dim, dim, st, num_out_rows, out, workspace, workspace_bytes,
                  mode, fixed, feat_dim, s);
}

extern "C" int apt_spmm_sum(int op, int dtype, const int64_t* coo_row, const int64_t* coo_col,
                            int64_t num_edges, const void* input, const void* edata,
                            int64_t edata_dim, int64_t feat_dim, const int64_t* coo_offset,
                            const int64_t* input_offset, const int64_t* output_offset,
                            int num_segments, int64_t num_out_rows, void* out,
                            void* workspace, size_t workspace_bytes, void* stream) {
  return apt_spmm_sum_known(op, dtype, coo_row, coo_col, num_edges, input, edata, edata_dim, feat_dim, coo_offset,
                            input_offset, output_offset, num_segments, num_out_rows, apt::kDevice, 0, out, workspace,
                            workspace_bytes, stream);
}

extern "C" int apt_sddmm(int op, int dtype, const int64_t* coo_row, const int64_t* coo_col,
                         int64_t num_edges, const void* lhs, const void* rhs, int64_t feat_dim,
                         const int64_t* coo_offset, const int64_t* lhs_offset,
                         const int64_t* rhs_offset, int num_segments, void* out, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(op == 0 || op == 1, "apt_sddmm: op %d", op);
  APT_CHECK_ARG(dtype >= APT_F32 && dtype <= APT_F16, "apt_sddmm: dtype %d", dtype);
  APT_CHECK_ARG(num_edges >= 0 && feat_dim > 0, "apt_sddmm: bad sizes");
  APT_CHECK_ARG(num_segments >= 1 && num_segments <= kMaxSegments,
                "apt_sddmm: %d segments outside [1,%d]", num_segments, kMaxSegments);
  if (num_edges == 0) return APT_OK;
  APT_CHECK_ARG(coo_row && coo_col && lhs && rhs && out && coo_offset && lhs_offset && rhs_offset,
                "apt_sddmm: null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  const size_t esz = elem_size(dtype);
  const SegTable st{coo_offset, lhs_offset, nullptr, num_segments};
  const int ve = slice_elems((uint64_t)(feat_dim * esz) | (uintptr_t)lhs | (uintptr_t)rhs | (uintptr_t)out, (int)esz);
  switch (dtype) {
    case APT_F32:
      return dispatch_sddmm<float>(op, ve, coo_row, coo_col, num_edges, lhs, rhs, feat_dim, st, rhs_offset, out, s);
    case APT_BF16:
      return dispatch_sddmm<__nv_bfloat16>(op, ve, coo_row, coo_col, num_edges, lhs, rhs, feat_dim, st, rhs_offset, out, s);
    default:
      return dispatch_sddmm<__half>(op, ve, coo_row, coo_col, num_edges, lhs, rhs, feat_dim, st, rhs_offset, out, s);
  }
}
