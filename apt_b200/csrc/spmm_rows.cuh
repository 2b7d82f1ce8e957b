// The row kernel of the SpMM and what it shares with the kernels that prepare a block for it.
//
// Every output row belongs to a group of lanes of one warp, which walks the row's edges, keeps the
// sums in fp32 registers and writes the row once: no float atomics, no zero-fill of the output.
//
//   lane split   `lpe` lanes cover one input row (VPL slices of up to 16 bytes each), `ep` edges of the
//                row are read side by side, and their partial sums meet in a shuffle butterfly at the
//                end. The second factor is for narrow rows that are too few to fill the chip side by side (row_split).
//   in flight    the loads of U edges (U * VPL slices a lane) are issued before any of them is added;
//                the next row's bounds and source indexes are fetched while this row's slices are
//                on their way, so that a short row costs one round of latency and not three. Full rounds carry
//                no predicate: a round is bound by its instruction count once the rows come out of L2 (lanes
//                beyond the row read its last slice again and are not written).
//   long rows    the reverse direction of a block gathers at its hubs: longer rows (`long_edges`) are cut into
//                items of about sqrt(edges) edges, at least kItemEdges, that whole warps take before the rows. Each
//                leaves its partial sums in scratch and the item that finishes last adds them in order. One
//                block of 1024 threads per long row, the form before this, kept 26 of 148 SMs busy for
//                62 us behind the row kernel.
//
// Wide rows of many edges have a kernel of their own (spmm_stream.cuh). Rows that are no whole slices may have been laid out anew (widen.cuh).
//
// Where a row's edges are (`mode`):
//   kFixed    every row has `fixed` consecutive edges: what a fanout sampler produces. No table.
//   kRanges   grouped by row, any length: range[] (k_edge_ranges)
//   kOrder    anything else: a counting sort by row leaves (source row, edge) pairs in order[]
//   kDevice   the probe kernel's verdict is read from device memory (apt_spmm_sum, which may not wait)
//
// What it measured is at rows_min_blocks.
#pragma once

#include <algorithm>

#include "rows.cuh"
#include "widen.cuh"

namespace apt {

constexpr int kMaxSegments = 64;
// kUMulW: one fp32 weight per edge and head. kDots: no sums, but every edge's dots of its input row with the output row's own.
enum { kCopyU = 0, kCopyE = 1, kUMulE = 2, kUAddE = 3, kUMulW = 4, kDots = 5 };
enum { kDevice = -1, kFixed = 0, kRanges = 1, kOrder = 2 };

// Rows of more edges are left to whole warps. A group narrower than a warp hands over earlier: its own pace is
// one round of latency per U edges.
constexpr int kLongRow = 128, kLongRowNarrow = 32;
constexpr int kItemEdges = 64;
constexpr int kLongRun = 64;     // runs of at least this many edges make the probe ask for the counting sort

struct SegTable {
  // first edge, first input row and first output row of every segment; null where a kernel has no use for them
  const int64_t* coo_off;
  const int64_t* in_off;
  const int64_t* out_off;
  int nseg;
};

// The probe's answer in one word, so that a single store delivers it to the host: rows (31 bits), mode (2), whether a few rows have many of the edges (1),
// sequence (30). Rows that do not fit (or are negative) answer mode 3.
__host__ __device__ inline int64_t probe_pack(int64_t rows, int mode, bool hubs, int64_t sequence) {
  return (sequence << 34) | ((int64_t)hubs << 33) | ((int64_t)mode << 31) | rows;
}
__host__ __device__ inline int64_t probe_rows(int64_t w) { return w & 0x7fffffff; }
__host__ __device__ inline int probe_mode(int64_t w) { return (int)(w >> 31) & 3; }
__host__ __device__ inline bool probe_hubs(int64_t w) { return w >> 33 & 1; }
__host__ __device__ inline int64_t probe_sequence(int64_t w) { return (int64_t)((uint64_t)w >> 34); }
constexpr int64_t kProbeSequences = (1 << 30) - 1;

struct SpmmWs {
  // zero when a call starts that groups edges or asks the device for the mode
  int64_t* result;      // [1] the probe's answer (probe_pack)
  unsigned long long* probe;   // what the blocks of the probe found (probe_votes)
  int32_t* num_items;   // [1]
  int32_t* num_slots;   // [1] slots of order[] given out
  int32_t* num_parts;   // [1] rows of part[] given out
  int32_t* cnt;         // [spread_rows(rows)] edges per row, at spread(row)
  int32_t* part_done;   // [max_parts] items of a row that have finished, at the row's first part
  size_t zero_bytes;
  // written before they are read
  int2* range;          // [rows] first and last slot (edge) of every row
  uint32_t* rank;       // [edges] position inside its row
  uint2* order;         // grouped by output row, see OrderKind
  int4* items;          // [max_items] row, first, last slot, part (-1: the row's only item)
  float* part;          // [part_floats] partial sums
  int64_t max_items, max_parts, part_floats;
};

constexpr uint32_t kNoRank = 0xffffffffu;     // rank of an edge that belongs to no row

// Where a row's counter is. Ids go by first occurrence, so the first rows are the ones that many edges share, and atomics on
// one line queue up in one slice of L2: with 32 neighbours to a line, the first line of a block of a million edges over 151 552
// sources gets 15 000 of them, one after another, which is what counting them took (27 us; sources at random 14). 32 rows
// that are 32 apart share a line instead (a tile of 1024 rows is transposed), the first one 4800: 27 -> 17 us.
__host__ __device__ inline uint32_t spread(uint32_t row) { return (row & ~1023u) | (row & 31u) << 5 | (row >> 5 & 31u); }
inline int64_t spread_rows(int64_t rows) { return (rows + 1023) / 1024 * 1024; }

// What the counting sort leaves in order[], a slot to an edge.
enum OrderKind {
  kByEdge = 0,      // uint2 (input row, edge), and items for long rows: k_spmm_rows
  kByRow = 1,       // uint2 (input row, output row): k_spmm_stream
  kByBoth = 2,      // uint4 (input row, output row, edge): k_spmm_stream with weights
};

__device__ __forceinline__ int seg_of(const int64_t* coo, int nseg, int64_t e) {
  int k = 0;
  while (k + 1 < nseg && coo[k + 1] <= e) ++k;
  return k;
}

__host__ __device__ inline int item_edges(int deg) {
  int per = kItemEdges;
  while ((int64_t)per * per < deg) per += 32;
  return per;
}

constexpr int64_t kRowsManyOrdered = 3 << 13;

// How rows are divided among lanes: slices of `ve` elements, `vpl` of them a lane.
struct RowSplit {
  int ve, vpl;
  int lpe, ep;       // lanes to an edge, edges side by side: powers of two, lpe * ep <= 32
  int long_edges;    // longer rows are whole warps' work (kOrder)
};
// ordered: the rows' edges come by a sort's list (kOrder), or may (kDevice).
inline RowSplit row_split(int64_t feat_dim, int ve, int64_t num_edges, int64_t num_rows, bool ordered) {
  RowSplit r;
  const int64_t nvec = feat_dim / ve;
  r.ve = ve;
  // one slice a lane while 32 lanes cover the row; two, then four, beyond (wider rows are walked in column blocks). Half as
  // many lanes with twice the slices, two edges side by side, take half the address arithmetic but more registers:
  // 64 -> 98 us for bf16 x 256.
  r.vpl = nvec <= 32 ? 1 : nvec <= 64 ? 2 : 4;
  r.lpe = pow2_ge(ceil_div(nvec, r.vpl));
  // Edges side by side: as many as fill the chip's lanes, never more than half the mean row, whose second half would idle those lanes. Where
  // the rows fill the chip by themselves they go side by side instead: no sums to join, and rows of 15 edges are walked in as many
  // steps by half the warps. us, as many edges as go -> rows first (42 727 x 15 edges unless it says so; forward | reverse):
  // bf16 x 128 32 -> 24.5 | 48 -> 36, x 64 22 -> 13 | 29.5 -> 24, fp32 x 64 30 -> 24 | 48 -> 36, x 32 21 -> 13.7 | 29 -> 23, 60 000 x 8 of bf16 x 10
  // 20.5 -> 8.1, 5 000 x 15 of fp32 x 64 6.7 -> 5.6; 1 000 x 15, which do not fill it, stay as they are (one by one 4.5 -> 5.1). Four
  // lanes to a row at least: with two, rows of very different lengths wait for one another (67 000 x 15 of bf16 x 4 11 -> 17 | 19 -> 27).
  // The edges of long rows stay side by side: in a list, rows of more than kLongRowNarrow edges would all become items, and many edges one
  // after another make the last wave of rows long. As many edges as go -> rows first, us: in a list fp32 x 32, 7 000 x 16 33 -> 33, x 20 34 -> 36; 15 000 x 16
  // 38 -> 37, x 20 40 -> 42, x 32 48 -> 54; 60 000 x 24 86 -> 82, x 28 92 -> 97, x 40 115 -> 161; one after another fp32 x 16, 15 000 x 30 21 -> 20.4, x 50
  // 24 -> 25, x 200 45 -> 59; 60 000 x 30 43 -> 32, x 50 54 -> 44.
  const int64_t longest = !ordered ? 40 : num_rows >= kRowsManyOrdered ? 24 : 16;
  const int most = pow2_le(num_edges / (num_rows * 2), 32 / r.lpe);
  r.ep = 1;
  while (r.ep < most && (num_edges > longest * num_rows || r.lpe * r.ep < 4 || num_rows * r.lpe * r.ep * 2 <= (int64_t)kNumSMs * 24 * 32)) r.ep <<= 1;
  r.long_edges = r.lpe * r.ep == 32 ? kLongRow : kLongRowNarrow;
  return r;
}

// What the blocks of a kernel that looks edges over found, a word each (k_gat_ranges). A word per block is written whatever it
// is, so that nothing has to be cleared in front; who needs the answer reads them all.
struct Verdict {
  const uint32_t* word;      // null: nothing was found
  int count;
};
constexpr int kVerdicts = 592;
// By all threads of a block.
__device__ __forceinline__ bool any_found(const Verdict& v) {
  if (!v.word) return false;
  uint32_t found = 0u;
  for (int t = threadIdx.x; t < v.count; t += blockDim.x) found |= v.word[t];
  return __syncthreads_or((int)found) != 0;
}

template <typename T>
struct RowArgs {
  const int64_t* row;
  const T* in;
  const T* edata;          // kUMulW: float[E][heads]
  int64_t edata_dim, feat_dim;
  SegTable st;
  int64_t num_rows, num_edges;
  SpmmWs ws;
  T* out;
  int mode, fixed;
  RowSplit split;
  int part_stride;         // floats per part
  Verdict none;            // found: no row has edges (kRanges)
  int32_t* status;         // flags of the call; null: the library's own word (apt_pending_flags)
  const int64_t* col;      // output row of an edge, inside its segment
  // kDots
  const T* own;            // the output rows' own
  float* dots;             // [E][heads]
  uint32_t num_in;         // input rows; ws.cnt and ws.rank count their edges on the way
  int64_t width;           // columns of an output row where input rows were widened to feat_dim; 0: feat_dim
};

// ---- which rows k_spmm_stream takes --------------------------------------------------------------
// The lines, us of the call by k_spmm_rows -> by k_spmm_stream on either side (15 edges a row, or 0 to 30 where it says so):
//   sorted edges, 98 304: gains from all sizes tried on: fp32 x 128, 65 535 edges 49 -> 37, 98 310 54 -> 42; x 256 50 -> 41, 54 -> 42
//   weighted, up to 512 bytes, 393 216: 300 000 edges bf16 4 x 64 30.5 -> 30.9, fp32 4 x 32 31.9 -> 30.4; 393 210 37.1 -> 35.2, 39.2 -> 33.9
//   above 512 bytes, 196 608: 135 000 edges fp32 4 x 64 22.0 -> 23.2, sums of fp32 x 256 23.9 -> 27.1; 196 605 27.4 -> 27.3, 27.7 -> 29.1 (0 to 30:
//     36.3 -> 35.6), bf16 x 512 33.0 -> 31.0; 300 000 39.2 -> 37.2, 35.4 -> 35.4, 45.7 -> 39.1
//   sums, up to 512 bytes, 655 360: 450 000 edges fp32 x 128 32.0 -> 30.8 (0 to 30: 43.5 -> 39.4), bf16 x 256 37.8 -> 34.2, fp32 x 72 30.8 -> 30.3; 655 365
//     44.6 -> 44.0 (60 -> 53), 50.5 -> 45.0, 38.5 -> 40.6 (54 -> 46); 1 013 760 70 -> 55 (96 -> 67), 77 -> 60, 58 -> 50. Rows that half fill the warp and have
//     the same number of edges each lose 5 to 8 % from there to about 800 000.
constexpr int kStreamBlocks = 2;
constexpr int stream_warps(bool one_slice) { return one_slice ? 12 : 10; }
constexpr int kStreamShared = 112 * 1024 - 2560;      // a block's, beside its barriers and segment tables
constexpr int kStreamHeads = 8, kStreamHeadsWide = 16;      // weights an edge can bring along; of wide rows behind the sort
constexpr int kStreamMinSlices = 17, kStreamStretch = 32;
constexpr int kStreamParts = 32;      // parts of a row that one warp adds up
constexpr int kStreamMinOrdered = 3 << 15, kStreamMinWide = 3 << 16, kStreamMinWeighted = 3 << 17, kStreamMinSums = 5 << 17;
constexpr int64_t kStreamMaxEdges = 0x7fffffff - 4096;      // a warp looks up to 159 slots ahead of the last one, in 31 bits
// Rows to a group; a warp has two groups on their way.
constexpr int stream_group(bool one_slice) { return one_slice ? 8 : 4; }

struct StreamPlan {
  int row_bytes, warp_bytes;
  int warps, shared;         // a block's
  int lph;                   // kDots: lanes to a head
};
inline int stream_lph(int64_t feat_dim, size_t esz, int heads) { return pow2_ge(ceil_div((int64_t)(feat_dim / heads * esz), 16), 64); }
inline bool stream_one_slice(int op, int64_t feat_dim, size_t esz, int heads) {
  return op == kDots ? heads * stream_lph(feat_dim, esz, heads) <= 32 : feat_dim * (int64_t)esz <= 512;
}
inline StreamPlan stream_plan(int op, int64_t feat_dim, size_t esz, int heads, bool widened = false) {
  StreamPlan p{};
  p.row_bytes = (int)(feat_dim * esz);
  p.lph = op == kDots ? stream_lph(feat_dim, esz, heads) : 32;
  p.warp_bytes = 2 * 8 * 512 + (op == kUMulW ? 64 * heads * 4 : 0);      // rows (two groups of eight of a slice a lane, four of two), weights
  if (widened) p.warp_bytes += stream_one_slice(op, feat_dim, esz, heads) ? 512 : 1024;      // the row that is written
  p.warps = std::min(stream_warps(stream_one_slice(op, feat_dim, esz, heads)), kStreamShared / p.warp_bytes);
  p.shared = p.warps * p.warp_bytes;
  return p;
}
// Floats of scratch for partial sums. k_spmm_rows: room for the longest rows of a power-law block at 256 columns; a row that finds
// none is one item. k_spmm_stream leaves up to two rows a warp, of up to 512 columns (12 to 15 MB): with six floats an edge as
// its only room 135 000 edges of bf16 x 512 had 79 of 296 blocks.
constexpr int kStreamMaxColumns = 512;
inline int64_t part_room(int64_t num_edges) {
  if (num_edges <= kItemEdges) return 1;
  const int64_t room = std::min<int64_t>(6 * num_edges + 1024, (int64_t)16 << 20);
  if (num_edges < kStreamMinOrdered) return room;
  return std::max(room, 2 * kStreamMaxColumns * std::min<int64_t>(num_edges / kStreamStretch, kNumSMs * kStreamBlocks * stream_warps(true)));
}
// Blocks of `warps` warps: a stretch is at least kStreamStretch edges, and behind the sort long enough for the partial sums to find room.
inline int stream_blocks(int64_t feat_dim, int64_t num_edges, int64_t part_floats, int warps, bool grouped) {
  int64_t least = kStreamStretch;
  if (!grouped) least = std::max(least, ceil_div((int64_t)2 * feat_dim * num_edges, part_floats));
  return (int)std::min<int64_t>(std::max<int64_t>(1, num_edges / (least * warps)), kNumSMs * kStreamBlocks);
}
// `slice`: bytes of the widest access to rows and results. `grouped`: the edges are (kFixed, kRanges).
// Where nobody knows (kDevice) the lines of edges in no order hold for grouped ones as well: with a launch of either kernel, of which one
// returns at once, every such call paid 2 us and 30 000 x 15 grouped edges of fp32 x 128 took 57 us instead of 50 (row kernel alone 54).
inline bool stream_fits(int op, int slice, int64_t feat_dim, size_t esz, int heads, int64_t num_edges, bool grouped) {
  const int64_t row = feat_dim * (int64_t)esz;
  if (slice != 16 || row < kStreamMinSlices * 16 || row > 64 * 16 || num_edges > kStreamMaxEdges) return false;
  if (heads > (!grouped && row > 512 && num_edges >= kStreamMinWide ? kStreamHeadsWide : kStreamHeads)) return false;
  const int64_t least = !grouped ? kStreamMinOrdered : row > 512 ? kStreamMinWide : op == kCopyU ? kStreamMinSums : kStreamMinWeighted;
  if (num_edges < least) return false;
  if (op != kDots) return op == kCopyU || op == kUMulW;
  const int lph = stream_lph(feat_dim, esz, heads);
  return lph >= 4 && lph * heads <= 64;
}
inline OrderKind order_kind(int op, int slice, int64_t feat_dim, size_t esz, int heads, int64_t num_edges) {
  if (!stream_fits(op, slice, feat_dim, esz, heads, num_edges, false)) return kByEdge;
  return op == kCopyU ? kByRow : kByBoth;
}

// One slice of one edge's contribution, in two steps so that the loads of several edges are issued
// before any of them is used.
template <typename T, int VE, int OP>
struct EdgeSlice {
  Raw<T, VE> x;                                           // input slice (kCopyE: the edge's own)
  Raw<T, (OP == kUMulE || OP == kUAddE) ? VE : 2 / sizeof(T) + 1> w;   // per-column edge values
  float s;                                                // per-head edge value
};

// `lane_in` and `lane_edata` point at the lane's column of row 0, `off` bytes before this slice.
template <typename T, int VE, int OP>
__device__ __forceinline__ void slice_load(EdgeSlice<T, VE, OP>& v, const RowArgs<T>& a, const T* lane_in, uint32_t off,
                                           const T* lane_edata, uint32_t row_bytes, uint32_t edata_bytes, uint32_t src, uint32_t e,
                                           int col, int per, int head) {
  v.x = load_raw<T, VE>(OP == kCopyE ? at_row(lane_edata, e, edata_bytes)
                                     : (const T*)((const char*)at_row(lane_in, src, row_bytes) + off));
  if constexpr (OP == kUMulE || OP == kUAddE) {
    if (per == 1) {
      v.w = load_raw<T, VE>(at_row(lane_edata, e, edata_bytes));
    } else if (head >= 0) {
      v.s = Elem<T>::to_f(*at_row(lane_edata, e, edata_bytes));
    } else {
      const T* const p = at_row(a.edata, e, edata_bytes);
      Pack<T, VE> w;
#pragma unroll
      for (int t = 0; t < VE; ++t) w.v[t] = p[(col + t) / per];
#pragma unroll
      for (int k = 0; k < (int)(sizeof(v.w.w) / 4); ++k)
        v.w.w[k] = sizeof(T) * VE < 4 ? (unsigned int)*(const unsigned short*)&w : ((const unsigned int*)&w)[k];
    }
  }
  if constexpr (OP == kUMulW) v.s = __ldg((const float*)at_row(lane_edata, e, edata_bytes));
}

template <typename T, int VE, int OP>
__device__ __forceinline__ void slice_add(Acc<VE>& acc, const EdgeSlice<T, VE, OP>& v, int per, int head) {
  if constexpr (OP == kUMulE) {
    if (per != 1 && head >= 0) {
      acc.fma(v.x, v.s);
    } else {
      acc.fma(v.x, v.w);
    }
  } else if constexpr (OP == kUAddE) {
    acc.add(v.x);
    if (per != 1 && head >= 0) {
      const F2 ss = f2_pack(v.s, v.s);
#pragma unroll
      for (int q = 0; q < Acc<VE>::P; ++q) acc.p[q] = f2_add(acc.p[q], ss);
    } else {
      acc.add(v.w);
    }
  } else if constexpr (OP == kUMulW) {
    acc.fma(v.x, v.s);
  } else {
    acc.add(v.x);
  }
}

// The slices of U edges, two and two, and what they come to: rows of many lanes take an edge at a time where they fill the chip (row_split), and a sum of 15
// edges one after another is a fifth further from 64 bits than of four side by side, one of 24 half as far again. fp32 x 64, 42 727 x 15 edges, 2-norm of the error over
// that of the sums: side by side 6.1e-8, one after another 7.4e-8, here 5.6e-8; x 32, 60 000 x 24 6.3e-8,
// 9.3e-8, 6.3e-8. Sums of the attention, fp32 4 x 16, 20 000 x 24, 1.06e-7, 1.20e-7, 1.02e-7. With fewer registers live it spills less as well (weighted fp32 316 -> 56 bytes).
constexpr bool in_pairs(int op) { return op == kCopyU || op == kCopyE || op == kUMulW; }      // (a value per column beside each slice: spills)
template <typename T, int VE, int OP, int U, int VPL>
__device__ __forceinline__ void slices_add(Acc<VE>& acc, const EdgeSlice<T, VE, OP> (&v)[U][VPL], int i, int per, int head) {
  Acc<VE> pair[U / 2];
#pragma unroll
  for (int u = 0; u < U / 2; ++u) {
    if constexpr (OP == kCopyU || OP == kCopyE) {
      pair[u].sum_of(v[2 * u][i].x, v[2 * u + 1][i].x);
    } else {
      pair[u].zero();
      slice_add<T, VE, OP>(pair[u], v[2 * u][i], per, head);
      slice_add<T, VE, OP>(pair[u], v[2 * u + 1][i], per, head);
    }
    if (!in_pairs(OP)) acc.add(pair[u]);
  }
  if (!in_pairs(OP)) return;
#pragma unroll
  for (int u = 1; u < U / 2; ++u) pair[0].add(pair[u]);
  acc.add(pair[0]);
}

// The sums of the edges read side by side meet, and the lanes of the first of them write the row's column block.
template <typename T, int VE, int VPL, int OP, bool WIDENED>
__device__ __forceinline__ void rows_write(const RowArgs<T>& a, Acc<VE> (&acc)[VPL], const int (&col)[VPL], const int (&head)[VPL], int d, int c0, int nvec, int lpe,
                                           int lpr, int vl, int epi, unsigned gmask) {
#pragma unroll 1
  for (int o = lpe; o < lpr; o <<= 1)
#pragma unroll
    for (int i = 0; i < VPL; ++i) acc[i].join(gmask, o);
  if (epi != 0) return;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    if (c0 + vl + i * lpe >= nvec) continue;
    if constexpr (WIDENED) {
      // weighted rows are widened head by head
      const int heads = OP == kUMulW ? (int)a.edata_dim : 1, h = OP == kUMulW ? head[i] : 0;
      const int from = OP == kUMulW ? (int)a.feat_dim / heads : 0, to = (int)a.width / heads;
      store_some<T, VE>(a.out + (int64_t)d * a.width + col[i] - h * (from - to), acc[i].template rounded<T>(), to - (col[i] - h * from));
    } else store_pack<T, VE>(a.out + (int64_t)d * a.feat_dim + col[i], acc[i].template rounded<T>());
  }
}

// Blocks an SM is to hold. The gather is bound by loads in flight, and the 64 (80) registers a thread of four (three)
// blocks hold the slices of plain sums without spilling; edge values and 8 elements a slice need more.
// 67 584 x 15 edges, bf16 x 256 (0.52 GB gathered, mostly out of L2): 89 us at one or two blocks, 65 at three, 63 at four;
// reverse 104 / 82 / 90 us. (fp32 x 256 behaved the same; rows of that many edges are k_spmm_stream's now.)
constexpr int rows_min_blocks(int op, int elems) {
  if (op == kCopyU || op == kCopyE || op == kUMulW) return elems <= 4 ? 4 : elems <= 8 ? 3 : 2;
  return elems <= 2 ? 3 : elems <= 8 ? 2 : 1;
}

// WIDE: a warp to an edge (lpe 32, ep 1), which leaves the geometry to the compiler and its registers to more warps.
// WIDENED: the input's rows are (widen.cuh), the result's are not.
template <typename T, int VE, int VPL, int OP, bool WIDE, bool WIDENED>
__global__ void __launch_bounds__(256, rows_min_blocks(OP, VE * VPL))
k_spmm_rows(const __grid_constant__ RowArgs<T> a) {
  wait_for_previous();
  constexpr int U = VPL >= 2 ? 2 : 4;
  __shared__ int64_t coo[kMaxSegments + 1], ioff[kMaxSegments + 1];
  int mode = a.mode, fixed = a.fixed;
  if (mode == kDevice) {
    const int64_t w = *a.ws.result;
    mode = probe_mode(w);
    fixed = mode == kFixed ? (int)(a.num_edges / a.num_rows) : 0;
  }
  if (mode != kOrder) {
    for (int t = threadIdx.x; t <= a.st.nseg; t += blockDim.x) {
      // no table: one segment whose rows start at 0
      coo[t] = a.st.coo_off ? a.st.coo_off[t] : 0;
      ioff[t] = a.st.in_off ? a.st.in_off[t] : 0;
    }
    __syncthreads();
  }
  const int lane = threadIdx.x & 31;
  const int lpe = WIDE ? 32 : a.split.lpe, vl = lane & (lpe - 1);
  const int nvec = (int)(a.feat_dim / VE);
  const int per = (int)(a.feat_dim / a.edata_dim);
  const uint32_t row_bytes = (uint32_t)(a.feat_dim * sizeof(T));
  const uint32_t ed_bytes = (uint32_t)(a.edata_dim * (OP == kUMulW ? sizeof(float) : sizeof(T)));
  const bool none = any_found(a.none);
  // rows and edges fit 31 bits; what is added to them is compared with what is left, or unsigned
  const uint32_t num_rows = (uint32_t)a.num_rows;
  const int warps = gridDim.x * (blockDim.x >> 5), warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int num_items = mode == kOrder ? min(*a.ws.num_items, (int)a.ws.max_items) : 0;
  // whole warps first take items, dealt from the last warp on (the first rows, often the longest, are the first warps': rows
  // of 32 bf16 columns in reverse 12.8 -> 9.1 us, of 4 x 64 with weights 115 -> 110) ...
  int it = warps - 1 - warp;
  bool items = it < num_items;
  // ... then groups of lanes take rows: lpr lanes, ep edges side by side
  int g_ep = items ? 32 / lpe : a.split.ep, g_lpr = lpe * g_ep, g_sub = lane & (g_lpr - 1), g_epi = g_sub / lpe;
  unsigned g_mask = g_lpr == 32 ? 0xffffffffu : (((1u << g_lpr) - 1u) << (lane - g_sub));
#define EP (WIDE ? 1 : g_ep)
#define LPR (WIDE ? 32 : g_lpr)
#define SUB (WIDE ? lane : g_sub)
#define EPI (WIDE ? 0 : g_epi)
#define GMASK (WIDE ? 0xffffffffu : g_mask)

  auto resolve = [&](int k, uint32_t& src, uint32_t& e) {
    if (mode == kOrder) {
      const uint2 o = a.ws.order[k];
      src = o.x;
      e = o.y;
    } else {
      e = (uint32_t)k;
      src = OP == kCopyE ? 0u : (uint32_t)(ioff[a.st.nseg > 1 ? seg_of(coo, a.st.nseg, k) : 0] + a.row[k]);
    }
  };
  auto bounds = [&](uint32_t d, int& b, int& e) {
    if (mode == kFixed) {
      b = (int)d * fixed;
      e = b + fixed;
    } else {
      const int2 r = none ? make_int2(0, 0) : a.ws.range[d];
      b = r.x;
      e = r.y;
    }
  };

  uint32_t d = 0, G = 0;
  int b = 0, e = 0, nb = 0, ne = 0, part = -1;
  uint32_t src = 0, eid = 0, nsrc = 0, neid = 0;
  auto start_item = [&]() {
    const int4 m = a.ws.items[it];
    d = (uint32_t)m.x;
    b = m.y;
    e = m.z;
    part = m.w;
    if (lane < e - b) resolve(b + lane, src, eid);
  };
  auto start_rows = [&]() {
    items = false;
    g_ep = a.split.ep, g_lpr = lpe * g_ep, g_sub = lane & (g_lpr - 1), g_epi = g_sub / lpe;
    g_mask = g_lpr == 32 ? 0xffffffffu : (((1u << g_lpr) - 1u) << (lane - g_sub));
    G = warps * (32 / LPR);
    d = warp * (32 / LPR) + lane / LPR;
    part = -1;
    if (d < num_rows) {
      bounds(d, b, e);
      if (SUB < e - b) resolve(b + SUB, src, eid);
    }
    if (d + G < num_rows) bounds(d + G, nb, ne);
  };
  if (items) start_item(); else start_rows();

  // the lane's columns: worked out once for rows of one column block (the divisions by the head width took a quarter of
  // a short row's instructions)
  const T *lane_in = nullptr, *lane_ed[VPL];
  uint32_t off[VPL];      // bytes from the lane's first slice; lanes past the row's last slice read their first one again
  int head[VPL], col[VPL], at_block = 0;
  auto set_block = [&](int c0) {
    at_block = c0;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      col[i] = (c0 + vl + i * lpe < nvec ? c0 + vl + i * lpe : i == 0 ? nvec - 1 : c0 + vl < nvec ? c0 + vl : nvec - 1) * VE;
      head[i] = (OP == kUMulW || (per > 1 && per % VE == 0)) ? col[i] / per : -1;
      off[i] = (uint32_t)((col[i] - col[0]) * (int)sizeof(T));
      lane_ed[i] = OP == kUMulW ? (const T*)((const float*)a.edata + head[i]) : a.edata + (head[i] >= 0 ? head[i] : col[i]);
    }
    lane_in = a.in + col[0];
  };
  set_block(0);

  while (items || d < num_rows) {
    int nnb = 0, nne = 0;
    if (!items) {
      // the next row's indexes and the bounds of the one after it are on their way while this one is summed
      if (d + G < num_rows && SUB < ne - nb) resolve(nb + SUB, nsrc, neid);
      if (d + 2 * G < num_rows) bounds(d + 2 * G, nnb, nne);
    }
    const bool skip = !items && mode == kOrder && e - b > a.split.long_edges;
#pragma unroll 1
    for (int c0 = 0; c0 < nvec && !skip; c0 += lpe * VPL) {
      if (c0 != at_block) set_block(c0);
      Acc<VE> acc[VPL];
#pragma unroll
      for (int i = 0; i < VPL; ++i) acc[i].zero();
      uint32_t my_src = src, my_e = eid;
#pragma unroll 1
      for (int left = e - b; left > 0; left -= LPR) {
        const int k0 = e - left;
        if (k0 != b && SUB < left) resolve(k0 + SUB, my_src, my_e);
        const int cnt = min(LPR, left);
        int j = EPI;
        const int full = cnt & ~(EP * U - 1);
#pragma unroll 1
        for (; j < full; j += EP * U) {
          EdgeSlice<T, VE, OP> v[U][VPL];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint32_t s = OP == kCopyE ? 0u : __shfl_sync(GMASK, my_src, j + u * EP, LPR);
            const uint32_t x = OP == kCopyU ? 0u : __shfl_sync(GMASK, my_e, j + u * EP, LPR);
#pragma unroll
            for (int i = 0; i < VPL; ++i) slice_load<T, VE, OP>(v[u][i], a, lane_in, off[i], lane_ed[i], row_bytes, ed_bytes, s, x, col[i], per, head[i]);
          }
          if constexpr (WIDE) {
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int i = 0; i < VPL; ++i) slice_add<T, VE, OP>(acc[i], v[u][i], per, head[i]);
          } else {
#pragma unroll
            for (int i = 0; i < VPL; ++i) slices_add<T, VE, OP, U, VPL>(acc[i], v, i, per, head[i]);
          }
        }
        if (full < cnt) {
          EdgeSlice<T, VE, OP> v[U][VPL];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint32_t s = OP == kCopyE ? 0u : __shfl_sync(GMASK, my_src, (j + u * EP) & (LPR - 1), LPR);
            const uint32_t x = OP == kCopyU ? 0u : __shfl_sync(GMASK, my_e, (j + u * EP) & (LPR - 1), LPR);
            if (j + u * EP < cnt) {
#pragma unroll
              for (int i = 0; i < VPL; ++i) slice_load<T, VE, OP>(v[u][i], a, lane_in, off[i], lane_ed[i], row_bytes, ed_bytes, s, x, col[i], per, head[i]);
            } else if constexpr (!WIDE && in_pairs(OP)) {
#pragma unroll
              for (int i = 0; i < VPL; ++i) v[u][i] = EdgeSlice<T, VE, OP>{};
            }
          }
          if constexpr (WIDE || !in_pairs(OP)) {
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (j + u * EP < cnt) {
#pragma unroll
                for (int i = 0; i < VPL; ++i) slice_add<T, VE, OP>(acc[i], v[u][i], per, head[i]);
              }
          } else {
#pragma unroll
            for (int i = 0; i < VPL; ++i) slices_add<T, VE, OP, U, VPL>(acc[i], v, i, per, head[i]);
          }
        }
      }
      int last = 1;
      if (part >= 0) {
        // several items to the row: leave the sums, and let the item that finishes last add them up in item order.
        // Only the last column block counts the item as finished.
        float* p = a.ws.part + (int64_t)part * a.part_stride;
#pragma unroll 1
        for (int o = lpe; o < LPR; o <<= 1)
#pragma unroll
          for (int i = 0; i < VPL; ++i) acc[i].join(GMASK, o);
        if (EPI == 0) {
#pragma unroll
          for (int i = 0; i < VPL; ++i) {
            if (c0 + vl + i * lpe >= nvec) continue;
#pragma unroll
            for (int t = 0; t < VE; ++t) __stcg(p + col[i] + t, acc[i].get(t));
          }
        }
        if (c0 + lpe * VPL < nvec) continue;
        last = 0;
        const int2 r = a.ws.range[d];
        const int size = item_edges(r.y - r.x), parts = (r.y - r.x + size - 1) / size;
        const int first = part - (b - r.x) / size;
        __threadfence();
        __syncwarp();
        if (lane == 0) last = atomicAdd(a.ws.part_done + first, 1) == parts - 1;
        last = __shfl_sync(0xffffffffu, last, 0);
        if (!last) break;
        __threadfence();
#pragma unroll 1
        for (int cc = 0; cc < nvec; cc += lpe * VPL) {
          if (cc != at_block) set_block(cc);
#pragma unroll
          for (int i = 0; i < VPL; ++i) {
            acc[i].zero();
#pragma unroll 1
            for (int q = EPI; q < parts; q += EP) {
              const float* src_part = a.ws.part + (int64_t)(first + q) * a.part_stride;
#pragma unroll
              for (int t = 0; t < VE; t += 2)
                acc[i].p[t / 2] = f2_add(acc[i].p[t / 2], f2_pack(__ldcg(src_part + col[i] + t), VE > 1 ? __ldcg(src_part + col[i] + (VE > 1 ? t + 1 : t)) : 0.f));
            }
          }
          c0 = cc;
          if (cc + lpe * VPL < nvec) {
            rows_write<T, VE, VPL, OP, WIDENED>(a, acc, col, head, d, c0, nvec, lpe, LPR, vl, EPI, GMASK);
          }
        }
      }
      rows_write<T, VE, VPL, OP, WIDENED>(a, acc, col, head, d, c0, nvec, lpe, LPR, vl, EPI, GMASK);
    }
    if (items) {
      it += warps;
      if (it < num_items) start_item(); else start_rows();
    } else {
      d += G;
      b = nb, e = ne, src = nsrc, eid = neid;
      nb = nnb, ne = nne;
    }
  }
#undef EP
#undef LPR
#undef SUB
#undef EPI
#undef GMASK
}

// ---- launch -----------------------------------------------------------------------
template <typename T, int VE, int VPL, int OP, bool WIDE, bool WIDENED>
static int launch_rows_kernel(const RowArgs<T>& a, cudaStream_t s) {
  static int occupancy[64] = {};
  int per_sm = 0;
  const int rc = blocks_per_sm(k_spmm_rows<T, VE, VPL, OP, WIDE, WIDENED>, 256, occupancy, &per_sm);
  if (rc != APT_OK) return rc;
  const int64_t want = ceil_div(a.num_rows, 256 / (a.split.lpe * a.split.ep));
  const int64_t wave = (int64_t)kNumSMs * per_sm;
  APT_FOLLOW((k_spmm_rows<T, VE, VPL, OP, WIDE, WIDENED>), (int)(want < wave ? want : wave), 256, 0, s, a);
  return APT_OK;
}

template <typename T, int VE, int OP, bool WIDENED = false>
static int launch_rows_vpl(const RowArgs<T>& a, cudaStream_t s) {
  // rows of two and four slices a lane are wide ones
  switch (a.split.vpl) {
    case 1:
      return a.split.lpe == 32 ? launch_rows_kernel<T, VE, 1, OP, true, WIDENED>(a, s) : launch_rows_kernel<T, VE, 1, OP, false, WIDENED>(a, s);
    case 2: return launch_rows_kernel<T, VE, 2, OP, true, WIDENED>(a, s);
    default: return launch_rows_kernel<T, VE, 4, OP, true, WIDENED>(a, s);
  }
}

template <typename T, int OP>
static int launch_stream(const RowArgs<T>& a, cudaStream_t s);     // spmm_stream.cuh

template <typename T, int OP>
static int launch_rows_ve(const RowArgs<T>& a, cudaStream_t s) {
  if constexpr (OP == kCopyU || OP == kUMulW) {
    if (stream_fits(OP, a.split.ve * (int)sizeof(T), a.feat_dim, sizeof(T), OP == kCopyU ? 1 : (int)a.edata_dim, a.num_edges, a.mode == kFixed || a.mode == kRanges)) return launch_stream<T, OP>(a, s);
  }
  if constexpr (OP == kCopyU || OP == kUMulW)
    if (a.width) return launch_rows_vpl<T, 16 / sizeof(T), OP, true>(a, s);
  switch (a.split.ve * (int)sizeof(T)) {
    case 16: return launch_rows_vpl<T, 16 / sizeof(T), OP>(a, s);
    case 8: return launch_rows_vpl<T, 8 / sizeof(T), OP>(a, s);
    case 4: return launch_rows_vpl<T, 4 / sizeof(T), OP>(a, s);
    default: return launch_rows_vpl<T, 1, OP>(a, s);
  }
}

// One translation unit per element type (spmm_f32.cu, spmm_bf16.cu, spmm_f16.cu) holds these.
template <typename T>
int launch_spmm_rows(int op, const RowArgs<T>& a, cudaStream_t s);

#define APT_DEFINE_SPMM_ROWS(T)                                                                          \
  template <>                                                                                            \
  int launch_spmm_rows<T>(int op, const RowArgs<T>& a, cudaStream_t s) {      \
    switch (op) {                                                                                        \
      case kCopyU: return launch_rows_ve<T, kCopyU>(a, s);                                \
      case kCopyE: return launch_rows_ve<T, kCopyE>(a, s);                                \
      case kUMulE: return launch_rows_ve<T, kUMulE>(a, s);                                \
      case kUAddE: return launch_rows_ve<T, kUAddE>(a, s);                                \
      case kDots: return launch_stream<T, kDots>(a, s);                                \
      default: return launch_rows_ve<T, kUMulW>(a, s);                                   \
    }                                                                                                    \
  }

// ---- shared by spmm.cu and gat.cu -----------------------------------------------------
constexpr int kStreamWaitPolls = 1 << 20;      // of an mbarrier, each of which may suspend for a while itself
int bulk_wait_polls();
int pending_word(int32_t** word);            // for flags of calls without a status word: see spmm.cu
// slot_bytes: of order[] (OrderKind).
size_t spmm_layout(int64_t num_rows, int64_t num_edges, char* base, SpmmWs* ws, int slot_bytes = 8);
// Counted edges (ws.cnt) to places: ws.range, and the items of long rows.
int launch_slots(int64_t num_rows, const SpmmWs& ws, int mode, OrderKind kind, int long_edges, int part_stride, cudaStream_t s);

}  // namespace apt
