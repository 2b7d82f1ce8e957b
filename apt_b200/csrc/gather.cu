// Cache-aware feature-row gather: one launch, no scratch.
//
// A warp takes a chunk of rows. One lane to a row looks the id up (p = feat_pos_map[id]: p >= 0 cache row, p < -1 row -p - 2 of the
// table in page-locked host memory, p == -1 no such row: zeros and a flag) and leaves the row's address in shared memory. In
// the result the chunk is one run of elements, which the warp copies from end to end, 8 of 32 lanes each in flight:
// rows of any width fill all lanes, and what is in flight does not depend on it. The division that finds an element's row is a
// multiplication.
//
// Rows one after another, the form before this, had a row of 33 to 127 elements as one load of 32 in flight, and a row of
// 33 took the steps of 64. us, that form -> this one (distinct rows, all cached unless it says so):
//   495 616 x 2 KiB     331 -> 320 (6.36 TB/s, 0.97 of the measured copy rate)
//   243 961 x 880 B     145 -> 76           243 961 x 882 B (2-byte elements)   172 -> 113
//   200 000 x 1 KiB     104 -> 68           200 000 x 1200 B                    144 -> 84
//   318 250 x 288 B      49 -> 40           318 250 x 292 B (4-byte elements)    66 -> 47
//   400 000 x 200 B (8-byte elements) 48 -> 41      400 000 x 66 B (2-byte elements)  70 -> 23
//   143 000 x 512 B, 2.7 % of them from host memory 50.7 -> 46.7
//
// Rows in host memory that begin or end inside a 32-byte sector are not part of the run (k_gather<V, true>, HostRow): two loads of it that
// share a sector, both on their way, have it cross the link twice. us, rows one after another (one load of 32 elements on its way, the next one finds the shared
// sector in L1), as part of the run -> by themselves:
//   from host memory all of them   12 000 x 402 B (2-byte elements) 138, 217 -> 113; 40 000 x 94 B (2) 150, 235 -> 145; 40 000 x 1202 B (2) 1147, 1678 -> 1035;
//     12 000 x 804 B (4) 225, 276 -> 213; 40 000 x 68 B (4) 127, 153 -> 129; 40 000 x 400 B (16) 352, 394 -> 353; 800 x 1998 B (2) 42, 54 -> 38
//   a tenth of them   5 438 x 402 B 9.8, 10.9 -> 10.1; 12 000 x 402 B 21, 21 -> 17; 40 000 x 68 B 17.8, 17.7 -> 17.1
// Bound by HBM, by the host link (64 bytes to a few KiB a request, about 50 M rows/s) and, small requests, by three dependent
// loads; rows of 2-byte elements by their loads and stores (copying 882-byte rows through shared memory in 16-byte vectors, shifted on the way
// out, took 93 instead of 113 us and rows below 512 bytes longer; two elements to a lane 135). Host rows of whole sectors by
// themselves, in front of the others, two at a time through shared memory: 143 000 x 512 B 90. Chunks of 16 KiB instead of kChunkBytes: 880 B 80, 1 KiB 71;
// of 2 KiB 89, 75.
//
// Rows are opaque bytes. An element V is the widest of 16/8/4/2/1 bytes that divides every row size, column offset
// and base address involved.
#include <string.h>

#include "common.cuh"

namespace apt {

constexpr int kGatherBlock = 256;
constexpr int kGatherWaves = 4;    // cap on the grid, in units of 148 x 8 blocks
constexpr int kGatherVectors = 8;  // elements a lane has in flight
constexpr int kChunkBytes = 4096;
constexpr int kGatherBlocks = 5;   // an SM (48 registers)
constexpr int kGatherBlocksNarrow = 6;   // of elements of 4 bytes or fewer (40)

template <typename V>
__device__ __forceinline__ V ld_vec(const V* p) { return __ldg(p); }
template <>
__device__ __forceinline__ uint4 ld_vec<uint4>(const uint4* p) { return ld_stream_16(p); }
template <typename V>
__device__ __forceinline__ void st_vec(V* p, V v) { *p = v; }
template <>
__device__ __forceinline__ void st_vec<uint4>(uint4* p, uint4 v) { st_stream_16(p, v); }
template <typename V>
__device__ __forceinline__ V zero_vec() { return V(0); }
template <>
__device__ __forceinline__ uint4 zero_vec<uint4>() { return make_uint4(0, 0, 0, 0); }
template <>
__device__ __forceinline__ uint2 zero_vec<uint2>() { return make_uint2(0, 0); }

// Rows [first, n) of the request, first from a device word when given.
__device__ __forceinline__ int64_t first_row(const int64_t* first_dev, int64_t n) {
  const int64_t f = first_dev ? *first_dev : 0;
  return f < 0 ? 0 : (f > n ? n : f);
}

struct GatherArgs {
  const int64_t* index;
  int64_t num_rows;
  const int64_t* num_rows_dev;
  const int64_t* first_row_dev;
  const int64_t* feat_pos_map;
  int64_t num_nodes;
  const char* dev_feats;
  int64_t num_dev_rows, dev_row_bytes;
  const char* uva_feats;
  int64_t num_uva_rows, uva_row_bytes, uva_col_offset_bytes;
  char* out;
  int32_t* status_word;
  Tagged counts;
};

// A warp's rows, one after another in the result: where each of them is. By all lanes; null: there is no such row, zeros. Returns the
// rows in host memory that are copied by themselves (a bit each).
__device__ __forceinline__ unsigned find_rows(const GatherArgs& a, int64_t r0, int rows, bool apart, const char** place, int lane, int& flags) {
  const char* row = nullptr;
  bool hosted = false;
  if (lane < rows) {
    const int64_t id = a.index[r0 + lane];
    if (id < 0 || id >= a.num_nodes) {
      flags |= APT_FLAG_ID_OUT_OF_RANGE;
    } else {
      const int64_t p = a.feat_pos_map[id];
      if (p == -1) {
        flags |= APT_FLAG_FEAT_NOT_EXIST;
      } else if (p >= a.num_dev_rows || (-p - 2) >= a.num_uva_rows) {
        flags |= APT_FLAG_ID_OUT_OF_RANGE;
      } else {
        row = p >= 0 ? a.dev_feats + p * a.dev_row_bytes : a.uva_feats + (-p - 2) * a.uva_row_bytes + a.uva_col_offset_bytes;
        hosted = p < 0 && apart;
      }
    }
  }
  __syncwarp();      // (the rows before have been read)
  place[lane] = row;
  return __ballot_sync(0xffffffffu, hosted);
}

// A row in host memory, by `lanes` lanes, a vector each at a time: whole 16-byte vectors from the 32-byte sector on that it begins in, so that none of
// the sectors that cross the link is asked for twice, put in place through shared memory. Places are behind the row's first sector.
template <typename V>
struct HostRow {
  const char* sector;
  uint32_t skew, end;      // the row's own bytes

  __device__ __forceinline__ HostRow(const GatherArgs& a, const char* row)
      : sector(row - ((uintptr_t)row & 31)), skew((uint32_t)(uintptr_t)row & 31u), end(row ? skew + (uint32_t)a.dev_row_bytes : 0u) {}
  __device__ __forceinline__ uint4 load(const GatherArgs& a, uint32_t p) const {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (p + 16 <= skew || p >= end) return v;
    const char* const from = sector + p;
    if (sizeof(V) == 16 || (from >= a.uva_feats && from + 16 <= a.uva_feats + a.num_uva_rows * a.uva_row_bytes)) return ld_stream_16((const uint4*)from);
    if constexpr (sizeof(V) < 16) {      // a vector that reaches beyond the table
      V* const part = (V*)&v;
#pragma unroll
      for (uint32_t t = 0; t < 16; t += sizeof(V))
        if (p + t >= skew && p + t < end) part[t / sizeof(V)] = __ldg((const V*)(from + t));
    }
    return v;
  }
  // by all lanes of the warp; lane c of the row's
  __device__ __forceinline__ void store(char* out, uint32_t at, uint4 v, uint4* stage, int lane, uint32_t c, uint32_t lanes) const {
    if constexpr (sizeof(V) == 16) {
      const uint32_t p = at + c * 16;
      if (p >= skew && p < end) st_stream_16((uint4*)(out + (p - skew)), v);
    } else {
      __syncwarp();      // (what was staged before has been read)
      stage[lane] = v;
      __syncwarp();
      const char* const from = (const char*)(stage + (lane - c));
      const uint32_t hi = min(at + lanes * 16, end);
#pragma unroll 4
      for (uint32_t q = max(at, skew) + c * (uint32_t)sizeof(V); q < hi; q += lanes * sizeof(V)) *(V*)(out + (q - skew)) = *(const V*)(from + (q - at));
    }
  }
};
// The `which`-th of the rows of a mask, or -1.
__device__ __forceinline__ int row_of_mask(unsigned mask, int which) {
  for (; which > 0; --which) mask &= mask - 1;
  return __ffs(mask) - 1;
}

enum ChunkKind { kOneRow, kRows, kRowsSkip };

// Elements [0, total) of a chunk. kRowsSkip: not those of the rows in `skip`.
template <typename V, ChunkKind KIND>
__device__ __forceinline__ void copy_chunk(uint32_t total, uint32_t elems, uint32_t inverse, const char* const* place, unsigned skip, V* dst, int lane) {
  constexpr int U = KIND == kRowsSkip ? kGatherVectors / 2 : kGatherVectors;      // (registers)
  const char* const only = KIND == kOneRow ? place[0] : nullptr;
  for (uint32_t e0 = 0; e0 < total; e0 += 32 * U) {
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t e = e0 + u * 32 + lane, r = KIND == kOneRow ? 0u : __umulhi(2 * e + 1, inverse);
      v[u] = zero_vec<V>();
      if (e < total && !(KIND == kRowsSkip && (skip >> r & 1u))) {
        const char* const from = KIND == kOneRow ? only : place[r];
        if (from) v[u] = ld_vec<V>((const V*)from + (KIND == kOneRow ? e : e - r * elems));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t e = e0 + u * 32 + lane;
      if (e < total && !(KIND == kRowsSkip && (skip >> __umulhi(2 * e + 1, inverse) & 1u))) st_vec<V>(dst + e0 + u * 32, v[u]);
    }
  }
}

template <typename V, bool APART>
__global__ void __launch_bounds__(kGatherBlock, sizeof(V) <= 4 ? kGatherBlocksNarrow : kGatherBlocks)
k_gather(const __grid_constant__ GatherArgs a, uint32_t elems, uint32_t inverse, uint32_t rows_per_chunk, int host_shift) {
  wait_for_previous();
  // the counts of a mini-batch leave with its rows: as a kernel in front they held the rows up for 4 us
  if (a.counts.host && blockIdx.x == 0) publish_tagged(a.counts);
  __shared__ const char* places[kGatherBlock / 32][32];
  __shared__ uint4 stages[APART ? kGatherBlock / 32 : 1][32];
  const int64_t num_rows = effective_n(a.num_rows, a.num_rows_dev);
  const uint32_t n = (uint32_t)num_rows, lane = threadIdx.x & 31;      // (below 2^31, and a step beyond it below 2^32)
  const char** const place = places[threadIdx.x >> 5];
  int flags = 0;
  for (uint32_t r0 = (uint32_t)first_row(a.first_row_dev, num_rows) + (blockIdx.x * (kGatherBlock / 32) + (threadIdx.x >> 5)) * rows_per_chunk; r0 < n;
       r0 += gridDim.x * (kGatherBlock / 32) * rows_per_chunk) {
    const uint32_t rows = min(rows_per_chunk, n - r0);
    const unsigned hosted = find_rows(a, r0, rows, APART, place, lane, flags);
    __syncwarp();
    // the first of the host's rows are on their way while the others are copied
    int mine = -1;
    uint4 ahead;
    if (APART && hosted) {
      mine = row_of_mask(hosted, lane >> host_shift);
      ahead = HostRow<V>(a, mine < 0 ? nullptr : place[mine]).load(a, (lane & ((1u << host_shift) - 1u)) * 16);
    }
    V* const dst = (V*)(a.out + r0 * a.dev_row_bytes) + lane;
    if (APART && hosted == 0xffffffffu >> (32 - rows)) {
    } else if (sizeof(V) < 16 && rows_per_chunk == 1) {
      copy_chunk<V, kOneRow>(elems, elems, inverse, place, 0u, dst, lane);
    } else if (APART && hosted) {
      copy_chunk<V, kRowsSkip>(rows * elems, elems, inverse, place, hosted, dst, lane);
    } else {
      copy_chunk<V, kRows>(rows * elems, elems, inverse, place, 0u, dst, lane);
    }
    if constexpr (APART) {
      const uint32_t host_lanes = 1u << host_shift, c = lane & (host_lanes - 1u);
      for (unsigned left = hosted; left;) {
        if (left != hosted) mine = row_of_mask(left, lane >> host_shift);
        const HostRow<V> row(a, mine < 0 ? nullptr : place[mine]);
        char* const out = a.out + ((int64_t)r0 + mine) * a.dev_row_bytes;
#pragma unroll 1
        for (uint32_t at = 0; at < (uint32_t)a.dev_row_bytes + 31; at += host_lanes * 16) {      // (once, where a row does not take all lanes)
          if (at || left != hosted) ahead = row.load(a, at + c * 16);
          row.store(out, at, ahead, stages[threadIdx.x >> 5], lane, c, host_lanes);
        }
        for (uint32_t k = 0; k < 32; k += host_lanes) left &= left - 1;
      }
    }
  }
  if (flags) atomicOr(a.status_word, flags);
}

static int vec_width(uint64_t bits) {
  for (int w = 16; w > 1; w >>= 1)
    if ((bits & (uint64_t)(w - 1)) == 0) return w;
  return 1;
}

// Blocks an SM for a gather that runs beside other kernels: enough reads over the host link for its full rate (one block's
// warps have 4 KiB each in flight, of the 80 KB that rate times latency asks of the whole chip), and room for the others,
// which at the full grid wait until it ends.
constexpr int kNarrowBlocks = 1;

static int gather_launch(const GatherArgs& a, cudaStream_t s, bool narrow = false) {
  uint64_t bits = (uint64_t)a.dev_row_bytes | (uintptr_t)a.out;
  if (a.num_dev_rows > 0) bits |= (uintptr_t)a.dev_feats;
  if (a.num_uva_rows > 0) bits |= (uint64_t)a.uva_row_bytes | (uint64_t)a.uva_col_offset_bytes | (uintptr_t)a.uva_feats;
  const int width = vec_width(bits);
  const int64_t elems = a.dev_row_bytes / width;
  // One row where every warp of the chip can have its own (a pass over several waits for the slowest, a row from the host); else as many
  // as fill the lanes or take up to kChunkBytes, while every warp of the chip has that many (and 32, a lane to look each up).
  int rows = 1;
  while (rows < 32 && (int64_t)rows * kNumSMs * 64 < a.num_rows && (rows * a.dev_row_bytes < 512 || 2 * rows * a.dev_row_bytes <= kChunkBytes))
    rows <<= 1;
  // (2 e + 1) / (2 elems) in 32 bits is the row of element e: exact while e < 2^18 and elems < 2^12, and rows that share a chunk have
  // 4096 bytes or fewer together
  const uint32_t inverse = rows > 1 ? (uint32_t)(((1ull << 31) + elems - 1) / elems) : 0u;
  int grid = wave_grid(ceil_div(a.num_rows, (int64_t)rows * (kGatherBlock / 32)), 8, kGatherWaves);
  if (narrow && grid > kNumSMs * kNarrowBlocks) grid = kNumSMs * kNarrowBlocks;
  // rows in host memory that end inside a 32-byte sector go by themselves
  const bool apart = a.num_uva_rows > 0 && ((((uint64_t)a.dev_row_bytes | (uint64_t)a.uva_row_bytes | (uint64_t)a.uva_col_offset_bytes | (uintptr_t)a.uva_feats) & 31) != 0);
  int host_shift = 2;      // lanes to a host row
  while (host_shift < 5 && (16 << host_shift) < a.dev_row_bytes + 31) ++host_shift;
  ProfScope prof("gather_hit", s);
#define APT_GATHER(V)                                                                                                   \
  if (apart) APT_FOLLOW((k_gather<V, true>), grid, kGatherBlock, 0, s, a, (uint32_t)elems, inverse, (uint32_t)rows, host_shift);    \
  else APT_FOLLOW((k_gather<V, false>), grid, kGatherBlock, 0, s, a, (uint32_t)elems, inverse, (uint32_t)rows, host_shift)
  switch (width) {
    case 16: APT_GATHER(uint4); break;
    case 8: APT_GATHER(uint2); break;
    case 4: APT_GATHER(uint32_t); break;
    case 2: APT_GATHER(uint16_t); break;
    default: APT_GATHER(uint8_t); break;
  }
#undef APT_GATHER
  return APT_OK;
}

static int gather_check(const char* who, const GatherArgs& a) {
  APT_CHECK_ARG(a.num_rows >= 0 && a.num_rows < (int64_t)0x7fffffff, "%s: bad num_rows", who);
  APT_CHECK_ARG(a.dev_row_bytes > 0 && a.num_dev_rows >= 0 && a.num_uva_rows >= 0 && a.num_nodes >= 0,
                "%s: bad table sizes", who);
  APT_CHECK_ARG(a.num_uva_rows == 0 || (a.uva_col_offset_bytes >= 0 &&
                                         a.uva_col_offset_bytes + a.dev_row_bytes <= a.uva_row_bytes),
                "%s: column window [%lld,+%lld) outside a %lld-byte host row", who,
                (long long)a.uva_col_offset_bytes, (long long)a.dev_row_bytes, (long long)a.uva_row_bytes);
  if (a.num_rows == 0) return APT_OK;
  APT_CHECK_ARG(a.index && a.feat_pos_map && a.out && a.status_word, "%s: null pointer", who);
  APT_CHECK_ARG((a.num_dev_rows == 0 || a.dev_feats) && (a.num_uva_rows == 0 || a.uva_feats),
                "%s: null feature table", who);
  return APT_OK;
}

}  // namespace apt

extern "C" int apt_set_tunable(const char* name, int64_t value) {
  using namespace apt;
  APT_CHECK_ARG(name, "apt_set_tunable: null name");
  // knobs of forms of the gather that are gone: taken, without effect, and said so, since a measurement would show nothing
  static const struct { const char* name; int64_t lo, hi; } retired[] = {
      {"gather_miss_mode", 0, 1}, {"gather_miss_blocks", 1, 65535}, {"gather_miss_kb_per_block", 0, 1 << 20},
      {"gather_hit_mode", 0, 2}, {"gather_hit_waves", 1, 64}};
  for (const auto& r : retired)
    if (!strcmp(name, r.name) && value >= r.lo && value <= r.hi) {
      fprintf(stderr, "apt_set_tunable: %s has no effect any more\n", name);
      return APT_OK;
    }
  if (!strcmp(name, "relabel_small") && value >= 0 && value <= 1) {
    set_relabel_small(value != 0);
    return APT_OK;
  }
  if (!strcmp(name, "bulk_wait_polls") && value >= 0 && value <= 1 << 20) {
    set_bulk_wait_polls((int)value);
    return APT_OK;
  }
  set_error("apt_set_tunable: unknown name or bad value: %s = %lld", name, (long long)value);
  return APT_ERR_BAD_ARG;
}

// The gather needs no scratch; the workspace argument and its (small) size stay for callers.
extern "C" size_t apt_gather_workspace_bytes(int64_t num_rows) { return num_rows < 0 ? 0 : 256; }

extern "C" int apt_gather_rows(const int64_t* index, int64_t num_rows,
                               const int64_t* num_rows_dev, const int64_t* feat_pos_map,
                               int64_t num_nodes, const void* dev_feats, int64_t num_dev_rows,
                               int64_t dev_row_bytes, const void* uva_feats,
                               int64_t num_uva_rows, int64_t uva_row_bytes,
                               int64_t uva_col_offset_bytes, void* out, void* workspace,
                               size_t workspace_bytes, int32_t* status_word, void* stream) {
  return apt_gather_rows_from(index, num_rows, num_rows_dev, nullptr, feat_pos_map, num_nodes, dev_feats,
                              num_dev_rows, dev_row_bytes, uva_feats, num_uva_rows, uva_row_bytes,
                              uva_col_offset_bytes, out, workspace, workspace_bytes, status_word, stream);
}

extern "C" int apt_gather_rows_from(const int64_t* index, int64_t num_rows,
                                    const int64_t* num_rows_dev, const int64_t* first_row_dev,
                                    const int64_t* feat_pos_map,
                                    int64_t num_nodes, const void* dev_feats, int64_t num_dev_rows,
                                    int64_t dev_row_bytes, const void* uva_feats,
                                    int64_t num_uva_rows, int64_t uva_row_bytes,
                                    int64_t uva_col_offset_bytes, void* out, void* workspace,
                                    size_t workspace_bytes, int32_t* status_word, void* stream) {
  using namespace apt;
  const GatherArgs a{index, num_rows, num_rows_dev, first_row_dev, feat_pos_map, num_nodes, (const char*)dev_feats,
                     num_dev_rows, dev_row_bytes, (const char*)uva_feats, num_uva_rows, uva_row_bytes,
                     uva_col_offset_bytes, (char*)out, status_word, Tagged{}};
  const int rc = gather_check("apt_gather_rows", a);
  if (rc != APT_OK || num_rows == 0) return rc;
  APT_CHECK_ARG(workspace && ((uintptr_t)workspace & 255) == 0,
                "apt_gather_rows: workspace must be non-null and 256-byte aligned");
  if (workspace_bytes < apt_gather_workspace_bytes(num_rows)) {
    set_error("apt_gather_rows: workspace %zu < %zu bytes", workspace_bytes, apt_gather_workspace_bytes(num_rows));
    return APT_ERR_CAPACITY;
  }
  return gather_launch(a, (cudaStream_t)stream);
}

extern "C" int apt_gather_rows_publish(const int64_t* index, int64_t num_rows, const int64_t* num_rows_dev, const int64_t* first_row_dev,
                                       const int64_t* feat_pos_map, int64_t num_nodes, const void* dev_feats, int64_t num_dev_rows,
                                       int64_t dev_row_bytes, const void* uva_feats, int64_t num_uva_rows, int64_t uva_row_bytes,
                                       int64_t uva_col_offset_bytes, void* out, int32_t* status_word, const int64_t* words, int count,
                                       const int64_t* last, const int64_t* sequence_dev, int64_t sequence, int64_t* host, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(words && last && host && count >= 1 && count <= 4096, "apt_gather_rows_publish: bad argument");
  const GatherArgs a{index, num_rows, num_rows_dev, first_row_dev, feat_pos_map, num_nodes, (const char*)dev_feats,
                     num_dev_rows, dev_row_bytes, (const char*)uva_feats, num_uva_rows, uva_row_bytes,
                     uva_col_offset_bytes, (char*)out, status_word, Tagged{words, count, last, sequence_dev, sequence, host}};
  const int rc = gather_check("apt_gather_rows_publish", a);
  if (rc != APT_OK) return rc;
  if (num_rows == 0) return apt_publish_tagged(words, count, last, sequence_dev, sequence, host, stream);
  return gather_launch(a, (cudaStream_t)stream);
}

extern "C" int apt_gather_rows_beside(const int64_t* index, int64_t num_rows,
                                    const int64_t* num_rows_dev, const int64_t* feat_pos_map,
                                    int64_t num_nodes, const void* dev_feats, int64_t num_dev_rows,
                                    int64_t dev_row_bytes, const void* uva_feats,
                                    int64_t num_uva_rows, int64_t uva_row_bytes,
                                    int64_t uva_col_offset_bytes, void* out, void* workspace,
                                    size_t workspace_bytes, int32_t* status_word, void* stream) {
  using namespace apt;
  const GatherArgs a{index, num_rows, num_rows_dev, nullptr, feat_pos_map, num_nodes, (const char*)dev_feats,
                     num_dev_rows, dev_row_bytes, (const char*)uva_feats, num_uva_rows, uva_row_bytes,
                     uva_col_offset_bytes, (char*)out, status_word, Tagged{}};
  const int rc = gather_check("apt_gather_rows", a);
  if (rc != APT_OK || num_rows == 0) return rc;
  APT_CHECK_ARG(workspace && ((uintptr_t)workspace & 255) == 0,
                "apt_gather_rows: workspace must be non-null and 256-byte aligned");
  if (workspace_bytes < apt_gather_workspace_bytes(num_rows)) {
    set_error("apt_gather_rows: workspace %zu < %zu bytes", workspace_bytes, apt_gather_workspace_bytes(num_rows));
    return APT_ERR_CAPACITY;
  }
  return gather_launch(a, (cudaStream_t)stream, true);
}

// The same without a workspace argument, for callers that must not allocate. The limit on the rows of a call dates from
// a form that kept its scratch in the library and is part of the interface.
namespace apt {
constexpr int64_t kStaticGatherMaxRows = 1 << 20;
}  // namespace apt

extern "C" int64_t apt_gather_static_max_rows(void) { return apt::kStaticGatherMaxRows; }

extern "C" int apt_gather_rows_static(const int64_t* index, int64_t num_rows,
                                      const int64_t* feat_pos_map, int64_t num_nodes,
                                      const void* dev_feats, int64_t num_dev_rows,
                                      int64_t dev_row_bytes, const void* uva_feats,
                                      int64_t num_uva_rows, int64_t uva_row_bytes,
                                      int64_t uva_col_offset_bytes, void* out,
                                      int32_t* status_word, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(num_rows >= 0, "apt_gather_rows_static: negative num_rows");
  if (num_rows > kStaticGatherMaxRows) {
    set_error("apt_gather_rows_static: %lld rows exceed the built-in scratch's limit of %lld rows per call (kept although the "
              "scratch is gone); split the request or use apt_gather_rows",
              (long long)num_rows, (long long)kStaticGatherMaxRows);
    return APT_ERR_CAPACITY;
  }
  const GatherArgs a{index, num_rows, nullptr, nullptr, feat_pos_map, num_nodes, (const char*)dev_feats,
                     num_dev_rows, dev_row_bytes, (const char*)uva_feats, num_uva_rows, uva_row_bytes,
                     uva_col_offset_bytes, (char*)out, status_word, Tagged{}};
  const int rc = gather_check("apt_gather_rows_static", a);
  if (rc != APT_OK || num_rows == 0) return rc;
  return gather_launch(a, (cudaStream_t)stream);
}
