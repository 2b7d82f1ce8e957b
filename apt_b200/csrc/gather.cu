// Cache-aware feature-row gather: one launch, no scratch.
//
// A warp takes a chunk of rows. One lane to a row looks the id up (p = feat_pos_map[id]: p >= 0 cache row, p < -1 row -p - 2 of the
// table in page-locked host memory, p == -1 no such row: zeros and a flag) and leaves the row's address in shared memory. In
// the result the chunk is one run of elements, which the warp copies from end to end, 8 of 32 lanes each in flight:
// rows of any width fill all lanes, and what is in flight does not depend on it. The division that finds an element's row is a
// multiplication.
//
// Rows one after another, the form before this, had a row of more than 32 elements as one load of 32 in flight, and a row of
// 33 took the steps of 64. us, that form -> this one (distinct rows, all cached unless it says so):
//   495 616 x 2 KiB     331 -> 320 (6.36 TB/s, 0.97 of the measured copy rate)
//   243 961 x 880 B     145 -> 76           243 961 x 882 B (2-byte elements)   172 -> 113
//   200 000 x 1 KiB     104 -> 68           200 000 x 1200 B                    144 -> 84
//   318 250 x 288 B      49 -> 40           318 250 x 292 B (4-byte elements)    66 -> 47
//   400 000 x 200 B (8-byte elements) 48 -> 41      400 000 x 66 B (2-byte elements)  70 -> 23
//   143 000 x 512 B, 2.7 % of them from host memory 50.7 -> 46.7
// Bound by HBM, by the host link (64 bytes to a few KiB a request, about 50 M rows/s) and, small requests, by three dependent
// loads; rows of 2-byte elements by their loads and stores (copying 882-byte rows through shared memory in 16-byte vectors, shifted on the way
// out, took 93 instead of 113 us and rows below 512 bytes longer; two elements to a lane 135). The host rows by themselves, in
// front of the others, two at a time through shared memory: 143 000 x 512 B 90. Chunks of 16 KiB instead of kChunkBytes: 880 B 80, 1 KiB 71;
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

// A warp's rows, one after another in the result: where each of them is. By all lanes; null: there is no such row, zeros.
__device__ __forceinline__ void find_rows(const GatherArgs& a, int64_t r0, int rows, const char** place, int lane, int& flags) {
  const char* row = nullptr;
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
      }
    }
  }
  __syncwarp();      // (the rows before have been read)
  place[lane] = row;
  __syncwarp();
}

template <typename V>
__global__ void __launch_bounds__(kGatherBlock, kGatherBlocks)
k_gather(const __grid_constant__ GatherArgs a, uint32_t elems, uint32_t inverse, int rows_per_chunk) {
  wait_for_previous();
  // the counts of a mini-batch leave with its rows: as a kernel in front they held the rows up for 4 us
  if (a.counts.host && blockIdx.x == 0) publish_tagged(a.counts);
  __shared__ const char* places[kGatherBlock / 32][32];
  const int64_t n = effective_n(a.num_rows, a.num_rows_dev), first = first_row(a.first_row_dev, n);
  const int lane = threadIdx.x & 31;
  const char** const place = places[threadIdx.x >> 5];
  const int64_t warps = (int64_t)gridDim.x * (kGatherBlock / 32);
  const int64_t warp = (int64_t)blockIdx.x * (kGatherBlock / 32) + (threadIdx.x >> 5);
  int flags = 0;
  for (int64_t r0 = first + warp * rows_per_chunk; r0 < n; r0 += warps * rows_per_chunk) {
    const int rows = (int)min((int64_t)rows_per_chunk, n - r0);
    find_rows(a, r0, rows, place, lane, flags);
    const uint32_t total = (uint32_t)rows * elems;
    V* const dst = (V*)(a.out + r0 * a.dev_row_bytes) + lane;
    for (uint32_t e0 = 0; e0 < total; e0 += 32 * kGatherVectors) {
      V v[kGatherVectors];
#pragma unroll
      for (int u = 0; u < kGatherVectors; ++u) {
        const uint32_t e = e0 + u * 32 + lane, r = __umulhi(2 * e + 1, inverse);
        v[u] = zero_vec<V>();
        if (e < total) {
          const char* const from = place[r];
          if (from) v[u] = ld_vec<V>((const V*)from + (e - r * elems));
        }
      }
#pragma unroll
      for (int u = 0; u < kGatherVectors; ++u)
        if (e0 + u * 32 + lane < total) st_vec<V>(dst + e0 + u * 32, v[u]);
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
  ProfScope prof("gather_hit", s);
  switch (width) {
    case 16: APT_FOLLOW(k_gather<uint4>, grid, kGatherBlock, 0, s, a, (uint32_t)elems, inverse, rows); break;
    case 8: APT_FOLLOW(k_gather<uint2>, grid, kGatherBlock, 0, s, a, (uint32_t)elems, inverse, rows); break;
    case 4: APT_FOLLOW(k_gather<uint32_t>, grid, kGatherBlock, 0, s, a, (uint32_t)elems, inverse, rows); break;
    case 2: APT_FOLLOW(k_gather<uint16_t>, grid, kGatherBlock, 0, s, a, (uint32_t)elems, inverse, rows); break;
    default: APT_FOLLOW(k_gather<uint8_t>, grid, kGatherBlock, 0, s, a, (uint32_t)elems, inverse, rows); break;
  }
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
