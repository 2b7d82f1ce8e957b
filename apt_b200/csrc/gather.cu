// Cache-aware feature-row gather: one launch, no scratch.
//
// A warp takes a chunk of rows. One lane to a row looks the id up (p = feat_pos_map[id]: p >= 0 cache row, p < -1 host row
// -p - 2, p == -1 no such row: zeros and a flag); the rows that live in page-locked host memory are copied first, then
// those of the cache, with four vectors (and, narrow rows, several rows) a lane in flight. The reads over the host
// link of all warps are outstanding together and beside the other warps' copies from HBM.
//
// Against the three kernels it replaces (decode ids and compact a miss list, copy the hits, copy the misses), B200:
//   495 616 rows x 2 KiB      357 -> 327 us (6.2 TB/s, 0.95 of the measured copy rate)
//   143 000 rows x 512 B      31 -> 28 us; with 2.7 % from host memory 72 -> 50 us
//   1 203 rows x 400 B, a tenth from host memory    15.5 -> 5.0 us
//   6 158 rows x 390 B (2-byte vectors)             26 -> 4.7 us
// and, in mini-batches that run beside one another on lanes, 7 470 -> 7 830 papers-shaped mini-batches a second. Bound
// by HBM, by the host link (64 bytes to a few KiB a request, about 50 M rows/s) and, small requests, by three dependent
// loads.
//
// Rows are opaque bytes. The vector width V is the widest of 16/8/4/2/1 bytes that divides every row size, column offset
// and base address involved.
#include <string.h>

#include "common.cuh"

namespace apt {

constexpr int kRowsPerGroup = 4;   // rows (or vectors of a long row) whose loads are in flight together
constexpr int kGatherBlock = 256;
constexpr int kGatherWaves = 4;    // cap on the grid, in units of 148 x 8 blocks

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

// A group of kRowsPerGroup rows a lane from those whose flag is set in `mask`: lpr lanes to a row of up to 32 vectors,
// 32 / lpr rows side by side. `p` is the lane's own row's position in the table, src_of finds the row there.
template <typename V>
struct RowGroup {
  V v[kRowsPerGroup];
  int row[kRowsPerGroup];     // row of the chunk, -1: none

  template <typename SRC>
  __device__ __forceinline__ void load(unsigned& mask, int64_t p, int chunks, int lpr, SRC src_of, int lane) {
    const int side = 32 / lpr, which = lane / lpr, c = lane & (lpr - 1);
#pragma unroll
    for (int k = 0; k < kRowsPerGroup; ++k) {
      // this lane's row is the `which`-th of the next `side` rows of the mask
      int mine = -1;
      for (int q = 0; q < side && mask; ++q) {
        const int l = __ffs(mask) - 1;
        mask &= mask - 1;
        if (q == which) mine = l;
      }
      const int64_t pk = __shfl_sync(0xffffffffu, p, mine < 0 ? 0 : mine);
      row[k] = c < chunks ? mine : -1;
      if (row[k] >= 0) v[k] = ld_vec<V>((const V*)src_of(pk) + c);
    }
  }
  __device__ __forceinline__ void store(char* out, int64_t first_row, int64_t row_bytes, int lpr, int lane) const {
    const int c = lane & (lpr - 1);
#pragma unroll
    for (int k = 0; k < kRowsPerGroup; ++k)
      if (row[k] >= 0) st_vec<V>((V*)(out + (first_row + row[k]) * row_bytes) + c, v[k]);
  }
};

// All rows of the mask; rows of more than 32 vectors one at a time, four vectors a lane in flight.
template <typename V, typename SRC>
__device__ __forceinline__ void copy_rows(unsigned mask, int64_t p, int64_t first_row, int chunks, int lpr, SRC src_of, char* out,
                                          int64_t row_bytes, int lane) {
  if (chunks <= 32) {
    while (mask) {
      RowGroup<V> g;
      g.load(mask, p, chunks, lpr, src_of, lane);
      g.store(out, first_row, row_bytes, lpr, lane);
    }
    return;
  }
  while (mask) {
    const int l = __ffs(mask) - 1;
    mask &= mask - 1;
    const V* const src = (const V*)src_of(__shfl_sync(0xffffffffu, p, l));
    V* const dst = (V*)(out + (first_row + l) * row_bytes);
    int c = lane;
    for (; c + 96 < chunks; c += 128) {
      V v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = ld_vec<V>(src + c + 32 * k);
#pragma unroll
      for (int k = 0; k < 4; ++k) st_vec<V>(dst + c + 32 * k, v[k]);
    }
    for (; c < chunks; c += 32) st_vec<V>(dst + c, ld_vec<V>(src + c));
  }
}

template <typename V>
__global__ void __launch_bounds__(kGatherBlock)
k_gather(const int64_t* __restrict__ index, int64_t n, const int64_t* __restrict__ n_dev, const int64_t* __restrict__ first_dev,
         const int64_t* __restrict__ pos_map, int64_t num_nodes, const char* __restrict__ dev_feats, int64_t num_dev_rows,
         const char* __restrict__ uva_feats, int64_t num_uva_rows, int64_t uva_row_bytes, int64_t col_offset_bytes,
         int64_t row_bytes, int rows_per_chunk, int lpr, char* __restrict__ out, int32_t* status, const Tagged counts) {
  wait_for_previous();
  // the counts of a mini-batch leave with its rows: as a kernel in front they held the rows up for 4 us
  if (counts.host && blockIdx.x == 0) publish_tagged(counts);
  n = effective_n(n, n_dev);
  const int64_t first = first_row(first_dev, n);
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (kGatherBlock / 32);
  const int64_t warp = (int64_t)blockIdx.x * (kGatherBlock / 32) + (threadIdx.x >> 5);
  const int chunks = (int)(row_bytes / (int64_t)sizeof(V));
  int flags = 0;
  for (int64_t r0 = first + warp * rows_per_chunk; r0 < n; r0 += warps * rows_per_chunk) {
    int64_t p = -2;
    const bool live = lane < rows_per_chunk && r0 + lane < n;
    if (live) {
      const int64_t id = index[r0 + lane];
      p = -1;
      if (id < 0 || id >= num_nodes) {
        flags |= APT_FLAG_ID_OUT_OF_RANGE;
      } else {
        p = pos_map[id];
        if (p == -1) {
          flags |= APT_FLAG_FEAT_NOT_EXIST;
        } else if (p >= num_dev_rows || (-p - 2) >= num_uva_rows) {
          flags |= APT_FLAG_ID_OUT_OF_RANGE;
          p = -1;
        }
      }
    }
    const unsigned hits = __ballot_sync(0xffffffffu, live && p >= 0);
    const unsigned misses = __ballot_sync(0xffffffffu, live && p < -1);
    unsigned none = __ballot_sync(0xffffffffu, live && p == -1);
    auto cached = [&](int64_t q) { return dev_feats + q * row_bytes; };
    auto hosted = [&](int64_t q) { return uva_feats + (-q - 2) * uva_row_bytes + col_offset_bytes; };
    // the reads over the host link first: they take longest, and the other warps' copies run meanwhile (holding them in
    // registers over this warp's own copies cost every request without misses a fifth)
    copy_rows<V>(misses, p, r0, chunks, lpr, hosted, out, row_bytes, lane);
    copy_rows<V>(hits, p, r0, chunks, lpr, cached, out, row_bytes, lane);
    while (none) {                 // no such row: zeros
      const int l = __ffs(none) - 1;
      none &= none - 1;
      for (int c = lane; c < chunks; c += 32) st_vec<V>((V*)(out + (r0 + l) * row_bytes) + c, zero_vec<V>());
    }
  }
  if (flags) atomicOr(status, flags);
}

static int vec_width(uint64_t bits) {
  for (int w = 16; w > 1; w >>= 1)
    if ((bits & (uint64_t)(w - 1)) == 0) return w;
  return 1;
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

// Blocks an SM for a gather that runs beside other kernels: enough reads over the host link for its full rate (one block's
// warps have 16 KiB each in flight, of the 80 KB that rate times latency asks of the whole chip), and room for the others,
// which at the full grid wait until it ends.
constexpr int kNarrowBlocks = 1;

static int gather_launch(const GatherArgs& a, cudaStream_t s, bool narrow = false) {
  uint64_t bits = (uint64_t)a.dev_row_bytes | (uintptr_t)a.out;
  if (a.num_dev_rows > 0) bits |= (uintptr_t)a.dev_feats;
  if (a.num_uva_rows > 0) bits |= (uint64_t)a.uva_row_bytes | (uint64_t)a.uva_col_offset_bytes | (uintptr_t)a.uva_feats;
  const int width = vec_width(bits);
  const int64_t vectors = a.dev_row_bytes / width;
  int lpr = 1;
  while (lpr < vectors && lpr < 32) lpr <<= 1;
  // chunks as large as leave every warp of the chip one: a small request wants all SMs, a large one few lookups
  const int64_t all_warps = (int64_t)kNumSMs * 8 * (kGatherBlock / 32);
  int per = 32 / lpr;
  while (per < 32 && (int64_t)per * all_warps < a.num_rows) per <<= 1;
  int grid = wave_grid(ceil_div(a.num_rows, (int64_t)per * (kGatherBlock / 32)), 8, kGatherWaves);
  if (narrow && grid > kNumSMs * kNarrowBlocks) grid = kNumSMs * kNarrowBlocks;
  ProfScope prof("gather_hit", s);
#define APT_GATHER(V)                                                                                                     \
  APT_FOLLOW(k_gather<V>, grid, kGatherBlock, 0, s, a.index, a.num_rows, a.num_rows_dev, a.first_row_dev, a.feat_pos_map, \
             a.num_nodes, a.dev_feats, a.num_dev_rows, a.uva_feats, a.num_uva_rows, a.uva_row_bytes,                      \
             a.uva_col_offset_bytes, a.dev_row_bytes, per, lpr, a.out, a.status_word, a.counts)
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
