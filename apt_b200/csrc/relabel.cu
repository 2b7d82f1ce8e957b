// Relabelling of a sampled layer: unique of cat(seeds, neighbours) in order of
// first occurrence, and the new id of every neighbour.
//
// One open-addressing table (linear probing, load <= 2/3) in the caller's
// workspace holds, per distinct id, the smallest position at which it occurs.
// An item is a "first occurrence" iff that minimum equals its own position;
// an ordered compaction turns the first-occurrence flags into new ids, which
// makes the result independent of the table layout and of thread scheduling.
// Three launches:
//
//   k_insert        items -> table (CAS on the key, atomicMin on the position),
//                   remembers each item's slot. When the layer is sampled by this
//                   library the sampling kernel does this itself
//                   (sample_replace_kernel<G, true>, apt_sample_relabel_csc) and the
//                   neighbour list is never read back.
//   k_first         which items are first occurrences: one bit an item, and the number of
//                   ones before every 32 items of a tile and in every tile. Leaves the
//                   position of an id's first occurrence beside every other item.
//   k_relabel       the new id of an id is the number of ones before its first occurrence: a
//                   tile's share (added up by every block in shared memory) plus a look at
//                   the bits. No block waits for another one; the form before this chained its
//                   tiles by a look-back and sent the ids through the table (1.08 M items:
//                   29 + 20 us). The first occurrence also empties its id's slot.
//
// Layers of up to 8192 items run in one block with the table in shared memory
// (k_relabel_small below).
//
// The table is empty between calls (apt_relabel_workspace_init empties it once,
// each call empties the slots it used), so a call costs what its own item count
// costs and no clearing pass is needed.
#include "sample_kernels.cuh"

namespace apt {

constexpr int kRelabelBlock = 1024;

static size_t relabel_bytes_for(int64_t items) {
  const int64_t n = items > 0 ? items : 1;
  return align_up((size_t)relabel_capacity(n) * sizeof(Slot), 256) + align_up((size_t)n * 4, 256) +
         align_up((size_t)(n / 32 + 1) * 8, 256) + (size_t)kMaxTiles * 4;
}

// The layout depends only on the size of the workspace, not on the call, so
// that "empty between calls" holds for one fixed slot region.
static bool relabel_layout(char* base, size_t bytes, RelabelWs* ws) {
  // 16 * 1.5 + 4 + 8 / 32 bytes per item plus the tiles: first guess, then shrink until it fits
  int64_t items = bytes > 20480 ? (int64_t)((bytes - 20480) / 283 * 10) : 0;
  while (items > 0 && relabel_bytes_for(items) > bytes) items -= 1 + items / 4096;
  ws->items_ws = items;
  if (items <= 0) return false;
  const size_t o_slot_of = align_up((size_t)relabel_capacity(items) * sizeof(Slot), 256);
  const size_t o_words = o_slot_of + align_up((size_t)items * 4, 256);
  ws->slots = (Slot*)base;
  ws->slot_of = (int32_t*)(base + o_slot_of);
  ws->words = (uint2*)(base + o_words);
  ws->tile_count = (int32_t*)(base + o_words + align_up((size_t)(items / 32 + 1) * 8, 256));
  return true;
}

__device__ __forceinline__ int64_t item_at(const int64_t* seeds, int64_t S,
                                           const int64_t* nbrs, int64_t i) {
  return i < S ? seeds[i] : nbrs[i - S];
}

// Pass 1 when the ids come from memory (apt_relabel_csc).
__global__ void __launch_bounds__(256)
k_insert(const int64_t* __restrict__ seeds, int64_t S_host, const int64_t* __restrict__ nbrs,
         int64_t M_host, const int64_t* __restrict__ S_dev, int64_t per_seed, RelabelWs ws,
         int32_t* status) {
  wait_for_previous();
  const RelabelDims d = relabel_dims(S_host, M_host, S_dev, per_seed);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int flags = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < d.n; i += stride)
    ws.slot_of[i] = table_insert(ws.slots, d.cap, item_at(seeds, d.S, nbrs, i), (uint32_t)i, &flags);
  if (flags) atomicOr(status, flags);
}

// ---- pass 2: first occurrences --------------------------------------------------------
// One block to a tile of 2^tile_shift (at least kSubTile) consecutive items.
constexpr int kFirstThreads = 256;
constexpr int kFirstItems = 4;
constexpr int kSubTile = kFirstThreads * kFirstItems;
static_assert(kSubTile / 32 == 32, "a sub-tile's words are scanned by one warp");

__global__ void __launch_bounds__(kFirstThreads)
k_first(int64_t S_host, int64_t M_host, const int64_t* __restrict__ S_dev, int64_t per_seed, RelabelWs ws, int tile_shift) {
  wait_for_previous();
  __shared__ uint32_t counts[32], bases[32];
  const RelabelDims d = relabel_dims(S_host, M_host, S_dev, per_seed);
  const int64_t first = (int64_t)blockIdx.x << tile_shift;
  if (first >= d.n) return;
  const int64_t last = min(d.n, first + ((int64_t)1 << tile_shift));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t running = 0;
  for (int64_t base = first; base < last; base += kSubTile) {
    int32_t slot[kFirstItems];
    uint32_t min_pos[kFirstItems];
    unsigned ones[kFirstItems];
#pragma unroll
    for (int k = 0; k < kFirstItems; ++k) {
      const int64_t i = base + k * kFirstThreads + threadIdx.x;
      slot[k] = i < last ? ws.slot_of[i] : -1;
    }
#pragma unroll
    for (int k = 0; k < kFirstItems; ++k) min_pos[k] = slot[k] >= 0 ? ws.slots[slot[k]].min_pos : kNoPos;
#pragma unroll
    for (int k = 0; k < kFirstItems; ++k) {
      const int64_t i = base + k * kFirstThreads + threadIdx.x;
      const bool one = slot[k] >= 0 && min_pos[k] == (uint32_t)i;
      ones[k] = __ballot_sync(0xffffffffu, one);
      if (lane == 0) counts[k * (kFirstThreads / 32) + warp] = __popc(ones[k]);
      if (slot[k] >= 0 && !one) ws.slot_of[i] = (int32_t)min_pos[k];
    }
    __syncthreads();
    if (warp == 0) {
      const uint32_t c = counts[lane];
      uint32_t upto = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += t;
      }
      bases[lane] = running + upto - c;
      running += __shfl_sync(0xffffffffu, upto, 31);
    }
    __syncthreads();
    if (lane < kFirstItems) {
      const int w = lane * (kFirstThreads / 32) + warp;
      unsigned mine = ones[0];
#pragma unroll
      for (int k = 1; k < kFirstItems; ++k)
        if (lane == k) mine = ones[k];
      if (base + w * 32 < last) ws.words[(base >> 5) + w] = make_uint2(bases[w], mine);
    }
  }
  if (threadIdx.x == 0) ws.tile_count[blockIdx.x] = (int32_t)running;
}

// ---- pass 3: new ids ------------------------------------------------------------------
// out_col (may be null): the position of each neighbour's seed, the other side of the block's edges.
__global__ void __launch_bounds__(256)
k_relabel(int64_t S_host, int64_t M_host, const int64_t* __restrict__ S_dev, int64_t per_seed, RelabelWs ws, int tile_shift,
          int64_t* __restrict__ out_unique, int64_t* __restrict__ out, int64_t* __restrict__ out_col,
          int64_t* __restrict__ out_num_unique, const RowTables tables, int32_t* status) {
  wait_for_previous();
  __shared__ int tile_base[kMaxTiles];
  __shared__ int scratch[33];
  const RelabelDims d = relabel_dims(S_host, M_host, S_dev, per_seed);
  const int tiles = (int)((d.n + ((int64_t)1 << tile_shift) - 1) >> tile_shift);
  const int each = (tiles + (int)blockDim.x - 1) / (int)blockDim.x;
  for (int t = threadIdx.x; t < tiles; t += blockDim.x) tile_base[t] = ws.tile_count[t];
  __syncthreads();
  int mine = 0;
  const int t0 = threadIdx.x * each, t1 = min(tiles, t0 + each);
  for (int t = t0; t < t1; ++t) mine += tile_base[t];
  int total;
  int at = block_exclusive_scan(mine, scratch, &total);
  for (int t = t0; t < t1; ++t) {
    const int c = tile_base[t];
    tile_base[t] = at;
    at += c;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *out_num_unique = total;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int K = 4;
  int flags = 0;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; base < d.n; base += stride * K) {
    int32_t v[K];
    uint2 word[K];
    unsigned long long key[K];
    bool one[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t i = base + k * stride;
      v[k] = i < d.n ? ws.slot_of[i] : -1;
      one[k] = v[k] >= 0 && (ws.words[i >> 5].y >> (i & 31) & 1u);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (v[k] < 0) continue;
      // where the id occurs first: here, or at the position that pass 2 left
      const uint32_t pos = one[k] ? (uint32_t)(base + k * stride) : (uint32_t)v[k];
      word[k] = ws.words[pos >> 5];
      if (one[k]) key[k] = ws.slots[v[k]].key;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t i = base + k * stride;
      if (i >= d.n) continue;
      if (out_col && i >= d.S) out_col[i - d.S] = (int64_t)((uint32_t)(i - d.S) / (uint32_t)per_seed);
      if (v[k] < 0) {
        if (i >= d.S) out[i - d.S] = -1;
        continue;
      }
      const uint32_t pos = one[k] ? (uint32_t)i : (uint32_t)v[k];
      const int64_t id = (int64_t)tile_base[pos >> tile_shift] + word[k].x + __popc(word[k].y & ((1u << (pos & 31)) - 1u));
      if (i >= d.S) out[i - d.S] = id;
      if (one[k]) {
        flags |= check_row(tables, (int64_t)key[k]);
        out_unique[id] = (int64_t)key[k];
        st_plain_16((uint4*)(ws.slots + v[k]), make_uint4(0xffffffffu, 0xffffffffu, kNoPos, 0xffffffffu));
      }
    }
  }
  if (flags) atomicOr(status, flags);
}

// ---- small layers: the whole relabelling in one block, table in shared memory ----------
// Up to kSmallItems items (the innermost hops of a mini-batch: 1024 seeds x (1 + 5)) fit a
// table of kSmallCap 16-byte slots in the 227 KB of shared memory of one SM together with
// each item's slot number. One block of 1024 threads then runs the three phases (insert,
// ordered compaction, relabel) with block barriers between them: no global table traffic,
// no clearing, one launch. (Drawing the neighbours inside this one block as well was measured
// slower than the separate sampling kernel: 28 us against 22 us for 1024 seeds x 5, because one
// block walks the dependent seed -> row -> neighbour loads in five rounds.) The order of first
// occurrence is decided by the minimum position per id exactly as in the multi-block path, so
// both give the same arrays.
static bool g_relabel_small = true;   // apt_set_tunable("relabel_small", 0) forces the multi-block path
void set_relabel_small(bool on) { g_relabel_small = on; }

constexpr int kSmallItems = 8192;
// behind a sampling kernel, which fills the table on its way, the one-block form only saves launches. Sampling and relabelling
// together, one block against the grid, fanout 5: 500 items 6.2 us against 9.8, 1536 8.0 / 11.0, 2048 8.5 / 12.2, 3072
// 10.0 / 12.1; fanout 15: 6.2 / 9.0, 8.2 / 9.8, 8.2 / 10.6, 9.8 / 10.8; relabelling of 6144 items 16.1 / 12.9
constexpr int kSmallSampled = 3072;
constexpr uint32_t kSmallCap = 12288;
constexpr uint16_t kSmallNoSlot = 0xffffu;
constexpr size_t kSmallSmem = (size_t)kSmallCap * sizeof(Slot) + (size_t)kSmallItems * sizeof(uint16_t);

// erase_nbrs: the neighbour list sits in the (otherwise unused) table region of the workspace and
// every entry is put back to all-ones once read, so that the table stays empty between calls.
__global__ void __launch_bounds__(kRelabelBlock)
k_relabel_small(const int64_t* __restrict__ seeds, int64_t S_host, int64_t* __restrict__ nbrs,
                int64_t M_host, const int64_t* __restrict__ S_dev, int64_t per_seed, int erase_nbrs,
                int64_t* __restrict__ out_unique, int64_t* __restrict__ out_relabeled, int64_t* __restrict__ out_col,
                int64_t* __restrict__ out_num_unique, const RowTables tables, int32_t* status) {
  wait_for_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int scratch[33];
  Slot* slots = (Slot*)smem;
  uint16_t* slot_of = (uint16_t*)(smem + (size_t)kSmallCap * sizeof(Slot));
  const RelabelDims d = relabel_dims(S_host, M_host, S_dev, per_seed);
  const int n = (int)d.n;
  for (uint32_t t = threadIdx.x; t < kSmallCap; t += blockDim.x) {
    slots[t].key = kEmptyKey;
    slots[t].min_pos = kNoPos;
    slots[t].pad = 0;
  }
  __syncthreads();
  int flags = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int64_t id = item_at(seeds, d.S, nbrs, i);
    if (erase_nbrs && i >= d.S) nbrs[i - d.S] = -1;
    if (id < 0) {   // not an id (see table_insert): no slot, relabelled to -1
      flags |= APT_FLAG_ID_OUT_OF_RANGE;
      slot_of[i] = kSmallNoSlot;
      continue;
    }
    const unsigned long long key = (unsigned long long)id;
    uint32_t pos = (uint32_t)(((uint64_t)hash_id(id) * kSmallCap) >> 32);
    for (;;) {   // at most kSmallItems of the kSmallCap slots are ever taken: an empty one is found
      Slot* s = slots + pos;
      unsigned long long prev = *(volatile unsigned long long*)&s->key;
      if (prev == kEmptyKey) prev = atomicCAS(&s->key, kEmptyKey, key);
      if (prev == kEmptyKey || prev == key) {
        atomicMin(&s->min_pos, (uint32_t)i);
        slot_of[i] = (uint16_t)pos;
        break;
      }
      pos = pos + 1 == kSmallCap ? 0 : pos + 1;
    }
  }
  __syncthreads();
  int running = 0;
  for (int base = 0; base < n; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int f = i < n && slot_of[i] != kSmallNoSlot && slots[slot_of[i]].min_pos == (uint32_t)i;
    int total;
    const int ex = block_exclusive_scan(f, scratch, &total);
    if (f) {
      const int id = running + ex;
      flags |= check_row(tables, (int64_t)slots[slot_of[i]].key);
      out_unique[id] = (int64_t)slots[slot_of[i]].key;
      slots[slot_of[i]].pad = (uint32_t)id;
    }
    running += total;
  }
  if (threadIdx.x == 0) *out_num_unique = running;
  if (flags) atomicOr(status, flags);
  __syncthreads();
  for (int i = (int)d.S + threadIdx.x; i < n; i += blockDim.x) {
    out_relabeled[i - d.S] = slot_of[i] == kSmallNoSlot ? (int64_t)-1 : (int64_t)slots[slot_of[i]].pad;
    if (out_col) out_col[i - d.S] = (int64_t)((uint32_t)(i - d.S) / (uint32_t)per_seed);
  }
}

static int set_small_smem() {
  static bool attr_set[64] = {};
  int dev = 0;
  APT_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && !attr_set[dev]) {
    APT_CUDA(cudaFuncSetAttribute(k_relabel_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
    attr_set[dev] = true;
  }
  return APT_OK;
}

// Passes 2 and 3 of the multi-block path (the table already holds every item).
static int first_and_relabel(int64_t num_seeds, int64_t num_neighbors, const int64_t* num_seeds_dev,
                             int64_t per_seed, const RelabelWs& ws, int64_t* out_unique, int64_t* out_relabeled,
                             int64_t* out_col, int64_t* out_num_unique, const RowTables& tables, int32_t* status_word,
                             cudaStream_t s) {
  const int64_t n = num_seeds + num_neighbors;
  int tile_shift = 10;
  while (ceil_div(n, (int64_t)1 << tile_shift) > kMaxTiles) ++tile_shift;
  APT_FOLLOW(k_first, (int)ceil_div(n, (int64_t)1 << tile_shift), kFirstThreads, 0, s, num_seeds, num_neighbors, num_seeds_dev,
             per_seed, ws, tile_shift);
  const int grid = wave_grid(ceil_div(n, 256 * 4), 8, 1);
  APT_FOLLOW(k_relabel, grid, 256, 0, s, num_seeds, num_neighbors, num_seeds_dev, per_seed, ws, tile_shift, out_unique,
             out_relabeled, out_col, out_num_unique, tables, status_word);
  return APT_OK;
}

}  // namespace apt

extern "C" size_t apt_relabel_workspace_bytes(int64_t num_items) {
  if (num_items < 0) return 0;
  // a little headroom so that the size-only layout always fits num_items
  return apt::relabel_bytes_for(num_items + num_items / 256 + 4096);
}

extern "C" int apt_relabel_workspace_init(void* workspace, size_t workspace_bytes, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(workspace && workspace_bytes > 0, "apt_relabel_workspace_init: null workspace");
  APT_CUDA(cudaMemsetAsync(workspace, 0xff, workspace_bytes, (cudaStream_t)stream));
  return APT_OK;
}

extern "C" int apt_relabel_csc(const int64_t* seeds, int64_t num_seeds,
                               const int64_t* num_seeds_dev, const int64_t* neighbors,
                               int64_t num_neighbors, void* workspace, size_t workspace_bytes,
                               int64_t* out_unique, int64_t* out_relabeled,
                               int64_t* out_num_unique, int32_t* status_word, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(num_seeds >= 0 && num_neighbors >= 0, "apt_relabel_csc: negative size");
  const int64_t n = num_seeds + num_neighbors;
  APT_CHECK_ARG(n < (int64_t)0x7f000000, "apt_relabel_csc: %lld items exceed the 31-bit position range",
                (long long)n);
  APT_CHECK_ARG(out_num_unique && status_word, "apt_relabel_csc: null output word");
  int64_t per_seed = 0;
  if (num_seeds_dev) {
    APT_CHECK_ARG(num_seeds > 0 && num_neighbors % num_seeds == 0,
                  "apt_relabel_csc: with a device-side seed count the neighbours must be a fixed number per seed");
    per_seed = num_neighbors / num_seeds;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    APT_CUDA(cudaMemsetAsync(out_num_unique, 0, sizeof(int64_t), s));
    return APT_OK;
  }
  APT_CHECK_ARG((num_seeds == 0 || seeds) && (num_neighbors == 0 || (neighbors && out_relabeled)) &&
                    out_unique && workspace,
                "apt_relabel_csc: null pointer");
  APT_CHECK_ARG(((uintptr_t)workspace & 255) == 0, "apt_relabel_csc: workspace must be 256-byte aligned");
  if (n <= kSmallItems && g_relabel_small) {
    const int rc = set_small_smem();
    if (rc != APT_OK) return rc;
    ProfScope prof("relabel", s);
    APT_FOLLOW(k_relabel_small, 1, kRelabelBlock, kSmallSmem, s, seeds, num_seeds, (int64_t*)neighbors, num_neighbors,
               num_seeds_dev, per_seed, 0, out_unique, out_relabeled, nullptr, out_num_unique, RowTables{},
               status_word);
    return APT_OK;
  }
  RelabelWs ws;
  if (!relabel_layout((char*)workspace, workspace_bytes, &ws) || ws.items_ws < n) {
    set_error("apt_relabel_csc: workspace of %zu bytes holds %lld items, %lld needed (apt_relabel_workspace_bytes)",
              workspace_bytes, (long long)ws.items_ws, (long long)n);
    return APT_ERR_CAPACITY;
  }
  ProfScope prof("relabel", s);
  APT_FOLLOW(k_insert, wave_grid(ceil_div(n, 256 * 2), 8, 2), 256, 0, s, seeds, num_seeds, neighbors, num_neighbors,
             num_seeds_dev, per_seed, ws, status_word);
  return first_and_relabel(num_seeds, num_neighbors, num_seeds_dev, per_seed, ws, out_unique, out_relabeled, nullptr,
                           out_num_unique, RowTables{}, status_word, s);
}

extern "C" int apt_sample_relabel_block(const int64_t* seeds, int64_t num_seeds, const int64_t* num_seeds_dev,
                                      int fanout, const int64_t* adj_pos_map, int64_t num_nodes,
                                      const int64_t* dev_indptr, const int64_t* dev_indices,
                                      const int64_t* uva_indptr, const int64_t* uva_indices, uint64_t key,
                                      uint32_t call_id, const int64_t* call_id_base_dev, void* workspace,
                                      size_t workspace_bytes, int64_t* out_neighbors, int64_t* out_unique,
                                      int64_t* out_relabeled, int64_t* out_col, int64_t* out_num_unique, const int64_t* feat_pos_map, int64_t feat_num_nodes,
                                        int64_t num_dev_rows, int64_t num_uva_rows, int32_t* status_word,
                                      void* stream) {
  using namespace apt;
  const RowTables tables{feat_pos_map, feat_num_nodes, num_dev_rows, num_uva_rows};
  APT_CHECK_ARG(num_seeds >= 0 && fanout > 0 && num_nodes >= 0,
                "apt_sample_relabel_csc: bad sizes (seeds %lld fanout %d)", (long long)num_seeds, fanout);
  const int64_t num_neighbors = num_seeds * fanout, n = num_seeds + num_neighbors;
  APT_CHECK_ARG(n < (int64_t)0x7f000000, "apt_sample_relabel_csc: %lld items exceed the 31-bit position range",
                (long long)n);
  APT_CHECK_ARG(out_num_unique && status_word, "apt_sample_relabel_csc: null output word");
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    APT_CUDA(cudaMemsetAsync(out_num_unique, 0, sizeof(int64_t), s));
    return APT_OK;
  }
  APT_CHECK_ARG(seeds && out_unique && out_relabeled && workspace && uva_indptr && uva_indices,
                "apt_sample_relabel_csc: null pointer");
  APT_CHECK_ARG(((uintptr_t)workspace & 255) == 0, "apt_sample_relabel_csc: workspace must be 256-byte aligned");
  const uint32_t k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32);
  const CscView g{adj_pos_map, num_nodes, dev_indptr, dev_indices, uva_indptr, uva_indices};
  RelabelWs ws;
  if (!relabel_layout((char*)workspace, workspace_bytes, &ws) || ws.items_ws < n) {
    set_error("apt_sample_relabel_csc: workspace of %zu bytes holds %lld items, %lld needed "
              "(apt_relabel_workspace_bytes)", workspace_bytes, (long long)ws.items_ws, (long long)n);
    return APT_ERR_CAPACITY;
  }
  const bool small = n <= kSmallSampled && g_relabel_small;
  // small layers: the neighbours go to the caller's array or, when it wants none, to the table region of the
  // workspace (16 bytes per slot, 1.5 slots per item: always room for 8 bytes per neighbour), which the
  // one-block kernel does not use and wipes again as it reads
  int64_t* nbr_buf = out_neighbors ? out_neighbors : (int64_t*)ws.slots;
  const SampleInsert ins{ws.slots, ws.slot_of};
  {
    ProfScope prof("sample", s);
#define APT_SAMPLE_INSERT(G)                                                                         \
  do {                                                                                               \
    const int grid = wave_grid(ceil_div(num_seeds, 256 / G), kSampleBlocks, num_seeds_dev ? 1 : kSampleWaves);                    \
    if (small)                                                                                       \
      APT_FOLLOW((sample_replace_kernel<G, false>), grid, 256, 0, s, seeds, num_seeds,               \
                 num_seeds_dev, fanout, g, k0, k1, call_id, call_id_base_dev, nbr_buf, status_word,  \
                 SampleInsert{nullptr, nullptr});                                                    \
    else                                                                                             \
      APT_FOLLOW((sample_replace_kernel<G, true>), grid, 256, 0, s, seeds, num_seeds, num_seeds_dev, \
                 fanout, g, k0, k1, call_id, call_id_base_dev, out_neighbors, status_word, ins);     \
  } while (0)
    if (fanout <= 8) {
      APT_SAMPLE_INSERT(8);
    } else if (fanout <= 16) {
      APT_SAMPLE_INSERT(16);
    } else {
      APT_SAMPLE_INSERT(32);
    }
#undef APT_SAMPLE_INSERT
  }
  ProfScope prof("relabel", s);
  if (small) {
    const int rc = set_small_smem();
    if (rc != APT_OK) return rc;
    APT_FOLLOW(k_relabel_small, 1, kRelabelBlock, kSmallSmem, s, seeds, num_seeds, nbr_buf, num_neighbors,
               num_seeds_dev, (int64_t)fanout, out_neighbors ? 0 : 1, out_unique, out_relabeled, out_col, out_num_unique,
               tables, status_word);
    return APT_OK;
  }
  return first_and_relabel(num_seeds, num_neighbors, num_seeds_dev, (int64_t)fanout, ws, out_unique, out_relabeled, out_col,
                           out_num_unique, tables, status_word, s);
}

extern "C" int apt_sample_relabel_csc(const int64_t* seeds, int64_t num_seeds, const int64_t* num_seeds_dev,
                                      int fanout, const int64_t* adj_pos_map, int64_t num_nodes,
                                      const int64_t* dev_indptr, const int64_t* dev_indices,
                                      const int64_t* uva_indptr, const int64_t* uva_indices, uint64_t key,
                                      uint32_t call_id, const int64_t* call_id_base_dev, void* workspace,
                                      size_t workspace_bytes, int64_t* out_neighbors, int64_t* out_unique,
                                      int64_t* out_relabeled, int64_t* out_num_unique, int32_t* status_word,
                                      void* stream) {
  return apt_sample_relabel_block(seeds, num_seeds, num_seeds_dev, fanout, adj_pos_map, num_nodes, dev_indptr, dev_indices,
                                  uva_indptr, uva_indices, key, call_id, call_id_base_dev, workspace, workspace_bytes,
                                  out_neighbors, out_unique, out_relabeled, nullptr, out_num_unique, nullptr, 0, 0, 0, status_word,
                                  stream);
}
