// Owner bucketing (stable partition of ids by owning rank) and the sorted
// unique + inverse over a bounded id range.
#include <algorithm>

#include "common.cuh"

namespace apt {

constexpr int kBucketBlock = 1024;

__global__ void __launch_bounds__(kBucketBlock)
k_bucket_count(const int64_t* __restrict__ ids, int64_t n, const int64_t* __restrict__ n_dev,
               const int64_t* __restrict__ min_vids, OwnerParams p,
               int32_t* __restrict__ hist /* [world_size][nblocks] */,
               int nblocks) {
  wait_for_previous();
  __shared__ int64_t mv[kMaxRanks + 1];
  __shared__ int cnt[kMaxRanks];
  n = effective_n(n, n_dev);
  if (threadIdx.x <= p.world_size) mv[threadIdx.x] = min_vids[threadIdx.x];
  if (threadIdx.x < kMaxRanks) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // one shared-memory add per bucket and warp instead of one per id
  const int b = i < n ? owner_of(ids[i], mv, p) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, b);
  if (b >= 0 && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cnt[b], __popc(peers));
  __syncthreads();
  if (threadIdx.x < p.world_size)
    hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] = cnt[threadIdx.x];
}

// Scatter. hist[k*nblocks + blk] (written by k_bucket_count) is the number of
// ids of block blk owned by rank k. The first output slot of bucket k's ids from
// this block is (ids of all lower buckets) + (ids of bucket k in lower blocks):
// warp k of the block sums row k of hist for that, so no scan kernel sits between
// the two passes. Block 0 also writes the bucket sizes (+ their total) and the
// inclusive offsets.
__global__ void __launch_bounds__(kBucketBlock)
k_bucket_scatter(const int64_t* __restrict__ ids, int64_t n, const int64_t* __restrict__ n_dev,
                 const int64_t* __restrict__ min_vids, OwnerParams p,
                 const int32_t* __restrict__ hist, int nblocks,
                 int64_t* __restrict__ sorted, int64_t* __restrict__ perm,
                 int64_t* __restrict__ sizes, int64_t* __restrict__ offsets) {
  wait_for_previous();
  __shared__ int64_t mv[kMaxRanks + 1];
  __shared__ int warp_cnt[kBucketBlock / 32][kMaxRanks];
  __shared__ int row_total[kMaxRanks], row_before[kMaxRanks], bucket_base[kMaxRanks];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  n = effective_n(n, n_dev);
  if (threadIdx.x <= p.world_size) mv[threadIdx.x] = min_vids[threadIdx.x];
  for (int t = threadIdx.x; t < (kBucketBlock / 32) * kMaxRanks; t += blockDim.x)
    (&warp_cnt[0][0])[t] = 0;
  if (warp < p.world_size) {
    const int32_t* row = hist + (int64_t)warp * nblocks;
    int tot = 0, before = 0;
    for (int t = lane; t < nblocks; t += 32) {
      const int c = row[t];
      tot += c;
      if (t < (int)blockIdx.x) before += c;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      tot += __shfl_down_sync(0xffffffffu, tot, d);
      before += __shfl_down_sync(0xffffffffu, before, d);
    }
    if (lane == 0) {
      row_total[warp] = tot;
      row_before[warp] = before;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int k = 0; k < p.world_size; ++k) {
      bucket_base[k] = run + row_before[k];
      run += row_total[k];
      if (blockIdx.x == 0) {
        sizes[k] = row_total[k];
        offsets[k] = run;
      }
    }
    if (blockIdx.x == 0) sizes[p.world_size] = run;
  }
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n;
  int64_t v = 0;
  int b = -1;
  if (live) {
    v = ids[i];
    b = owner_of(v, mv, p);
  }
  // Rank of this lane among the lanes of its warp that share its bucket.
  const unsigned peers = __match_any_sync(0xffffffffu, b);
  const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
  if (live && rank_in_warp == 0) warp_cnt[warp][b] = __popc(peers);
  __syncthreads();
  // Exclusive scan over warps for each bucket (32 warps x <=32 buckets).
  if (threadIdx.x < kMaxRanks) {
    int run = 0;
    for (int w = 0; w < kBucketBlock / 32; ++w) {
      const int c = warp_cnt[w][threadIdx.x];
      warp_cnt[w][threadIdx.x] = run;
      run += c;
    }
  }
  __syncthreads();
  if (live) {
    const int64_t slot = (int64_t)bucket_base[b] + warp_cnt[warp][b] + rank_in_warp;
    sorted[slot] = v;
    perm[i] = slot;
  }
}

// One rank owns every id: the partition is the input, in one launch.
__global__ void __launch_bounds__(256)
k_bucket_one_rank(const int64_t* __restrict__ ids, int64_t n, const int64_t* __restrict__ n_dev, int64_t* __restrict__ sorted,
                  int64_t* __restrict__ perm, int64_t* __restrict__ sizes, int64_t* __restrict__ offsets) {
  wait_for_previous();
  n = effective_n(n, n_dev);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    sorted[i] = ids[i];
    perm[i] = i;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) sizes[0] = sizes[1] = offsets[0] = n;
}

// out = cat(a[0:na], b[0:nb]) with both lengths taken from device words (the input nodes of an
// SNP-GAT mini-batch: the local destination nodes followed by the ids received from the peers,
// python/npc/sampler.py:230).
__global__ void __launch_bounds__(256)
k_concat_ids(const int64_t* __restrict__ a, int64_t na, const int64_t* __restrict__ na_dev,
             const int64_t* __restrict__ b, int64_t nb, const int64_t* __restrict__ nb_dev,
             int64_t* __restrict__ out, int64_t* __restrict__ out_count, const RowTables tables, int32_t* status) {
  wait_for_previous();
  na = effective_n(na, na_dev);
  nb = effective_n(nb, nb_dev);
  const int64_t total = na + nb;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int flags = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int64_t id = i < na ? a[i] : b[i - na];
    out[i] = id;
    flags |= check_row(tables, id);
  }
  if (flags) atomicOr(status, flags);
  if (out_count && blockIdx.x == 0 && threadIdx.x == 0) *out_count = total;
}

// ------------------------------------------------------------ sorted unique
// A two-level bitmap over the id range stands in for the sort: level 0 has one
// bit per id, level 1 one bit per level-0 word that is not zero. Counting,
// ranking and emitting walk level 1 only (range/1024 words), so the cost of a
// call follows the number of ids, not the width of the range. Both levels are
// all-zero between calls: the pass that emits the ids also clears what it read.
// Three launches: mark (and count per tile of words), emit (ranks, ids, clear), inverse. The last can be enqueued beside what is made of the
// distinct ids, and leaves other things that take the same ids (OneRank, ListOf): us of a mini-batch, papers-shaped 218 -> 216, with
// source-split sampling for attention 231 -> 224. (The list written by the emit, whose lanes have several ids one after another to look up: 242.)
constexpr int kUniqBlock = 256;
constexpr int kSharedTiles = 1024;    // up to here a block adds its counts up in shared memory first
constexpr int kGroup = 256;           // tiles whose counts are added up once more where there are many
constexpr int kManyTiles = 8192;      // (every block of the emit reads the counts before its own: 32 a thread here)

// Ids set per tile; all zero between calls.
struct TileCounts {
  int32_t* tile;       // [tiles]
  int32_t* group;      // [tiles / kGroup + 1], used above kManyTiles
  int tiles;
  int shift;           // level-0 word -> tile
};

// The number of ids: `n`, or the device's count of groups of `per`.
__device__ __forceinline__ int64_t ids_of(int64_t n, const int64_t* n_dev, int64_t per) {
  if (!n_dev) return n;
  const int64_t v = *n_dev * per;
  return v < 0 ? 0 : min(v, n);
}

// Runs of lanes whose ids share a word (the virtual ids of a sampled hop come in runs of its fanout) are joined
// first: one atomic a run. 23 000 ids in runs of 25: 24 us with one an id.
__global__ void __launch_bounds__(256)
k_uniq_mark(const int64_t* __restrict__ ids, int64_t n, const int64_t* __restrict__ n_dev, int64_t per,
            int64_t lo, int64_t hi, uint32_t* __restrict__ l0, uint32_t* __restrict__ l1,
            TileCounts counts, int32_t* status) {
  wait_for_previous();
  __shared__ int here[kSharedTiles];
  const bool shared = counts.tiles <= kSharedTiles;
  if (shared) {
    for (int t = threadIdx.x; t < counts.tiles; t += 256) here[t] = 0;
    __syncthreads();
  }
  n = ids_of(n, n_dev, per);
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int flags = 0;
  // whole warps iterate together
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i - lane < n; i += stride) {
    uint32_t w = 0xffffffffu, bits = 0u;      // words of the range number less than 2^31
    if (i < n) {
      const int64_t v = ids[i];
      if (v < lo || v >= hi) {
        flags |= APT_FLAG_ID_OUT_OF_RANGE;
      } else {
        w = (uint32_t)((v - lo) >> 5);
        bits = 1u << ((v - lo) & 31);
      }
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t w2 = __shfl_down_sync(0xffffffffu, w, o), b2 = __shfl_down_sync(0xffffffffu, bits, o);
      if (lane + o < 32 && w2 == w) bits |= b2;
    }
    const uint32_t before = __shfl_up_sync(0xffffffffu, w, 1);
    if (w == 0xffffffffu || (lane > 0 && before == w)) continue;
    if ((*(volatile uint32_t*)(l0 + w) & bits) == bits) continue;
    const uint32_t old = atomicOr(l0 + w, bits);
    if (old == 0) atomicOr(l1 + (w >> 5), 1u << (w & 31));  // first bit of this word
    const int set = __popc(bits & ~old);
    if (!set) continue;
    const uint32_t tile = w >> counts.shift;
    if (shared) {
      atomicAdd(here + tile, set);
    } else {
      atomicAdd(counts.tile + tile, set);
      if (counts.tiles > kManyTiles) atomicAdd(counts.group + tile / kGroup, set);
    }
  }
  if (flags) atomicOr(status, flags);
  if (!shared) return;
  __syncthreads();
  for (int t = threadIdx.x; t < counts.tiles; t += 256)
    if (here[t]) atomicAdd(counts.tile + t, here[t]);
}

// Ranking, emitting and clearing in one launch. A block (a tile) has 8 * `per_warp` consecutive level-1 words, dealt to
// its warps in turn (a dense run of ids in a wide range is a few neighbouring words), a lane to each. A lane with few
// level-0 words below its own (a wide range) walks them itself, all loads in flight; where there are many the warp's lanes
// take the 32 words together, one level-1 word after another (a dense range: a million ids below one thousand level-1
// words; one thread to a word walked 1024 ids alone, 75 to 430 us). The first rank of a tile is the sum of the counts
// the marks left for the tiles before it, read beside the tile's own words: with counts found here and chained by a
// decoupled look-back the launch took 11 us instead of 4 (67 584 ids of 111 million), most of it waiting in
// turn for the ticket, the look-back's windows and the closing counter.
// info[w] = (rank of the word's first id, its bits).
// 16 words: 50 000 ids of 8.2 million, six to a level-1 word on average, take 5.0 us; with 8 a sixth of the lanes went the
// warp's way and it took 11.7.
constexpr int kOwnWords = 16, kOwnIds = 32;

__global__ void __launch_bounds__(kUniqBlock)
k_uniq_emit(uint32_t* __restrict__ l0, uint32_t* __restrict__ l1, int64_t nwords1, int per_warp,
            int64_t lo, const TileCounts tc, uint2* __restrict__ info, int64_t* __restrict__ out_unique,
            int64_t* __restrict__ out_num_unique) {
  wait_for_previous();
  constexpr int W = kUniqBlock / 32;
  __shared__ uint32_t counts[kUniqBlock];
  __shared__ int scratch[33], s_before[W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tile = blockIdx.x;
  const int64_t first = (int64_t)tile * W * per_warp + warp;      // word of lane k: first + k * W
  const int64_t w1 = first + lane * W;
  const uint32_t mine = lane < per_warp && w1 < nwords1 ? l1[w1] : 0u;
  int before = 0;
  {
    const bool many = tc.tiles > kManyTiles;
    const int start = many ? tile / kGroup * kGroup : 0;
    for (int t = start + threadIdx.x; t < tile; t += kUniqBlock) before += tc.tile[t];
    if (many)
      for (int t = threadIdx.x; t < tile / kGroup; t += kUniqBlock) before += tc.group[t];
  }
  uint32_t word[kOwnWords], count = 0;
  const bool few = __popc(mine) <= kOwnWords;
  uint32_t rest = mine;
#pragma unroll
  for (int q = 0; q < kOwnWords; ++q) {
    word[q] = few && rest ? l0[(w1 << 5) + __ffs(rest) - 1] : 0u;
    rest &= rest - 1;
  }
#pragma unroll
  for (int q = 0; q < kOwnWords; ++q) count += __popc(word[q]);
  for (unsigned m = __ballot_sync(0xffffffffu, !few); m; m &= m - 1) {
    const int k = __ffs(m) - 1;
    const uint32_t mask = __shfl_sync(0xffffffffu, mine, k);
    const uint32_t c = __reduce_add_sync(0xffffffffu, mask >> lane & 1u ? __popc(l0[((first + k * W) << 5) + lane]) : 0u);
    if (lane == k) count = c;
  }
  // ranks inside the block, in the order of the words
  counts[lane * W + warp] = count;
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) s_before[warp] = before;
  __syncthreads();
  int total_i;
  const int before_word = block_exclusive_scan((int)counts[threadIdx.x], scratch, &total_i);
  counts[threadIdx.x] = (uint32_t)before_word;
  const uint32_t total = (uint32_t)total_i;
  __syncthreads();
  int64_t base = 0;
#pragma unroll
  for (int q = 0; q < W; ++q) base += s_before[q];
  if (tile == (int)gridDim.x - 1 && threadIdx.x == 0) *out_num_unique = base + total;
  int64_t at = base + counts[lane * W + warp];      // rank of the first id below this lane's word
  const bool own = few && count <= kOwnIds;
  for (unsigned m = __ballot_sync(0xffffffffu, !own); m; m &= m - 1) {
    const int k = __ffs(m) - 1;
    const uint32_t mask = __shfl_sync(0xffffffffu, mine, k);
    const int64_t start = __shfl_sync(0xffffffffu, at, k);
    const int64_t w = ((first + k * W) << 5) + lane;
    const uint32_t bits = mask >> lane & 1u ? l0[w] : 0u;
    uint32_t upto = __popc(bits);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    const uint32_t here = upto - __popc(bits);
    if (bits) {
      info[w] = make_uint2((uint32_t)(start + here), bits);
      l0[w] = 0u;
    }
    // the ids of one level-0 word at a time, a lane to a bit
    for (uint32_t q = mask; q; q &= q - 1) {
      const int j = __ffs(q) - 1;
      const uint32_t x = __shfl_sync(0xffffffffu, bits, j), rank = __shfl_sync(0xffffffffu, here, j);
      if (x >> lane & 1u) out_unique[start + rank + __popc(x & ((1u << lane) - 1u))] = lo + ((((first + k * W) << 5) + j) << 5) + lane;
    }
  }
  if (own) {
    rest = mine;
#pragma unroll
    for (int q = 0; q < kOwnWords; ++q) {
      if (!rest) break;
      const int64_t w = (w1 << 5) + __ffs(rest) - 1;
      rest &= rest - 1;
      info[w] = make_uint2((uint32_t)at, word[q]);
      l0[w] = 0u;
      for (uint32_t bits = word[q]; bits; bits &= bits - 1) out_unique[at++] = lo + (w << 5) + __ffs(bits) - 1;
    }
  }
  if (lane < per_warp && mine) l1[w1] = 0u;
}

// The distinct ids behind `head`'s, in a list of their own (as the inverse's launch makes it, a launch for the list alone, 4 us of a
// source-split mini-batch's chain, is not needed). all null: no such list.
struct ListOf {
  const int64_t* head;
  int64_t num_head;
  const int64_t* num_head_dev;
  const int64_t* unique;
  int64_t num_unique;
  const int64_t* num_unique_dev;
  int64_t* all;
  int64_t* num_all;
  RowTables tables;      // of a gather of the list's rows
};

// What a bucketing by owner leaves in a world of one rank: ids [0, count) where they are. all null: nothing.
struct OneRank {
  int64_t* perm;
  int64_t num;
  const int64_t* num_dev;      // null: as many as there are ids
  int64_t *sizes, *offsets;
};

__global__ void __launch_bounds__(256)
k_uniq_inverse(const int64_t* __restrict__ ids, int64_t n, const int64_t* __restrict__ n_dev, int64_t per,
               int64_t lo, int64_t hi, const uint2* __restrict__ info, TileCounts counts, int64_t* __restrict__ out_inverse, const OneRank one,
               const ListOf list, int32_t* status) {
  wait_for_previous();
  n = ids_of(n, n_dev, per);
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = i; t < counts.tiles; t += stride) {      // the emit is done with them
    counts.tile[t] = 0;
    if (t % kGroup == 0) counts.group[t / kGroup] = 0;
  }
  if (one.perm) {
    const int64_t count = one.num_dev ? effective_n(one.num, one.num_dev) : n;
    for (int64_t t = i; t < count; t += stride) one.perm[t] = t;
    if (i == 0) one.sizes[0] = one.sizes[1] = one.offsets[0] = count;
  }
  if (list.all) {
    const int64_t heads = effective_n(list.num_head, list.num_head_dev), total = heads + effective_n(list.num_unique, list.num_unique_dev);
    if (i == 0 && list.num_all) *list.num_all = total;
    int flags = 0;
    for (int64_t t = i; t < total; t += stride) {
      const int64_t v = t < heads ? list.head[t] : list.unique[t - heads];
      list.all[t] = v;
      flags |= check_row(list.tables, v);
    }
    if (flags) atomicOr(status, flags);
  }
  for (; i < n; i += stride) {
    const int64_t v = ids[i];
    if (v < lo || v >= hi) {
      out_inverse[i] = -1;
      continue;
    }
    const int64_t r = v - lo;
    const uint2 w = info[r >> 5];
    out_inverse[i] = (int64_t)w.x + __popc(w.y & ((1u << (r & 31)) - 1u));
  }
}

}  // namespace apt

extern "C" size_t apt_bucket_workspace_bytes(int64_t num_ids, int world_size) {
  if (num_ids < 0 || world_size < 1) return 0;
  const int64_t nblocks = apt::ceil_div(num_ids > 0 ? num_ids : 1, apt::kBucketBlock);
  return apt::align_up((size_t)(nblocks * world_size + 1) * 4, 256);
}

extern "C" int apt_bucket_by_owner(const int64_t* ids, int64_t num_ids,
                                   const int64_t* num_ids_dev, const int64_t* min_vids, int world_size,
                                   int64_t shuffle_id_offset, int rank,
                                   int node_beg, int node_end, void* workspace,
                                   size_t workspace_bytes, int64_t* out_sorted,
                                   int64_t* out_perm, int64_t* out_bucket_sizes,
                                   int64_t* out_bucket_offsets, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(world_size >= 1 && world_size <= kMaxRanks,
                "apt_bucket_by_owner: world_size %d outside [1,%d]", world_size, kMaxRanks);
  APT_CHECK_ARG(num_ids >= 0 && num_ids < (int64_t)0x7fffffff, "apt_bucket_by_owner: bad num_ids");
  APT_CHECK_ARG(min_vids && out_bucket_sizes && out_bucket_offsets,
                "apt_bucket_by_owner: null pointer");
  APT_CHECK_ARG(rank >= 0 && rank < world_size && shuffle_id_offset >= 0 &&
                    shuffle_id_offset < world_size,
                "apt_bucket_by_owner: rank/offset outside the world");
  cudaStream_t s = (cudaStream_t)stream;
  if (num_ids == 0) {
    APT_CUDA(cudaMemsetAsync(out_bucket_sizes, 0, sizeof(int64_t) * (world_size + 1), s));
    APT_CUDA(cudaMemsetAsync(out_bucket_offsets, 0, sizeof(int64_t) * world_size, s));
    return APT_OK;
  }
  APT_CHECK_ARG(ids && out_sorted && out_perm && workspace, "apt_bucket_by_owner: null pointer");
  const size_t need = apt_bucket_workspace_bytes(num_ids, world_size);
  if (workspace_bytes < need) {
    set_error("apt_bucket_by_owner: workspace %zu < %zu bytes", workspace_bytes, need);
    return APT_ERR_CAPACITY;
  }
  OwnerParams p;
  p.world_size = world_size;
  p.shuffle_id_offset = (int)shuffle_id_offset;
  p.rank = rank;
  p.node_beg = node_beg;
  p.node_end = node_end;
  const int nblocks = (int)ceil_div(num_ids, kBucketBlock);
  int32_t* hist = (int32_t*)workspace;
  ProfScope prof("bucket", s);
  if (world_size == 1) {
    APT_FOLLOW(k_bucket_one_rank, wave_grid(ceil_div(num_ids, 256), 8, 1), 256, 0, s, ids, num_ids, num_ids_dev, out_sorted,
               out_perm, out_bucket_sizes, out_bucket_offsets);
    return APT_OK;
  }
  APT_FOLLOW(k_bucket_count, nblocks, kBucketBlock, 0, s, ids, num_ids, num_ids_dev, min_vids, p, hist, nblocks);
  APT_FOLLOW(k_bucket_scatter, nblocks, kBucketBlock, 0, s, ids, num_ids, num_ids_dev, min_vids, p, hist,
             nblocks, out_sorted, out_perm, out_bucket_sizes, out_bucket_offsets);
  return APT_OK;
}

namespace apt {
struct UniqWs {
  uint32_t* l0;           // [nwords0] one bit per id
  uint32_t* l1;           // [nwords1] one bit per level-0 word
  uint2* info;            // [nwords1 * 32] rank of the word's first id and its bits, of the words the call set
  TileCounts counts;
  int64_t nwords1;
  int nblocks, per_warp;
};
static size_t uniq_layout(int64_t range, char* base, UniqWs* ws) {
  const int64_t nwords0 = ceil_div(range > 0 ? range : 1, 32);
  const int64_t nwords1 = ceil_div(nwords0, 32);
  // level-1 words a warp: few enough that a narrow range still spreads over the SMs, 32 at most
  int per_warp = 1;
  while (per_warp < 32 && (int64_t)per_warp * kNumSMs * (kUniqBlock / 32) < nwords1) per_warp <<= 1;
  const int nblocks = (int)ceil_div(nwords1, (int64_t)per_warp * (kUniqBlock / 32));
  const size_t b0 = align_up((size_t)nwords1 * 32 * 4, 256);  // level 0, padded to whole level-1 words
  const size_t b1 = align_up((size_t)nwords1 * 4, 256);
  const size_t b2 = align_up((size_t)nwords1 * 32 * 8, 256);
  const size_t b3 = align_up((size_t)nblocks * 4, 256);
  const size_t b4 = align_up((size_t)(nblocks / kGroup + 1) * 4, 256);
  if (ws) {
    ws->l0 = (uint32_t*)base;
    ws->l1 = (uint32_t*)(base + b0);
    ws->info = (uint2*)(base + b0 + b1);
    int shift = 5 + 3;      // 32 level-0 words to a level-1 word, 8 warps
    for (int k = per_warp; k > 1; k >>= 1) ++shift;
    ws->counts = TileCounts{(int32_t*)(base + b0 + b1 + b2), (int32_t*)(base + b0 + b1 + b2 + b3), nblocks, shift};
    ws->nwords1 = nwords1;
    ws->nblocks = nblocks;
    ws->per_warp = per_warp;
  }
  return b0 + b1 + b2 + b3 + b4;
}
}  // namespace apt

extern "C" size_t apt_unique_workspace_bytes(int64_t id_range) {
  if (id_range < 0) return 0;
  return apt::uniq_layout(id_range, nullptr, nullptr);
}

extern "C" int apt_unique_workspace_init(void* workspace, size_t workspace_bytes, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(workspace && workspace_bytes > 0, "apt_unique_workspace_init: null workspace");
  APT_CUDA(cudaMemsetAsync(workspace, 0, workspace_bytes, (cudaStream_t)stream));
  return APT_OK;
}

namespace apt {
static int uniq_check(const char* who, const int64_t* ids, int64_t num_ids, int64_t lo, int64_t hi, void* workspace, size_t workspace_bytes,
                      const void* out, UniqWs* ws) {
  APT_CHECK_ARG(ids && workspace && out, "%s: null pointer", who);
  const size_t need = uniq_layout(hi - lo, (char*)workspace, ws);
  if (workspace_bytes < need) {
    set_error("%s: workspace %zu < %zu bytes", who, workspace_bytes, need);
    return APT_ERR_CAPACITY;
  }
  return APT_OK;
}
static int uniq_sizes(const char* who, int64_t num_ids, int64_t lo, int64_t hi) {
  APT_CHECK_ARG(num_ids >= 0 && hi >= lo, "%s: bad sizes", who);
  APT_CHECK_ARG(hi - lo < ((int64_t)1 << 36), "%s: id range too wide for a bitmap", who);
  return APT_OK;
}
static int uniq_ids(const int64_t* ids, int64_t num_ids, const int64_t* num_ids_dev, int64_t per, int64_t lo, int64_t hi, const UniqWs& ws,
                    int64_t* out_unique, int64_t* out_num_unique, int32_t* status_word, cudaStream_t s) {
  APT_FOLLOW(k_uniq_mark, wave_grid(ceil_div(num_ids, 256), 8, 1), 256, 0, s, ids, num_ids, num_ids_dev, per, lo, hi, ws.l0, ws.l1, ws.counts,
             status_word);
  APT_FOLLOW(k_uniq_emit, ws.nblocks, kUniqBlock, 0, s, ws.l0, ws.l1, ws.nwords1, ws.per_warp, lo, ws.counts, ws.info, out_unique,
             out_num_unique);
  return APT_OK;
}
static int uniq_inverse(const int64_t* ids, int64_t num_ids, const int64_t* num_ids_dev, int64_t per, int64_t lo, int64_t hi, const UniqWs& ws,
                        int64_t* out_inverse, const OneRank& one, const ListOf& list, int32_t* status_word, cudaStream_t s) {
  const int64_t most = std::max(num_ids, list.all ? list.num_head + list.num_unique : 0);
  APT_FOLLOW(k_uniq_inverse, wave_grid(ceil_div(most, 256), 8, 1), 256, 0, s, ids, num_ids, num_ids_dev, per, lo, hi, ws.info, ws.counts,
             out_inverse, one, list, status_word);
  return APT_OK;
}
}  // namespace apt

extern "C" int apt_unique_sorted(const int64_t* ids, int64_t num_ids,
                                 const int64_t* num_ids_dev, int64_t id_lo,
                                 int64_t id_hi, void* workspace, size_t workspace_bytes,
                                 int64_t* out_unique, int64_t* out_inverse,
                                 int64_t* out_num_unique, int32_t* status_word,
                                 void* stream) {
  using namespace apt;
  int rc = uniq_sizes("apt_unique_sorted", num_ids, id_lo, id_hi);
  if (rc != APT_OK) return rc;
  APT_CHECK_ARG(out_num_unique && status_word, "apt_unique_sorted: null output word");
  cudaStream_t s = (cudaStream_t)stream;
  if (num_ids == 0 || id_hi == id_lo) {
    APT_CUDA(cudaMemsetAsync(out_num_unique, 0, sizeof(int64_t), s));
    if (num_ids > 0) {
      APT_CHECK_ARG(out_inverse, "apt_unique_sorted: null pointer");
      APT_CUDA(cudaMemsetAsync(out_inverse, 0xff, sizeof(int64_t) * num_ids, s));
    }
    return APT_OK;
  }
  UniqWs ws;
  rc = uniq_check("apt_unique_sorted", ids, num_ids, id_lo, id_hi, workspace, workspace_bytes, out_unique && out_inverse ? out_unique : nullptr, &ws);
  if (rc != APT_OK) return rc;
  ProfScope prof("unique_sorted", s);
  rc = uniq_ids(ids, num_ids, num_ids_dev, 1, id_lo, id_hi, ws, out_unique, out_num_unique, status_word, s);
  return rc != APT_OK ? rc : uniq_inverse(ids, num_ids, num_ids_dev, 1, id_lo, id_hi, ws, out_inverse, OneRank{}, ListOf{}, status_word, s);
}

extern "C" int apt_unique_ids(const int64_t* ids, int64_t num_ids, const int64_t* num_ids_dev, int64_t ids_per, int64_t id_lo, int64_t id_hi,
                              void* workspace, size_t workspace_bytes, int64_t* out_unique, int64_t* out_num_unique, int32_t* status_word,
                              void* stream) {
  using namespace apt;
  int rc = uniq_sizes("apt_unique_ids", num_ids, id_lo, id_hi);
  if (rc != APT_OK) return rc;
  APT_CHECK_ARG(out_num_unique && status_word && ids_per >= 1, "apt_unique_ids: bad argument");
  cudaStream_t s = (cudaStream_t)stream;
  if (num_ids == 0 || id_hi == id_lo) {
    APT_CUDA(cudaMemsetAsync(out_num_unique, 0, sizeof(int64_t), s));
    return APT_OK;
  }
  UniqWs ws;
  rc = uniq_check("apt_unique_ids", ids, num_ids, id_lo, id_hi, workspace, workspace_bytes, out_unique, &ws);
  if (rc != APT_OK) return rc;
  ProfScope prof("unique_sorted", s);
  return uniq_ids(ids, num_ids, num_ids_dev, ids_per, id_lo, id_hi, ws, out_unique, out_num_unique, status_word, s);
}

extern "C" int apt_unique_inverse(const int64_t* ids, int64_t num_ids, const int64_t* num_ids_dev, int64_t ids_per, int64_t id_lo, int64_t id_hi,
                                  void* workspace, size_t workspace_bytes, int64_t* out_inverse, const int64_t* unique, int64_t num_unique,
                                  const int64_t* num_unique_dev, int64_t* out_perm, int64_t* out_bucket_sizes, int64_t* out_bucket_offsets,
                                  const int64_t* head, int64_t num_head, const int64_t* num_head_dev, int64_t* out_all, int64_t* out_num_all,
                                  const int64_t* feat_pos_map, int64_t feat_num_nodes, int64_t num_dev_rows, int64_t num_uva_rows,
                                  int32_t* status_word, void* stream) {
  using namespace apt;
  int rc = uniq_sizes("apt_unique_inverse", num_ids, id_lo, id_hi);
  if (rc != APT_OK) return rc;
  APT_CHECK_ARG(ids_per >= 1 && (num_ids == 0 || out_inverse) && num_unique >= 0 && (num_unique == 0 || unique), "apt_unique_inverse: bad argument");
  APT_CHECK_ARG(!out_bucket_sizes == !out_bucket_offsets && !out_bucket_sizes == !out_perm, "apt_unique_inverse: null pointer");
  APT_CHECK_ARG(!out_all || (num_head >= 0 && (num_head == 0 || head) && num_unique_dev && status_word), "apt_unique_inverse: bad list");
  cudaStream_t s = (cudaStream_t)stream;
  if (num_ids == 0 || id_hi == id_lo) {
    if (num_ids > 0) APT_CUDA(cudaMemsetAsync(out_inverse, 0xff, sizeof(int64_t) * num_ids, s));
    if (out_bucket_sizes)      // (of distinct ids: there are none; of the ids themselves, if there are any)
      APT_FOLLOW(k_bucket_one_rank, 1, 256, 0, s, ids, num_unique_dev ? 0 : num_ids, num_unique_dev ? nullptr : num_ids_dev, out_perm, out_perm,
                 out_bucket_sizes, out_bucket_offsets);
    return out_all ? apt_concat_row_ids(head, num_head, num_head_dev, nullptr, 0, nullptr, out_all, out_num_all, feat_pos_map, feat_num_nodes,
                                        num_dev_rows, num_uva_rows, status_word, stream) : APT_OK;
  }
  UniqWs ws;
  rc = uniq_check("apt_unique_inverse", ids, num_ids, id_lo, id_hi, workspace, workspace_bytes, out_inverse, &ws);
  if (rc != APT_OK) return rc;
  ProfScope prof("unique_sorted", s);
  const OneRank one{out_perm, num_unique, num_unique_dev, out_bucket_sizes, out_bucket_offsets};
  const ListOf list{head, num_head, num_head_dev, unique, num_unique, num_unique_dev, out_all, out_num_all,
                    RowTables{feat_pos_map, feat_num_nodes, num_dev_rows, num_uva_rows}};
  return uniq_inverse(ids, num_ids, num_ids_dev, ids_per, id_lo, id_hi, ws, out_inverse, one, list, status_word, s);
}

extern "C" int apt_concat_ids(const int64_t* a, int64_t num_a, const int64_t* num_a_dev, const int64_t* b,
                              int64_t num_b, const int64_t* num_b_dev, int64_t* out, int64_t* out_count_dev,
                              void* stream) {
  return apt_concat_row_ids(a, num_a, num_a_dev, b, num_b, num_b_dev, out, out_count_dev, nullptr, 0, 0, 0, nullptr, stream);
}

extern "C" int apt_concat_row_ids(const int64_t* a, int64_t num_a, const int64_t* num_a_dev, const int64_t* b,
                                  int64_t num_b, const int64_t* num_b_dev, int64_t* out, int64_t* out_count_dev,
                                  const int64_t* feat_pos_map, int64_t feat_num_nodes, int64_t num_dev_rows,
                                  int64_t num_uva_rows, int32_t* status_word, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(!feat_pos_map || status_word, "apt_concat_ids: null status word");
  APT_CHECK_ARG(num_a >= 0 && num_b >= 0 && (num_a == 0 || a) && (num_b == 0 || b), "apt_concat_ids: bad argument");
  APT_CHECK_ARG(out || num_a + num_b == 0, "apt_concat_ids: null output");
  cudaStream_t s = (cudaStream_t)stream;
  if (num_a + num_b == 0) {
    if (out_count_dev) APT_CUDA(cudaMemsetAsync(out_count_dev, 0, sizeof(int64_t), s));
    return APT_OK;
  }
  APT_FOLLOW(k_concat_ids, wave_grid(ceil_div(num_a + num_b, 256), 8, 1), 256, 0, s, a, num_a, num_a_dev, b, num_b,
             num_b_dev, out, out_count_dev, RowTables{feat_pos_map, feat_num_nodes, num_dev_rows, num_uva_rows}, status_word);
  return APT_OK;
}
