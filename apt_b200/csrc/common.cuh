// Shared device/host helpers of libapt_b200: error plumbing, launch counting,
// optional per-kernel event timing, Philox4x32-10, 16-byte row movers and a
// block-wide exclusive scan.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/apt_b200.h"

namespace apt {

// ---------------------------------------------------------------- host side
void set_error(const char* fmt, ...);
void count_launch();
// RAII bracket that records events around one tagged kernel when profiling is on.
struct ProfScope {
  ProfScope(const char* tag, cudaStream_t s);
  ~ProfScope();
  const char* tag;
  cudaStream_t stream;
  int slot;
};

#define APT_CHECK_ARG(cond, ...)        \
  do {                                  \
    if (!(cond)) {                      \
      apt::set_error(__VA_ARGS__);      \
      return APT_ERR_BAD_ARG;           \
    }                                   \
  } while (0)

#define APT_CUDA(call)                                                        \
  do {                                                                        \
    cudaError_t e__ = (call);                                                 \
    if (e__ != cudaSuccess) {                                                 \
      apt::set_error("%s:%d %s -> %s", __FILE__, __LINE__, #call,             \
                     cudaGetErrorString(e__));                                \
      return APT_ERR_CUDA;                                                    \
    }                                                                         \
  } while (0)

// Launch + count + launch-error check (cudaPeekAtLastError keeps sticky
// errors visible to the caller's own checks).
#define APT_LAUNCH(kernel, grid, block, smem, stream, ...)                    \
  do {                                                                        \
    kernel<<<(grid), (block), (smem), (stream)>>>(__VA_ARGS__);               \
    apt::count_launch();                                                      \
    cudaError_t e__ = cudaPeekAtLastError();                                  \
    if (e__ != cudaSuccess) {                                                 \
      apt::set_error("%s:%d launch of %s -> %s", __FILE__, __LINE__, #kernel, \
                     cudaGetErrorString(e__));                                \
      return APT_ERR_CUDA;                                                    \
    }                                                                         \
  } while (0)

inline dim3 as_grid(int64_t blocks) { return dim3((unsigned)blocks); }
inline dim3 as_grid(dim3 grid) { return grid; }

// The same for a kernel that opens with wait_for_previous(): its launch overlaps the end of the kernel before it on the
// stream (programmatic dependent launch), in captured graphs too. Chains of kernels of a few microseconds are what this
// framework's mini-batches consist of: three edge operators over 61 310 edges 38 -> 31 us, a data-parallel batch 151 -> 135.
#define APT_FOLLOW(kernel, grid_, block_, smem_, stream_, ...)                \
  do {                                                                        \
    cudaLaunchAttribute attr__ = {};                                          \
    attr__.id = cudaLaunchAttributeProgrammaticStreamSerialization;           \
    attr__.val.programmaticStreamSerializationAllowed = 1;                    \
    cudaLaunchConfig_t cfg__ = {};                                            \
    cfg__.gridDim = as_grid(grid_);                                  \
    cfg__.blockDim = dim3((unsigned)(block_));                                \
    cfg__.dynamicSmemBytes = (smem_);                                         \
    cfg__.stream = (stream_);                                                 \
    cfg__.attrs = &attr__;                                                    \
    cfg__.numAttrs = 1;                                                       \
    const cudaError_t e__ = cudaLaunchKernelEx(&cfg__, kernel, __VA_ARGS__);  \
    apt::count_launch();                                                      \
    if (e__ != cudaSuccess) {                                                 \
      apt::set_error("%s:%d launch of %s -> %s", __FILE__, __LINE__, #kernel, \
                     cudaGetErrorString(e__));                                \
      return APT_ERR_CUDA;                                                    \
    }                                                                         \
  } while (0)

void set_relabel_small(bool on);   // relabel.cu: one-block shared-memory path for small layers
void set_bulk_wait_polls(int polls);   // spmm.cu: bound of k_spmm_stream's waits

// The tag of a sequence number (Tagged). A plain value's upper half is all zeros or all ones: no tag is, whatever the number, so that
// words which were read already are never taken for an answer. Numbers 2^30 apart share one.
__host__ __device__ inline uint32_t tag_of(int64_t sequence) { return ((uint32_t)sequence & 0x3fffffffu) | 0x40000000u; }

// While another thread captures a stream, or this one does, calls that might synchronise are refused and end the capture. For
// those that do not touch the captured work (page-locked memory of the library's own, asking a stream how it stands).
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

constexpr int kNumSMs = 148;  // B200: 2 dies x 74 SMs

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Grid for a grid-stride kernel: enough blocks for `work_blocks`, rounded up
// to whole waves of `per_sm` resident blocks on each of the 148 SMs, capped
// at `max_waves` waves.
inline int wave_grid(int64_t work_blocks, int per_sm, int max_waves = 8) {
  if (work_blocks < 1) work_blocks = 1;
  const int64_t wave = (int64_t)kNumSMs * per_sm;
  int64_t waves = ceil_div(work_blocks, wave);
  if (waves > max_waves) waves = max_waves;
  int64_t g = work_blocks < wave ? work_blocks : waves * wave;
  return (int)g;
}

// -------------------------------------------------------------- device side
#ifdef __CUDACC__

// Philox4x32-10 (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3",
// SC'11). Counter-based: the same (key, counter) gives the same four words on
// the GPU and in the CPU oracle.
struct Philox4 {
  uint32_t w[4];
};

__host__ __device__ inline Philox4 philox4x32_10(uint32_t c0, uint32_t c1,
                                                 uint32_t c2, uint32_t c3,
                                                 uint32_t k0, uint32_t k1) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)M0 * c0;
    const uint64_t p1 = (uint64_t)M1 * c2;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0;
    const uint32_t n1 = (uint32_t)p1;
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
    const uint32_t n3 = (uint32_t)p0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += W0; k1 += W1;
  }
  Philox4 out;
  out.w[0] = c0; out.w[1] = c1; out.w[2] = c2; out.w[3] = c3;
  return out;
}

__device__ __forceinline__ uint4 ld_stream_16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void st_stream_16(void* p, uint4 v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x),
               "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
// Plain (coherent) 16-byte store: used for stores into a peer GPU's memory.
__device__ __forceinline__ void st_plain_16(void* p, uint4 v) {
  asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x),
               "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
// Coherent 16-byte load (no .nc): for memory another GPU has just written.
__device__ __forceinline__ uint4 ld_plain_16(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// Two 8-byte words in one load that is not served from L1: for words that other blocks change meanwhile.
__device__ __forceinline__ ulonglong2 ld_volatile_2x8(const void* p) {
  ulonglong2 v;
  asm volatile("ld.volatile.global.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr int kMaxRanks = 32;

struct OwnerParams {
  int world_size;
  int shuffle_id_offset;
  int rank, node_beg, node_end;
};

// Owner of id v: the last rank d with min_vids[d] <= v, starting from
// shuffle_id_offset; owners outside this machine's rank window fall back to
// the calling rank.
__device__ __forceinline__ int owner_of(int64_t v, const int64_t* mv, const OwnerParams& p) {
  int d = p.shuffle_id_offset;
  while (d + 1 < p.world_size && mv[d + 1] <= v) ++d;
  if (d < p.node_beg || d >= p.node_end) d = p.rank;
  return d;
}

// A word block (of 32-bit values) on its way to page-locked host memory, the tag of a sequence number in the upper half of every
// word: the host polls for that, and nothing has to be ordered on the way. (A fence for a sequence number behind them all waits for
// the host link, 2 us when it is idle and up to 50 beside a gather's reads.) By all threads of a block.
struct Tagged {
  const int64_t* words;
  int count;
  const int64_t* last;            // the last word is taken from here
  const int64_t* sequence_dev;    // null: `sequence`
  int64_t sequence;
  int64_t* host;                  // null: nothing is published
};
__device__ __forceinline__ void publish_tagged(const Tagged& p) {
  const int64_t tag = (int64_t)tag_of(p.sequence_dev ? *p.sequence_dev : p.sequence) << 32;
  volatile int64_t* const host = p.host;
  for (int t = threadIdx.x; t < p.count; t += blockDim.x)
    host[t] = tag | ((t == p.count - 1 ? *(const volatile int64_t*)p.last : p.words[t]) & 0xffffffffll);
}

// Where the rows of a gather come from, for the kernels that make its ids: they look an id up as soon as they have it
// and flag what the gather would flag (no table: pos_map null), so that the flags are there before the rows are.
struct RowTables {
  const int64_t* pos_map;
  int64_t num_nodes, num_dev_rows, num_uva_rows;
};
__device__ __forceinline__ int check_row(const RowTables& t, int64_t id) {
  if (!t.pos_map) return 0;
  if (id < 0 || id >= t.num_nodes) return APT_FLAG_ID_OUT_OF_RANGE;
  const int64_t p = t.pos_map[id];
  if (p == -1) return APT_FLAG_FEAT_NOT_EXIST;
  return p >= t.num_dev_rows || (-p - 2) >= t.num_uva_rows ? APT_FLAG_ID_OUT_OF_RANGE : 0;
}

// First statement of every kernel launched with APT_FOLLOW: until the kernels before it are done and what they wrote can
// be read. None of them announces its end early (griddepcontrol.launch_dependents): this kernel's blocks would then sit
// on an SM beside blocks that still read lines about to be rewritten, and a load through the read-only path may find
// the old line in L1. Waiting for their exit gives the same times.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Sizes may live on the device: an operator chained behind another one takes
// its element count from a device word (what the previous kernel produced), so
// that the host never has to wait for it. `n_host` is then only an upper bound
// that sized the grid and the buffers.
__device__ __forceinline__ int64_t effective_n(int64_t n_host, const int64_t* n_dev) {
  if (!n_dev) return n_host;
  const int64_t v = *n_dev;
  return v < 0 ? 0 : (v < n_host ? v : n_host);
}

// Exclusive scan of one int per thread over a block of up to 1024 threads.
// Returns the thread's exclusive prefix; *total gets the block sum (all threads).
// `warp_sums` is a shared array of 33 ints. Ends with a __syncthreads().
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums,
                                                    int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    int s = lane < nw ? warp_sums[lane] : 0;
    int sinc = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, sinc, d);
      if (lane >= d) sinc += t;
    }
    warp_sums[lane] = sinc - s;  // exclusive warp offset
    if (lane == 31) warp_sums[32] = sinc;
  }
  __syncthreads();
  const int res = warp_sums[warp] + inc - v;
  *total = warp_sums[32];
  __syncthreads();
  return res;
}

#endif  // __CUDACC__

}  // namespace apt
