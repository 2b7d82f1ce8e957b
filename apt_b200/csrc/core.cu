// Process-wide plumbing of libapt_b200: last-error text, launch counter and
// the optional event-based per-kernel timer.
#include <stdarg.h>
#include <string.h>

#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"

namespace apt {

static thread_local char g_err[512] = "";
static std::atomic<int64_t> g_launches{0};

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// ---- profiler: a growing list of (tag, begin, end) event pairs.
struct ProfRec {
  const char* tag;
  cudaEvent_t beg, end;
};
static std::atomic<int> g_prof_on{0};
static std::mutex g_prof_mu;
static std::vector<ProfRec> g_prof;
static const size_t kProfMax = 1 << 16;

// Events are pooled: after a read they go back to the free list, so a steady
// loop creates no events.
static std::vector<cudaEvent_t> g_free_events;

static bool take_event(cudaEvent_t* ev) {
  if (!g_free_events.empty()) {
    *ev = g_free_events.back();
    g_free_events.pop_back();
    return true;
  }
  return cudaEventCreate(ev) == cudaSuccess;
}

ProfScope::ProfScope(const char* t, cudaStream_t s) : tag(t), stream(s), slot(-1) {
  if (!g_prof_on.load(std::memory_order_relaxed)) return;
  std::lock_guard<std::mutex> lk(g_prof_mu);
  if (g_prof.size() >= kProfMax) return;
  ProfRec r;
  r.tag = t;
  if (!take_event(&r.beg)) return;
  if (!take_event(&r.end)) {
    g_free_events.push_back(r.beg);
    return;
  }
  cudaEventRecord(r.beg, s);
  g_prof.push_back(r);
  slot = (int)g_prof.size() - 1;
}
ProfScope::~ProfScope() {
  if (slot < 0) return;
  std::lock_guard<std::mutex> lk(g_prof_mu);
  if ((size_t)slot < g_prof.size()) cudaEventRecord(g_prof[slot].end, stream);
}

// The word block goes to page-locked host memory, a sequence number behind it last: the host polls for that, which
// takes the place of a copy, an event and a wake-up.
__global__ void __launch_bounds__(256)
k_publish_words(const int64_t* __restrict__ words, int count, const int64_t* __restrict__ last, const int64_t* __restrict__ sequence_dev,
                int64_t sequence, volatile int64_t* host) {
  wait_for_previous();
  if (threadIdx.x == 0 && sequence_dev) sequence = *sequence_dev;
  for (int t = threadIdx.x; t < count; t += blockDim.x) host[t] = last && t == count - 1 ? *last : words[t];
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) host[count] = sequence;
}

__global__ void __launch_bounds__(256)
k_publish_tagged(const Tagged p) {
  wait_for_previous();
  publish_tagged(p);
}

// Several arrays of words to places of their own: the tensors of a mini-batch that leave buffers much longer than they are, in
// one launch (a clone each is an operator call and a copy).
constexpr int kCopyParts = 24;
struct WordCopies {
  const int64_t* src[kCopyParts];
  int64_t* dst[kCopyParts];
  int64_t count[kCopyParts];
};
__global__ void __launch_bounds__(256)
k_copy_words(const __grid_constant__ WordCopies c) {
  wait_for_previous();
  constexpr int K = 4;
  const int64_t* const src = c.src[blockIdx.y];
  int64_t* const dst = c.dst[blockIdx.y];
  const int64_t n = c.count[blockIdx.y], stride = (int64_t)gridDim.x * 256;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += K * stride) {
    int64_t v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = i + k * stride < n ? src[i + k * stride] : 0;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (i + k * stride < n) dst[i + k * stride] = v[k];
  }
}

// What a replay starts from, in one kernel in front of it: the seeds, the call-id base and the sequence number of its
// counts. (A copy of the seeds, and one of the two words inside the graph, cost a launch more on the host and put a copy
// engine between kernels twice.)
__global__ void __launch_bounds__(256)
k_stage_replay(const int64_t* __restrict__ seeds, int64_t n, int64_t* __restrict__ seeds_buf, int64_t call_base, int64_t sequence,
               int64_t* __restrict__ words) {
  wait_for_previous();
  for (int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x; t < n; t += (int64_t)gridDim.x * 256) seeds_buf[t] = seeds[t];
  if (blockIdx.x == 0 && threadIdx.x < 2) words[threadIdx.x] = threadIdx.x ? sequence : call_base;
}

}  // namespace apt

extern "C" {

int apt_publish_words(const int64_t* words, int count, const int64_t* sequence_dev, int64_t sequence, int64_t* host,
                      void* stream) {
  return apt_publish_words_from(words, count, nullptr, sequence_dev, sequence, host, stream);
}

int apt_publish_words_from(const int64_t* words, int count, const int64_t* last, const int64_t* sequence_dev, int64_t sequence,
                           int64_t* host, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(words && host && count >= 0 && count <= 4096, "apt_publish_words: bad argument");
  APT_FOLLOW(k_publish_words, 1, 256, 0, (cudaStream_t)stream, words, count, last, sequence_dev, sequence, host);
  return APT_OK;
}

int apt_copy_words(const int64_t* const* src, int64_t* const* dst, const int64_t* counts, int num, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(num >= 0 && (num == 0 || (src && dst && counts)), "apt_copy_words: bad argument");
  for (int k0 = 0; k0 < num; k0 += kCopyParts) {
    WordCopies c{};
    const int parts = num - k0 < kCopyParts ? num - k0 : kCopyParts;
    int64_t most = 0;
    for (int k = 0; k < parts; ++k) {
      c.src[k] = src[k0 + k], c.dst[k] = dst[k0 + k], c.count[k] = counts[k0 + k];
      APT_CHECK_ARG(c.count[k] >= 0 && (c.count[k] == 0 || (c.src[k] && c.dst[k])), "apt_copy_words: bad part");
      if (c.count[k] > most) most = c.count[k];
    }
    if (most == 0) continue;
    const int64_t want = ceil_div(most, 1024), fit = (int64_t)kNumSMs * 8 / parts;
    APT_FOLLOW(k_copy_words, dim3((unsigned)(want < fit ? want : fit), (unsigned)parts), 256, 0, (cudaStream_t)stream, c);
  }
  return APT_OK;
}

int apt_stage_replay(const int64_t* seeds, int64_t num_seeds, int64_t* seeds_buf, int64_t call_base, int64_t sequence,
                     int64_t* words, void* stream) {
  using namespace apt;
  APT_CHECK_ARG(num_seeds >= 0 && words && (num_seeds == 0 || (seeds && seeds_buf)), "apt_stage_replay: bad argument");
  APT_FOLLOW(k_stage_replay, wave_grid(ceil_div(num_seeds, 256), 4, 1), 256, 0, (cudaStream_t)stream, seeds, num_seeds,
             seeds_buf, call_base, sequence, words);
  return APT_OK;
}

int apt_publish_tagged(const int64_t* words, int count, const int64_t* last, const int64_t* sequence_dev, int64_t sequence, int64_t* host,
                       void* stream) {
  using namespace apt;
  APT_CHECK_ARG(words && last && host && count >= 1 && count <= 4096, "apt_publish_tagged: bad argument");
  APT_FOLLOW(k_publish_tagged, 1, 256, 0, (cudaStream_t)stream, (Tagged{words, count, last, sequence_dev, sequence, host}));
  return APT_OK;
}

static int wait_for_word(const char* who, const volatile int64_t* word, int shift, int64_t sequence, void* stream) {
  for (int64_t spin = 1; (int64_t)((uint64_t)*word >> shift) != sequence; ++spin) {
    if ((spin & 0x3fff) == 0) {
      // now and then the stream is asked, so that an error on it ends the wait
      apt::RelaxedCapture relaxed;
      const cudaError_t e = cudaStreamQuery((cudaStream_t)stream);
      if (e == cudaErrorNotReady) continue;
      APT_CUDA(e);
      if ((int64_t)((uint64_t)*word >> shift) == sequence) break;
      apt::set_error("%s: the stream is idle and the words have not arrived", who);
      return APT_ERR_TIMEOUT;
    }
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
  }
  return APT_OK;
}

int apt_wait_published(const int64_t* host, int count, int64_t sequence, void* stream) {
  APT_CHECK_ARG(host && count >= 0, "apt_wait_published: bad argument");
  return wait_for_word("apt_wait_published", host + count, 0, sequence, stream);
}

int apt_wait_tagged(int64_t* host, int count, int64_t sequence, void* stream) {
  APT_CHECK_ARG(host && count >= 1, "apt_wait_tagged: bad argument");
  for (int t = count - 1; t >= 0; --t) {
    const int rc = wait_for_word("apt_wait_tagged", host + t, 32, apt::tag_of(sequence), stream);
    if (rc != APT_OK) return rc;
    host[t] = (int32_t)host[t];
  }
  return APT_OK;
}

const char* apt_last_error(void) { return apt::g_err; }
int apt_version(void) { return 100; }
int64_t apt_launch_count(void) { return apt::g_launches.load(); }
void apt_launch_count_reset(void) { apt::g_launches.store(0); }

int apt_memcpy_async(void* dst, const void* src, size_t nbytes, void* stream) {
  if (nbytes == 0) return APT_OK;
  APT_CHECK_ARG(dst && src, "apt_memcpy_async: null pointer");
  APT_CUDA(cudaMemcpyAsync(dst, src, nbytes, cudaMemcpyDefault, (cudaStream_t)stream));
  return APT_OK;
}

int apt_profile_enable(int on) {
  apt::g_prof_on.store(on ? 1 : 0);
  return APT_OK;
}

int apt_profile_read(const char* tag, double* total_ms, int64_t* launches) {
  APT_CHECK_ARG(tag && total_ms && launches, "apt_profile_read: null argument");
  std::lock_guard<std::mutex> lk(apt::g_prof_mu);
  double ms = 0.0;
  int64_t n = 0;
  std::vector<apt::ProfRec> keep;
  for (auto& r : apt::g_prof) {
    if (strcmp(r.tag, tag) != 0) {
      keep.push_back(r);
      continue;
    }
    float t = 0.f;
    cudaError_t e = cudaEventSynchronize(r.end);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&t, r.beg, r.end);
    apt::g_free_events.push_back(r.beg);
    apt::g_free_events.push_back(r.end);
    if (e != cudaSuccess) {
      apt::set_error("apt_profile_read(%s): %s", tag, cudaGetErrorString(e));
      apt::g_prof.swap(keep);
      return APT_ERR_CUDA;
    }
    ms += t;
    ++n;
  }
  apt::g_prof.swap(keep);
  *total_ms = ms;
  *launches = n;
  return APT_OK;
}

}  // extern "C"
