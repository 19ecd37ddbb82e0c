// Exclusive prefix sums, and the small host helpers of kernels.cuh.
//
// The scan is the usual three phases: every CTA reduces its chunk, one CTA
// scans the chunk totals, every CTA rescans its chunk from its total. Up to
// kSmallMax values (most of the path's scans: block totals, cell indexes) it is
// one CTA with every value in registers: one launch instead of three.
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <vector>

#include "kernels.cuh"

namespace sifg {

std::atomic<uint64_t> g_kernel_launches{0};

constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr uint32_t kScanChunk = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums,
                                                         uint32_t& total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= (unsigned)d) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t w = lane < (unsigned)nw ? warp_sums[lane] : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= (unsigned)d) w += y;
    }
    if (lane < (unsigned)nw) warp_sums[lane] = w;
  }
  __syncthreads();
  total = warp_sums[(blockDim.x >> 5) - 1];
  const uint32_t before = warp ? warp_sums[warp - 1] : 0u;
  __syncthreads();
  return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t* __restrict__ d,
                                                                   uint32_t n,
                                                                   uint32_t* __restrict__ sums) {
  __shared__ uint32_t ws[32];
  const uint32_t base = blockIdx.x * kScanChunk;
  uint32_t acc = 0;
  for (int k = 0; k < kScanItems; k++) {
    const uint32_t i = base + k * kScanThreads + threadIdx.x;
    if (i < n) acc += d[i];
  }
  uint32_t total;
  block_exclusive_scan(acc, ws, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(uint32_t* __restrict__ sums,
                                                                 uint32_t m) {
  __shared__ uint32_t ws[32];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < m; base += kScanThreads) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < m ? sums[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(v, ws, total);
    if (i < m) sums[i] = carry + ex;
    carry += total;
  }
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(uint32_t* __restrict__ d,
                                                                  uint32_t n,
                                                                  const uint32_t* __restrict__ sums) {
  __shared__ uint32_t ws[32];
  const uint32_t base = blockIdx.x * kScanChunk;
  // Each thread owns kScanItems consecutive entries.
  const uint32_t first = base + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t acc = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const uint32_t i = first + k;
    v[k] = i < n ? d[i] : 0u;
    acc += v[k];
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan(acc, ws, total) + sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const uint32_t i = first + k;
    if (i < n) d[i] = run;
    run += v[k];
  }
}

// One CTA for up to kSmallMax values: each warp holds kSmallPer consecutive
// ones in registers, sixteen bytes a load, scans them by itself, and one
// exchange of the warps' totals places them. The scans of the path's block
// totals and cell indexes sit between dependent launches, so this CTA's latency
// is theirs: every load is in flight before the first is used, and there are
// two barriers whatever the count. (By chunks of 4,096 with a block scan each:
// 19 us for the 16,385 block totals of a 512^3 list, and three launches for a
// void index of 32,769 cells.)
// last_zero: d[n - 1] is taken as 0 (not read); total, when set, receives the
// sum of all n. d is 16-byte aligned.
constexpr int kSmallT = 1024;
constexpr uint32_t kSmallRows = 9;                     // 128 values a row
constexpr uint32_t kSmallPer = kSmallRows * 128;       // a warp's
constexpr uint32_t kSmallMax = kSmallT / 32 * kSmallPer;
__global__ void __launch_bounds__(kSmallT) scan_small_kernel(uint32_t* __restrict__ d, uint32_t n,
                                                             bool last_zero, uint32_t rows,
                                                             uint32_t* __restrict__ total_out) {
  __shared__ uint32_t ws[kSmallT / 32];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t base = warp * rows * 128 + lane * 4;
  uint4 v[kSmallRows];
#pragma unroll
  for (uint32_t r = 0; r < kSmallRows; r++) {
    const uint32_t i = base + r * 128;
    v[r] = make_uint4(0, 0, 0, 0);
    if (r >= rows) continue;
    if (i + 4 < n) {  // none of the four is the last value
      v[r] = *reinterpret_cast<const uint4*>(d + i);
    } else {
      const uint32_t end = last_zero ? n - 1 : n;
      if (i < end) v[r].x = d[i];
      if (i + 1 < end) v[r].y = d[i + 1];
      if (i + 2 < end) v[r].z = d[i + 2];
      if (i + 3 < end) v[r].w = d[i + 3];
    }
  }
  uint32_t run = 0;  // the warp's values before row r
#pragma unroll
  for (uint32_t r = 0; r < kSmallRows; r++) {
    if (r >= rows) break;
    const uint32_t sum = v[r].x + v[r].y + v[r].z + v[r].w;
    uint32_t x = sum;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, k);
      if (lane >= (unsigned)k) x += y;
    }
    const uint32_t e = run + x - sum;
    run += __shfl_sync(0xffffffffu, x, 31);
    const uint4 q = v[r];
    v[r] = make_uint4(e, e + q.x, e + q.x + q.y, e + q.x + q.y + q.z);
  }
  if (lane == 0) ws[warp] = run;
  __syncthreads();
  const uint32_t mine = ws[lane];
  uint32_t x = mine;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, k);
    if (lane >= (unsigned)k) x += y;
  }
  const uint32_t before = __shfl_sync(0xffffffffu, x - mine, warp);
  if (total_out && threadIdx.x == 31) *total_out = x;
#pragma unroll
  for (uint32_t r = 0; r < kSmallRows; r++) {
    if (r >= rows) break;
    const uint32_t i = base + r * 128;
    const uint4 q = make_uint4(v[r].x + before, v[r].y + before, v[r].z + before, v[r].w + before);
    if (i + 3 < n) {
      *reinterpret_cast<uint4*>(d + i) = q;
    } else {
      if (i < n) d[i] = q.x;
      if (i + 1 < n) d[i + 1] = q.y;
      if (i + 2 < n) d[i + 2] = q.z;
    }
  }
}

static void scan_small(uint32_t* d, uint32_t n, bool last_zero, uint32_t* total, cudaStream_t st) {
  const uint32_t rows = (n + kSmallT / 32 * 128 - 1) / (kSmallT / 32 * 128);
  scan_small_kernel<<<1, kSmallT, 0, st>>>(d, n, last_zero, rows, total);
  SIFG_LAUNCH_CHECK();
}

static bool scan_is_small(const uint32_t* d, uint32_t n) {
  return n <= kSmallMax && (uintptr_t)d % 16 == 0;
}

__global__ void store_last_kernel(const uint32_t* __restrict__ d, uint32_t i,
                                  uint32_t* __restrict__ out) {
  *out = d[i];
}

uint32_t scan_sums_needed(uint32_t n) { return (n + kScanChunk - 1) / kScanChunk; }

void exclusive_scan_u32(uint32_t* data, uint32_t n, cudaStream_t st, uint32_t* sums_scratch) {
  if (n == 0) return;
  if (scan_is_small(data, n)) {
    scan_small(data, n, false, nullptr, st);
    return;
  }
  const uint32_t blocks = (n + kScanChunk - 1) / kScanChunk;
  thread_local DevBuf sums;  // chunk totals; small; one per host thread driving a stream
  uint32_t* s = sums_scratch ? sums_scratch
                             : (uint32_t*)sums.ensure((size_t)blocks * sizeof(uint32_t));
  scan_reduce_kernel<<<blocks, kScanThreads, 0, st>>>(data, n, s);
  SIFG_LAUNCH_CHECK();
  scan_sums_kernel<<<1, kScanThreads, 0, st>>>(s, blocks);
  SIFG_LAUNCH_CHECK();
  scan_apply_kernel<<<blocks, kScanThreads, 0, st>>>(data, n, s);
  SIFG_LAUNCH_CHECK();
}

void exclusive_scan_total(uint32_t* data, uint32_t nb, uint32_t* total, cudaStream_t st) {
  const uint32_t n = nb + 1;
  if (scan_is_small(data, n)) {
    // One launch: data[nb] taken as zero, the total written as the scan ends.
    scan_small(data, n, true, total, st);
    return;
  }
  SIFG_CUDA(cudaMemsetAsync(data + nb, 0, sizeof(uint32_t), st));
  exclusive_scan_u32(data, n, st);
  store_last_kernel<<<1, 1, 0, st>>>(data, nb, total);
  SIFG_LAUNCH_CHECK();
}

// --- helpers ---

void* DevBuf::ensure(size_t want) {
  if (want <= bytes && ptr) return ptr;
  release();
  size_t b = want < 256 ? 256 : want;
  SIFG_CUDA(cudaMalloc(&ptr, b));
  bytes = b;
  return ptr;
}

void DevBuf::release() {
  if (ptr) cudaFree(ptr);
  ptr = nullptr;
  bytes = 0;
}

// Timing events are kept for reuse, per device, instead of being created and
// destroyed for every span (a run records a few hundred). The pool and its
// lock are never destroyed: timers held by static objects return their
// events at exit, in no fixed order with other files' statics.
static std::mutex& event_mu() {
  static std::mutex* m = new std::mutex;
  return *m;
}
static std::map<int, std::vector<cudaEvent_t>>& event_pool() {
  static auto* p = new std::map<int, std::vector<cudaEvent_t>>;
  return *p;
}

static cudaEvent_t take_event() {
  int dev = 0;
  SIFG_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lk(event_mu());
    auto& pool = event_pool()[dev];
    if (!pool.empty()) {
      const cudaEvent_t e = pool.back();
      pool.pop_back();
      return e;
    }
  }
  cudaEvent_t e;
  SIFG_CUDA(cudaEventCreate(&e));
  return e;
}

static void give_event(cudaEvent_t e) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaEventDestroy(e);
    return;
  }
  std::lock_guard<std::mutex> lk(event_mu());
  event_pool()[dev].push_back(e);
}

void event_pool_clear() {
  std::lock_guard<std::mutex> lk(event_mu());
  for (auto& [dev, pool] : event_pool())
    for (cudaEvent_t e : pool) cudaEventDestroy(e);
  event_pool().clear();
}

void KernelTimer::begin(cudaStream_t st) {
  const cudaEvent_t e = take_event();
  starts.push_back(e);
  open = (int)starts.size() - 1;
  SIFG_CUDA(cudaEventRecord(e, st));
}

void KernelTimer::end(cudaStream_t st) {
  const cudaEvent_t e = take_event();
  stops.push_back(e);
  open = -1;
  SIFG_CUDA(cudaEventRecord(e, st));
}

double KernelTimer::total_ms() {
  double t = 0.0;
  for (size_t i = 0; i < stops.size() && i < starts.size(); i++) {
    SIFG_CUDA(cudaEventSynchronize(stops[i]));
    float ms = 0.f;
    SIFG_CUDA(cudaEventElapsedTime(&ms, starts[i], stops[i]));
    t += ms;
  }
  return t;
}

void KernelTimer::reset() {
  for (auto e : starts) give_event(e);
  for (auto e : stops) give_event(e);
  starts.clear();
  stops.clear();
  open = -1;
}

KernelTimer::~KernelTimer() { reset(); }

}  // namespace sifg
