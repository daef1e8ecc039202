// Shared host utilities: thread-local error text and a device exclusive scan.
#include "common.cuh"
#include "device_limits.h"
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <iterator>
#include <map>
#include <mutex>

namespace impes {

static thread_local std::string g_last_error;

void set_last_error(const std::string& msg) { g_last_error = msg; }

static std::atomic<unsigned long long> g_launches{0};
static thread_local unsigned long long t_launches = 0;   // this host thread's launches
void count_launch() {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  ++t_launches;
}
void count_launches(long long n) {
  g_launches.fetch_add((unsigned long long)n, std::memory_order_relaxed);
  t_launches += (unsigned long long)n;
}
unsigned long long launches() { return g_launches.load(std::memory_order_relaxed); }
unsigned long long thread_launches() { return t_launches; }

namespace {
int current_device() {
  int dev = 0;
  IMPES_CUDA(cudaGetDevice(&dev));
  return dev;
}
}  // namespace
void raise_smem_limit(const void* kernel, size_t bytes) {
  static DeviceLimits limits;
  limits.raise(current_device(), kernel, bytes, [&](size_t v) {
    IMPES_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v));
  });
}
void allow_wide_cluster(const void* kernel) {
  static DeviceLimits limits;
  limits.raise(current_device(), kernel, 1, [&](size_t) {
    IMPES_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  });
}
int num_sms() {
  constexpr int kDevices = 128;
  static std::atomic<int> sms[kDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) dev = 0;
  int n = sms[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    sms[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}
namespace {
thread_local Arena* t_arena = nullptr;
}
Arena* Arena::current() { return t_arena; }
Arena::Scope::Scope(Arena& a) : before(t_arena) { t_arena = &a; }
Arena::Scope::~Scope() { t_arena = before; }

Arena::~Arena() {
  for (Chunk& c : chunks_) cudaFree(c.base);
}

void* Arena::take(size_t bytes) {
  const size_t need = (bytes + kAlign - 1) / kAlign * kAlign;
  Chunk* best = nullptr;
  std::map<size_t, size_t>::iterator at;
  for (Chunk& c : chunks_)             // the smallest free piece that holds it
    for (auto it = c.free.begin(); it != c.free.end(); ++it)
      if (it->second >= need && (!best || it->second < at->second)) {
        best = &c;
        at = it;
      }
  if (!best) {
    const size_t size = std::max(need, next_);
    void* base = nullptr;
    if (cudaMalloc(&base, size) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    next_ = std::min<size_t>(next_ * 2, 64u << 20);
    chunks_.push_back(Chunk{static_cast<char*>(base), size, {}});
    best = &chunks_.back();
    at = best->free.emplace(0, size).first;
  }
  const size_t off = at->first, len = at->second;
  best->free.erase(at);
  if (len > need) best->free.emplace(off + need, len - need);
  return best->base + off;
}

void Arena::give(void* p, size_t bytes) {
  const size_t len = (bytes + kAlign - 1) / kAlign * kAlign;
  for (Chunk& c : chunks_) {
    if (p < c.base || p >= c.base + c.size) continue;
    auto it = c.free.emplace(static_cast<size_t>(static_cast<char*>(p) - c.base), len).first;
    auto next = std::next(it);
    if (next != c.free.end() && it->first + it->second == next->first) {
      it->second += next->second;
      c.free.erase(next);
    }
    if (it != c.free.begin()) {
      auto prev = std::prev(it);
      if (prev->first + prev->second == it->first) {
        prev->second += it->second;
        c.free.erase(it);
      }
    }
    return;
  }
}

void Arena::trim() {
  for (size_t q = chunks_.size(); q-- > 0;) {
    Chunk& c = chunks_[q];
    if (c.free.size() == 1 && c.free.begin()->second == c.size) {
      cudaFree(c.base);
      chunks_.erase(chunks_.begin() + q);
    }
  }
}

const char* last_error_cstr() { return g_last_error.c_str(); }

bool stream_capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return st != cudaStreamCaptureStatusNone;
}

bool pdl_enabled() {
  static const bool on = [] {
    const char* ev = getenv("IMPES_NO_PDL");
    return !(ev && ev[0] == '1');
  }();
  return on;
}

namespace {
__global__ void k_fence() {}
}  // namespace
void pdl_fence(cudaStream_t s) {
  k_fence<<<1, 32, 0, s>>>(); count_launch();
  IMPES_CHECK_LAUNCH();
}

PhaseTimers& timers() {
  static PhaseTimers t;
  return t;
}

namespace {
constexpr int kScanBlock = 1024;

// Phase 1: per-block inclusive scan in shared memory; block totals to `sums`.
__global__ void k_scan_block(const int* __restrict__ in, int* __restrict__ out, int n,
                             int* __restrict__ sums) {
  __shared__ int s[kScanBlock];
  int i = blockIdx.x * kScanBlock + threadIdx.x;
  int v = (i < n) ? in[i] : 0;
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < kScanBlock; o <<= 1) {
    int t = (threadIdx.x >= (unsigned)o) ? s[threadIdx.x - o] : 0;
    __syncthreads();
    s[threadIdx.x] += t;
    __syncthreads();
  }
  if (i < n) out[i] = s[threadIdx.x] - v;  // exclusive
  if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = s[threadIdx.x];
}

// Phase 2: add the scanned block offsets; last element gets the total.
__global__ void k_scan_add(int* __restrict__ out, int n, const int* __restrict__ offs) {
  int i = blockIdx.x * kScanBlock + threadIdx.x;
  if (i < n) out[i] += offs[blockIdx.x];
}
__global__ void k_scan_total(const int* __restrict__ in, int* __restrict__ out, int n) {
  out[n] = (n > 0) ? out[n - 1] + in[n - 1] : 0;
}
}  // namespace

void exclusive_scan_i32_dev(const int* d_in, int* d_out, int n, cudaStream_t stream) {
  if (n <= 0) {
    IMPES_CUDA(cudaMemsetAsync(d_out, 0, sizeof(int), stream));
    return;
  }
  int nb = (n + kScanBlock - 1) / kScanBlock;
  DBuf<int> sums(nb), offs(nb + 1);
  k_scan_block<<<nb, kScanBlock, 0, stream>>>(d_in, d_out, n, sums.p); ::impes::count_launch();
  IMPES_CHECK_LAUNCH();
  if (nb > 1) {
    exclusive_scan_i32_dev(sums.p, offs.p, nb, stream);
    k_scan_add<<<nb, kScanBlock, 0, stream>>>(d_out, n, offs.p); ::impes::count_launch();
    IMPES_CHECK_LAUNCH();
  }
  k_scan_total<<<1, 1, 0, stream>>>(d_in, d_out, n); ::impes::count_launch();
  IMPES_CHECK_LAUNCH();
  // temporaries are freed at scope exit: make sure the kernels using them ran
  IMPES_CUDA(cudaStreamSynchronize(stream));
}

int exclusive_scan_i32(const int* d_in, int* d_out, int n, cudaStream_t stream) {
  exclusive_scan_i32_dev(d_in, d_out, n, stream);
  int total = 0;
  IMPES_CUDA(cudaMemcpyAsync(&total, d_out + n, sizeof(int), cudaMemcpyDeviceToHost, stream));
  IMPES_CUDA(cudaStreamSynchronize(stream));
  return total;
}

}  // namespace impes
