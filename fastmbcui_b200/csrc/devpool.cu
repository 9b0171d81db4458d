#include "devpool.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "cuda_util.h"

namespace mbc {

namespace {

constexpr int kMaxDevices = 64;
constexpr size_t kBound = (size_t)8 << 30;  // idle bytes a pool keeps: at most this and a sixteenth of the device
// ... while a quarter of the device is free besides (others, such as a tensor
// library's allocator, come first), looked at as a plan or solver ends, but not
// again within this time: the question takes the driver 0.1 ms and more
constexpr size_t kRoom = 4;
constexpr std::chrono::milliseconds kLook(200);

// Idle cudaMalloc blocks of one device, by size.  (The driver's own
// stream-ordered pools hand out kept memory as fast, but take 5 ms per GB to
// grow, ten times cudaMalloc.)
struct Pool {
  std::mutex mu;
  struct Block {
    void *ptr;
    uint64_t seq;  // order of release: the oldest goes first when the bound is met
  };
  std::multimap<size_t, Block> idle;
  size_t idle_bytes = 0, bound = 0;
  std::chrono::steady_clock::time_point looked{};  // at the device's free memory
  uint64_t seq = 0;
};
Pool g_pools[kMaxDevices];
std::atomic<int64_t> g_alive{0};

// sizes in steps of an eighth of their power of two (small) or 2 MB, so that
// the buffers of the next pose's solver fit those of the last
size_t rounded(size_t b)
{
  if (b < 4096) return (b + 511) / 512 * 512;
  if (b >= (size_t)16 << 20) return (b + ((size_t)2 << 20) - 1) / ((size_t)2 << 20) * ((size_t)2 << 20);
  size_t step = 512;
  while (step * 16 < b) step *= 2;
  return (b + step - 1) / step * step;
}

// frees idle blocks, the oldest first, until at most `keep` bytes are left;
// the pool's device is current and its mutex held
void trim(Pool &p, size_t keep)
{
  while (p.idle_bytes > keep && !p.idle.empty()) {
    auto old = p.idle.begin();
    for (auto it = p.idle.begin(); it != p.idle.end(); ++it)
      if (it->second.seq < old->second.seq) old = it;
    cudaFree(old->second.ptr);
    p.idle_bytes -= old->first;
    p.idle.erase(old);
  }
}

struct DeviceGuard {  // a device made current for a while
  int prev = -1;
  explicit DeviceGuard(int dev)
  {
    if (cudaGetDevice(&prev) != cudaSuccess || prev == dev) prev = -1;
    else cudaSetDevice(dev);
  }
  ~DeviceGuard()
  {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

thread_local cudaStream_t t_stream = nullptr;
thread_local bool t_in_call = false;

}  // namespace

CallScope::CallScope(cudaStream_t st) : st_(st), prev_(t_stream), had_(t_in_call)
{
  t_stream = st;
  t_in_call = true;
}

CallScope::~CallScope()
{
  t_stream = prev_;
  t_in_call = had_;
}

mbc_status CallScope::end(mbc_status s)
{
  if (s != MBC_OK) cudaStreamSynchronize(st_);  // the first error stands
  return s;
}

void DevMem::release()
{
  if (!ptr) return;
  if (t_in_call) cudaStreamSynchronize(t_stream);
  if (dev_ < 0) {
    cudaFree(ptr);
  } else {
    Pool &p = g_pools[dev_];
    DeviceGuard on(dev_);
    std::lock_guard<std::mutex> lk(p.mu);
    if (size_ > p.bound) {
      cudaFree(ptr);
    } else {
      trim(p, p.bound - size_);
      try {
        p.idle.emplace(size_, Pool::Block{ptr, ++p.seq});
        p.idle_bytes += size_;
      } catch (const std::bad_alloc &) {  // a destructor may be the caller
        cudaFree(ptr);
      }
    }
  }
  ptr = nullptr;
  bytes = size_ = 0;
  dev_ = -1;
}

mbc_status DevMem::reserve(size_t b)
{
  if (b <= bytes && ptr) return MBC_OK;
  release();
  if (b == 0) b = 16;
  int dev = -1;
  MBC_CK(cudaGetDevice(&dev));
  Pool *p = dev >= 0 && dev < kMaxDevices ? &g_pools[dev] : nullptr;
  std::unique_lock<std::mutex> lk;
  if (p) lk = std::unique_lock<std::mutex>(p->mu);
  dev_ = -1;
  size_ = b;
  if (pooled_ && p) {
    if (p->bound == 0) {
      size_t free_b = 0, total_b = 0;
      MBC_CK(cudaMemGetInfo(&free_b, &total_b));
      p->bound = std::min<size_t>(kBound, total_b / 16);
    }
    dev_ = dev;
    size_ = rounded(b);
    auto it = p->idle.lower_bound(size_);
    if (it != p->idle.end() && it->first <= size_ + size_ / 8) {
      ptr = it->second.ptr;
      size_ = it->first;
      p->idle_bytes -= it->first;
      p->idle.erase(it);
    }
  }
  cudaError_t e = ptr ? cudaSuccess : cudaMalloc(&ptr, size_);
  if (e == cudaErrorMemoryAllocation && p && !p->idle.empty()) {
    // the pool's idle memory goes before any allocation of the library fails
    cudaGetLastError();
    trim(*p, 0);
    e = cudaMalloc(&ptr, size_);
  }
  if (e != cudaSuccess) {
    ptr = nullptr;
    size_ = 0;
    dev_ = -1;
    cudaGetLastError();
    return fail(MBC_NO_MEMORY, std::string("device allocation of ") + std::to_string(b) + " bytes: " + cudaGetErrorString(e));
  }
  bytes = b;
  return MBC_OK;
}

mbc_status DevMem::reserve_spare(size_t b)
{
  constexpr size_t kSmall = (size_t)64 << 20;  // not asked about
  if ((b > bytes || !ptr) && b > kSmall) {
    size_t free_b = 0, total_b = 0;
    MBC_CK(device_free_bytes(&free_b, &total_b));
    if (free_b < b + std::max((size_t)4 << 30, total_b / 10)) {
      release();
      return fail(MBC_NO_MEMORY, "no spare device memory");
    }
  }
  return reserve(b);
}

cudaError_t device_free_bytes(size_t *free_b, size_t *total_b)
{
  const cudaError_t e = cudaMemGetInfo(free_b, total_b);
  int dev = -1;
  if (e != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return e;
  std::lock_guard<std::mutex> lk(g_pools[dev].mu);
  *free_b += g_pools[dev].idle_bytes;
  return cudaSuccess;
}

void pool_retain() { ++g_alive; }

void pool_drop()
{
  const bool last = --g_alive == 0;
  for (int d = 0; d < kMaxDevices; ++d) {
    std::lock_guard<std::mutex> lk(g_pools[d].mu);
    if (g_pools[d].idle.empty()) continue;
    DeviceGuard on(d);
    if (!last) {
      const auto now = std::chrono::steady_clock::now();
      size_t free_b = 0, total_b = 0;
      if (now - g_pools[d].looked < kLook) continue;
      g_pools[d].looked = now;
      if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && free_b >= total_b / kRoom) continue;
    }
    trim(g_pools[d], 0);
  }
}

namespace {

// pinned flags: one page for all solvers, 16-byte slots
constexpr int kSlots = 256;
std::mutex g_flag_mu;
int32_t *g_flag_page = nullptr;
std::vector<int32_t *> g_flag_free;

}  // namespace

int32_t *pinned_flags()
{
  std::lock_guard<std::mutex> lk(g_flag_mu);
  if (!g_flag_page) {
    try {
      g_flag_free.reserve(kSlots);  // no later push allocates
    } catch (const std::bad_alloc &) {
      return nullptr;
    }
    if (cudaHostAlloc((void **)&g_flag_page, sizeof(int32_t) * 4 * kSlots, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      g_flag_page = nullptr;
      return nullptr;
    }
    for (int k = kSlots - 1; k >= 0; --k) g_flag_free.push_back(g_flag_page + 4 * k);
  }
  int32_t *p = nullptr;
  if (!g_flag_free.empty()) {
    p = g_flag_free.back();
    g_flag_free.pop_back();
  } else if (cudaHostAlloc((void **)&p, sizeof(int32_t) * 4, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
  }
  return p;
}

void pinned_flags_release(int32_t *p)
{
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_flag_mu);
  if (g_flag_page && p >= g_flag_page && p < g_flag_page + 4 * kSlots) g_flag_free.push_back(p);
  else cudaFreeHost(p);
}

}  // namespace mbc
