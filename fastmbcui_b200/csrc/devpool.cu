#include "devpool.h"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "cuda_util.h"

namespace mbc {

namespace {

constexpr int kMaxDevices = 64;
constexpr size_t kBound = (size_t)8 << 30;  // idle bytes a pool keeps: at most this and a sixteenth of the device

// One memory pool and one stream per device.  Every allocation and every
// release is ordered on that stream and the allocating thread waits for it
// (it is idle but for them), so memory released by one thread may go to a
// solver of another thread and stream.
struct Pool {
  std::once_flag once;
  std::atomic<cudaMemPool_t> pool{nullptr};
  cudaStream_t st = nullptr;
};
Pool g_pools[kMaxDevices];
std::atomic<int64_t> g_alive{0};

// the pool of a device (made on first use with the device current), or NULL
// where the device has no stream-ordered allocator
Pool *pool_of(int dev)
{
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  Pool &p = g_pools[dev];
  std::call_once(p.once, [&] {
    int ok = 0;
    size_t free_b = 0, total_b = 0;
    if (cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, dev) != cudaSuccess || !ok ||
        cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t mp = nullptr;
    cudaStream_t st = nullptr;
    uint64_t keep = std::min<size_t>(kBound, total_b / 16);
    if (cudaMemPoolCreate(&mp, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(mp, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
        cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      if (mp) cudaMemPoolDestroy(mp);
      return;
    }
    p.st = st;
    p.pool = mp;
  });
  return p.pool ? &p : nullptr;
}

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
    int cur = -1;
    if (cudaGetDevice(&cur) == cudaSuccess && cur != dev_) cudaSetDevice(dev_);
    cudaFreeAsync(ptr, p.st);
    if (cur >= 0 && cur != dev_) cudaSetDevice(cur);
  }
  ptr = nullptr;
  bytes = 0;
  dev_ = -1;
}

mbc_status DevMem::reserve(size_t b)
{
  if (b <= bytes && ptr) return MBC_OK;
  release();
  if (b == 0) b = 16;
  int dev = -1;
  MBC_CK(cudaGetDevice(&dev));
  Pool *p = pooled_ ? pool_of(dev) : nullptr;
  cudaError_t e = cudaSuccess;
  if (p) {
    e = cudaMallocFromPoolAsync(&ptr, b, p->pool, p->st);
    if (e == cudaErrorMemoryAllocation) {
      // give the idle memory back and try once more
      cudaGetLastError();
      cudaStreamSynchronize(p->st);
      cudaMemPoolTrimTo(p->pool, 0);
      e = cudaMallocFromPoolAsync(&ptr, b, p->pool, p->st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(p->st);
    dev_ = dev;
  } else {
    e = cudaMalloc(&ptr, b);
    dev_ = -1;
  }
  if (e != cudaSuccess) {
    ptr = nullptr;
    dev_ = -1;
    cudaGetLastError();
    return fail(MBC_NO_MEMORY, std::string("device allocation of ") + std::to_string(b) + " bytes: " + cudaGetErrorString(e));
  }
  bytes = b;
  return MBC_OK;
}

cudaError_t device_free_bytes(size_t *free_b, size_t *total_b)
{
  cudaError_t e = cudaMemGetInfo(free_b, total_b);
  if (e != cudaSuccess) return e;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return cudaSuccess;
  if (Pool *p = pool_of(dev)) {
    uint64_t held = 0, used = 0;
    if (cudaMemPoolGetAttribute(p->pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
        cudaMemPoolGetAttribute(p->pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess && held > used)
      *free_b += (size_t)(held - used);
  }
  return cudaSuccess;
}

void pool_retain() { ++g_alive; }

void pool_drop()
{
  if (--g_alive != 0) return;
  int cur = -1;
  bool moved = false;
  for (int d = 0; d < kMaxDevices; ++d) {
    Pool &p = g_pools[d];
    if (!p.pool) continue;
    if (cur < 0 && cudaGetDevice(&cur) != cudaSuccess) return;
    if (d != cur) {
      cudaSetDevice(d);
      moved = true;
    }
    cudaStreamSynchronize(p.st);
    cudaMemPoolTrimTo(p.pool, 0);
  }
  if (moved) cudaSetDevice(cur);
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
