// The device memory pool (devpool.cu, compiled as host code) against a fake
// CUDA runtime: two devices of a given size, allocations counted, streams
// that record when they are waited for.  Run with the name of one check.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "devpool.h"

// ---- the fake runtime ----
namespace {

constexpr size_t kGiB = (size_t)1 << 30;
size_t g_total = 64 * kGiB, g_other[2] = {0, 0};  // device size, memory of other users
std::map<void *, std::pair<size_t, int>> g_live;  // size, device
uintptr_t g_next = 1 << 20;
int g_mallocs = 0, g_frees = 0, g_host = 0;
std::vector<cudaStream_t> g_waited;
thread_local int t_dev = 0;
bool g_fail_new = false;

size_t used(int dev)
{
  size_t s = g_other[dev];
  for (auto &e : g_live)
    if (e.second.second == dev) s += e.second.first;
  return s;
}

}  // namespace

void *operator new(size_t n)
{
  if (g_fail_new) throw std::bad_alloc();
  if (void *p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaGetDevice(int *d)
{
  *d = t_dev;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d)
{
  t_dev = d;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n)
{
  if (used(t_dev) + n > g_total) return cudaErrorMemoryAllocation;
  *p = (void *)g_next;
  g_next += n + 512;
  g_live[*p] = {n, t_dev};
  ++g_mallocs;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
  if (!g_live.erase(p)) {
    std::fprintf(stderr, "cudaFree of %p, which is not allocated\n", p);
    std::exit(1);
  }
  ++g_frees;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t)
{
  *t = g_total;
  *f = g_total - used(t_dev);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
  g_waited.push_back(st);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
  *p = std::malloc(n);
  ++g_host;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
  std::free(p);
  --g_host;
  return cudaSuccess;
}
}

namespace mbc {
mbc_status fail(mbc_status s, const std::string &) { return s; }
}  // namespace mbc

#define CHECK(x)                                                     \
  do {                                                               \
    if (!(x)) {                                                      \
      std::fprintf(stderr, "line %d: %s\n", __LINE__, #x);           \
      std::exit(1);                                                  \
    }                                                                \
  } while (0)

using mbc::DevMem;

namespace {

const size_t MiB = (size_t)1 << 20;

// what is released serves the next request of about its size, of any thread;
// another device's does not; the last user's end gives everything back
void reuse()
{
  {
    mbc::PoolUser user;
    void *a, *b;
    {
      DevMem x, y;
      CHECK(x.reserve(100 * MiB) == MBC_OK && y.reserve(3000) == MBC_OK);
      a = x.ptr, b = y.ptr;
    }
    CHECK(g_mallocs == 2 && g_frees == 0);
    std::thread([&] {
      DevMem x, y;
      CHECK(x.reserve(99 * MiB) == MBC_OK && y.reserve(2900) == MBC_OK);
      CHECK(x.ptr == a && y.ptr == b && g_mallocs == 2);
      DevMem z;  // a kept block is not given for a request far smaller than it
      CHECK(z.reserve(10 * MiB) == MBC_OK && g_mallocs == 3);
    }).join();
    std::thread([&] {
      t_dev = 1;
      DevMem x;
      CHECK(x.reserve(100 * MiB) == MBC_OK && g_mallocs == 4);
    }).join();
    size_t f, t;
    CHECK(mbc::device_free_bytes(&f, &t) == cudaSuccess && f == g_total);  // idle memory counts as free
  }
  CHECK(g_live.empty() && t_dev == 0);
}

// at most a sixteenth of the device is kept (4 of 64 GiB), the oldest goes
// first, and a block above the bound is not kept
void bound()
{
  mbc::PoolUser user;
  void *first;
  {
    DevMem a, b, c;
    CHECK(a.reserve(2 * kGiB) == MBC_OK && b.reserve(2 * kGiB) == MBC_OK && c.reserve(2 * kGiB) == MBC_OK);
    first = c.ptr;  // destroyed first
  }
  CHECK(g_live.size() == 2 && !g_live.count(first));
  {
    DevMem a;
    CHECK(a.reserve(5 * kGiB) == MBC_OK);
  }
  CHECK(used(0) == 4 * kGiB);
}

// an allocation that would fail takes the idle memory
void trim()
{
  mbc::PoolUser user;
  {
    DevMem a;
    CHECK(a.reserve(3 * kGiB) == MBC_OK);
  }
  DevMem big;
  CHECK(big.reserve(63 * kGiB) == MBC_OK && g_live.size() == 1);
  DevMem more;
  CHECK(more.reserve(2 * kGiB) == MBC_NO_MEMORY && !more.ptr);
  CHECK(more.reserve(kGiB) == MBC_OK);
}

// ... also one that does not come from the pool itself
void trim_unpooled()
{
  mbc::PoolUser user;
  {
    DevMem a;
    CHECK(a.reserve(3 * kGiB) == MBC_OK);
  }
  DevMem big(false);
  CHECK(big.reserve(63 * kGiB) == MBC_OK && g_live.size() == 1);
  big.release();
  CHECK(g_live.empty());
}

// what a kept object holds between its calls is no reason to keep idle memory
void leave()
{
  mbc::PoolUser *kept = new mbc::PoolUser();
  DevMem own;
  {
    mbc::PoolUser call;
    DevMem a;
    CHECK(own.reserve(MiB) == MBC_OK && a.reserve(kGiB) == MBC_OK);
    a.release();
    CHECK(g_live.size() == 2);
    kept->leave();
    CHECK(g_live.size() == 2);
  }
  CHECK(g_live.size() == 1 && own.ptr);
  {
    mbc::PoolUser end;
    own.release();
    delete kept;  // counted once
    CHECK(g_live.size() == 1);
  }
  CHECK(g_live.empty());
}

// memory that a call can do without leaves 4 GiB or a tenth of the device, idle
// memory counted as free; 64 MB are always given
void spare()
{
  mbc::PoolUser user;
  {
    DevMem a;
    CHECK(a.reserve(2 * kGiB) == MBC_OK);
  }
  g_other[0] = 54 * kGiB;  // 10 of 64 GiB free, 2 of them idle
  DevMem x;
  CHECK(x.reserve_spare(3 * kGiB) == MBC_OK);
  CHECK(x.reserve_spare(3 * kGiB) == MBC_OK);  // has it already
  CHECK(x.reserve_spare(5 * kGiB) == MBC_NO_MEMORY && !x.ptr && !x.bytes);
  g_other[0] = 59 * kGiB;
  CHECK(x.reserve_spare(kGiB) == MBC_NO_MEMORY && x.reserve_spare(64 * MiB) == MBC_OK);
}

// with less than a quarter of the device free nothing idle outlives a solver
void room()
{
  mbc::PoolUser user;
  for (size_t others : {40 * kGiB, 50 * kGiB}) {
    std::this_thread::sleep_for(std::chrono::milliseconds(250));  // it is looked at five times a second
    g_other[0] = others;
    {
      mbc::PoolUser solver;
      DevMem a;
      CHECK(a.reserve(2 * kGiB) == MBC_OK);
    }
    CHECK(used(0) == others + (others == 40 * kGiB ? 2 * kGiB : 0));
  }
  CHECK(t_dev == 0);
}

// inside a call a release waits for the call's stream, a failing call for its
// work; outside of calls nothing waits
void waits()
{
  mbc::PoolUser user;
  cudaStream_t st = (cudaStream_t)64;
  {
    mbc::CallScope scope(st);
    DevMem a;
    CHECK(a.reserve(MiB) == MBC_OK && a.reserve(2 * MiB) == MBC_OK && g_waited.size() == 1 && g_waited[0] == st);
    CHECK(scope.end(MBC_OK) == MBC_OK && g_waited.size() == 1);
    CHECK(scope.end(MBC_BAD_ARG) == MBC_BAD_ARG && g_waited.size() == 2);
  }
  CHECK(g_waited.size() == 3);  // a's release, still inside the scope
  {
    DevMem a;
    CHECK(a.reserve(MiB) == MBC_OK);
  }
  CHECK(g_waited.size() == 3);
}

// no host memory for the pool's lists: the block is freed, nothing is thrown
void host_memory()
{
  mbc::PoolUser user;
  {
    DevMem a;
    CHECK(a.reserve(MiB) == MBC_OK);
    g_fail_new = true;
  }
  CHECK(mbc::pinned_flags() == nullptr);
  g_fail_new = false;
  CHECK(g_live.empty());
  int32_t *p = mbc::pinned_flags();
  CHECK(p != nullptr);
  g_fail_new = true;
  mbc::pinned_flags_release(p);
  g_fail_new = false;
  CHECK(mbc::pinned_flags() == p && g_host == 1);
}

}  // namespace

int main(int argc, char **argv)
{
  const std::map<std::string, void (*)()> checks = {
      {"reuse", reuse}, {"bound", bound}, {"trim", trim}, {"trim_unpooled", trim_unpooled}, {"leave", leave},
      {"room", room}, {"spare", spare}, {"waits", waits}, {"host_memory", host_memory}};
  auto it = checks.find(argc > 1 ? argv[1] : "");
  if (it == checks.end()) return 2;
  it->second();
  std::puts("ok");
  return 0;
}
