// Device memory of the solvers, from a bounded pool per device.
//
// A solver lives for one pose of a moving scene and owns some forty buffers,
// up to gigabytes of digit planes.  cudaMalloc and cudaFree map and unmap
// each of them and cudaFree waits for the device: 9 of 25 ms of a 3000-point
// FP64 solve and 15 of 190 ms of a 24000-point step went to them.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "mbc_internal.h"

namespace mbc {

// The stream of the library call that this thread is in.  Buffers that are
// released inside a call (a workspace that grows, a local one that ends) wait
// for it first; so does a call that ends with an error, which may have left
// work in flight.  Every call that succeeds ends with its stream synchronised,
// so buffers released outside a call (the solver's end) are idle.
class CallScope {
 public:
  explicit CallScope(cudaStream_t st);
  ~CallScope();
  CallScope(const CallScope &) = delete;
  CallScope &operator=(const CallScope &) = delete;
  // the call's result on its way out
  mbc_status end(mbc_status s);

 private:
  cudaStream_t st_, prev_;
  bool had_;
};

// Owned device allocation that only grows; memory of the current device's
// pool.  The pool keeps what is released, at most 8 GiB and a sixteenth of the
// device, for the next solver of any thread and stream.  It gives all of it
// back when an allocation of this library would fail, when a plan or solver
// ends on a device with less than a quarter free, and once no plan and no
// solver is alive but those that an operator context keeps between its calls.
struct DevMem {
  void *ptr = nullptr;
  size_t bytes = 0;
  DevMem() = default;
  // pooled = false: cudaMalloc and cudaFree (which waits for the device), for
  // objects whose calls return with work in flight
  explicit DevMem(bool pooled) : pooled_(pooled) {}
  DevMem(const DevMem &) = delete;
  DevMem &operator=(const DevMem &) = delete;
  ~DevMem() { release(); }
  mbc_status reserve(size_t b);
  // ... for memory that only makes a call faster (the parts of split
  // reductions): refused where it would take the room that the call's other
  // buffers may need, 4 GiB or a tenth of the device
  mbc_status reserve_spare(size_t b);
  void release();

 private:
  size_t size_ = 0;  // of the allocation
  bool pooled_ = true;
  int dev_ = -1;  // device of the pool, -1: cudaMalloc
};

// Free memory of the current device, the pool's idle memory included.
cudaError_t device_free_bytes(size_t *free_b, size_t *total_b);

// Four pinned host words for the flags a solver polls (NULL: none to be had).
int32_t *pinned_flags();
void pinned_flags_release(int32_t *p);

}  // namespace mbc
