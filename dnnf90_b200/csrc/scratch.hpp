// scratch.hpp - device scratch of one call, from a stream-ordered pool.
//
// A call that needs device memory only while it runs takes it from one pool
// per device, private to the library (cudaMallocAsync), instead of
// cudaMalloc / cudaFree, which wait for the whole device and map fresh pages
// on every call (0.75 ms for a 7 MB operand).  The pool is bounded: a call ends
// with what it holds beyond POOL_KEEP bytes given back, and scratch_trim
// (called when a network is freed) returns the rest.  The
// allocations are ordered on the caller's stream, so calls of several
// threads and streams share the pool safely.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace dnnf90 {

constexpr size_t POOL_KEEP = (size_t)512 << 20;

// device memory for work enqueued on st, released (in stream order) when the
// object goes out of scope; null after a failure
class DevScratch {
 public:
  DevScratch() = default;
  ~DevScratch() { release(); }
  DevScratch(const DevScratch &) = delete;
  DevScratch &operator=(const DevScratch &) = delete;
  cudaError_t take(size_t bytes, cudaStream_t st);
  void release();
  template <typename T>
  T *as() const { return (T *)p_; }

 private:
  void *p_ = nullptr;
  cudaStream_t st_ = nullptr;
};

// returns what the current device's pool holds unused
void scratch_trim();

// One page of pinned, device-mapped host memory of the process, through
// which calls read small results back without a staged copy.  Its users hold
// the library's lock from the write to the read.  Null if it cannot be had.
constexpr int PIN_DOUBLES = 64;
double *pinned_page();

// resident blocks of kernel k per SM, asked of the runtime once per (device,
// kernel, threads, shared memory): the query costs more than a launch
int blocks_per_sm(const void *k, int threads, size_t smem);

}  // namespace dnnf90
