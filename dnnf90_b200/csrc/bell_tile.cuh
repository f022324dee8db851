// bell_tile.cuh - what the register-tiled Bell kernels of both precisions
// share (bell_tile.cu, bell_tile64.cu): the index maps of a tile, staging
// helpers and launch helpers.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "engine.hpp"
#include "scratch.hpp"

namespace dnnf90 {
namespace {

// ------------------------------------------------------------ tile algebra
// entries of a tile of side L in td dimensions, and the graded index maps
__host__ __device__ constexpr int tsize(int td, int L) { return td == 2 ? L * (L + 1) / 2 : L; }
__host__ __device__ constexpr int tdeg(int td, int e) {
  int s = 0;
  if (td == 1) return e;
  while ((s + 1) * (s + 2) / 2 <= e) ++s;
  return s;
}
__host__ __device__ constexpr int tsecond(int td, int e) {
  return td == 1 ? 0 : e - tdeg(2, e) * (tdeg(2, e) + 1) / 2;
}
__host__ __device__ constexpr int tfirst(int td, int e) {
  return td == 1 ? e : tdeg(2, e) - tsecond(2, e);
}
__host__ __device__ constexpr int tindex(int td, int a1, int a2) {
  return td == 1 ? a1 : (a1 + a2) * (a1 + a2 + 1) / 2 + a2;
}
// index of the sum of entries e and c
__host__ __device__ constexpr int tadd(int td, int e, int c) {
  return tindex(td, tfirst(td, e) + tfirst(td, c), tsecond(td, e) + tsecond(td, c));
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void cp16(void *dst, const void *src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
               "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// copy of n 32-bit words of a table into shared memory
__device__ __forceinline__ void copy_words(void *dst, const void *src, int nwords) {
  for (int i = threadIdx.x; i < nwords; i += blockDim.x)
    ((uint32_t *)dst)[i] = __ldg((const uint32_t *)src + i);
}

// items [it0, it1) of this block: a contiguous share of npts * gy items,
// item = point + npts * (32-neuron tile)
__device__ __forceinline__ void block_items(long nitem, long &it0, long &it1) {
  it0 = (long)blockIdx.x * nitem / gridDim.x;
  it1 = (long)(blockIdx.x + 1) * nitem / gridDim.x;
}

int grid_for(const void *k, int threads, size_t smem, long items) {
  const long g = (long)grid_sms() * blocks_per_sm(k, threads, smem);
  return (int)std::max(1L, std::min(g, items));
}

#define CKT(x)                                                         \
  do {                                                                 \
    cudaError_t e_ = (x);                                              \
    if (e_ != cudaSuccess) {                                           \
      set_error(std::string("bell_tile: ") + cudaGetErrorString(e_));  \
      return RC_DEVICE;                                                \
    }                                                                  \
  } while (0)

}  // namespace
}  // namespace dnnf90
