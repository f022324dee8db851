// plan_block.hpp - the device tables of one network in one allocation.
//
// A table set's plans are some fifty small tables.  One cudaMalloc and one
// blocking copy for each took as long as building them, so they are gathered
// on the host first and go over together.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

namespace dnnf90 {

class PlanBlock {
 public:
  // a copy of h; upload sets *d to its place on the device
  template <typename T>
  void add(T **d, const std::vector<T> &h) {
    const size_t at = (host_.size() + 255) / 256 * 256, bytes = h.size() * sizeof(T);
    host_.resize(at + std::max<size_t>(bytes, 16));
    if (bytes) std::memcpy(host_.data() + at, h.data(), bytes);
    puts_.push_back({(void **)d, at});
  }
  // one allocation, *base, for the caller to free
  cudaError_t upload(void **base) {
    *base = nullptr;
    cudaError_t e = cudaMalloc(base, std::max<size_t>(host_.size(), 16));
    if (e == cudaSuccess && !host_.empty())
      e = cudaMemcpy(*base, host_.data(), host_.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      if (*base) cudaFree(*base);
      *base = nullptr;
      return e;
    }
    for (const Put &p : puts_) *p.d = (char *)*base + p.at;
    return e;
  }

 private:
  struct Put {
    void **d;
    size_t at;
  };
  std::vector<unsigned char> host_;
  std::vector<Put> puts_;
};

}  // namespace dnnf90
