// arena.cuh -- device memory of a handle (network, learned correction).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace gpg {

// One device block for all the arrays of a handle: a handle is made and freed in
// one allocation each (a network's 23 took 0.8 ms to free).  add() the arrays,
// those to be zero-filled first, then allocate().
class Arena {
 public:
  template <typename T>
  void add(T *&p, size_t count) {
    slots_.push_back({reinterpret_cast<void **>(&p), size_});
    size_ += (count * sizeof(T) + 255) / 256 * 256;
  }
  void zeroed_to_here() { zero_ = size_; }
  cudaError_t allocate(void **block) {
    cudaError_t e = cudaMalloc(block, size_);
    if (e != cudaSuccess) {
      cudaGetLastError();  // reported by this call alone
      *block = nullptr;
      return e;
    }
    for (const Slot &s : slots_) *s.p = static_cast<char *>(*block) + s.at;
    return cudaMemset(*block, 0, zero_);
  }

 private:
  struct Slot {
    void **p;
    size_t at;
  };
  std::vector<Slot> slots_;
  size_t size_ = 0, zero_ = 0;
};

// whether the device runs the tensor-core kernels (compute capability 10.x); its
// number in *major and *minor (cudaGetDeviceProperties would take 3 ms)
inline cudaError_t compute_capability(int device, int *major, int *minor) {
  cudaError_t e = cudaDeviceGetAttribute(major, cudaDevAttrComputeCapabilityMajor, device);
  return e != cudaSuccess ? e : cudaDeviceGetAttribute(minor, cudaDevAttrComputeCapabilityMinor, device);
}

}  // namespace gpg
