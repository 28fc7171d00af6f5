// What a context has set for, or asked about, its kernels. A shared-memory limit
// or an occupancy belongs to one device, so it is kept in the context and not in
// the process: with contexts on two devices each device has its own.
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>

#include <unordered_map>

namespace lfx {

class KernelAttrs {
 public:
  // dynamic shared memory of a launch of kern: up to `bytes` from now on
  cudaError_t allow_smem(const void* kern, size_t bytes) {
    size_t& have = smem_[kern];
    if (have >= bytes) return cudaSuccess;
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) have = bytes;
    return e;
  }
  // a number that depends on the device and the kernel alone
  template <class Ask>
  int once(const void* kern, Ask ask) {
    const auto it = number_.find(kern);
    if (it != number_.end()) return it->second;
    return number_[kern] = ask();
  }

 private:
  std::unordered_map<const void*, size_t> smem_;
  std::unordered_map<const void*, int> number_;
};

}  // namespace lfx
