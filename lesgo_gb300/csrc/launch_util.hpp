// Errors and launch helpers shared by the translation units.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>

#include "lesgo_gpu.h"

namespace lesgo {

struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define CK(x)                                                                                 \
  do {                                                                                        \
    cudaError_t e_ = (x);                                                                     \
    if (e_ != cudaSuccess)                                                                    \
      throw Error(e_ == cudaErrorMemoryAllocation ? LESGO_ERR_NOMEM : LESGO_ERR_CUDA,         \
                  std::string(#x) + ": " + cudaGetErrorString(e_));                           \
  } while (0)

// A kernel's dynamic shared-memory limit (cudaFuncAttributeMaxDynamicSharedMemorySize)
// belongs to the function, not to a launch, and a replayed CUDA graph
// launches its kernel nodes against the value current at replay.  Handles
// of different grids share the kernel instances, so a handle that set a
// smaller limit than another handle's captured node needs would break that
// node's replay.  The limit is therefore only ever raised, per device,
// under a lock (handles may live on several host threads).
inline void raise_smem_limit(const void* kern, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> limit;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  size_t& cur = limit[{dev, kern}];
  if (bytes <= cur) return;
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  cur = bytes;
}

}  // namespace lesgo
