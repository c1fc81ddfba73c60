// launch_limits.h -- how many CTAs of a kernel fit an SM, per device.
//
// A kernel's limit of dynamic shared memory belongs to a device, not to the
// process: it is raised once on every device that launches the kernel, to the
// most that device allows, so that a launch on one thread never sees another
// thread's smaller limit.
#pragma once

#include <cuda_runtime_api.h>

#include <map>
#include <mutex>
#include <string>

#include "aed_internal.h"

namespace aed {

// Of one kernel (a static object beside its launch).
class KernelLimits {
 public:
  // CTAs of `threads` threads with `dyn` bytes of dynamic shared memory that an
  // SM of the current device holds; 0: none, negative: an error code.
  int ctas_per_sm(const void* kern, int threads, size_t dyn) {
    std::lock_guard<std::mutex> lk(mu_);
    Device* d = nullptr;
    if (const int rc = device(kern, &d)) return rc;
    if (dyn > d->most) return 0;
    const auto key = std::make_pair(threads, dyn);
    auto it = d->ctas.find(key);
    if (it == d->ctas.end()) {
      int n = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(&n, kern, threads, dyn, 0) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
      }
      it = d->ctas.emplace(key, n < 0 ? 0 : n).first;
    }
    return it->second;
  }
  // The most dynamic shared memory a CTA of the kernel may take on the current device.
  int most_dynamic(const void* kern, size_t* most) {
    std::lock_guard<std::mutex> lk(mu_);
    Device* d = nullptr;
    const int rc = device(kern, &d);
    *most = rc ? 0 : d->most;
    return rc;
  }

 private:
  struct Device {
    size_t most = 0;
    std::map<std::pair<int, size_t>, int> ctas;  // by (threads, dynamic shared memory)
  };
  int device(const void* kern, Device** out) {
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    auto it = devices_.find(dev);
    if (e == cudaSuccess && it == devices_.end()) {
      Device d;
      cudaFuncAttributes fa{};
      e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kern);
      if (e == cudaSuccess && optin > (int)fa.sharedSizeBytes) {
        d.most = (size_t)optin - fa.sharedSizeBytes;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d.most);
      }
      if (e == cudaSuccess) it = devices_.emplace(dev, d).first;
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(AED_ERR_CUDA, std::string("kernel shared memory limit: ") + cudaGetErrorString(e));
    }
    *out = &it->second;
    return AED_OK;
  }
  std::mutex mu_;
  std::map<int, Device> devices_;
};

}  // namespace aed
