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
#include <vector>

#include "aed_internal.h"

namespace aed {

// The device that a DeviceGuard of this thread has made current (-1: none).
inline thread_local int t_guarded_device = -1;

// Of one kernel (a static object beside its launch; a launch-bound product asks
// on every call, so the few entries are searched in turn).
class KernelLimits {
 public:
  // CTAs of `threads` threads with `dyn` bytes of dynamic shared memory that an
  // SM of the current device holds; 0: none, negative: an error code.
  int ctas_per_sm(const void* kern, int threads, size_t dyn) {
    std::lock_guard<std::mutex> lk(mu_);
    const int dev = current();
    for (const Shape& s : shapes_)
      if (s.dev == dev && s.threads == threads && s.dyn == dyn) return s.ctas;
    size_t most = 0;
    if (const int rc = raise(kern, dev, &most)) return rc;
    int n = 0;
    if (dyn <= most &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(&n, kern, threads, dyn, 0) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    shapes_.push_back({dev, threads, dyn, n < 0 ? 0 : n});
    return shapes_.back().ctas;
  }
  // The most dynamic shared memory a CTA of the kernel may take on the current device.
  int most_dynamic(const void* kern, size_t* most) {
    std::lock_guard<std::mutex> lk(mu_);
    return raise(kern, current(), most);
  }

 private:
  struct Shape {
    int dev, threads;
    size_t dyn;
    int ctas;
  };
  static int current() {
    int dev = t_guarded_device;
    if (dev < 0) cudaGetDevice(&dev);
    return dev;
  }
  int raise(const void* kern, int dev, size_t* most) {
    *most = 0;
    auto it = most_.find(dev);
    if (it == most_.end()) {
      int optin = 0;
      size_t bytes = 0;
      cudaFuncAttributes fa{};
      cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kern);
      if (e == cudaSuccess && optin > (int)fa.sharedSizeBytes) {
        bytes = (size_t)optin - fa.sharedSizeBytes;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      }
      if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(AED_ERR_CUDA, std::string("kernel shared memory limit: ") + cudaGetErrorString(e));
      }
      it = most_.emplace(dev, bytes).first;
    }
    *most = it->second;
    return AED_OK;
  }
  std::mutex mu_;
  std::vector<Shape> shapes_;
  std::map<int, size_t> most_;  // by device: the raised limit
};

}  // namespace aed
