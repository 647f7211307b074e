// A set-up that belongs to a device (kernel attributes): run once on each
// device that comes to need it, with that device current.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <set>

namespace vs {

class OncePerDevice {
 public:
  // f() unless it has succeeded on this device; its error if it fails, and the
  // next call tries again
  template <class F>
  cudaError_t run(int device, F&& f) {
    std::lock_guard<std::mutex> lock(mu_);
    if (done_.count(device)) return cudaSuccess;
    const cudaError_t e = f();
    if (e == cudaSuccess) done_.insert(device);
    return e;
  }

 private:
  std::mutex mu_;
  std::set<int> done_;
};

}  // namespace vs
