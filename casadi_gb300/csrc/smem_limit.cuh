// Dynamic shared memory limits of kernels, raised once per kernel and device.
//
// A kernel's limit (cudaFuncAttributeMaxDynamicSharedMemorySize) belongs to the function on a
// device, not to a launch: a launch that asks for more than the limit standing at that moment fails.
// Written per launch, one thread's smaller size could land between another thread's larger one and
// its launch. So each is raised to the most the device allows, when the kernel is first used there,
// and never written again.
#pragma once
#include <mutex>
#include <unordered_map>

namespace cgb {

class SmemLimits {
 public:
  // raise(): 0 on success. Called once per kernel and device (again after a failure).
  template <class F>
  int once(const void* kernel, int device, F raise) {
    std::lock_guard<std::mutex> lk(mtx_);
    unsigned long long& devices = raised_[kernel];
    const unsigned long long bit =
        device >= 0 && device < 64 ? 1ull << device : 0;  // others: each time, to the same value
    if (devices & bit) return 0;
    const int e = raise();
    if (e == 0) devices |= bit;
    return e;
  }

 private:
  std::mutex mtx_;
  std::unordered_map<const void*, unsigned long long> raised_;  // kernel -> devices
};

}  // namespace cgb
