// What is set once a device and not once a process: a kernel's attributes belong to the device that is current when they are set.
#pragma once
#include <atomic>

class PerDevice {
 public:
  // Runs set() (0: done) unless it has succeeded for this device before; other threads may run it at the same time.
  template <typename Set> int once(int device, Set set) {
    const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int rc = set();
    if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<unsigned long long> done_{0};
};

#ifdef __CUDACC__
// Lets `kernel` be launched with `bytes` of dynamic shared memory on the current device.
template <typename F> static inline int qv_allow_smem(F kernel, size_t bytes, PerDevice& devices) {
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess) device = -1;
  return devices.once(device, [&] { return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
}
#endif
