// What a process does once on every CUDA device. A kernel's dynamic shared-memory
// limit is an attribute of the device that is current when it is set, so a flag per
// process leaves the second device's launches at 48 KB.
#pragma once

#include <stdint.h>

#include <atomic>

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#endif

namespace plum {

class OncePerDevice {
 public:
  // set() (0: done) until it has succeeded on `device`; its result, else 0. Threads
  // that come at once may each set: the same value.
  template <class Set>
  int run(int device, Set set) {
    const bool known = device >= 0 && device < 64;
    const uint64_t bit = known ? 1ull << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int rc = (int)set();
    if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

#if defined(__CUDACC__)
// Every call of the library selects its context's device first, through use_device, so
// what runs inside the call knows the device without asking (asking took 0.1 us, three
// to four times in a host move or a growth step).
inline thread_local int t_device = 0;

inline cudaError_t use_device(int device) {
  t_device = device;
  return cudaSetDevice(device);
}

// Allows `kernel` that much dynamic shared memory on the call's device. `once`: the
// kernel's own.
template <class Kernel>
inline cudaError_t allow_smem(OncePerDevice& once, Kernel* kernel, size_t bytes) {
  return (cudaError_t)once.run(t_device, [&] {
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  });
}

// SMs of the call's device.
inline int device_sms() {
  static std::atomic<int> known[64];
  const int dev = t_device;
  int sms = 0;
  if (dev >= 0 && dev < 64) sms = known[dev].load(std::memory_order_relaxed);
  if (sms > 0) return sms;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) return 152;
  if (dev >= 0 && dev < 64) known[dev].store(sms, std::memory_order_relaxed);
  return sms;
}
#endif

}  // namespace plum
