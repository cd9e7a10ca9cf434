// Kernels that use more than 48 KB of dynamic shared memory have to be allowed it, on every device that runs them.
#pragma once
#include <mutex>

// What a kernel has been allowed so far, by device.  Safe with several threads: the limit is only ever raised, under a lock.
class SmemAllowance {
 public:
  // set(bytes) sets the kernel's limit on the current device, which is `device`, and returns an error code (0: none).  It is
  // not called again for what has been allowed before (so not while a stream that has seen the launch before is captured).
  template <typename Set>
  int raise(int device, int bytes, Set set) {
    if (bytes <= 48 * 1024) return 0;
    std::lock_guard<std::mutex> hold(lock_);
    const bool kept = device >= 0 && device < DEVICES;
    if (kept && bytes <= allowed_[device]) return 0;
    const int err = set(bytes);
    if (err == 0 && kept) allowed_[device] = bytes;
    return err;
  }

 private:
  static constexpr int DEVICES = 64;
  std::mutex lock_;
  int allowed_[DEVICES] = {};
};

#ifdef __CUDACC__
template <typename Kernel>
inline cudaError_t allow_smem(Kernel kernel, size_t bytes, SmemAllowance& allowance) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  return (cudaError_t)allowance.raise(device, (int)bytes, [&](int most) {
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  });
}
#endif
