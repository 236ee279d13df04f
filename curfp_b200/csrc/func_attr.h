// func_attr.h — settings a kernel needs once on every device it runs on
// (cudaFuncSetAttribute applies to the current device alone).
#pragma once
#include <atomic>
#include <cstdint>

namespace rfp {

// Runs set() unless it has succeeded for the device before.  A failure is not
// remembered: the next call tries again.  Devices past 63 set it every time.
class OncePerDevice {
 public:
  template <class F>
  bool operator()(int device, F&& set) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return true;
    if (!set()) return false;
    done_.fetch_or(bit, std::memory_order_release);
    return true;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

#ifdef __CUDACC__
// Opts a kernel into `bytes` of dynamic shared memory on the handle's device.
template <typename K>
inline bool smem_attr(OncePerDevice& once, int device, K kernel, int bytes) {
  return once(device, [&] {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
        cudaSuccess)
      return true;
    cudaGetLastError();
    return false;
  });
}
#endif

}  // namespace rfp
