// What the library asks of a device or sets on it once: a kernel's attributes
// (cudaFuncSetAttribute holds for the current device only), the number of its
// SMs, how many CTAs it holds at once.
#pragma once

#include <cuda_runtime.h>

#include <mutex>

namespace silt {

inline int current_device() {
    int dev = 0;
    cudaGetDevice(&dev);
    return dev;
}

template <class T>
class PerDevice {
    static constexpr int KEPT = 64;  // device ordinals with a value of their own; beyond, it is made on each call
    std::once_flag once_[KEPT];
    T value_[KEPT] = {};

  public:
    // The value of device `dev`, which is current: make(dev), called on the first use there.
    T of(int dev, T (*make)(int)) {
        if (dev < 0 || dev >= KEPT) return make(dev);
        std::call_once(once_[dev], [this, dev, make] { value_[dev] = make(dev); });
        return value_[dev];
    }
};

inline int query_sm_count(int dev) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) return n;
    cudaGetLastError();
    return 148;
}

// Dynamic shared memory for the kernel on the current device. A refusal is the
// result alone, not the thread's last error.
template <class... KArgs>
cudaError_t allow_smem(void (*kernel)(KArgs...), size_t bytes) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace silt
