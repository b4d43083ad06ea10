// What launchers ask of the device. The dynamic shared memory above 48 KB that a kernel may be launched with is set per device. A launcher keeps one of these per
// kernel: the limit is set at the kernel's first launch on each device of the process and remembered by device.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>

namespace gi {

class SharedLimit {
  public:
    // Lets `kernel` have `bytes` on the current device; the runtime's answer where it refuses. For several threads at once.
    cudaError_t allow(const void* kernel, int bytes) {
        int device = 0;
        cudaError_t e = cudaGetDevice(&device);
        const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;      // (further devices: set at every launch)
        if (e == cudaSuccess && !(set_.load(std::memory_order_relaxed) & bit)) {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (e == cudaSuccess) set_.fetch_or(bit, std::memory_order_relaxed);
        }
        if (e != cudaSuccess) cudaGetLastError();      // the caller reports it: it must not show up at the next launch
        return e;
    }

  private:
    std::atomic<unsigned long long> set_{0};
};

// Multiprocessors of the current device.
inline int sm_count() {
    int sms = 0, device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms > 0 ? sms : 1;
}

}  // namespace gi
