// Set-up that holds for one device (a kernel's shared-memory opt-in), done once for each device that the
// process uses, on the current one; a set-up that failed is tried again.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace mvr {

class PerDevice {
public:
    template <class F>
    cudaError_t operator()(F f)
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 0 || dev >= kDevices) return f();
        if (done_[dev].load(std::memory_order_acquire)) return cudaSuccess;
        e = f();  // by several threads at once: the same values
        if (e == cudaSuccess) done_[dev].store(true, std::memory_order_release);
        return e;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<bool> done_[kDevices] = {};
};

}  // namespace mvr
