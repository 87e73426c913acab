// Work done once for each CUDA device a process uses (a kernel's shared-memory
// limit, a memory pool): such state belongs to the device that is current when
// it is set up, not to the process.
#pragma once

#include <cuda_runtime_api.h>

#include <mutex>

namespace rtgb {

constexpr int kMaxDevices = 64;

class OncePerDevice {
public:
    // Runs make(device) for the current device unless it has succeeded there
    // before; safe to call from several threads.
    template <typename Make>
    cudaError_t run(Make make) {
        int device = 0;
        if (const cudaError_t e = cudaGetDevice(&device); e != cudaSuccess) return e;
        if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> lock(mutex_);
        if (done_[device]) return cudaSuccess;
        const cudaError_t e = make(device);
        done_[device] = e == cudaSuccess;
        return e;
    }

private:
    std::mutex mutex_;
    bool done_[kMaxDevices] = {};
};

}  // namespace rtgb
