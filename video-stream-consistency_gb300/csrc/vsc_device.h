// Per-device state of the launch code: function attributes such as the opt-in to
// large dynamic shared memory belong to a device (its context), not to the process.
#pragma once

#include <cuda_runtime_api.h>

#include <mutex>

namespace vsc {

constexpr int kMaxDevices = 64;

// What prepare(&value) made on the current device, made at the first use on each
// device.  Only a success is kept: after a failure the next call tries again.
template <class T>
class PerDevice {
public:
    template <class F>
    cudaError_t get(F&& prepare, T* out)
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess)
            return e;
        if (dev < 0 || dev >= kMaxDevices)
            return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> lock(mu_);
        if (!ready_[dev]) {
            if ((e = prepare(&value_[dev])) != cudaSuccess)
                return e;
            ready_[dev] = true;
        }
        *out = value_[dev];
        return cudaSuccess;
    }

private:
    std::mutex mu_;
    bool ready_[kMaxDevices] = {};
    T value_[kMaxDevices] = {};
};

}  // namespace vsc
