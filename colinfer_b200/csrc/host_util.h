// host_util.h -- what the launching side of several kernels shares.
#pragma once
#include <cuda_runtime.h>
#include <mutex>

constexpr int kMaxDevices = 64;

// Lets a kernel be launched with up to `bytes` of dynamic shared memory on the current device.  The limit belongs to the kernel,
// not to a launch: set to what each call needs, one thread could lower it between another thread's setting and its launch.  So
// it is set once per device, to the most that any call asks for.
class SmemOptIn {
public:
    cudaError_t operator()(const void* kernel, int bytes) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> lock(guard_);
        if (done_[dev]) return cudaSuccess;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        done_[dev] = e == cudaSuccess;
        return e;
    }

private:
    std::mutex guard_;
    bool done_[kMaxDevices] = {};
};
