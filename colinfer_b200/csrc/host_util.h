// host_util.h -- what the launching side of several kernels shares.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <mutex>
#include <unordered_map>

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

// What an occupancy query answered, by a key of the caller's that holds everything the answer depends on: up to three queries a
// call, 0.3 us each, are saved.  Bounded: beyond MOST answers it starts over.
class Remembered {
public:
    template <class F> int operator()(uint64_t key, F query) {   // an answer below 0 (an error) is not kept
        std::lock_guard<std::mutex> lock(guard_);
        const auto it = known_.find(key);
        if (it != known_.end()) return it->second;
        const int n = query();
        if (n < 0) return n;
        if (known_.size() >= MOST) known_.clear();
        known_.emplace(key, n);
        return n;
    }

private:
    static constexpr size_t MOST = 4096;
    std::mutex guard_;
    std::unordered_map<uint64_t, int> known_;
};
