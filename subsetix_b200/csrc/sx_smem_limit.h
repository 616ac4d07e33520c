// Dynamic shared memory limit of a kernel.  The limit belongs to the device, so what has
// been raised is remembered per device, and under a lock: a thread with a smaller request
// must not lower what another thread has raised and is about to launch with.
#pragma once

#include <cuda_runtime_api.h>
#include <mutex>

class SxSmemLimit {
public:
    // Lets `kernel` (always the same) take `bytes` on the current device.
    cudaError_t raise(const void* kernel, int bytes)
    {
        int device = 0;
        cudaError_t err = cudaGetDevice(&device);
        if (err != cudaSuccess) return err;
        std::lock_guard<std::mutex> hold(lock_);
        const bool known = device >= 0 && device < DEVICES;  // the others are raised every time
        if (known && bytes <= raised_[device]) return cudaSuccess;
        err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (err == cudaSuccess && known) raised_[device] = bytes;
        return err;
    }

private:
    static constexpr int DEVICES = 64;
    std::mutex lock_;
    int raised_[DEVICES] = {};
};
