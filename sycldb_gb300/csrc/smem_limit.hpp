// A kernel's dynamic shared memory above 48 KB has to be allowed per device.
// One SmemLimit (a static beside the launch) remembers the devices on which
// its kernels have been allowed theirs; a refusal is not remembered.  Safe with
// several threads and devices.
#pragma once

#include <atomic>
#include <cstdint>

#include <cuda_runtime_api.h>

namespace sdb {

class SmemLimit {
public:
    // Lets the kernels use up to `bytes` (the same on every call of one object)
    // on the calling thread's current device.  False when the device refuses.
    template <class... Kernel>
    bool allow(int bytes, Kernel... kernels)
    {
        int dev = -1;
        bool ok = cudaGetDevice(&dev) == cudaSuccess && dev >= 0;
        const uint64_t bit = ok && dev < 64 ? 1ull << dev : 0;  // devices past 63: asked each time
        if (allowed_.load(std::memory_order_acquire) & bit) return true;
        ((ok = ok && cudaFuncSetAttribute(reinterpret_cast<const void *>(kernels),
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess),
         ...);
        if (ok) allowed_.fetch_or(bit, std::memory_order_release);
        else cudaGetLastError();
        return ok;
    }

private:
    std::atomic<uint64_t> allowed_{0};  // bit d: device d
};

}  // namespace sdb
