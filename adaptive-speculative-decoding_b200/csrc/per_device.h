// What host code does once per device and process: kernel attributes, module loads, device limits.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

namespace asd {

int set_error(const char* fmt, ...);     // records the message, returns -1

// cudaFuncSetAttribute and module loads are per device.  `run` calls `set` on the current device until one call of it has returned 0;
// a thread that meets another's call on its device waits for its end, so that no first launch overtakes the attribute it needs.
// Devices do not wait for one another: a module load may wait for its device, whose kernels may wait for a rank on another one.
class PerDeviceOnce {
public:
    template <typename F>
    int run(F&& set) {
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = 1ull << (dev & 63);
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        std::lock_guard<std::mutex> hold(lock_[dev & 63]);
        if (done_.load(std::memory_order_relaxed) & bit) return 0;
        const int rc = set();
        if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
        return rc;
    }

private:
    std::atomic<unsigned long long> done_{0};
    std::mutex lock_[64];
};

// the statements (which may return -1, as ASD_CUDA does) once per device, in a function that returns -1 on failure
#define ASD_ONCE(once, ...)                  \
    do {                                     \
        if ((once).run([&]() -> int {        \
                __VA_ARGS__;                 \
                return 0;                    \
            }))                              \
            return -1;                       \
    } while (0)

struct DeviceLimits {
    int sms = 0, smem_optin = 0;         // multiprocessors; shared memory that a block may ask for
};

// of the current device: no thread sees one of them without the other
inline int device_limits(DeviceLimits* out) {
    static PerDeviceOnce once;
    static DeviceLimits known[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    DeviceLimits& d = known[dev & 63];
    if (e == cudaSuccess)
        once.run([&]() -> int {
            e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            return e == cudaSuccess ? 0 : -1;
        });
    if (e != cudaSuccess) return set_error("the device's limits cannot be read: %s", cudaGetErrorString(e));
    *out = d;
    return 0;
}

// lets launches of fn ask for all the shared memory that its static part leaves.  Once per device: set to each launch's own size, a
// smaller launch on another thread takes it back before a larger one has started.
template <typename F>
int allow_max_smem(F* fn) {
    DeviceLimits dev;
    cudaFuncAttributes fa;
    if (device_limits(&dev)) return -1;
    cudaError_t e = cudaFuncGetAttributes(&fa, fn);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.smem_optin - (int)fa.sharedSizeBytes);
    return e == cudaSuccess ? 0 : set_error("shared memory of a kernel: %s", cudaGetErrorString(e));
}

}  // namespace asd
