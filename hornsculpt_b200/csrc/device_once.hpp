// Once-per-device initialisation. __constant__ tables live separately on each
// device, so an upload done on device 0 leaves device 1's copy all zero: the
// flag must be per device ordinal, and the check-and-set must be serialised
// because sessions on several host threads may upload at the same time.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <stdexcept>
#include <string>
#include <utility>

namespace hsb {

inline int currentDevice() {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("CUDA current device: ") + cudaGetErrorString(e));
    if (device < 0 || device >= 256)
        throw std::runtime_error("CUDA device ordinal out of range.");
    return device;
}

class PerDeviceOnce {
  public:
    // Runs `init` unless it has already completed on the current device. A
    // throwing `init` leaves the device unmarked, so the next call retries.
    template <class F> void run(F &&init) {
        const int device = currentDevice();
        std::lock_guard<std::mutex> lock(mutex_);
        if (done_[device])
            return;
        init();
        done_[device] = true;
    }

  private:
    static constexpr int kMaxDevices = 256;
    std::mutex mutex_;
    bool done_[kMaxDevices] = {};
};

// A per-device value computed once by `make` (a device attribute, a schedulable
// cluster size); a thrown `make` leaves the device unset.
template <class V> class PerDeviceValue {
  public:
    template <class F> V get(F &&make) {
        const int device = currentDevice();
        std::lock_guard<std::mutex> lock(mutex_);
        if (!set_[device]) {
            value_[device] = make();
            set_[device] = true;
        }
        return value_[device];
    }

  private:
    std::mutex mutex_;
    bool set_[256] = {};
    V value_[256] = {};
};

// Lets `kernel` take the dynamic shared memory the device offers beyond the
// default 48 KB. The limit belongs to the kernel function, so every session,
// thread and launch size shares it: it is raised once per device, to all the
// device can give, and never set to the need of one launch, which another
// launch may exceed.
inline void allowSharedMemory(const void *kernel) {
    static std::mutex mutex;
    static std::set<std::pair<int, const void *>> allowed;
    const int device = currentDevice();
    std::lock_guard<std::mutex> lock(mutex);
    if (allowed.count({device, kernel}))
        return;
    cudaFuncAttributes own{};
    int most = 0;
    cudaError_t e = cudaFuncGetAttributes(&own, kernel);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - int(own.sharedSizeBytes));
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("CUDA shared memory limit: ") + cudaGetErrorString(e));
    allowed.emplace(device, kernel);
}
template <class... P> void allowSharedMemory(void (*kernel)(P...)) {
    allowSharedMemory(reinterpret_cast<const void *>(kernel));
}

// Multiprocessors of the current device.
inline int smCount() {
    static PerDeviceValue<int> count;
    return count.get([]() {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, currentDevice()) != cudaSuccess || n <= 0)
            n = 148;
        return n;
    });
}

}  // namespace hsb
