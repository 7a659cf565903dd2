// What a launch asks the runtime about the current device, asked once per device: a Linear of a short prompt is 3 us of GPU time, and its queries took as long on the host.
// And whether kernels may be launched programmatically, for both libraries.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>

namespace device_info {

constexpr int MAX_DEVICES = 64;

inline int current() {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}
// SMs of the current device, 0: unknown
inline int sm_count() {
    static std::atomic<int> known[MAX_DEVICES];
    const int dev = current();
    if (dev >= 0 && dev < MAX_DEVICES && known[dev].load(std::memory_order_relaxed) > 0) return known[dev].load(std::memory_order_relaxed);
    int sms = 0;
    if (dev < 0 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (dev < MAX_DEVICES) known[dev].store(sms, std::memory_order_relaxed);
    return sms;
}
// Allows launches of Kernel with up to `bytes` of dynamic shared memory on the current device; `bytes` is the same in every call of an instantiation.
template <auto Kernel>
inline cudaError_t allow_shared(int bytes) {
    static std::atomic<uint64_t> done{0};
    const int dev = current();
    const uint64_t bit = dev >= 0 && dev < MAX_DEVICES ? (uint64_t)1 << dev : 0;
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
    return e;
}

// MB200_PDL=0: no kernel begins before its predecessor in the stream has ended
inline bool pdl_enabled() {
    static const bool on = [] {
        const char* e = getenv("MB200_PDL");
        return !(e != nullptr && e[0] == '0');
    }();
    return on;
}

}  // namespace device_info
