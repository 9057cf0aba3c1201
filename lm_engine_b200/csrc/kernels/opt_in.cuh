// Launch attributes of kernels (dynamic shared memory beyond 48 KB, clusters of 16).  They belong to a device's copy of
// the kernel, so they are set once on every device that launches it and not once per process.
#pragma once
#include <atomic>

namespace lme {

// One attribute with one value per kernel: threads that come here together set the same value.
template <auto Kern>
inline bool opt_in(cudaFuncAttribute attr, int value) {
    static std::atomic<unsigned long long> done{0};     // a bit per device
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return false;
    const unsigned long long bit = device < 64 ? 1ull << device : 0ull;
    if (done.load(std::memory_order_acquire) & bit) return true;
    if (cudaFuncSetAttribute(Kern, attr, value) != cudaSuccess) return false;
    done.fetch_or(bit, std::memory_order_release);
    return true;
}

}  // namespace lme
