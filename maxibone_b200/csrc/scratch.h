// Device scratch kept between calls: one grow-only buffer per device, for the synchronous
// entry points around the diffusion (morphology, field combination, field histograms).
// They are called over and over with the same sizes, and mapping memory afresh costs
// 0.3 to 0.5 ms for the smallest buffer and tens of milliseconds for gigabytes.  A call
// holds its device's buffer, locked, until its work on the device is done.
// maxi_release_cached_memory() frees it.
#pragma once

#include <stddef.h>

#include <mutex>

namespace maxi {

// Locks the current device's scratch, grows it to `bytes` and returns it (256-byte aligned) in
// *p; a maxi_status.  `what` names the caller in the error of a failed allocation.
int acquire_scratch(size_t bytes, std::unique_lock<std::mutex> &lock, void **p, const char *what);
template <typename T>
int acquire_scratch(size_t bytes, std::unique_lock<std::mutex> &lock, T **p, const char *what) {
    void *v = nullptr;
    const int rc = acquire_scratch(bytes, lock, &v, what);
    *p = static_cast<T *>(v);
    return rc;
}

void release_scratch();

}  // namespace maxi
