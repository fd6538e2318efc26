// Device memory of the synchronous entry points around the diffusion, kept between calls:
// they are called over and over with the same sizes, and mapping memory afresh costs 0.3 to
// 0.5 ms for the smallest buffer and tens of milliseconds for gigabytes.
//
//   * The field steps (combination, field histogram) take a buffer out of a list and put it back
//     once their work on the device is done; one that no kept buffer is large enough for is
//     allocated in the order of its stream.  Calls of several threads thus run side by side.  At
//     most kSpareKept bytes are kept per device.
//   * The sphere morphology, whose scratch goes with the volume, has one grow-only buffer per
//     device.  A call holds it, locked, until its work on the device is done.
//
// maxi_release_cached_memory() frees both; an allocation of the library that finds no room frees
// the list's buffers first (with_room).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <mutex>

namespace maxi {

// The keys of the field histogram's largest batch (512 MB) with its tables.
constexpr size_t kSpareKept = size_t(576) << 20;

// A buffer of the current device, for work on `st`.  Put back by give_back(), which waits for
// that work.
class SpareBuffer {
public:
    // A maxi_status; `what` names the caller in the error of a failed allocation.
    int take(size_t bytes, cudaStream_t st, const char *what);
    // Waits for the stream and puts the buffer back.
    cudaError_t give_back();
    uint8_t *data() const { return static_cast<uint8_t *>(p_); }
    SpareBuffer() = default;
    SpareBuffer(const SpareBuffer &) = delete;
    ~SpareBuffer() { give_back(); }

private:
    void *p_ = nullptr;
    size_t bytes_ = 0;
    int device_ = 0;
    cudaStream_t st_ = nullptr;
};

// Frees the current device's spare buffers.
void free_spare_buffers();

// alloc(), and once more without the spare buffers if there was no room.
template <typename F>
cudaError_t with_room(F &&alloc) {
    cudaError_t e = alloc();
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    free_spare_buffers();
    return alloc();
}

// Locks the current device's buffer, grows it to `bytes` and returns it (256-byte aligned) in
// *p; a maxi_status.
int acquire_scratch(size_t bytes, std::unique_lock<std::mutex> &lock, void **p, const char *what);
template <typename T>
int acquire_scratch(size_t bytes, std::unique_lock<std::mutex> &lock, T **p, const char *what) {
    void *v = nullptr;
    const int rc = acquire_scratch(bytes, lock, &v, what);
    *p = static_cast<T *>(v);
    return rc;
}

// Frees the morphology's buffers and the spare ones, of every device.
void release_scratch();

}  // namespace maxi
