// Device memory kept between calls (scratch.h).
#include "scratch.h"

#include <algorithm>
#include <map>
#include <vector>

#include "host_util.h"

namespace maxi {
namespace {

struct Scratch {
    std::mutex mu;
    void *buf = nullptr;
    size_t bytes = 0;
    void drop() {
        if (!buf) return;
        cudaDeviceSynchronize();  // earlier calls' work on the buffer
        cudaFree(buf);
        buf = nullptr;
        bytes = 0;
    }
};
std::mutex g_scratch_mu;
std::map<int, Scratch *> g_scratch;

// The least size of a spare buffer, which a call's tables fit.
constexpr size_t kSmallSpare = size_t(1) << 20;

struct Spare {
    void *p;
    size_t bytes;
};
struct Spares {
    std::vector<Spare> idle;  // by size
    size_t kept = 0;
    Spare remove(size_t i) {
        const Spare s = idle[i];
        idle.erase(idle.begin() + i);
        kept -= s.bytes;
        return s;
    }
};
std::mutex g_spares_mu;
std::map<int, Spares> g_spares;

}  // namespace

int SpareBuffer::take(size_t bytes, cudaStream_t st, const char *what) {
    cudaError_t e = cudaGetDevice(&device_);
    if (e != cudaSuccess) return set_cuda_error(e, "cudaGetDevice");
    // These calls wait for their stream and cannot be captured.  Refused here, as memory allocated
    // in a capture belongs to its graph and must not come into the list.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(st, &capture);
    if (e == cudaSuccess && capture != cudaStreamCaptureStatusNone) e = cudaErrorStreamCaptureUnsupported;
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_cuda_error(e, what);
    }
    bytes = std::max(bytes, kSmallSpare);
    Spare too_small{};
    {
        std::lock_guard<std::mutex> lk(g_spares_mu);
        Spares &s = g_spares[device_];
        size_t i = 0;
        while (i < s.idle.size() && s.idle[i].bytes < bytes) i++;
        // (a small request leaves the large buffers to those that need them)
        if (i < s.idle.size() && (bytes > kSmallSpare || s.idle[i].bytes == kSmallSpare)) {
            const Spare fits = s.remove(i);
            p_ = fits.p, bytes_ = fits.bytes, st_ = st;
            return MAXI_OK;
        }
        if (i > 0 && s.idle[i - 1].bytes > kSmallSpare) too_small = s.remove(i - 1);  // the new one takes its place
    }
    if (too_small.p) cudaFreeAsync(too_small.p, st);
    void *p = nullptr;
    if (with_room([&] { return cudaMallocAsync(&p, bytes, st); }) != cudaSuccess) {
        cudaGetLastError();
        return set_error(MAXI_ERR_OUT_OF_MEMORY, "could not allocate %zu bytes of %s scratch", bytes, what);
    }
    p_ = p, bytes_ = bytes, st_ = st;
    return MAXI_OK;
}

cudaError_t SpareBuffer::give_back() {
    if (!p_) return cudaSuccess;
    const cudaError_t e = cudaStreamSynchronize(st_);
    try {
        std::lock_guard<std::mutex> lk(g_spares_mu);
        Spares &s = g_spares[device_];
        if (s.kept + bytes_ <= kSpareKept) {
            size_t i = 0;
            while (i < s.idle.size() && s.idle[i].bytes < bytes_) i++;
            s.idle.insert(s.idle.begin() + i, Spare{p_, bytes_});
            s.kept += bytes_;
            p_ = nullptr;
        }
    } catch (...) {
        // no room in the list: the buffer is freed
    }
    if (p_) cudaFreeAsync(p_, st_);
    p_ = nullptr;
    return e;
}

void free_spare_buffers() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    std::vector<Spare> idle;
    {
        std::lock_guard<std::mutex> lk(g_spares_mu);
        Spares &s = g_spares[dev];
        idle.swap(s.idle);
        s.kept = 0;
    }
    for (const Spare &s : idle) cudaFree(s.p);
}

int acquire_scratch(size_t bytes, std::unique_lock<std::mutex> &lock, void **p, const char *what) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_cuda_error(e, "cudaGetDevice");
    Scratch *s;
    {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        Scratch *&slot = g_scratch[dev];
        if (!slot) slot = new Scratch();
        s = slot;
    }
    lock = std::unique_lock<std::mutex>(s->mu);
    if (s->bytes < bytes) {
        s->drop();
        if (with_room([&] { return cudaMalloc(&s->buf, bytes); }) != cudaSuccess) {
            cudaGetLastError();
            s->buf = nullptr;
            return set_error(MAXI_ERR_OUT_OF_MEMORY, "could not allocate %zu bytes of %s scratch", bytes, what);
        }
        s->bytes = bytes;
    }
    *p = s->buf;
    return MAXI_OK;
}

void release_scratch() {
    {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        for (auto &kv : g_scratch) {
            std::lock_guard<std::mutex> lk2(kv.second->mu);
            kv.second->drop();
        }
    }
    std::map<int, Spares> all;
    {
        std::lock_guard<std::mutex> lk(g_spares_mu);
        all.swap(g_spares);
    }
    for (auto &kv : all)
        for (const Spare &s : kv.second.idle) cudaFree(s.p);
}

}  // namespace maxi
