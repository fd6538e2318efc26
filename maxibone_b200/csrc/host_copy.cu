// Staged host <-> device copies for pageable caller buffers (host_copy.h).
#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace maxi {

namespace {

constexpr size_t kChunk = size_t(1) << 20;  // bytes per staging buffer (2 MB: 10.5 against 9.4 ms below)
constexpr int kMaxWorkers = 8;             // host threads of a copy, two buffers each
constexpr int kMaxKept = 2 * kMaxWorkers;  // buffers kept between calls (16 MB)

// Pinned staging buffers kept between calls: allocating them cost more than the copies they
// serve (64 MB: 30 to 60 ms to page-lock and 11 to release; a 360 x 400 x 416 call of 10
// repetitions took 53 ms with them and takes 9.4 without, 3 of them kernels).  A copy takes buffers out of the list and puts them back;
// what a concurrent copy finds missing it allocates, and beyond kMaxKept frees again.
std::mutex g_staging_mu;
std::vector<void *> g_staging_free;

cudaError_t take_buffers(int n, std::vector<void *> &out) {
    {
        std::lock_guard<std::mutex> lk(g_staging_mu);
        g_staging_free.reserve(kMaxKept);  // so that putting buffers back cannot fail
        out.reserve(n);
        while ((int) out.size() < n && !g_staging_free.empty()) {
            out.push_back(g_staging_free.back());
            g_staging_free.pop_back();
        }
    }
    while ((int) out.size() < n) {
        void *p = nullptr;
        const cudaError_t e = cudaHostAlloc(&p, kChunk, cudaHostAllocPortable);
        if (e != cudaSuccess) return e;
        out.push_back(p);
    }
    return cudaSuccess;
}

void return_buffers(std::vector<void *> &bufs) {
    for (void *p : bufs) {
        {
            std::lock_guard<std::mutex> lk(g_staging_mu);
            if ((int) g_staging_free.size() < kMaxKept) {
                g_staging_free.push_back(p);
                p = nullptr;
            }
        }
        if (p) cudaFreeHost(p);
    }
    bufs.clear();
}

// Runs worker(w, first buffer, second buffer) for w < n on n host threads (the calling
// thread among them, and in place of threads that cannot be started); the first error.
template <typename F>
cudaError_t run_workers(size_t chunks, F &&worker) try {
    const unsigned hc = std::thread::hardware_concurrency();
    const int n = (int) std::min<size_t>(chunks, std::max(1u, std::min<unsigned>(kMaxWorkers, hc ? hc : 1u)));
    std::vector<void *> bufs;
    cudaError_t e = take_buffers(2 * n, bufs);
    int dev = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return_buffers(bufs);
        return e;
    }
    std::atomic<int> first{(int) cudaSuccess};
    auto run = [&](int w) {
        cudaError_t we = cudaSetDevice(dev);
        if (we == cudaSuccess) we = worker(w, n, bufs[2 * w], bufs[2 * w + 1]);
        int none = (int) cudaSuccess;
        if (we != cudaSuccess) first.compare_exchange_strong(none, (int) we);
    };
    std::vector<std::thread> pool;
    int started = 1;
    try {
        pool.reserve(n);
        for (; started < n; started++) pool.emplace_back(run, started);
    } catch (...) {
        // no more threads: this one takes the rest
    }
    run(0);
    for (int w = started; w < n; w++) run(w);
    for (auto &t : pool) t.join();
    return_buffers(bufs);
    return (cudaError_t) first.load();
} catch (...) {
    return cudaErrorMemoryAllocation;  // no room for the lists, before any thread or copy
}

// The two buffers of a worker with an event each ("the copy from or to it is done"); waits
// for both before it goes.
struct Pair {
    void *buf[2];
    cudaEvent_t ev[2] = {nullptr, nullptr};
    Pair(void *a, void *b) : buf{a, b} {}
    cudaError_t init() {
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < 2 && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
        return e;
    }
    ~Pair() {
        for (cudaEvent_t e : ev)
            if (e) {
                cudaEventSynchronize(e);
                cudaEventDestroy(e);
            }
    }
};

}  // namespace

bool host_pageable(const void *p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Worker w of n takes chunks w, w + n, ...: while one of its chunks crosses, it fills (or
// empties) its other buffer.
cudaError_t copy_to_device_staged(void *d_dst, const void *h_src, size_t n, cudaStream_t st) {
    const size_t chunks = (n + kChunk - 1) / kChunk;
    cudaError_t e = run_workers(chunks, [&](int w, int workers, void *a, void *b) {
        Pair s(a, b);
        cudaError_t e = s.init();
        int k = 0;
        for (size_t c = w; e == cudaSuccess && c < chunks; c += workers, k ^= 1) {
            const size_t off = c * kChunk, len = std::min(kChunk, n - off);
            if ((e = cudaEventSynchronize(s.ev[k])) != cudaSuccess) break;  // the buffer's previous chunk has crossed
            std::memcpy(s.buf[k], static_cast<const char *>(h_src) + off, len);
            if ((e = cudaMemcpyAsync(static_cast<char *>(d_dst) + off, s.buf[k], len, cudaMemcpyHostToDevice, st)) == cudaSuccess)
                e = cudaEventRecord(s.ev[k], st);
        }
        return e;
    });
    const cudaError_t e2 = cudaStreamSynchronize(st);
    return e != cudaSuccess ? e : e2;
}

cudaError_t copy_to_host_staged(void *h_dst, const void *d_src, size_t n, cudaStream_t st) {
    const size_t chunks = (n + kChunk - 1) / kChunk;
    return run_workers(chunks, [&](int w, int workers, void *a, void *b) {
        Pair s(a, b);
        cudaError_t e = s.init();
        auto fetch = [&](size_t c, int k) {
            const size_t off = c * kChunk, len = std::min(kChunk, n - off);
            if ((e = cudaMemcpyAsync(s.buf[k], static_cast<const char *>(d_src) + off, len, cudaMemcpyDeviceToHost, st)) == cudaSuccess)
                e = cudaEventRecord(s.ev[k], st);
        };
        int k = 0;
        if (e == cudaSuccess && (size_t) w < chunks) fetch(w, k);
        for (size_t c = w; e == cudaSuccess && c < chunks; c += workers, k ^= 1) {
            if (c + workers < chunks) fetch(c + workers, k ^ 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(s.ev[k]);
            if (e == cudaSuccess) {
                const size_t off = c * kChunk;
                std::memcpy(static_cast<char *>(h_dst) + off, s.buf[k], std::min(kChunk, n - off));
            }
        }
        return e;
    });
}

StagingBuffer::StagingBuffer() {
    if (take_buffers(1, bufs_) != cudaSuccess) cudaGetLastError();
}

StagingBuffer::~StagingBuffer() { return_buffers(bufs_); }

void release_staging_buffers() {
    std::vector<void *> bufs;
    {
        std::lock_guard<std::mutex> lk(g_staging_mu);
        bufs.swap(g_staging_free);
    }
    for (void *p : bufs) cudaFreeHost(p);
}

}  // namespace maxi
