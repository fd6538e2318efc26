// Device scratch kept between calls (scratch.h).
#include "scratch.h"

#include <map>

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

}  // namespace

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
        if (cudaMalloc(&s->buf, bytes) != cudaSuccess) {
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
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    for (auto &kv : g_scratch) {
        std::lock_guard<std::mutex> lk2(kv.second->mu);
        kv.second->drop();
    }
}

}  // namespace maxi
