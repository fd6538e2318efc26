// Launching the kernels whose shared memory goes with the call, and launches that overlap the
// end of the one before them.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace maxi {

// The most dynamic shared memory of a kernel without static shared memory on sm_100 (227 KB).
constexpr int kMaxDynamicSmem = 232448;

// Lets a launch of the kernel have `bytes` of dynamic shared memory.  The limit belongs to the
// kernel and the device, not to the launch: set to a call's own size, it could fall below what
// another thread was about to launch with, so it is the same on every call.
template <typename... Params>
cudaError_t allow_dynamic_smem(void (*kernel)(Params...), int bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;  // allowed anyway
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
}

// Launches `kernel`; `overlap`: with programmatic stream serialization, its blocks may come up
// once every block of the launch before it has called pass_prepare() or ended.
template <typename... Params, typename... Args>
cudaError_t launch_pass(void (*kernel)(Params...), bool overlap, int64_t grid, int threads, int smem, cudaStream_t st,
                        const Args &...args) {
    cudaError_t e = allow_dynamic_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned) grid);
    cfg.blockDim = dim3((unsigned) threads);
    cfg.dynamicSmemBytes = (size_t) smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// In an overlapped launch's blocks: the next launch's blocks may come up; wait until the launch
// before is complete and its writes are visible.  Every block waits, so a launch that is complete
// has all earlier ones behind it.  Without the launch attribute both do nothing.
__device__ __forceinline__ void pass_prepare() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pass_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace maxi
