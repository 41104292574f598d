// dg_host.h -- host-side helpers shared by the kernel launchers.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <utility>

namespace dg {

// cudaFuncSetAttribute acts on the current device, so a kernel's dynamic
// shared-memory limit is raised once per device.  `done` is the caller's
// record for that one kernel: a bit per device ordinal (ordinals past 63 set
// the attribute on every call).  Safe to call from several threads.
template <class Kernel>
inline cudaError_t ensure_dynamic_smem(Kernel kern, int bytes, std::atomic<unsigned long long> &done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

// A launch that may begin while the one before it in the stream (`overlap`)
// is still running: that one lets its dependents go, and the kernel itself
// waits for it where it has to.
template <class... Params, class... Args>
inline cudaError_t launch_after(void (*kern)(Params...), int blocks, int threads, int smem, cudaStream_t st,
                                bool overlap, Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace dg
