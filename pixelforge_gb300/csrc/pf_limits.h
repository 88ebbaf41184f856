/*
 * pf_limits.h - how many CTAs of a kernel with dynamic shared memory fit on
 * an SM, and the limits such a launch needs.
 *
 * Host code only (CUDA runtime C API), safe with several threads and devices.
 */
#ifndef PF_LIMITS_H
#define PF_LIMITS_H

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <mutex>

#define PF_LIMITS_KEPT 64

/* CTAs of `kernel` with `block` threads and `smem` bytes of dynamic shared
 * memory that fit on an SM of the current device, its shared-memory limits
 * set.  Asked of the driver once per device, kernel and size: the calls for
 * every launch of a frame take about as long as a small frame's kernel.  The
 * last PF_LIMITS_KEPT answers are kept (the sizes are powers of two and row
 * widths by 256 pixels: a device asks for about 40).
 *
 * A kernel's limit is only ever raised, whatever is still kept: a launch
 * follows this call outside the lock, so a limit that followed the sizes
 * could be lowered under another thread's launch.  (It is raised to what is
 * asked for: with all that the device allows, five of seven workloads measured
 * about 1 us longer, sphere1080 156.6 against 155.1, next to the noise.) */
inline cudaError_t pfd_ctas_per_sm(const void *kernel, int block, size_t smem, bool maxShared, int &fit)
{
    struct Known { const void *kernel; int dev, block, fit; size_t smem; };
    static std::mutex m;
    static Known known[PF_LIMITS_KEPT];
    static int count = 0, next = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(m);
    for (int i = 0; i < count; i++) {
        const Known &k = known[i];
        if (k.kernel == kernel && k.dev == dev && k.block == block && k.smem == smem) { fit = k.fit; return cudaSuccess; }
    }
    cudaFuncAttributes at;
    e = cudaFuncGetAttributes(&at, kernel);
    if (e == cudaSuccess && smem > (size_t)at.maxDynamicSharedSizeBytes)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && maxShared)                 /* the CTAs' shared memory, not L1, bounds how many fit on an SM */
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, block, smem);
    if (e == cudaSuccess) {
        known[next] = Known{ kernel, dev, block, fit, smem };
        next = (next + 1) % PF_LIMITS_KEPT;
        count = count < PF_LIMITS_KEPT ? count + 1 : count;
    }
    return e;
}

#endif /* PF_LIMITS_H */
