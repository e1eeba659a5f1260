/* Host side of a launch: what belongs to a device rather than to the process.
 *
 * A solver is bound to the device that it was made on, and one process may
 * drive several devices, or reset one.  A kernel's shared-memory limit is an
 * attribute of the kernel on the current device, lost with its context, so it
 * is set before every launch that needs it; the SM count is asked of the
 * current device; the resident blocks per SM, a slower question, are kept per
 * device.  Plain runtime calls only, so that this file compiles without a
 * device compiler. */
#ifndef OV_HOST_H
#define OV_HOST_H

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>

#include <atomic>

namespace ov {

/* the SM count of the current device */
inline cudaError_t device_sms(int* sms)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess && *sms <= 0)
        e = cudaErrorInvalidDevice;
    return e;
}

/* lets `kern` take smem bytes of dynamic shared memory on the current device
   (the default 48 KB also hold the kernels' static words) */
inline cudaError_t allow_smem(const void* kern, size_t smem)
{
    if (smem <= 40 * 1024)
        return cudaSuccess;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

/* A kernel's resident blocks per SM, by device: block size and count in one
   word, so that threads that launch for the first time together read all of
   it or nothing.  Devices beyond the last slot ask every time. */
struct Residency {
    static constexpr int DEVICES = 32;
    std::atomic<uint64_t> slot[DEVICES];
};

/* blocks of `kern` that the current device holds at a time, after allow_smem */
inline cudaError_t resident_blocks(Residency& r, const void* kern, int block, size_t smem, int* resident)
{
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = device_sms(&sms);
    if (e == cudaSuccess)
        e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    const bool kept = dev >= 0 && dev < Residency::DEVICES;
    const uint64_t word = kept ? r.slot[dev].load() : 0u;
    if (word >> 32 == (uint64_t)block) {
        per_sm = (int)(word & 0xffffffffu);
    } else {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem);
        if (e != cudaSuccess)
            return e;
        if (per_sm < 1)
            per_sm = 1;
        if (kept)
            r.slot[dev].store((uint64_t)block << 32 | (uint64_t)per_sm);
    }
    *resident = sms * per_sm;
    return cudaSuccess;
}

}  // namespace ov

#endif /* OV_HOST_H */
