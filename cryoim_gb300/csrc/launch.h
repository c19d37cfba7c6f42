// launch.h — what launchers ask of the device.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace cryoim {

// Allows kern the dynamic shared memory of a launch that wants `bytes` of it, beside the kernel's own
// static memory: up to 48 KB in all every kernel may have, more takes an attribute of the kernel, a state
// of the device that every lane, context and host thread launches under.  So it is only ever set to
// the most that a block of this kernel can have: with each launch's own size, one thread could lower
// it between another's call and its launch, which the device would then refuse.
inline cudaError_t allow_smem_of(const void* kern, size_t bytes) {
    if (bytes <= 16 * 1024) return cudaSuccess;  // (no kernel with dynamic memory has 32 KB of its own beside it)
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return e;
    if (bytes + fa.sharedSizeBytes <= 48 * 1024) return cudaSuccess;
    if (fa.maxDynamicSharedSizeBytes > 48 * 1024 && bytes <= (size_t)fa.maxDynamicSharedSizeBytes) return cudaSuccess;
    int dev = 0, most = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
    const int room = most - (int)fa.sharedSizeBytes;
    if (room < 0 || bytes > (size_t)room) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, room);
}
template <class... A>
cudaError_t allow_smem(void (*kern)(A...), size_t bytes) {
    return allow_smem_of(reinterpret_cast<const void*>(kern), bytes);
}

// the current device's SMs (152 where it cannot be asked: the launch will say why)
inline int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 152;
    return n;
}

}  // namespace cryoim
