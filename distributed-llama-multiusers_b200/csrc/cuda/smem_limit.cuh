// How much dynamic shared memory a kernel may be launched with is a setting of each device: raised there the first time, and whenever a launch needs more.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

extern void dl_set_error(const char* fmt, ...);

struct SmemLimit { std::atomic<int> bytes[64] = {}; };       // one per kernel: what each device has been given
// 0, or the negated CUDA error (dl_last_error)
template <typename K>
static int dl_smem_limit(const char* who, K kernel, size_t bytes, SmemLimit& given, int dev = -1) {      // dev: the current device where the caller knows it
    cudaError_t e = dev >= 0 ? cudaSuccess : cudaGetDevice(&dev);
    if (e == cudaSuccess && dev < 64 && given.bytes[dev] >= (int)bytes) return 0;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) { dl_set_error("%s smem attr: %s", who, cudaGetErrorString(e)); return -(int)e; }
    if (dev < 64) given.bytes[dev] = (int)bytes;
    return 0;
}
