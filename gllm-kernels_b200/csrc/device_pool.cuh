// Device memory of weights and scratch.
//
// cudaMalloc and cudaFree each cost tens to hundreds of microseconds and cudaFree waits for the device, which is nothing for a
// model's weights but most of the time of a call whose activations are quantized and uploaded like a weight
// (gllmk_gemm_fp4: W[14336, 4096] x 2048 tokens 850 - 1360 us, 600 of them here).  Freed weight buffers of up to 64 MB
// therefore stay with the library, at most 128 MB per device, until the last context of the device is freed or one of the
// library's own allocations fails.
// A buffer that is taken again may still be read by kernels its last owner launched, on any stream: the taker waits for the
// device once.  Only an upload from device memory takes one (it has to wait for the device anyway); an upload from the host
// waits for nothing, so that it also works beside a stream capture of another thread, and its time is the bus's.
// An allocation has the size that was asked for.  A buffer serves smaller requests too, as long as it is no more than an eighth
// (or 64 KB) larger: activations whose token counts differ a little share buffers, and no weight holds much more than it needs.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>
#include <vector>

namespace gllmk {

constexpr size_t POOL_MAX_BLOCK = (size_t)64 << 20, POOL_MAX_BYTES = (size_t)128 << 20;
struct DevicePool {
    struct Block { void *p; size_t bytes; };
    std::mutex mu;
    std::vector<Block> blocks;  // oldest first
    size_t held = 0;
    int contexts = 0;
};
inline DevicePool &pool_of(int device) {
    static DevicePool *pools = new DevicePool[64];  // never destroyed: weights may be freed while the process ends
    return pools[device & 63];
}
inline void pool_trim(int device) {
    DevicePool &p = pool_of(device);
    std::lock_guard<std::mutex> l(p.mu);
    for (const DevicePool::Block &b : p.blocks) cudaFree(b.p);
    p.blocks.clear();
    p.held = 0;
}
// cudaMalloc on the current device, `device`; when memory is short, once more without the idle buffers.
inline cudaError_t device_malloc(int device, void **out, size_t bytes) {
    cudaError_t e = cudaMalloc(out, bytes);
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        pool_trim(device);
        e = cudaMalloc(out, bytes);
    }
    return e;
}
// A buffer of at least *bytes, which receives its size.  reuse: it may be a freed one; *waited is set if it is (the device has been
// waited for).
inline cudaError_t pool_take(int device, size_t *bytes, void **out, bool reuse, bool *waited) {
    *out = nullptr;
    if (reuse) {
        DevicePool &p = pool_of(device);
        std::lock_guard<std::mutex> l(p.mu);
        const size_t slack = *bytes / 8 > (size_t)65536 ? *bytes / 8 : (size_t)65536;
        size_t best = p.blocks.size();
        for (size_t i = 0; i < p.blocks.size(); i++)
            if (p.blocks[i].bytes >= *bytes && p.blocks[i].bytes - *bytes <= slack && (best == p.blocks.size() || p.blocks[i].bytes < p.blocks[best].bytes))
                best = i;
        if (best != p.blocks.size()) {
            *out = p.blocks[best].p;
            *bytes = p.blocks[best].bytes;
            p.held -= *bytes;
            p.blocks.erase(p.blocks.begin() + (ptrdiff_t)best);
        }
    }
    if (*out) {
        const cudaError_t e = cudaDeviceSynchronize();
        if (e == cudaSuccess) *waited = true;
        else cudaFree(*out), *out = nullptr;
        return e;
    }
    return device_malloc(device, out, *bytes);
}
inline void pool_put(int device, void *ptr, size_t bytes) {
    if (!ptr) return;
    DevicePool &p = pool_of(device);
    std::lock_guard<std::mutex> l(p.mu);
    if (bytes > POOL_MAX_BLOCK || p.contexts == 0) {
        cudaFree(ptr);
        return;
    }
    while (p.held + bytes > POOL_MAX_BYTES) {
        cudaFree(p.blocks.front().p);
        p.held -= p.blocks.front().bytes;
        p.blocks.erase(p.blocks.begin());
    }
    p.blocks.push_back({ptr, bytes});
    p.held += bytes;
}

}  // namespace gllmk
