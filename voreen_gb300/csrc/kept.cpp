// Device memory that a context keeps between calls (vrc_internal.h).
#include <cuda_runtime.h>

#include <utility>

#include "vrc_internal.h"

namespace vrc {

void* KeptMemory::take(Kind k, size_t need, size_t most, size_t* got) {
    std::lock_guard<std::mutex> g(lock);
    Block& b = blocks[k];
    if (!b.p || b.bytes < need || b.bytes > most) return nullptr;
    void* p = b.p;
    *got = b.bytes;
    b = Block{};
    return p;
}

void KeptMemory::put(Kind k, void* p, size_t bytes, size_t limit) {
    if (bytes <= limit) {
        std::lock_guard<std::mutex> g(lock);
        if (!closed) {
            std::swap(blocks[k].p, p);
            blocks[k].bytes = bytes;
        }
    }
    cudaFree(p);
}

cudaError_t KeptMemory::scratch(size_t best, size_t least, void** p, size_t* got) {
    void* small = nullptr;  // freed first: beside it the larger one might not fit
    bool ask;
    {
        std::lock_guard<std::mutex> g(lock);
        Block& b = blocks[SCRATCH];
        ask = best != refused;
        if (b.p && b.bytes >= (ask ? best : least)) {
            *p = b.p;
            *got = b.bytes;
            b = Block{};
            return cudaSuccess;
        }
        std::swap(small, b.p);
        b = Block{};
    }
    cudaFree(small);
    if (ask) {
        const cudaError_t e = device_alloc_bytes(*this, p, *got = best);
        if (e != cudaErrorMemoryAllocation) return e;
        std::lock_guard<std::mutex> g(lock);
        refused = best;
    }
    return device_alloc_bytes(*this, p, *got = least);
}

bool KeptMemory::give_back(bool close) {
    Block all[KINDS];
    {
        std::lock_guard<std::mutex> g(lock);
        std::swap(all, blocks);
        refused = 0;
        closed = closed || close;
    }
    bool any = false;
    for (Block& b : all) {
        any = any || b.p;
        cudaFree(b.p);
    }
    return any;
}

size_t KeptMemory::held() {
    std::lock_guard<std::mutex> g(lock);
    size_t n = 0;
    for (const Block& b : blocks) n += b.bytes;
    return n;
}

cudaError_t device_alloc_bytes(KeptMemory& kept, void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) return e;
    const bool again = e == cudaErrorMemoryAllocation && kept.give_back();
    if (again) e = cudaMalloc(p, bytes);
    cudaGetLastError();  // an error is the caller's to report, not the next launch's
    return e;
}

}  // namespace vrc
