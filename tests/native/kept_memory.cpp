// KeptMemory and device_alloc (kept.cpp) on a counting stand-in for the device
// allocator: who owns a block when, and that nothing is lost or freed twice.
#include <cuda_runtime.h>

#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "../../voreen_gb300/csrc/vrc_internal.h"

namespace {
std::mutex m;
std::set<void*> live;
size_t room = SIZE_MAX;  // bytes the allocator still has
std::set<std::pair<void*, size_t>> sizes;
int mallocs = 0;
cudaError_t last = cudaSuccess;
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> g(m);
    ++mallocs;
    if (n > room) return last = cudaErrorMemoryAllocation;
    room -= n;
    *p = std::malloc(1);
    live.insert(*p);
    sizes.insert({*p, n});
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> g(m);
    assert(live.erase(p) == 1);
    for (auto it = sizes.begin(); it != sizes.end(); ++it)
        if (it->first == p) {
            room += it->second;
            sizes.erase(it);
            break;
        }
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
}

using K = vrc::KeptMemory;

static void* block(K& kept, size_t n) {
    void* p = nullptr;
    assert(vrc::device_alloc(kept, &p, n) == cudaSuccess);
    return p;
}

int main() {
    {
        K kept;
        size_t got = 0;
        assert(!kept.take(K::VOLUME, 1, SIZE_MAX, &got) && !kept.give_back());
        void* a = block(kept, 100);
        kept.put(K::VOLUME, a, 100, 1000);
        assert(kept.held() == 100);
        assert(!kept.take(K::VOLUME, 101, SIZE_MAX, &got));  // too small
        assert(!kept.take(K::VOLUME, 40, 99, &got));         // too large
        assert(!kept.take(K::STAGE, 1, SIZE_MAX, &got));     // another kind
        assert(kept.take(K::VOLUME, 60, 100, &got) == a && got == 100 && kept.held() == 0);
        assert(!kept.take(K::VOLUME, 60, 100, &got));        // once
        kept.put(K::VOLUME, a, 100, 1000);
        void* b = block(kept, 200);
        kept.put(K::VOLUME, b, 200, 1000);  // the last one stays
        assert(kept.held() == 200 && live.count(b) && live.size() == 1);
        kept.put(K::STAGE, block(kept, 2000), 2000, 1000);  // over the limit
        assert(kept.held() == 200 && live.size() == 1);
        kept.put(K::STAGE, block(kept, 300), 300, 1000);
        assert(kept.held() == 500 && live.size() == 2);
        assert(kept.give_back() && kept.held() == 0 && live.empty());
        kept.put(K::VOLUME, block(kept, 7), 7, 1000);  // still open
        assert(kept.held() == 7);
        assert(kept.give_back(true) && live.empty());
        kept.put(K::VOLUME, block(kept, 7), 7, 1000);  // a volume that outlives its context
        assert(kept.held() == 0 && live.empty());
    }
    {
        K kept;
        room = 1000;
        kept.put(K::VOLUME, block(kept, 600), 600, 1000);
        kept.put(K::STAGE, block(kept, 100), 100, 1000);
        void* a = block(kept, 300);  // fits beside them
        assert(kept.held() == 700);
        void* b = block(kept, 650);  // only once they are given back
        assert(kept.held() == 0 && live.size() == 2 && last == cudaSuccess);
        mallocs = 0;
        void* c = nullptr;
        assert(vrc::device_alloc(kept, &c, 100) == cudaErrorMemoryAllocation && !c);
        assert(mallocs == 1 && last == cudaSuccess);  // nothing kept: tried once, and the error taken back
        cudaFree(a);
        cudaFree(b);
        assert(room == 1000 && live.empty());
        room = SIZE_MAX;
    }
    {
        K kept;
        void* p = nullptr;
        size_t got = 0;
        auto use = [&](size_t best, size_t least) {
            mallocs = 0;
            p = nullptr;
            const cudaError_t e = kept.scratch(best, least, &p, &got);
            assert(last == cudaSuccess);
            if (e == cudaSuccess) kept.put(K::SCRATCH, p, got, SIZE_MAX);
            return e;
        };
        room = 1000;
        assert(use(400, 200) == cudaSuccess && got == 400 && mallocs == 1);
        assert(use(400, 200) == cudaSuccess && got == 400 && mallocs == 0);  // again: nothing allocated
        assert(use(100, 50) == cudaSuccess && got == 400 && mallocs == 0);
        assert(use(900, 450) == cudaSuccess && got == 900 && mallocs == 1);  // beside the 400 it would not fit
        assert(use(1200, 600) == cudaSuccess && got == 600 && mallocs == 2);  // refused: the smaller one
        assert(use(1200, 600) == cudaSuccess && got == 600 && mallocs == 0);  // and not asked for again
        assert(use(1200, 600) == cudaSuccess && got == 600 && mallocs == 0);
        assert(use(2400, 1100) == cudaErrorMemoryAllocation && kept.held() == 0);
        assert(use(1200, 600) == cudaSuccess && got == 600);
        room += 1000;
        assert(use(1200, 600) == cudaSuccess && got == 600 && mallocs == 0);
        kept.give_back();  // room may have been made since
        assert(use(1200, 600) == cudaSuccess && got == 1200 && mallocs == 1);
        kept.give_back(true);
        assert(live.empty());
        room = SIZE_MAX;
    }
    {
        K kept;
        std::vector<std::thread> threads;
        for (int t = 0; t < 4; ++t)
            threads.emplace_back([&kept, t] {
                for (int i = 0; i < 2000; ++i) {
                    size_t got = 0;
                    void* p = kept.take(t & 1 ? K::VOLUME : K::STAGE, 10, 20, &got);
                    if (!p) p = block(kept, got = 10 + i % 11);
                    kept.put(t & 1 ? K::VOLUME : K::STAGE, p, got, 18);
                    if (i % 100 == 0) kept.give_back();
                }
            });
        for (auto& t : threads) t.join();
        kept.give_back(true);
        assert(live.empty());
    }
    std::puts("kept_memory ok");
}
