// Pinned host blocks, kept for the next context when one gives its own back.  The driver takes 1.4 to
// 4 ms for a block however small it is: every context's third solve, which pins its staging, cost
// 3.5 ms (32^3; 0.86 unrecorded).  Kept are blocks of up to 1 MB, 8 MB in all.
#include <cuda.h>   // CUcontext and CUresult (the types only)

#include <map>
#include <mutex>

#include "internal.h"

namespace ddagpu {

namespace {

constexpr size_t kLeast = 64 << 10, kMost = 1 << 20, kHeld = 8 << 20;

struct Kept {
    std::mutex mu;
    std::multimap<std::pair<unsigned long long, size_t>, void *> blocks;   // by CUDA context and size
    size_t bytes = 0;
};

Kept &kept()
{
    static Kept *k = new Kept;   // contexts may outlive static objects
    return *k;
}

// Identity of the current CUDA context: a block is valid in the one that it was made in, which a
// device reset ends.  0 if the driver does not say; nothing is kept then.
unsigned long long context_id()
{
    using Get = CUresult (*)(CUcontext, unsigned long long *);
    static const Get get = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        const cudaError_t e = cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? reinterpret_cast<Get>(f) : nullptr;
    }();
    unsigned long long id = 0;
    return get && get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

}  // namespace

cudaError_t pinned_take(size_t bytes, unsigned char **p, size_t *size)
{
    size_t n = kLeast;
    while (n < bytes && n < kMost) n *= 2;
    if (n < bytes) n = bytes;
    if (n <= kMost) {
        const unsigned long long id = context_id();
        Kept &k = kept();
        std::lock_guard<std::mutex> lk(k.mu);
        const auto it = k.blocks.lower_bound({id, n});
        if (id && it != k.blocks.end() && it->first.first == id) {
            *p = static_cast<unsigned char *>(it->second);
            *size = it->first.second;
            k.bytes -= *size;
            k.blocks.erase(it);
            return cudaSuccess;
        }
    }
    *size = n;
    return cudaHostAlloc((void **)p, n, cudaHostAllocPortable);
}

void pinned_give(unsigned char *p, size_t size)
{
    if (!p) return;
    if (size <= kMost) {
        const unsigned long long id = context_id();
        Kept &k = kept();
        std::lock_guard<std::mutex> lk(k.mu);
        if (id && k.bytes + size <= kHeld) {
            k.blocks.insert({{id, size}, p});
            k.bytes += size;
            return;
        }
    }
    cudaFreeHost(p);
}

}  // namespace ddagpu
