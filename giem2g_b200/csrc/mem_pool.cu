// Temporary device memory of an operator's set-up, from a stream-ordered pool of its own.
//
// A frequency's set-up allocates and frees its weights, bases and transform buffers.  With cudaMalloc and cudaFree
// that is page mapping and a device synchronisation per buffer: at 64x64x16 more than half of the set-up's time.  The
// pool keeps up to kPoolKeep bytes mapped between calls (the whole set-up at 64x64x16, 250 MB); beyond that,
// synchronisation points give the memory back, and the operator's end gives back all of it.  Every buffer is used and
// freed on the operator's own stream.
#include "common.cuh"
#include "ie_internal.h"

namespace {
constexpr unsigned long long kPoolKeep = 512ull << 20;
}

int g2_pool_alloc(cudaMemPool_t *pool, void **p, size_t bytes, cudaStream_t st)
{
    *p = nullptr;
    if (!*pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        G2_CUDA_CHECK(cudaGetDevice(&props.location.id));
        G2_CUDA_CHECK(cudaMemPoolCreate(pool, &props));
        unsigned long long keep = kPoolKeep;
        G2_CUDA_CHECK(cudaMemPoolSetAttribute(*pool, cudaMemPoolAttrReleaseThreshold, &keep));
    }
    G2_CUDA_CHECK(cudaMallocFromPoolAsync(p, bytes ? bytes : 1, *pool, st));
    return G2_OK;
}
void g2_pool_free(void *p, cudaStream_t st)
{
    if (p) cudaFreeAsync(p, st);
}
