// Temporary device memory of the operators' set-up: one stream-ordered pool per device.
//
// A frequency's set-up allocates and frees its weights, bases and transform buffers.  With cudaMalloc and cudaFree
// that is page mapping and a device synchronisation per buffer: at 64x64x16 more than half of the set-up's time.  The
// pool keeps up to kPoolKeep bytes mapped between calls (two such set-ups, or the receivers' weights at that grid), and the
// end of the device's last operator gives back all of it.  Every buffer is used and freed on one stream, its operator's.
//
// What would not fit into kPoolKeep beside the buffers in use comes from cudaMalloc: the pool would map it and unmap it for
// each use, at a third of cudaMalloc's speed.  Tensor + transform at 128x128x32 (1.1 GB each for the spatial tensor and its x
// transform, 0.4 GB of weights): all from the pool 15 + 21 ms, all above 256 MB from cudaMalloc 9.7 + 6.8, by this rule
// 8.7 + 6.9; at 64x128x27 5.2 + 5.6, 3.8 + 2.7, 3.8 + 1.9; the receivers' tensor at 64x64x16 3.8, 4.8, 3.8.
#include <mutex>
#include <unordered_set>
#include "common.cuh"
#include "ie_internal.h"

struct G2Pool {
    cudaMemPool_t pool = nullptr;
    int refs = 0;
    int dev = 0;
    unsigned long long ctx = 0;
};

namespace {
constexpr unsigned long long kPoolKeep = 512ull << 20;
constexpr size_t kSmall = 1ull << 20;  // not worth asking for
constexpr int kMaxDevices = 64;

std::mutex g_mu;
G2Pool *g_pool[kMaxDevices] = {};       // the device's pool while an operator holds it
std::unordered_set<void *> g_direct;    // buffers from cudaMalloc

// The current context's number (the driver's cuCtxGetId, reached through the runtime); 0 if the driver has none.  A device
// reset ends a context and its pools without the operators' doing.
unsigned long long context_id()
{
    typedef int (*Fn)(void *, unsigned long long *);
    static const Fn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
                        q == cudaDriverEntryPointSuccess;
        return ok ? reinterpret_cast<Fn>(p) : nullptr;
    }();
    unsigned long long id = 0;
    return fn && fn(nullptr, &id) == 0 ? id : 0;
}

int acquire(G2Pool **ref)
{
    int dev = 0;
    G2_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return G2_ERR_UNSUPPORTED;
    const unsigned long long ctx = context_id();
    if (!g_pool[dev] || g_pool[dev]->ctx != ctx) {  // a pool of an ended context stays with its operators
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        G2_CUDA_CHECK(cudaMemPoolCreate(&pool, &props));
        unsigned long long keep = kPoolKeep;
        const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) cudaMemPoolDestroy(pool);
        G2_CUDA_CHECK(e);
        g_pool[dev] = new G2Pool{pool, 0, dev, ctx};
    }
    *ref = g_pool[dev];
    (*ref)->refs++;
    return G2_OK;
}
}  // namespace

int g2_pool_alloc(G2Pool **ref, void **p, size_t bytes, cudaStream_t st)
{
    *p = nullptr;
    if (!*ref) {
        std::lock_guard<std::mutex> lk(g_mu);
        const int rc = acquire(ref);
        if (rc) return rc;
    }
    unsigned long long used = 0;
    if (bytes > kSmall) G2_CUDA_CHECK(cudaMemPoolGetAttribute((*ref)->pool, cudaMemPoolAttrUsedMemCurrent, &used));
    if (used + bytes > kPoolKeep) {
        G2_CUDA_CHECK(cudaMalloc(p, bytes));
        std::lock_guard<std::mutex> lk(g_mu);
        g_direct.insert(*p);
        return G2_OK;
    }
    G2_CUDA_CHECK(cudaMallocFromPoolAsync(p, bytes ? bytes : 1, (*ref)->pool, st));
    return G2_OK;
}

void g2_pool_free(void *p, cudaStream_t st)
{
    if (!p) return;
    bool direct;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        direct = g_direct.erase(p) > 0;
    }
    if (direct) {
        cudaStreamSynchronize(st);
        cudaFree(p);
    } else {
        cudaFreeAsync(p, st);
    }
}

void g2_pool_release(G2Pool **ref)
{
    G2Pool *k = *ref;
    *ref = nullptr;
    if (!k) return;
    std::lock_guard<std::mutex> lk(g_mu);
    if (--k->refs > 0) return;
    if (g_pool[k->dev] == k) g_pool[k->dev] = nullptr;
    if (context_id() == k->ctx) cudaMemPoolDestroy(k->pool);
    delete k;
}
