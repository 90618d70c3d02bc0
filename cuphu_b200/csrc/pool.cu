/*
 * pool.cu -- the library's stream-ordered device memory.
 *
 * cudaMallocAsync on a device's default pool returns the memory to the driver
 * whenever the caller synchronises (its release threshold is 0), so every
 * call after a synchronisation mapped its scratch anew: 16 ms for a cost
 * build whose kernels take 60 us.  The library keeps a pool of its own per
 * device, created at first use, that holds on to at most kPoolKeep bytes
 * across synchronisations; cuphu_release_workspace gives them back.  The
 * allocations stay stream-ordered, so calls on several streams and threads
 * never share a live block, and nothing outside the library is reconfigured.
 */
#include "common.cuh"

#include <mutex>

namespace cuphu {
namespace {
constexpr unsigned long long kPoolKeep = 1ull << 30;
constexpr int kDevs = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kDevs];

cudaMemPool_t pool_of(int dev)
{
    if (dev < 0 || dev >= kDevs) return nullptr;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        unsigned long long keep = kPoolKeep;
        /* the first use may lie inside a stream capture, of this thread or another, which a call
         * that is not stream-ordered would invalidate; making a pool touches no stream */
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        const bool relaxed = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) p = nullptr;
        if (p) cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        if (relaxed) cudaThreadExchangeStreamCaptureMode(&mode);
        cudaGetLastError();
        g_pool[dev] = p;
    }
    return g_pool[dev];
}
}  // namespace

void *pool_alloc(size_t bytes, cudaStream_t s)
{
    int dev = 0;
    void *p = nullptr;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    cudaMemPool_t pool = pool_of(dev);
    const cudaError_t e = pool ? cudaMallocFromPoolAsync(&p, bytes, pool, s)
                               : cudaMallocAsync(&p, bytes, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

void pool_trim(int dev)
{
    if (dev < 0 || dev >= kDevs) return;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (g_pool[dev] && cudaMemPoolTrimTo(g_pool[dev], 0) != cudaSuccess) cudaGetLastError();
}

}  // namespace cuphu
