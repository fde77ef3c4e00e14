// The library's stream-ordered scratch pools (see stream_buffer.h).
#include "util/stream_buffer.h"

#include <mutex>

namespace gs_native {

namespace {

constexpr int kDevices = 64;
std::mutex g_mutex;
cudaMemPool_t g_pools[kDevices] = {};

// The current device's pool, made at its first use.
cudaMemPool_t DevicePool() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_pools[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
        unsigned long long keep = kPoolBytes;
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return nullptr;
        }
        g_pools[device] = pool;
    }
    return g_pools[device];
}

}  // namespace

StreamBuffer::~StreamBuffer() {
    if (data_) cudaFreeAsync(data_, stream_);
}

bool StreamBuffer::Allocate(size_t bytes) {
    if (data_) return false;
    const cudaMemPool_t pool = DevicePool();
    if (!pool) return false;
    return cudaMallocFromPoolAsync(&data_, bytes ? bytes : 1, pool, stream_) == cudaSuccess;
}

void ReleaseStreamPools() {
    std::lock_guard<std::mutex> lock(g_mutex);
    for (cudaMemPool_t pool : g_pools)
        if (pool) cudaMemPoolTrimTo(pool, 0);
}

}  // namespace gs_native
