// The library's stream-ordered scratch pools (see stream_buffer.h).
#include "util/stream_buffer.h"

#include <cuda.h>

#include <map>
#include <mutex>

namespace gs_native {

namespace {

std::mutex g_mutex;
// By context: a context's reset takes its pool with it, and the next one has another id.
std::map<unsigned long long, cudaMemPool_t> g_pools;

// Id of the calling thread's context, which is made current first where none is; 0 on
// failure.
unsigned long long ContextId() {
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static const GetId get_id = [] {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult found;
        const bool ok = cudaGetDriverEntryPointByVersion("cuCtxGetId", &entry, 12000, cudaEnableDefault, &found) ==
                            cudaSuccess &&
                        found == cudaDriverEntryPointSuccess;
        return ok ? reinterpret_cast<GetId>(entry) : nullptr;
    }();
    unsigned long long id = 0;
    if (!get_id) return 0;
    if (get_id(nullptr, &id) == CUDA_SUCCESS) return id;
    return cudaFree(nullptr) == cudaSuccess && get_id(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// The current context's pool, made at its first use.
cudaMemPool_t ContextPool() {
    const unsigned long long id = ContextId();
    int device = 0;
    if (id == 0 || cudaGetDevice(&device) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(g_mutex);
    const auto known = g_pools.find(id);
    if (known != g_pools.end()) return known->second;
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
    g_pools[id] = pool;
    return pool;
}

}  // namespace

StreamBuffer::~StreamBuffer() {
    if (data_) cudaFreeAsync(data_, stream_);
}

bool StreamBuffer::Allocate(size_t bytes) {
    if (data_) return false;
    const cudaMemPool_t pool = ContextPool();
    if (!pool) return false;
    return cudaMallocFromPoolAsync(&data_, bytes ? bytes : 1, pool, stream_) == cudaSuccess;
}

void ReleaseStreamPool() {
    const unsigned long long id = ContextId();
    std::lock_guard<std::mutex> lock(g_mutex);
    const auto known = g_pools.find(id);
    if (known != g_pools.end()) cudaMemPoolTrimTo(known->second, 0);
}

}  // namespace gs_native
