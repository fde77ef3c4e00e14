// Allocation hook of the stage classes (see device_array.h).
#include "util/device_array.h"

#include <atomic>

#include "util/stream_buffer.h"

namespace gs_native {

namespace {
std::atomic<DeviceAllocFn> g_alloc_hook{nullptr};
}  // namespace

void SetDeviceAllocHook(DeviceAllocFn fn) { g_alloc_hook.store(fn); }

cudaError_t DeviceAlloc(void** ptr, size_t bytes) {
    DeviceAllocFn fn = g_alloc_hook.load();
    if (fn) return fn(ptr, bytes);
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e == cudaErrorMemoryAllocation) {
        // what the scratch pool keeps may be what is missing
        cudaGetLastError();
        ReleaseStreamPool();
        e = cudaMalloc(ptr, bytes);
    }
    return e;
}

}  // namespace gs_native
