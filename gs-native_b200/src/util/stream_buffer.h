// Device scratch of one call, allocated and freed in stream order.
//
// The stateless entry points (spatial permutation, evaluation metrics) need scratch
// that no object of the caller holds. cudaMalloc and cudaFree synchronise the device
// and take the driver's locks (2.3 ms of a 2.8 ms permutation of 1.2M Gaussians, and
// tens of milliseconds beside other processes), so the scratch comes from a memory
// pool of the library's own, one per context: stream-ordered, so it is safe with any
// number of threads and streams, and a device reset leaves nothing behind that a later
// call would use. At most kPoolBytes stay reserved between calls; ReleaseStreamPool
// gives those back too, and DeviceAlloc calls it before it reports that memory has run
// out. A call that needs more than kPoolBytes (a permutation of more than 4.1M
// Gaussians) maps the block anew each time: 320 us at 6.0M Gaussians.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace gs_native {

constexpr size_t kPoolBytes = size_t{64} << 20;

class StreamBuffer {
public:
    explicit StreamBuffer(cudaStream_t stream) : stream_(stream) {}
    ~StreamBuffer();
    StreamBuffer(const StreamBuffer&) = delete;
    StreamBuffer& operator=(const StreamBuffer&) = delete;

    // Once per buffer.
    bool Allocate(size_t bytes);
    unsigned char* get() const { return static_cast<unsigned char*>(data_); }

private:
    cudaStream_t stream_;
    void* data_ = nullptr;
};

// Gives the unused memory of the current context's pool back to its device.
void ReleaseStreamPool();

}  // namespace gs_native
