// gs_native::SpatialOrder over the Morton-key, sort and gather kernels.
#include "core/spatial/spatial_order.h"

#include <algorithm>

#include "kernels.h"

namespace gs_native {

namespace {
size_t ArrayBytes(int count) { return (static_cast<size_t>(count) * sizeof(uint32_t) + 255) & ~static_cast<size_t>(255); }
}  // namespace

// keys and ids (two of each), the bounds, the sort's scratch
size_t SpatialOrder::WorkspaceBytes(int count) {
    return 4 * ArrayBytes(count) + 256 + gsn::radix_sort_scratch_bytes(count);
}

const uint32_t* SpatialOrder::ComputeIn(unsigned char* work, const float* params, int count, cudaStream_t stream) {
    const size_t array = ArrayBytes(count);
    uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(work), reinterpret_cast<uint32_t*>(work + array)};
    uint32_t* ids[2] = {reinterpret_cast<uint32_t*>(work + 2 * array), reinterpret_cast<uint32_t*>(work + 3 * array)};
    auto* bounds = reinterpret_cast<uint32_t*>(work + 4 * array);
    if (gsn::launch_morton_keys(params, count, bounds, keys[0], stream) != GSN_OK) return nullptr;
    bool in_alt = false;
    const gsn::RadixSortScratch scratch = gsn::radix_sort_scratch(work + 4 * array + 256);
    if (gsn::launch_radix_sort(keys[0], ids[0], keys[1], ids[1], true, count, nullptr, 0, 30, scratch, &in_alt,
                               stream) != GSN_OK)
        return nullptr;
    return ids[in_alt ? 1 : 0];
}

bool SpatialOrder::Compute(const float* params, int count) {
    if (!params || count <= 0 || !work_.Reserve(WorkspaceBytes(count))) return false;
    const uint32_t* perm = ComputeIn(work_.get(), params, count, stream_);
    if (!perm) return false;
    perm_ = perm;
    count_ = count;
    return true;
}

bool SpatialOrder::Apply(float* params, int count, bool bf16_sh, const int* parents) {
    if (!params || count != count_ || !perm_) return false;
    const size_t floats = static_cast<size_t>(count) * (bf16_sh ? GSN_SH_INDEX + 24 : GSN_PARAM_COUNT);
    if (!block_.Reserve(floats) || !parents_.Reserve(static_cast<size_t>(count))) return false;
    if (gsn::launch_gather_gaussians(params, block_.get(), perm_, count, bf16_sh, stream_) != GSN_OK ||
        cudaMemcpyAsync(params, block_.get(), floats * sizeof(float), cudaMemcpyDeviceToDevice, stream_) !=
            cudaSuccess ||
        gsn::launch_compose_parents(parents, perm_, count, parents_.get(), stream_) != GSN_OK)
        return false;
    return true;
}

bool SpatialOrder::Compose(const int* parents, int* out) {
    if (!out || !perm_) return false;
    return gsn::launch_compose_parents(parents, perm_, count_, out, stream_) == GSN_OK;
}

}  // namespace gs_native
