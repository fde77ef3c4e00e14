// Spatial (Morton) ordering of the Gaussians and the gathers that apply it.
//
// A permutation of the Gaussians changes no result (every kernel is per
// Gaussian, per record or per pixel, and tile lists are ordered by depth, then
// id: reordering ids only changes which of two equal-depth Gaussians comes
// first, exactly as the reference's own ordering after a density step does).
// It does change locality: with the ids in Morton order of their means, the
// Gaussians of one view occupy long id runs, so a visibility-masked update
// (GaussianUpdateArgs::sparse) skips whole 32-byte sectors of the SoA rows, and
// the per-record gathers and gradient atomics of a tile hit nearby addresses.
//
// Keys: 10 bits per axis of the position inside the bounding box of all
// finite means (a device min/max reduction), interleaved z-y-x into 30 bits.
#include "common.cuh"
#include "kernels.h"

namespace gsn {

namespace {

// Order-preserving float <-> unsigned map for the min reductions.
__device__ __forceinline__ uint32_t ordered(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float unordered(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? u & 0x7FFFFFFFu : ~u);
}

constexpr int kBoundsBlocks = 148 * 2;

// bounds[0..2]: smallest ordered coordinates of the finite means; bounds[3..5]:
// smallest complements (the largest coordinates), all initialised by one memset to
// 0xFF. Six global atomics per block: with six per warp of 1,184 blocks the
// atomics queued on one L2 line (42 us at 1.2M Gaussians).
__global__ void __launch_bounds__(256) position_bounds(const float* __restrict__ params, int n,
                                                       uint32_t* __restrict__ bounds) {
    __shared__ uint32_t s[6];
    if (threadIdx.x < 6) s[threadIdx.x] = 0xFFFFFFFFu;
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
#pragma unroll 4
    for (int64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float x = params[static_cast<int64_t>(a) * n + i];
            if (isfinite(x)) {
                lo[a] = fminf(lo[a], x);
                hi[a] = fmaxf(hi[a], x);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, ordered(lo[a]));
        const uint32_t h = __reduce_min_sync(0xffffffffu, ~ordered(hi[a]));
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&s[a], l);
            atomicMin(&s[3 + a], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMin(bounds + threadIdx.x, s[threadIdx.x]);
}

__device__ __forceinline__ uint32_t spread10(uint32_t x) {
    x &= 0x3FFu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

__global__ void __launch_bounds__(256) morton_keys(const float* __restrict__ params, int n,
                                                   const uint32_t* __restrict__ bounds,
                                                   uint32_t* __restrict__ keys) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float lo = unordered(bounds[a]), hi = unordered(~bounds[3 + a]);
        const float x = params[static_cast<int64_t>(a) * n + i];
        const float span = hi - lo;
        float f = span > 0.0f ? (x - lo) / span : 0.0f;
        f = isfinite(f) ? fminf(fmaxf(f, 0.0f), 1.0f) : 1.0f;
        q[a] = static_cast<uint32_t>(f * 1023.0f + 0.5f);
    }
    keys[i] = spread10(q[0]) | (spread10(q[1]) << 1) | (spread10(q[2]) << 2);
}

// Rows of 32-bit words: dst[r][i] = src[r][perm[i]]. A random permutation reads a
// 32-byte sector per word, so the gather is bound by L2 sector traffic and by how
// many of those reads are in flight: a thread takes kGatherItems Gaussians
// (strided by the block, so loads of perm and stores stay coalesced) of kGatherRows
// rows and issues all of its gathers together.
constexpr int kGatherItems = 4, kGatherRows = 2;

__global__ void __launch_bounds__(256) gather_rows(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                                                   const uint32_t* __restrict__ perm, int n, int rows) {
    const int64_t first = static_cast<int64_t>(blockIdx.x) * (256 * kGatherItems) + threadIdx.x;
    const int row0 = blockIdx.y * kGatherRows;
    uint32_t from[kGatherItems], v[kGatherRows][kGatherItems];
#pragma unroll
    for (int k = 0; k < kGatherItems; ++k) from[k] = first + 256 * k < n ? perm[first + 256 * k] : 0u;
#pragma unroll
    for (int r = 0; r < kGatherRows; ++r)
#pragma unroll
        for (int k = 0; k < kGatherItems; ++k)
            v[r][k] = row0 + r < rows ? src[static_cast<int64_t>(row0 + r) * n + from[k]] : 0u;
#pragma unroll
    for (int r = 0; r < kGatherRows; ++r)
#pragma unroll
        for (int k = 0; k < kGatherItems; ++k)
            if (row0 + r < rows && first + 256 * k < n) dst[static_cast<int64_t>(row0 + r) * n + first + 256 * k] = v[r][k];
}

__global__ void __launch_bounds__(256) compose_parents(const int* __restrict__ parents,
                                                       const uint32_t* __restrict__ perm, int n,
                                                       int* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int p = static_cast<int>(perm[i]);
    out[i] = parents ? parents[p] : p;
}

}  // namespace

int launch_morton_keys(const float* params, int n, uint32_t* bounds, uint32_t* keys, cudaStream_t stream) {
    if (n <= 0) return GSN_OK;
    if (!params || !bounds || !keys) return GSN_ERR_INVALID_ARGUMENT;
    if (cudaMemsetAsync(bounds, 0xFF, 6 * sizeof(uint32_t), stream) != cudaSuccess) return GSN_ERR_CUDA;
    position_bounds<<<min(ceil_div(n, 256), kBoundsBlocks), 256, 0, stream>>>(params, n, bounds);
    morton_keys<<<ceil_div(n, 256), 256, 0, stream>>>(params, n, bounds, keys);
    return launched(2);
}

int launch_gather_gaussians(const float* src, float* dst, const uint32_t* perm, int n, bool bf16_sh,
                            cudaStream_t stream) {
    if (n <= 0) return GSN_OK;
    if (!src || !dst || !perm) return GSN_ERR_INVALID_ARGUMENT;
    // one 32-bit word per (physical row, Gaussian) in both layouts
    const int rows = bf16_sh ? kPrecisionPhysicalRows : kParams;
    const dim3 grid(ceil_div(n, 256 * kGatherItems), ceil_div(rows, kGatherRows));
    gather_rows<<<grid, 256, 0, stream>>>(reinterpret_cast<const uint32_t*>(src), reinterpret_cast<uint32_t*>(dst),
                                          perm, n, rows);
    return launched(1);
}

int launch_compose_parents(const int* parents, const uint32_t* perm, int n, int* out, cudaStream_t stream) {
    if (n <= 0) return GSN_OK;
    if (!perm || !out) return GSN_ERR_INVALID_ARGUMENT;
    compose_parents<<<ceil_div(n, 256), 256, 0, stream>>>(parents, perm, n, out);
    return launched(1);
}

}  // namespace gsn
