// (h) LBVH 3-nearest-neighbour search for the initial Gaussian scales.
//
// Same result as ComputeMeanDist2Cuda (knn.cu:16-255): for every point the mean
// of its (up to) three smallest squared distances to the other points, 0 when
// there are fewer than two points. The structure is a linear BVH: 30-bit Hilbert
// codes over the bounding box, a stable radix sort (sort.cu), the points copied
// into that order, buckets of 8 consecutive points as leaves and boxes of 32
// children above them (three levels at 100k points, two launches to build).
//
// A warp answers 32 consecutive (so mostly neighbouring) points together. It
// starts from the distances among its own points, which already bound the third
// neighbour closely, then walks the tree once for all of them: the 32 lanes test
// a node's 32 child boxes against the warp's bounding box at once, the child on
// the warp's own path is entered first, and a leaf's points are read once for 32
// queries. Along a Hilbert curve neighbours in order are neighbours in space; a Morton
// order's jumps gave single warps boxes with 6,467 of the 12,500 leaves in reach (191
// at most so), and those warps decided the time: a search of 100k points of a volume
// and two shells took 377 us with it and takes 186 us. A thread-per-point walk of a
// binary tree of the same leaves spent its time on divergent, dependent loads (order,
// then point): 2,433 us.
//
// Squared distances are evaluated without contraction ((dx*dx + dy*dy) + dz*dz,
// each rounded) and ties go to the smaller index, so the neighbour indices equal
// those of an exhaustive FP32 search whatever the order of the walk.
#include <float.h>

#include "common.cuh"
#include "kernels.h"
#include "knn_kernels.h"

namespace gsn {

namespace {

constexpr int kMaxLevels = 7;  // 8 x 32^6 points
}  // namespace

// Box counts per level (0: the leaves) and where each level starts in lo / hi.
struct KnnTree {
    int levels;
    int count[kMaxLevels];
    int offset[kMaxLevels];
};

namespace {

KnnTree knn_tree(int n) {
    KnnTree t{};
    t.count[0] = (n + 7) / 8;
    t.levels = 1;
    while (t.count[t.levels - 1] > 32) {
        t.count[t.levels] = (t.count[t.levels - 1] + 31) / 32;
        t.offset[t.levels] = t.offset[t.levels - 1] + t.count[t.levels - 1];
        ++t.levels;
    }
    return t;
}

constexpr int kThreads = 256;
constexpr int kQueryThreads = 64;  // two independent warps: small blocks even out the tail
constexpr int kBucket = 8;         // points per leaf
constexpr int kFan = 32;           // children per box

// Smallest / largest corner over groups of W consecutive lanes.
template <int W>
__device__ __forceinline__ void box_reduce(float3& mn, float3& mx) {
#pragma unroll
    for (int o = W / 2; o; o >>= 1) {
        mn.x = fminf(mn.x, __shfl_xor_sync(0xffffffffu, mn.x, o));
        mn.y = fminf(mn.y, __shfl_xor_sync(0xffffffffu, mn.y, o));
        mn.z = fminf(mn.z, __shfl_xor_sync(0xffffffffu, mn.z, o));
        mx.x = fmaxf(mx.x, __shfl_xor_sync(0xffffffffu, mx.x, o));
        mx.y = fmaxf(mx.y, __shfl_xor_sync(0xffffffffu, mx.y, o));
        mx.z = fmaxf(mx.z, __shfl_xor_sync(0xffffffffu, mx.z, o));
    }
}

__device__ __forceinline__ unsigned int spread10(unsigned int v) {
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__device__ __forceinline__ unsigned int float_to_ordered(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float ordered_to_float(unsigned int u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// bounds[0..2]: smallest ordered coordinates; bounds[3..5]: smallest complements,
// so one memset to 0xFF initialises all six.
__global__ void bounds_kernel(const float* __restrict__ pts, int n, unsigned int* bounds) {
    pdl_begin();
    __shared__ unsigned int s[6];
    if (threadIdx.x < 6) s[threadIdx.x] = 0xFFFFFFFFu;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const unsigned int o = i < n ? float_to_ordered(pts[3ll * i + a]) : 0u;
        const unsigned int lo = __reduce_min_sync(0xffffffffu, i < n ? o : 0xFFFFFFFFu);
        const unsigned int hi = __reduce_min_sync(0xffffffffu, i < n ? ~o : 0xFFFFFFFFu);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&s[a], lo);
            atomicMin(&s[3 + a], hi);
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMin(bounds + threadIdx.x, s[threadIdx.x]);
}

// Position of a cell along the Hilbert curve of 2^10 cells per axis (J. Skilling,
// "Programming the Hilbert curve", 2004: axes to transposed index).
__device__ __forceinline__ uint32_t hilbert30(uint32_t x[3]) {
#pragma unroll
    for (uint32_t q = 1u << 9; q > 1u; q >>= 1) {
        const uint32_t low = q - 1u;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (x[i] & q) {
                x[0] ^= low;
            } else {
                const uint32_t t = (x[0] ^ x[i]) & low;
                x[0] ^= t;
                x[i] ^= t;
            }
        }
    }
    x[1] ^= x[0];
    x[2] ^= x[1];
    uint32_t t = 0;
#pragma unroll
    for (uint32_t q = 1u << 9; q > 1u; q >>= 1)
        if (x[2] & q) t ^= q - 1u;
    return (spread10(x[0] ^ t) << 2) | (spread10(x[1] ^ t) << 1) | spread10(x[2] ^ t);
}

__global__ void curve_kernel(const float* __restrict__ pts, int n, const unsigned int* __restrict__ bounds,
                             uint32_t* __restrict__ keys) {
    pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float lo = ordered_to_float(bounds[a]), hi = ordered_to_float(~bounds[3 + a]);
        float ext = hi - lo;
        float t = ext > 0.0f ? (pts[3ll * i + a] - lo) / ext : 0.0f;
        c[a] = static_cast<uint32_t>(fminf(fmaxf(t * 1023.0f, 0.0f), 1023.0f));
    }
    keys[i] = hilbert30(c);
}

// The points in curve order with their index as the fourth word, the leaf boxes
// (8 points each) and the boxes of 32 leaves: one block covers 256 points, which
// is one box of the level above the leaves.
__global__ void __launch_bounds__(kThreads) leaves_kernel(const float* __restrict__ pts,
                                                          const uint32_t* __restrict__ order, int n, KnnTree tree,
                                                          float4* __restrict__ sorted, float4* __restrict__ lo,
                                                          float4* __restrict__ hi) {
    static_assert(kThreads == kBucket * kFan, "a block is one second-level box");
    pdl_begin();
    __shared__ float3 s_lo[kFan], s_hi[kFan];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float3 mn = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), mx = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    if (i < n) {
        const uint32_t id = order[i];
        const float* p = pts + 3ll * id;
        const float x = p[0], y = p[1], z = p[2];
        sorted[i] = make_float4(x, y, z, __uint_as_float(id));
        // as a running fminf / fmaxf from +-FLT_MAX: a NaN coordinate widens nothing
        mn = make_float3(fminf(mn.x, x), fminf(mn.y, y), fminf(mn.z, z));
        mx = make_float3(fmaxf(mx.x, x), fmaxf(mx.y, y), fmaxf(mx.z, z));
    }
    box_reduce<kBucket>(mn, mx);
    if ((threadIdx.x & (kBucket - 1)) == 0) {
        const int leaf = i / kBucket;
        s_lo[threadIdx.x / kBucket] = mn;
        s_hi[threadIdx.x / kBucket] = mx;
        if (leaf < tree.count[0]) {
            lo[leaf] = make_float4(mn.x, mn.y, mn.z, 0.0f);
            hi[leaf] = make_float4(mx.x, mx.y, mx.z, 0.0f);
        }
    }
    if (tree.levels == 1) return;
    __syncthreads();
    if (threadIdx.x < kFan) {
        mn = s_lo[threadIdx.x];
        mx = s_hi[threadIdx.x];
        box_reduce<kFan>(mn, mx);
        if (threadIdx.x == 0) {
            lo[tree.offset[1] + blockIdx.x] = make_float4(mn.x, mn.y, mn.z, 0.0f);
            hi[tree.offset[1] + blockIdx.x] = make_float4(mx.x, mx.y, mx.z, 0.0f);
        }
    }
}

// The levels above: one block, a warp per box.
__global__ void __launch_bounds__(1024) levels_kernel(KnnTree tree, float4* lo, float4* hi) {
    pdl_begin();
    const int lane = threadIdx.x & 31;
    for (int level = 2; level < tree.levels; ++level) {
        for (int node = threadIdx.x >> 5; node < tree.count[level]; node += 32) {
            float3 mn = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), mx = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
            const int child = node * kFan + lane;
            if (child < tree.count[level - 1]) {
                const float4 a = lo[tree.offset[level - 1] + child], b = hi[tree.offset[level - 1] + child];
                mn = make_float3(a.x, a.y, a.z);
                mx = make_float3(b.x, b.y, b.z);
            }
            box_reduce<kFan>(mn, mx);
            if (lane == 0) {
                lo[tree.offset[level] + node] = make_float4(mn.x, mn.y, mn.z, 0.0f);
                hi[tree.offset[level] + node] = make_float4(mx.x, mx.y, mx.z, 0.0f);
            }
        }
        __syncthreads();  // the block's own global writes are visible to it
    }
}

// Squared distance of the box [plo, phi] (a point when equal) to a node's box.
// Each difference, square and sum is monotonic under rounding, so the distance of
// a box is never above that of a point inside it.
__device__ __forceinline__ float box_distance(float3 plo, float3 phi, float3 lo, float3 hi) {
    const float x = fmaxf(fmaxf(lo.x - phi.x, plo.x - hi.x), 0.0f);
    const float y = fmaxf(fmaxf(lo.y - phi.y, plo.y - hi.y), 0.0f);
    const float z = fmaxf(fmaxf(lo.z - phi.z, plo.z - hi.z), 0.0f);
    return fmaf(z, z, fmaf(y, y, x * x));
}

// Exact squared distance in FP32 without contraction: ((dx*dx + dy*dy) + dz*dz).
__device__ __forceinline__ float sq_distance(float3 p, float x, float y, float z) {
    const float dx = __fsub_rn(p.x, x), dy = __fsub_rn(p.y, y), dz = __fsub_rn(p.z, z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

struct Best3 {
    float d[3];
    int i[3];
    __device__ __forceinline__ void init() {
        d[0] = d[1] = d[2] = FLT_MAX;
        i[0] = i[1] = i[2] = -1;
    }
    __device__ __forceinline__ bool better(float dist, int idx, int k) const {
        return dist < d[k] || (dist == d[k] && (i[k] < 0 || idx < i[k]));
    }
    __device__ __forceinline__ void insert(float dist, int idx) {
        if (!better(dist, idx, 2)) return;
        if (better(dist, idx, 1)) {
            d[2] = d[1];
            i[2] = i[1];
            if (better(dist, idx, 0)) {
                d[1] = d[0];
                i[1] = i[0];
                d[0] = dist;
                i[0] = idx;
            } else {
                d[1] = dist;
                i[1] = idx;
            }
        } else {
            d[2] = dist;
            i[2] = idx;
        }
    }
};

// 32 queries per warp (see the top). A lane whose coordinates are not finite has
// no neighbour (every distance is infinite or NaN) and takes no part in the walk.
__global__ void __launch_bounds__(kQueryThreads) query_kernel(const float4* __restrict__ sorted, int n, KnnTree tree,
                                                              const float4* __restrict__ lo,
                                                              const float4* __restrict__ hi,
                                                              float* __restrict__ mean_dist2,
                                                              int* __restrict__ neighbors) {
    pdl_begin();
    constexpr uint32_t kAll = 0xffffffffu;
    const int rank = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = rank >> 5;
    if (warp * 32 >= n) return;
    float4 me = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (rank < n) me = sorted[rank];
    const float3 p = make_float3(me.x, me.y, me.z);
    const int self = __float_as_int(me.w);
    const bool active = rank < n && isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
    float3 qlo = active ? p : make_float3(FLT_MAX, FLT_MAX, FLT_MAX);
    float3 qhi = active ? p : make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    box_reduce<32>(qlo, qhi);
    Best3 best;
    best.init();
    const int mine = min(32, n - warp * 32);
    for (int k = 0; k < mine; ++k) {
        const float x = __shfl_sync(kAll, p.x, k), y = __shfl_sync(kAll, p.y, k), z = __shfl_sync(kAll, p.z, k);
        const int other = __shfl_sync(kAll, self, k);
        const float d = sq_distance(p, x, y, z);
        if (k != lane && d <= best.d[2]) best.insert(d, other);
    }
    // boxes are pruned against the current third distance widened by a few ulps,
    // so rounding of the box distance can never drop a tying candidate
    float bound = active ? best.d[2] * 1.000004f : -1.0f;
    int level = tree.levels - 1, base = 0;
    uint32_t masks[kMaxLevels];
    int bases[kMaxLevels];
    // this lane's child of `base`'s node at `level`: its box stays in registers, so that
    // testing a child against every lane's point is six shuffles and no load
    float3 clo = make_float3(0.0f, 0.0f, 0.0f), chi = clo;
    auto load_children = [&]() {
        const int child = min(base + lane, tree.count[level] - 1);
        const float4 l = lo[tree.offset[level] + child], h = hi[tree.offset[level] + child];
        clo = make_float3(l.x, l.y, l.z);
        chi = make_float3(h.x, h.y, h.z);
    };
    // the children whose box is within the warp's largest bound of the warp's box
    auto candidates = [&]() {
        load_children();
        const float widest = __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(fmaxf(bound, 0.0f))));
        return __ballot_sync(kAll, base + lane < tree.count[level] && box_distance(qlo, qhi, clo, chi) <= widest);
    };
    uint32_t mask = candidates();
    while (true) {
        if (mask == 0) {
            if (++level >= tree.levels) break;
            mask = masks[level];
            base = bases[level];
            if (mask) load_children();
            continue;
        }
        // the child that holds this warp's own points first: its neighbours tighten the bounds
        const int own = static_cast<int>((static_cast<int64_t>(warp) * 32 / kBucket) >> (5 * level)) - base;
        const int c = own >= 0 && own < kFan && ((mask >> own) & 1u) ? own : __ffs(mask) - 1;
        mask &= ~(1u << c);
        const int node = base + c;
        if (level == 0 && node / (32 / kBucket) == warp) continue;  // the warp's own points, already done
        const float3 l = make_float3(__shfl_sync(kAll, clo.x, c), __shfl_sync(kAll, clo.y, c), __shfl_sync(kAll, clo.z, c));
        const float3 h = make_float3(__shfl_sync(kAll, chi.x, c), __shfl_sync(kAll, chi.y, c), __shfl_sync(kAll, chi.z, c));
        if (!__any_sync(kAll, box_distance(p, p, l, h) <= bound)) continue;
        if (level > 0) {
            masks[level] = mask;
            bases[level] = base;
            --level;
            base = node * kFan;
            mask = candidates();
            continue;
        }
        const int first = node * kBucket;
        float4 q[kBucket];
#pragma unroll
        for (int k = 0; k < kBucket; ++k) q[k] = sorted[min(first + k, n - 1)];
#pragma unroll
        for (int k = 0; k < kBucket; ++k) {
            const float d = sq_distance(p, q[k].x, q[k].y, q[k].z);
            if (first + k < n && d <= best.d[2]) best.insert(d, __float_as_int(q[k].w));
        }
        if (active) bound = best.d[2] * 1.000004f;
    }
    if (rank >= n) return;
    const int found = n - 1 < 3 ? n - 1 : 3;
    float mean = 0.0f;
    if (found == 3) mean = (best.d[0] + best.d[1] + best.d[2]) / 3.0f;
    else if (found == 2) mean = (best.d[0] + best.d[1]) / 2.0f;
    else if (found == 1) mean = best.d[0];
    mean_dist2[self] = mean;
    if (neighbors)
#pragma unroll
        for (int k = 0; k < 3; ++k) neighbors[3ll * self + k] = k < found ? best.i[k] : -1;
}

inline int grid_for(int64_t n) { return static_cast<int>(n > 0 ? (n + kThreads - 1) / kThreads : 1); }

}  // namespace

KnnLayout knn_layout(int n) {
    KnnLayout L;
    const KnnTree tree = knn_tree(n > 0 ? n : 1);
    const size_t boxes = static_cast<size_t>(tree.offset[tree.levels - 1]) + tree.count[tree.levels - 1];
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t at = off;
        off += (bytes + 255) & ~static_cast<size_t>(255);
        return at;
    };
    L.bounds = take(6 * sizeof(unsigned int));
    L.keys = take(sizeof(uint32_t) * static_cast<size_t>(n));
    L.keys_alt = take(sizeof(uint32_t) * static_cast<size_t>(n));
    L.ids = take(sizeof(uint32_t) * static_cast<size_t>(n));
    L.ids_alt = take(sizeof(uint32_t) * static_cast<size_t>(n));
    L.sorted = take(sizeof(float4) * static_cast<size_t>(n));
    L.lo = take(sizeof(float4) * boxes);
    L.hi = take(sizeof(float4) * boxes);
    L.sort = take(radix_sort_scratch_bytes(n));
    L.total = off;
    return L;
}

int launch_knn3(const float* points, int n, float* mean_dist2, int* neighbors, void* workspace, cudaStream_t s) {
    if (n <= 0) return GSN_OK;
    if (n < 2) {
        if (cudaMemsetAsync(mean_dist2, 0, sizeof(float) * n, s) != cudaSuccess) return GSN_ERR_CUDA;
        if (neighbors && cudaMemsetAsync(neighbors, 0xFF, sizeof(int) * 3 * n, s) != cudaSuccess) return GSN_ERR_CUDA;
        return GSN_OK;
    }
    const KnnLayout L = knn_layout(n);
    const KnnTree tree = knn_tree(n);
    char* w = static_cast<char*>(workspace);
    auto* bounds = reinterpret_cast<unsigned int*>(w + L.bounds);
    auto* keys = reinterpret_cast<uint32_t*>(w + L.keys);
    auto* keys_alt = reinterpret_cast<uint32_t*>(w + L.keys_alt);
    auto* ids = reinterpret_cast<uint32_t*>(w + L.ids);
    auto* ids_alt = reinterpret_cast<uint32_t*>(w + L.ids_alt);
    auto* sorted = reinterpret_cast<float4*>(w + L.sorted);
    auto* lo = reinterpret_cast<float4*>(w + L.lo);
    auto* hi = reinterpret_cast<float4*>(w + L.hi);
    if (cudaMemsetAsync(bounds, 0xFF, 6 * sizeof(unsigned int), s) != cudaSuccess) return GSN_ERR_CUDA;
    launch_step(bounds_kernel, grid_for(n), kThreads, 0, s, points, n, bounds);
    launch_step(curve_kernel, grid_for(n), kThreads, 0, s, points, n, bounds, keys);
    int launches = 2;
    bool alt = false;
    RadixSortScratch scratch = radix_sort_scratch(w + L.sort);
    int st = launch_radix_sort(keys, ids, keys_alt, ids_alt, true, n, nullptr, 0, 30, scratch, &alt, s);
    if (st != GSN_OK) return st;
    const uint32_t* order = alt ? ids_alt : ids;
    launch_step(leaves_kernel, grid_for(n), kThreads, 0, s, points, order, n, tree, sorted, lo, hi);
    ++launches;
    if (tree.levels > 2) {
        launch_step(levels_kernel, 1, 1024, 0, s, tree, lo, hi);
        ++launches;
    }
    launch_step(query_kernel, static_cast<int>((static_cast<int64_t>(n) + kQueryThreads - 1) / kQueryThreads),
                kQueryThreads, 0, s, sorted, n, tree, lo, hi, mean_dist2, neighbors);
    ++launches;
    return launched(launches);
}

}  // namespace gsn
