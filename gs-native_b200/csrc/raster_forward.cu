// (c) Per-tile front-to-back alpha blending.
//
// One CTA of 128 threads per 16x16 tile, one warp per 8x8 quadrant and two pixels
// per lane (four rows apart). The tile's sorted records are staged into shared
// memory in batches of 128, one per thread; while a batch is blended every thread
// already holds its slot of the next one in registers, so the id -> record gather
// overlaps the blend.
//
// Per batch each warp tests the records against its quadrant (raster_common.cuh
// region_hit: can the record's alpha >= 1/255 ellipse reach it?) with four ballots
// and walks only the set bits, in order; per pixel, powers below the record's alpha
// floor are rejected before expf. Both tests only drop evaluations the exact
// per-pixel test would have skipped, so the result is unchanged. A CTA stops as
// soon as all of its pixels are saturated.
//
// The loop is bound by instruction issue (83 % of the slots), so what counts is the
// pixel slots evaluated per pair taken - 1.91 with 16x8 strips and the ellipse's
// bounding box, 1.29 with 8x8 quadrants and the ellipse at 1.2M Gaussians and
// 1600x1064, 3.07 and 1.93 at 300k and 979x546 - and the instructions of a visit: the
// walk is the same for every lane (no per-lane exit), a record is three shared loads
// at one address, and the records a pixel took are kept as one bit mask per 32. Four
// warps per tile also shorten the serial walk of a long list where the frame has few
// tiles. Exact form at 1.2M 370 -> 272 us, fast form at 3.0M and 2048x1360 321 -> 290
// us, at 100k and 800x532 197 -> 140 us, exact at 4,096 and 128x128 63 -> 23 us.
//
// The exact form evaluates the per-pixel arithmetic (power, alpha clamp at
// 0.99, the 1/255 skip and the 1e-4 transmittance stop) exactly as the
// reference does (renderer.cu:273-338), so images are bit-identical for
// identical inputs. The fast form takes alpha as ex2 of the power in log2
// units with the opacity folded in (raster_common.cuh fast_record: two FMAs and
// one MUFU per pixel, one compare for the 1/255 test) and updates the
// transmittance as T - alpha T; every pixel is evaluated branch-free. Besides the
// image the kernel records, per pixel, how many records were consumed up to its
// last contribution; the backward pass takes its replay's take set from it.
// A counting variant (RasterForwardArgs::pair_count) also sums the pairs taken.
#include "raster_common.cuh"
#include "kernels.h"

namespace gsn {

namespace {

// A record as it is staged: 48 bytes, so one address serves its three shared loads,
// and 16-byte loads of consecutive records by consecutive lanes meet no bank twice.
struct Record {
    float2 mean;
    float2 color_rg;
    float4 conic;     // exact form: conic + opacity; fast form: fast_record terms
    float color_b;
    float floor;      // exact form: the alpha floor
    float limit;      // cull_limit, in the units of `conic`
    float unused;
};
static_assert(sizeof(Record) == 48, "three 16-byte words");

struct Fetched {
    float2 mean;
    float4 conic;
    float3 color;
};

__device__ __forceinline__ Fetched fetch(const RasterForwardArgs& a, int64_t r, int64_t end) {
    Fetched s;
    if (r < end) {
        uint32_t id = __ldg(a.tile_ids + r);
        s.mean = __ldg(a.means + id);
        s.conic = __ldg(a.conic_opacity + id);
        const float* c = reinterpret_cast<const float*>(a.colors) + 3ull * id;
        s.color = make_float3(__ldg(c), __ldg(c + 1), __ldg(c + 2));
    } else {
        s.mean = make_float2(0.f, 0.f);
        s.conic = make_float4(0.f, 0.f, 0.f, 0.f);
        s.color = make_float3(0.f, 0.f, 0.f);
    }
    return s;
}

template <bool kFast>
__device__ __forceinline__ void stage(const Fetched& f, Record* dst) {
    const float limit = cull_limit(f.mean, f.conic);
    float4* out = reinterpret_cast<float4*>(dst);
    out[0] = make_float4(f.mean.x, f.mean.y, f.color.x, f.color.y);
    out[1] = kFast ? fast_record(f.conic) : f.conic;
    out[2] = make_float4(f.color.z, kFast ? 0.0f : alpha_floor(f.conic.w), kFast ? limit * (0.5f * kLog2e) : limit, 0.0f);
}

constexpr int kForwardWarps = 4;
constexpr int kForwardThreads = 32 * kForwardWarps;
constexpr int kForwardPix = kTilePixels / kForwardThreads;  // rows y0 + 4p of the warp's quadrant
static_assert(kRasterBatch == kForwardThreads, "one staged record per thread");

template <bool kFast, bool kCount>
__global__ void __launch_bounds__(kForwardThreads) raster_forward_kernel(RasterForwardArgs a) {
    pdl_begin();
    __shared__ __align__(16) Record s_rec[kRasterBatch];
    __shared__ int s_bound;

    const int t = threadIdx.x;
    const int lane = t & 31;
    const int warp = t >> 5;
    const int tile = blockIdx.x;
    const int qx = (tile % a.cam.tile_count_x) * kTile + 8 * (warp & 1);
    const int qy = (tile / a.cam.tile_count_x) * kTile + 8 * (warp >> 1);
    const float sx0 = static_cast<float>(qx), sx1 = sx0 + 7.0f;
    const float sy0 = static_cast<float>(qy), sy1 = sy0 + 7.0f;
    const int px = qx + (lane & 7), py0 = qy + (lane >> 3);
    const float fx = static_cast<float>(px);
    float fy[kForwardPix];
    bool done[kForwardPix];
    float T[kForwardPix];
    float3 C[kForwardPix];
    int consumed[kForwardPix];
    unsigned int pairs = 0;  // kCount: pairs this thread's pixels took
#pragma unroll
    for (int p = 0; p < kForwardPix; ++p) {
        fy[p] = static_cast<float>(py0 + 4 * p);
        done[p] = !(px < a.cam.width && py0 + 4 * p < a.cam.height);
        T[p] = 1.0f;
        C[p] = make_float3(0.f, 0.f, 0.f);
        consumed[p] = 0;
    }

    const int64_t begin = a.tile_offsets[tile];
    const int64_t end = a.tile_offsets[tile + 1];
    // the take flags' plane of this warp's half of the tile (rows 0-7 or 8-15)
    uint32_t* plane = a.record_warps ? a.record_warps + (warp >> 1) * a.record_words : nullptr;

    Fetched next = fetch(a, begin + t, end);
    for (int64_t base = begin; base < end; base += kRasterBatch) {
        bool mine = true;
#pragma unroll
        for (int p = 0; p < kForwardPix; ++p) mine = mine && done[p];
        if (__syncthreads_and(mine)) break;
        if (a.checkpoints && base > begin) {
            float4* state =
                a.checkpoints + checkpoint_slot(begin, static_cast<int>(base - begin)) * kTilePixels;
            const int in_tile = (8 * (warp >> 1) + (lane >> 3)) * kTile + 8 * (warp & 1) + (lane & 7);
#pragma unroll
            for (int p = 0; p < kForwardPix; ++p)
                state[in_tile + 4 * p * kTile] = make_float4(T[p], C[p].x, C[p].y, C[p].z);
        }
        stage<kFast>(next, s_rec + t);
        __syncthreads();
        next = fetch(a, base + kRasterBatch + t, end);
        const int batch = static_cast<int>(min(static_cast<int64_t>(kRasterBatch), end - base));
        const int rel = static_cast<int>(base - begin);
#pragma unroll 1
        for (int k = 0; k < kRasterBatch / 32; ++k) {
            const int jl = k * 32 + lane;
            bool hit = jl < batch;
            if (hit) {
                const Record& c = s_rec[jl];
                const float4 q = c.conic;
                hit = kFast ? region_hit(c.mean, -q.x, -q.y, -q.z, c.limit, sx0, sx1, sy0, sy1)
                            : region_hit(c.mean, q.x, 2.0f * q.y, q.z, c.limit, sx0, sx1, sy0, sy1);
            }
            uint32_t m = __ballot_sync(0xffffffffu, hit);
            if (__all_sync(0xffffffffu, done[0] && done[1])) break;
            // records of this chunk that each pixel took, one bit each
            uint32_t took[kForwardPix] = {};
            while (m) {  // the same for every lane
                const uint32_t bit = m & (0u - m);
                m ^= bit;
                const Record& c = s_rec[k * 32 + 31 - __clz(bit)];
                const float4 head = reinterpret_cast<const float4*>(&c)[0];
                const float4 q = c.conic;
                const float dx = head.x - fx;
                const float cb = c.color_b;
                // every pixel is evaluated branch-free, so the dependency chains
                // interleave; one that does not take the record changes nothing
                if constexpr (kFast) {
                    // fast_record terms (raster_common.cuh), the same expressions as
                    // the fast backward; scalar arithmetic: this loop is bound by the
                    // ALU pipe, which the register moves of packed pairs would load
                    // further
                    const float Ax = fmaf(q.x * dx, dx, q.w), Bx = q.y * dx;
#pragma unroll
                    for (int p = 0; p < kForwardPix; ++p) {
                        const float dy = head.y - fy[p];
                        const float pw2 = fmaf(fmaf(q.z, dy, Bx), dy, Ax);
                        const bool take = !done[p] && pw2 >= kLog2AlphaMin;
                        const float alpha = take ? fminf(kAlphaMax, ex2_approx(pw2)) : 0.0f;
                        float w = alpha * T[p];
                        // a live pixel's T stays >= 1e-4, so only a taken record can
                        // stop it, and a pixel that was already done has w = 0: the
                        // updated done flag alone decides whether w counts
                        done[p] = done[p] || T[p] - w < kTransmittanceMin;
                        w = done[p] ? 0.0f : w;
                        C[p].x = fmaf(head.z, w, C[p].x);
                        C[p].y = fmaf(head.w, w, C[p].y);
                        C[p].z = fmaf(cb, w, C[p].z);
                        T[p] -= w;  // T (1 - alpha) as T - alpha T; unchanged at the stop
                        // alpha >= 1/255 and T >= 1e-4 make a taken record's w > 0
                        if (w > 0.0f) took[p] |= bit;
                    }
                } else {
                    const float lim = c.floor;
                    const Power power(q, dx);
#pragma unroll
                    for (int p = 0; p < kForwardPix; ++p) {
                        const float pw = power.at(head.y - fy[p]);
                        const bool act = !done[p] && !(pw > 0.0f) && !(pw < lim);
                        const float alpha = fminf(kAlphaMax, gaussian_weight(q.w, pw));
                        bool take = act && !(alpha < kAlphaMin);
                        const float nextT = T[p] * (1.0f - alpha);
                        const bool stop = take && nextT < kTransmittanceMin;
                        done[p] = done[p] || stop;
                        take = take && !stop;
                        const float w = alpha * T[p];
                        if (take) {
                            C[p].x = fmaf(head.z, w, C[p].x);
                            C[p].y = fmaf(head.w, w, C[p].y);
                            C[p].z = fmaf(cb, w, C[p].z);
                            T[p] = nextT;
                            took[p] |= bit;
                        }
                    }
                }
            }
#pragma unroll
            for (int p = 0; p < kForwardPix; ++p) {
                if (took[p]) consumed[p] = rel + k * 32 + 32 - __clz(took[p]);
                if (kCount) pairs += __popc(took[p]);
            }
            if (plane) {
                // this quadrant's take flags of the chunk's 32 records, one bit
                // each, into the plane at the records' global positions
                const uint32_t any = __reduce_or_sync(0xffffffffu, took[0] | took[1]);
                if (lane == 0 && any) {
                    const int64_t r0 = base + k * 32;
                    const int off = static_cast<int>(r0 & 31);
                    atomicOr(plane + (r0 >> 5), any << off);
                    // only where a flag falls there: past the last record the word may not exist
                    const uint32_t over = off ? any >> (32 - off) : 0u;
                    if (over) atomicOr(plane + (r0 >> 5) + 1, over);
                }
            }
        }
    }
    if (a.tile_bounds) {
        int most = 0;
#pragma unroll
        for (int p = 0; p < kForwardPix; ++p) most = max(most, consumed[p]);
        most = __reduce_max_sync(0xffffffffu, most);
        if (t == 0) s_bound = 0;
        __syncthreads();
        if (lane == 0) atomicMax(&s_bound, most);
        __syncthreads();
        if (t == 0) a.tile_bounds[tile] = s_bound;
    }
    if (kCount) {
        const unsigned long long warp_pairs = __reduce_add_sync(0xffffffffu, pairs);
        if (lane == 0 && warp_pairs) atomicAdd(a.pair_count, warp_pairs);
    }
#pragma unroll
    for (int p = 0; p < kForwardPix; ++p) {
        if (!(px < a.cam.width && py0 + 4 * p < a.cam.height)) continue;
        const int64_t pix = static_cast<int64_t>(py0 + 4 * p) * a.cam.width + px;
        float* out = a.image + pix * 3;
        out[0] = C[p].x + T[p] * a.background.x;
        out[1] = C[p].y + T[p] * a.background.y;
        out[2] = C[p].z + T[p] * a.background.z;
        if (a.final_transmittance) a.final_transmittance[pix] = T[p];
        if (a.contributors) a.contributors[pix] = consumed[p];
    }
}

}  // namespace

size_t checkpoint_blocks(int64_t records) { return static_cast<size_t>(records) / kSegment; }

int launch_raster_forward(const RasterForwardArgs& a, cudaStream_t stream) {
    int64_t tiles = static_cast<int64_t>(a.cam.tile_count_x) * a.cam.tile_count_y;
    if (tiles <= 0) return GSN_OK;
    const unsigned grid = static_cast<unsigned>(tiles);
    if (a.pair_count) {
        if (a.fast) launch_step(raster_forward_kernel<true, true>, grid, kForwardThreads, 0, stream, a);
        else launch_step(raster_forward_kernel<false, true>, grid, kForwardThreads, 0, stream, a);
    } else if (a.fast) {
        launch_step(raster_forward_kernel<true, false>, grid, kForwardThreads, 0, stream, a);
    } else {
        launch_step(raster_forward_kernel<false, false>, grid, kForwardThreads, 0, stream, a);
    }
    return launched(1);
}

}  // namespace gsn
