// (d) Analytic backward of the per-tile blend.
//
// One warp per 16x16 tile, eight pixels per lane as four packed pairs, replaying the
// tile's records front to back against each pixel's final colour like the reference
// (solver.cu:325-466), with these changes:
//   * the take set is the forward pass's: records [0, limit) of a tile hold every
//     record a pixel took (limit = the per-pixel contributor count the forward
//     records), so a pixel takes record idx when idx < limit and the per-pixel alpha
//     test passes; the transmittance stop needs no replay;
//   * only the records some pixel of the tile took (the forward's take flags) are
//     visited, in batches of 32 staged in shared memory;
//   * a lane sums the contributions of its eight pixels in registers, so one warp
//     reduction serves 256 pixel-record pairs; pixels are evaluated branch-free (a
//     pixel that does not take a record gets alpha = 0, which zeroes its terms) in
//     packed FP32x2 arithmetic (one instruction per two operations, each half rounded
//     as its scalar form), so their dependency chains interleave;
//   * the 11 per-record values are summed over the lanes through shared memory: each
//     lane stores its shares as a column, and after every second record 22 lanes add
//     one row of 32 each (eight 16-byte loads), about 27 instructions per record where
//     a butterfly reduce-scatter takes 55; the sums leave with three 16-byte vector
//     reductions per record;
//   * the colour term of dL/dalpha is carried per pixel as one scalar: the
//     gradient-weighted colour in front of the record minus the gradient-weighted
//     final colour;
//   * per-record factors leave the per-pixel loop: d(cov a) and d(cov c) are
//     accumulated without the power's factor 1/2 and d(opacity logit) without the
//     sigmoid's (1 - o), applied once per record before the reduction;
//   * the fast form evaluates alpha as ex2 of the power in log2 units with the opacity
//     folded in (two FMAs, one MUFU per pixel; raster_common.cuh fast_record), takes a
//     pixel on one compare and divides by (1 - alpha) through the hardware reciprocal;
//     the exact form keeps the reference's power expression, expf and the correctly
//     rounded reciprocal;
//   * where the frame has few tiles (the forward wrote checkpoints: T and the colour of
//     every pixel after each kSegment records of its tile), a tile's list is cut into
//     segments that run as independent warps, each starting from its checkpoint: kSegment
//     records each where they are enough for the list, equal shares of whole kSegments
//     where it is longer. A serial walk per tile left 11 warps per SM on 1,700 tiles of
//     800 records, and the longest list decided the time; with the rest of a longer list
//     on the last warp, 100k faint Gaussians on 250x180 took 14,080 us in the exact form
//     (two warps per tile: 12,990) instead of 2,484;
//   * a segment is a warp's whole work (a loop over segments made the compiler hold every
//     pixel's inputs across it: 168 registers, or spills at 128, and 25 % more time).
//   * the exact form skips the pairs of a quadrant that the record's ellipse does not
//     reach (93 -> 67 us at 4,096 Gaussians and 128x128, neutral at 1.2M); in the fast
//     form the branches cost more than the skipped arithmetic (468 -> 506 us at 3.0M).
// Bound by instruction issue at 16 warps per SM (116 registers). Exact form at 1.2M
// Gaussians and 1600x1064 602 -> 582 us, at 4,096 and 128x128 130 -> 67 us; fast form at
// 3.0M and 2048x1360 487 -> 468 us, at 100k and 800x532 320 -> 260 us.
// Per-Gaussian output (12 floats, Gaussian-major): d(u, v), d(cov a, b, c),
// d(opacity logit), d(r, g, b), sum|du|, sum|dv|, 0.
#include <algorithm>

#include "raster_common.cuh"
#include "kernels.h"

namespace gsn {

namespace {

constexpr int kVals = 12;
constexpr int kFields = 11;     // values of a record that are not padding
constexpr int kSumRow = 36;     // a value's 32 lanes, padded: rows 16 bytes apart in the banks
constexpr int kPairs = 4;       // pixel pairs per lane

// Where pair h of a lane lies in the tile. Exact form: one pair in each 8x8 quadrant,
// so that a quadrant out of a record's reach is a pair to skip; fast form: four pairs
// down one column, which share the column's terms.
template <bool kFast>
struct PairLayout {
    static __device__ __forceinline__ int lane_x(int lane) { return kFast ? lane & 15 : lane & 7; }
    static __device__ __forceinline__ int lane_y(int lane) { return kFast ? lane >> 4 : lane >> 3; }
    static __device__ __forceinline__ constexpr int column(int h) { return kFast ? 0 : 8 * (h & 1); }
    static __device__ __forceinline__ constexpr int row(int h) { return kFast ? 4 * h : 8 * (h >> 1); }
    static constexpr int kStep = kFast ? 2 : 4;  // between the pair's two rows
};
constexpr int kBatch = 32;      // records staged per batch (one per lane)

template <bool kFast>
__global__ void __launch_bounds__(32, 16) raster_backward_kernel(RasterBackwardArgs a) {
    pdl_begin();
    __shared__ uint32_t s_id[kBatch];
    __shared__ float2 s_mean[kBatch];
    __shared__ float4 s_conic[kBatch];
    __shared__ float4 s_aux[kBatch];  // fast form: fast_record terms; exact form: the alpha floor in x
    __shared__ float3 s_color[kBatch];
    __shared__ __align__(16) float s_acc[kBatch * kVals];
    __shared__ __align__(16) float s_sum[2 * kFields * kSumRow];

    const int lane = threadIdx.x;
    const int tile = blockIdx.x;
    const int64_t begin = a.tile_offsets[tile];
    // records [0, bound) hold every record a pixel of the tile took; within the tile's
    // list also where the camera has tiles that the last frame had not, whose bounds and
    // offsets are of different frames
    const int bound = static_cast<int>(
        min(static_cast<int64_t>(a.tile_bounds[tile]), a.tile_offsets[tile + 1] - begin));
    // this warp's segment of it: kSegment records, or an equal share of whole kSegments
    // where the list is longer than those. The reduction of equal values tells the compiler
    // that they are equal: with `from` in a uniform register the kernel takes 116 registers
    // instead of 126, with which the exact form is 3 % slower
    const int span = kSegment * static_cast<int>(gridDim.y);
    int length = kSegment;
    if (bound > span) length = kSegment * ((bound + span - 1) / span);
    length = __reduce_max_sync(0xffffffffu, length);
    const int from = static_cast<int>(blockIdx.y) * length;
    if (from >= bound) return;
    const int to = min(bound, from + length);
    const int tx = tile % a.cam.tile_count_x, ty = tile / a.cam.tile_count_x;
    using Layout = PairLayout<kFast>;
    const int x0 = tx * kTile + Layout::lane_x(lane), y0 = ty * kTile + Layout::lane_y(lane);
    const float fx0 = static_cast<float>(x0), ny0 = -static_cast<float>(y0);
    for (int k = lane; k < kBatch; k += 32) s_acc[k * kVals + 11] = 0.0f;  // the padding slot

    // per pixel pair: T, P - S (P = dL/dcolour . colour in front of the
    // record, S = dL/dcolour . final colour) and dL/dcolour
    float2 T2[kPairs], P2[kPairs], gI2[kPairs][3];
    int limit[2 * kPairs];
    const float4* checkpoint = nullptr;
    if (from > 0) checkpoint = a.checkpoints + checkpoint_slot(begin, from) * kTilePixels;
#pragma unroll
    for (int p = 0; p < 2 * kPairs; ++p) {
        const int px = x0 + Layout::column(p >> 1), py = y0 + Layout::row(p >> 1) + Layout::kStep * (p & 1);
        float gi[3] = {0.0f, 0.0f, 0.0f};
        float S = 0.0f, T = 1.0f, P = 0.0f;
        limit[p] = 0;
        if (px < a.cam.width && py < a.cam.height) {
            const int64_t pix = static_cast<int64_t>(py) * a.cam.width + px;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                gi[c] = a.image_grad[pix * 3 + c];
                S += gi[c] * a.image[pix * 3 + c];
            }
            limit[p] = a.contributors[pix];
            if (checkpoint) {
                const float4 state = checkpoint[(py - ty * kTile) * kTile + px - tx * kTile];
                T = state.x;
                P = gi[0] * state.y + gi[1] * state.z + gi[2] * state.w;
            }
        }
        const int h = p >> 1;
        if (p & 1) {
            P2[h].y = P - S;
            T2[h].y = T;
#pragma unroll
            for (int c = 0; c < 3; ++c) gI2[h][c].y = gi[c];
        } else {
            P2[h].x = P - S;
            T2[h].x = T;
#pragma unroll
            for (int c = 0; c < 3; ++c) gI2[h][c].x = gi[c];
        }
    }
    for (int rel = from; rel < to; rel += kBatch) {
        const int batch = min(kBatch, to - rel);
        // stage one record per lane; the quadrants that a record some pixel of the tile
        // took in the forward pass can reach become four ballots (the fast form: all four)
        bool flag[kPairs] = {};
        if (lane < batch) {
            const int64_t r = begin + rel + lane;
            const uint32_t id = __ldg(a.tile_ids + r);
            s_id[lane] = id;
            const float2 mean = __ldg(a.means + id);
            const float4 q = __ldg(a.conic_opacity + id);
            s_mean[lane] = mean;
            s_conic[lane] = q;
            const float* c = reinterpret_cast<const float*>(a.colors) + 3ull * id;
            s_color[lane] = make_float3(__ldg(c), __ldg(c + 1), __ldg(c + 2));
            s_aux[lane] = kFast ? fast_record(q) : make_float4(alpha_floor(q.w), 0.0f, 0.0f, 0.0f);
            if (((a.record_warps[r >> 5] | a.record_warps[a.record_words + (r >> 5)]) >> (r & 31)) & 1u) {
                const float limit_q = cull_limit(mean, q);
#pragma unroll
                for (int h = 0; h < kPairs; ++h) {
                    const float qx = static_cast<float>(tx * kTile + 8 * (h & 1));
                    const float qy = static_cast<float>(ty * kTile + 8 * (h >> 1));
                    flag[h] = kFast || region_hit(mean, q.x, 2.0f * q.y, q.z, limit_q, qx, qx + 7.0f, qy, qy + 7.0f);
                }
            }
        }
        uint32_t reach[kPairs];
#pragma unroll
        for (int h = 0; h < kPairs; ++h) reach[h] = __ballot_sync(0xffffffffu, flag[h]);
        uint32_t m = (reach[0] | reach[1]) | (reach[2] | reach[3]);
        const uint32_t taken = m;
        __syncwarp();
        int parity = 0, previous = 0;
        while (m) {
            const uint32_t bit = m & (0u - m);
            m ^= bit;
            const int j = 31 - __clz(bit);
            const int idx = rel + j;
            const float2 mu = s_mean[j];
            const float4 q = s_conic[j];
            const float3 col = s_color[j];
            const float4 aux = s_aux[j];
            const float2 m1 = pk(-1.0f), one = pk(1.0f);
            float2 acc[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) acc[i] = pk(0.0f);
            float abs_u = 0.0f, abs_v = 0.0f;
#pragma unroll
            for (int h = 0; h < kPairs; ++h) {
                if (!kFast && !(reach[h] & bit)) continue;  // the same for every lane
                const float dx = mu.x - (fx0 + static_cast<float>(Layout::column(h)));
                const float qxdx = q.x * dx, qydx = q.y * dx;
                // -y of the pair's pixels, exact in fp32
                const float2 ny = add2(pk(ny0), make_float2(-static_cast<float>(Layout::row(h)),
                                                            -static_cast<float>(Layout::row(h) + Layout::kStep)));
                const float2 dy = add2(pk(mu.y), ny);
                float2 alpha;
                if constexpr (kFast) {
                    const float Ax = fmaf(aux.x * dx, dx, aux.w), Bx = aux.y * dx;
                    const float2 pw2 = fma2(fma2(pk(aux.z), dy, pk(Bx)), dy, pk(Ax));
                    const bool take0 = idx < limit[2 * h] && pw2.x >= kLog2AlphaMin;
                    const bool take1 = idx < limit[2 * h + 1] && pw2.y >= kLog2AlphaMin;
                    alpha.x = take0 ? fminf(kAlphaMax, ex2_approx(pw2.x)) : 0.0f;
                    alpha.y = take1 ? fminf(kAlphaMax, ex2_approx(pw2.y)) : 0.0f;
                } else {
                    const Power power(q, dx);
                    const float pw0 = power.at(dy.x), pw1 = power.at(dy.y);
                    const float raw0 = gaussian_weight(q.w, pw0);
                    const float raw1 = gaussian_weight(q.w, pw1);
                    const bool take0 = idx < limit[2 * h] && !(pw0 > 0.0f) && !(pw0 < aux.x) &&
                                       !(raw0 < kAlphaMin);
                    const bool take1 = idx < limit[2 * h + 1] && !(pw1 > 0.0f) && !(pw1 < aux.x) &&
                                       !(raw1 < kAlphaMin);
                    alpha.x = take0 ? fminf(kAlphaMax, raw0) : 0.0f;
                    alpha.y = take1 ? fminf(kAlphaMax, raw1) : 0.0f;
                }
                // d alpha / d power: raw below the clamp, 0 when clamped or not taken
                const float2 r = make_float2(alpha.x < kAlphaMax ? alpha.x : 0.0f,
                                             alpha.y < kAlphaMax ? alpha.y : 0.0f);
                const float2 w = mul2(alpha, T2[h]);
                const float2 om = fma2(alpha, m1, one);  // 1 - alpha
                const float2 inv = make_float2(one_over<kFast>(om.x), one_over<kFast>(om.y));
                float2 G = mul2(gI2[h][0], pk(col.x));
                G = fma2(gI2[h][1], pk(col.y), G);
                G = fma2(gI2[h][2], pk(col.z), G);
                // dL/dalpha = (dL/dC . (colour in front + T c - final)) / (1 - alpha)
                const float2 dalpha = mul2(fma2(T2[h], G, P2[h]), inv);
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[6 + c] = fma2(w, gI2[h][c], acc[6 + c]);
                const float2 common = mul2(dalpha, r);
                const float2 qx = fma2(pk(q.y), dy, pk(qxdx));
                const float2 qy = fma2(pk(q.z), dy, pk(qydx));
                const float2 cqx = mul2(common, qx), cqy = mul2(common, qy);
                acc[0] = fma2(cqx, m1, acc[0]);
                acc[1] = fma2(cqy, m1, acc[1]);
                acc[2] = fma2(cqx, qx, acc[2]);  // halved once per record below
                acc[3] = fma2(cqx, qy, acc[3]);
                acc[4] = fma2(cqy, qy, acc[4]);  // halved once per record below
                acc[5] = add2(acc[5], common);   // times (1 - o) once per record below
                abs_u += fabsf(cqx.x) + fabsf(cqx.y);
                abs_v += fabsf(cqy.x) + fabsf(cqy.y);
                P2[h] = fma2(w, G, P2[h]);
                // T (1 - alpha): the forward's expression in each form (unchanged at alpha = 0)
                T2[h] = kFast ? fma2(w, m1, T2[h]) : mul2(T2[h], om);
            }
            // this lane's share of the record's 11 values, into the columns of
            // s_sum: d(cov a) and d(cov c) carry the factor 1/2 of the power,
            // the opacity logit the sigmoid's derivative o (1 - o) / o (exact)
            float* column = s_sum + parity * (kFields * kSumRow) + lane;
            column[0 * kSumRow] = acc[0].x + acc[0].y;
            column[1 * kSumRow] = acc[1].x + acc[1].y;
            column[2 * kSumRow] = 0.5f * (acc[2].x + acc[2].y);
            column[3 * kSumRow] = acc[3].x + acc[3].y;
            column[4 * kSumRow] = 0.5f * (acc[4].x + acc[4].y);
            column[5 * kSumRow] = (1.0f - q.w) * (acc[5].x + acc[5].y);
            column[6 * kSumRow] = acc[6].x + acc[6].y;
            column[7 * kSumRow] = acc[7].x + acc[7].y;
            column[8 * kSumRow] = acc[8].x + acc[8].y;
            column[9 * kSumRow] = abs_u;
            column[10 * kSumRow] = abs_v;
            // every second record (and at the batch's last): one lane per value adds
            // the 32 lanes' shares
            if (parity == 0 && m) {
                previous = j;
                parity = 1;
                continue;
            }
            __syncwarp();
            if (lane < kFields * (parity + 1)) {
                const float4* row = reinterpret_cast<const float4*>(s_sum + lane * kSumRow);
                float2 even = pk(0.0f), odd = pk(0.0f);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 x = row[i];
                    even = add2(even, make_float2(x.x, x.y));
                    odd = add2(odd, make_float2(x.z, x.w));
                }
                even = add2(even, odd);
                // rows 0..10 hold the pair's first record, 11..21 its second
                const int slot = parity == 1 && lane < kFields ? previous : j;
                s_acc[slot * kVals + (lane < kFields ? lane : lane - kFields)] = even.x + even.y;
            }
            parity = 0;
            __syncwarp();
        }
        for (int k = lane; k < kBatch * (kVals / 4); k += 32) {
            const int j = k / (kVals / 4);
            if ((taken >> j) & 1u)
                red_add_v4(a.grad_out + static_cast<int64_t>(s_id[j]) * kVals + 4 * (k % (kVals / 4)),
                           reinterpret_cast<const float4*>(s_acc)[k]);
        }
        __syncwarp();
    }
}

}  // namespace

int launch_raster_backward(const RasterBackwardArgs& a, cudaStream_t stream) {
    int64_t tiles = static_cast<int64_t>(a.cam.tile_count_x) * a.cam.tile_count_y;
    if (tiles <= 0) return GSN_OK;
    if (!a.contributors || !a.tile_bounds || !a.record_warps || (reinterpret_cast<uintptr_t>(a.grad_out) & 15) != 0)
        return GSN_ERR_INVALID_ARGUMENT;
    // warps per tile: enough to fill the GPU (one whose segment lies past the tile's
    // bound leaves at once), at least four at kCheckpointTiles
    static_assert(kSegmentWarps / kCheckpointTiles >= 2, "a frame with checkpoints has segments");
    const int64_t parts = a.checkpoints ? std::min<int64_t>(16, kSegmentWarps / tiles) : 1;
    const dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(parts));
    if (a.fast) launch_step(raster_backward_kernel<true>, grid, 32, 0, stream, a);
    else launch_step(raster_backward_kernel<false>, grid, 32, 0, stream, a);
    return launched(1);
}

}  // namespace gsn
