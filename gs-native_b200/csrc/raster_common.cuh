// Shared pieces of the forward and backward tile kernels.
#pragma once

#include "common.cuh"

namespace gsn {

constexpr int kRasterBatch = 128;  // records the forward stages at a time

// Frames with few tiles: the forward writes every pixel's transmittance and colour
// after each kSegment records of its tile, so that the backward pass can run the
// segments of a long list side by side.
constexpr int kSegment = 128;      // a batch of the forward pass
constexpr int kSegmentWarps = 16384;  // warps a segmented launch aims at (7 times 148 SMs x 16 resident, about)
static_assert(kSegment == kRasterBatch, "checkpoints are written between batches");

// Where the checkpoint before record `at` (a positive multiple of kSegment) of a tile's
// list lies, in blocks of 256 pixels. Each stands for a record, of which a tile's next is
// kSegment further on; the next tile begins behind all of them and starts with a stride
// of its own, so no two share a slot, and the last one is below records / kSegment.
__device__ __forceinline__ int64_t checkpoint_slot(int64_t tile_begin, int at) {
    return tile_begin / kSegment + at / kSegment - 1;
}

// Which records can matter to a rectangle of pixels. With conic (A, B, C) and
// opacity o, alpha >= 1/255 needs q(d) = A dx^2 + 2 B dx dy + C dy^2 <= 2 ln(255 o).
// The bound is widened (by 2 %, 0.05 and a term in the conic's condition number
// kappa) for the rounding of the per-pixel float evaluation, which can reach a few
// ulps of A dx^2 + C dy^2 (up to ~kappa q), so a culled record is one the exact
// per-pixel test would have skipped for every pixel of the rectangle: culling never
// changes a result.
//
// The widened bound: negative for a record that can never pass (255 o <= 1),
// infinite for a degenerate or non-finite one.
__device__ __forceinline__ float cull_limit(float2 mean, float4 q) {
    const float inf = __int_as_float(0x7f800000);
    const float lo = 255.0f * q.w;
    if (!(lo > 1.0f)) return -1.0f;
    const float det = q.x * q.z - q.y * q.y;
    const float tr = 0.5f * (q.x + q.z);
    const float disc = sqrtf(fmaxf(tr * tr - det, 0.0f));
    const float kappa = (tr + disc) / fmaxf(tr - disc, 1e-30f);
    float Q = 2.0f * __logf(lo) * (1.02f + 1e-6f * kappa) + 0.05f;
    if (!(q.x > 0.0f) || !(q.z > 0.0f) || !(det > 0.0f) || !(kappa < 1e5f) || !isfinite(mean.x) || !isfinite(mean.y))
        Q = inf;
    return Q;
}

// Can a record reach alpha >= 1/255 at a pixel of [x0, x1] x [y0, y1]? The ellipse
// form a dx^2 + b dx dy + c dy^2 takes its minimum over the rectangle at the mean,
// where that lies inside, and else on one of the (at most two) edges that face it:
// on each at the clamped point of the line of smallest q for a fixed dx (slope
// -b / 2c) or a fixed dy. Both candidates are values at points of the rectangle, so
// their minimum is the minimum over it (an approximate slope moves it in the second
// order only). limit is the bound in the units of (a, b, c); its widening covers the
// rounding here too, which stays a few ulps of kappa q. NaN counts as reached. Tighter than the bounding box of the ellipse:
// at 1.2M Gaussians and 1600x1064 a 16x8 strip visits 217 records per tile instead
// of 284 (208 of them are taken by a pixel), an 8x8 quadrant 384 instead of 517.
__device__ __forceinline__ bool region_hit(float2 mean, float a, float b, float c, float limit, float x0,
                                           float x1, float y0, float y1) {
    const float lx = x0 - mean.x, hx = x1 - mean.x, ly = y0 - mean.y, hy = y1 - mean.y;
    const float dx = fminf(fmaxf(0.0f, lx), hx), dy = fminf(fmaxf(0.0f, ly), hy);
    const float slope_y = __fdividef(-0.5f * b, c), slope_x = __fdividef(-0.5f * b, a);
    const float ey = fminf(fmaxf(slope_y * dx, ly), hy), ex = fminf(fmaxf(slope_x * dy, lx), hx);
    const float q1 = fmaf(fmaf(c, ey, b * dx), ey, a * dx * dx);
    const float q2 = fmaf(fmaf(a, ex, b * dy), ex, c * dy * dy);
    return !(fminf(q1, q2) > limit);
}

// Power below which alpha = min(0.99, o * expf(power)) is certainly < 1/255:
// power < -ln(255 o) - 1e-3 gives o * e^power < e^-0.001 / 255, a relative gap
// far wider than the rounding of expf and of the product. -inf disables the test.
__device__ __forceinline__ float alpha_floor(float opacity) {
    float lo = 255.0f * opacity;
    if (!(lo > 0.0f) || !isfinite(lo)) return -__int_as_float(0x7f800000);
    return -logf(lo) - 1e-3f;
}

// Gaussian power -(A dx^2 + C dy^2) / 2 - B dx dy of a record at the pixels of
// one column (shared dx), the exact form: the reference's expression
// (renderer.cu:300-303) with its contraction written out, so that every kernel that
// evaluates it rounds alike, images match bit for bit whichever kernel renders them
// and the backward pass takes what the forward took. The fast forms have their own
// (fast_record below).
struct Power {
    float dx, qx, qydx, qz;
    __device__ __forceinline__ Power(float4 q, float delta_x) {
        dx = delta_x;
        qx = __fmul_rn(q.x, dx);
        qydx = __fmul_rn(q.y, dx);
        qz = q.z;
    }
    __device__ __forceinline__ float at(float dy) const {
        const float t = __fmaf_rn(qx, dx, __fmul_rn(__fmul_rn(qz, dy), dy));
        return __fmaf_rn(-0.5f, t, -__fmul_rn(qydx, dy));
    }
};

// o * e^power of the exact form, with the reference's expf.
__device__ __forceinline__ float gaussian_weight(float opacity, float power) { return opacity * expf(power); }

// 1 / x for x in [0.01, 1] (one minus a clamped alpha): the correctly rounded
// reciprocal in the exact form, the single hardware approximation (PTX
// rcp.approx, within an ulp) in the fast form.
template <bool kFast>
__device__ __forceinline__ float one_over(float x) {
    if (!kFast) return __frcp_rn(x);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Fast-form record terms. The fast forms evaluate a record's alpha as
// ex2(pw2) with pw2 = log2(o) + log2(e) * power, the Gaussian power in log2
// units with the opacity folded in: per record k = (-log2(e) A / 2,
// -log2(e) B, -log2(e) C / 2, log2(o)), per (thread, record) the column terms
// Ax = k.x dx^2 + k.w and Bx = k.y dx, per pixel two FMAs
// pw2 = (k.z dy + Bx) dy + Ax and one MUFU ex2. A pixel takes the record when
// alpha >= 1/255, i.e. pw2 >= log2(1/255) (one compare; false for NaN; a
// record with o < 1/255 never passes since pw2 <= log2(o)). The reference's
// second test, power > 0, only catches rounding: projected conics are
// positive definite (the 2D covariance carries +0.3 on its diagonal and
// det <= 0 is culled), so the true power is never positive; the fast forms
// drop it, as evaluating it against log2(o) would reject pixels within an ulp
// of a Gaussian's centre. The forward and backward fast kernels share these
// expressions, so their take decisions agree.
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLog2AlphaMin = -7.9943534368588578f;  // log2(1/255)

__device__ __forceinline__ float4 fast_record(float4 q) {
    return make_float4(-0.5f * kLog2e * q.x, -kLog2e * q.y, -0.5f * kLog2e * q.z, log2f(q.w));
}

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Packed FP32x2 arithmetic (sm_100: one instruction performs two IEEE
// round-to-nearest operations, each rounded as its scalar form). The fast forms
// evaluate a thread's four pixels as two pairs (pixels 2h and 2h + 1) with
// these, which halves the issue slots of their per-pixel arithmetic.
__device__ __forceinline__ float2 pk(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

}  // namespace gsn
