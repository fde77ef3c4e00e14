// Learned density policy: a 16 -> 64 -> 64 -> 4 MLP (ReLU, softmax over
// keep / clone / split / prune) with fp16 working weights and fp32 arithmetic.
//
// Weights, flat (kMlpParams floats): W1[64][16], b1[64], W2[64][64], b2[64],
// W3[4][64], b3[4]. Training keeps an fp32 master copy and Adam moments; the
// forward and backward passes read the fp16 copy (mixed precision).
//
// Both passes are bound by FP32 FMA issue (15,104 multiply-adds per trained
// sample, 5,376 per inferred one), so they run as register-tiled GEMMs: a CTA of
// 256 threads takes tiles of 128 samples, keeps the activations of a tile
// feature-major in shared memory and the weights (widened to fp32 once per CTA)
// beside them, and every thread forms an 8 x 4 block of a layer's outputs: three
// 16-byte shared loads per 32 FMAs, two of them the same for the whole warp. (4 x 4
// blocks, two loads per 16 FMAs, were bound by shared memory: 294 us per fit step and
// 119 us per inference of 300k samples against 277 and 98.) CTAs are persistent; a
// training CTA holds its share of the weight gradients in registers over all of
// its tiles and adds them to the global fp32 gradient once, in 16-byte vector
// reductions; the next tile's inputs are loaded while a tile is computed. One thread
// per sample with its vectors in shared memory (two shared loads and a widening per
// FMA, 5,508 atomics per 128 samples) took 1,620 and 149 us; four fit steps and an
// inference went from 7,029 to 1,208 us (FP32 FMA floor 0.53 ms).
#include <cuda_fp16.h>

#include "common.cuh"
#include "mlp.h"

namespace gsn {

namespace {

constexpr int kIn = 16, kHid = 64, kOut = 4;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid;
constexpr int kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kOut * kHid;
static_assert(kOffB3 + kOut == kMlpParams, "weight layout");

constexpr int kMlpThreads = 256;
constexpr int kSampleTile = 128;       // samples per tile
constexpr int kRow = kSampleTile + 4;  // padded row: rows 16 bytes apart in the banks
constexpr int kW3Row = kHid + 4;

// The weights in fp32, shared by the CTA. W1 and W2 are stored input-major for the
// forward products; training adds W2 output-major for the backward one.
struct Weights {
    float w1[kIn * kHid];
    float w2[kHid * kHid];
    float w3[kOut * kW3Row];
    float b1[kHid], b2[kHid], b3[kOut];
};

__device__ __forceinline__ void load_weights(const __half* __restrict__ src, Weights& w) {
    for (int i = threadIdx.x; i < kMlpParams; i += kMlpThreads) {
        const float v = __half2float(src[i]);
        if (i < kOffB1) w.w1[(i % kIn) * kHid + i / kIn] = v;
        else if (i < kOffW2) w.b1[i - kOffB1] = v;
        else if (i < kOffB2) w.w2[((i - kOffW2) % kHid) * kHid + (i - kOffW2) / kHid] = v;
        else if (i < kOffW3) w.b2[i - kOffB2] = v;
        else if (i < kOffB3) w.w3[((i - kOffW3) / kHid) * kW3Row + (i - kOffW3) % kHid] = v;
        else w.b3[i - kOffB3] = v;
    }
}

// This thread's 8 x 4 block: rows row0 .. row0 + 7 of a layer (the same for a warp),
// samples col0 .. col0 + 3.
constexpr int kBlockRows = 8;

struct Block {
    int row0, col0;
    __device__ __forceinline__ Block() {
        row0 = kBlockRows * (threadIdx.x >> 5);
        col0 = 4 * (threadIdx.x & 31);
    }
};
static_assert(kBlockRows * (kMlpThreads / 32) == kHid && 4 * 32 == kSampleTile, "one block per thread");

// acc[i][j] += sum over k of w[k][row0 + i] * x[k][col0 + j], k ascending.
template <int K>
__device__ __forceinline__ void block_product(const float* __restrict__ w, const float* __restrict__ x, const Block& b,
                                              float acc[kBlockRows][4]) {
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
        const float4 a0 = *reinterpret_cast<const float4*>(w + k * kHid + b.row0);
        const float4 a1 = *reinterpret_cast<const float4*>(w + k * kHid + b.row0 + 4);
        const float4 v = *reinterpret_cast<const float4*>(x + k * kRow + b.col0);
        const float ai[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, vj[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < kBlockRows; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ai[i], vj[j], acc[i][j]);
    }
}

__device__ __forceinline__ void store_rows(float* dst, const Block& b, const float v[kBlockRows][4]) {
#pragma unroll
    for (int i = 0; i < kBlockRows; ++i)
        *reinterpret_cast<float4*>(dst + (b.row0 + i) * kRow + b.col0) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
}

// relu(bias + w x) of one layer into `out` (rows of kRow) and, as this thread's
// block, into h.
template <int K>
__device__ __forceinline__ void layer(const float* w, const float* bias, const float* x, const Block& b, float* out,
                                      float h[kBlockRows][4]) {
#pragma unroll
    for (int i = 0; i < kBlockRows; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) h[i][j] = bias[b.row0 + i];
    block_product<K>(w, x, b, h);
#pragma unroll
    for (int i = 0; i < kBlockRows; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) h[i][j] = fmaxf(h[i][j], 0.0f);
    store_rows(out, b, h);
}

// A tile's features on their way to shared memory (zeros past n): loaded ahead of the
// tile's turn, stored feature-major at it.
struct TileFeatures {
    static constexpr int kPer = kSampleTile * kIn / kMlpThreads;
    float v[kPer];
    __device__ __forceinline__ void load(const float* __restrict__ features, int64_t first, int n) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int i = threadIdx.x + u * kMlpThreads;
            v[u] = first + i / kIn < n ? features[first * kIn + i] : 0.0f;
        }
    }
    __device__ __forceinline__ void store(float* f) const {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int i = threadIdx.x + u * kMlpThreads;
            f[(i % kIn) * kRow + i / kIn] = v[u];
        }
    }
};

// Output a = t & 3 of the two samples 2 (t >> 2) and 2 (t >> 2) + 1, then all four
// outputs of both by the quad of threads that shares them.
__device__ __forceinline__ void tile_logits(const Weights& w, const float* __restrict__ h2, float logit[2][kOut]) {
    const int a = threadIdx.x & 3;
    float p0 = w.b3[a], p1 = p0;
    const float* wr = w.w3 + a * kW3Row;
    const float* hr = h2 + 2 * (threadIdx.x >> 2);
#pragma unroll 4
    for (int o = 0; o < kHid; o += 4) {
        const float4 q = *reinterpret_cast<const float4*>(wr + o);
        const float qi[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 v = *reinterpret_cast<const float2*>(hr + (o + i) * kRow);
            p0 = fmaf(qi[i], v.x, p0);
            p1 = fmaf(qi[i], v.y, p1);
        }
    }
    const int quad = threadIdx.x & 28;
#pragma unroll
    for (int q = 0; q < kOut; ++q) {
        logit[0][q] = __shfl_sync(0xffffffffu, p0, quad | q);
        logit[1][q] = __shfl_sync(0xffffffffu, p1, quad | q);
    }
}

__device__ __forceinline__ float pick(const float v[kOut], int a) {
    return a == 0 ? v[0] : a == 1 ? v[1] : a == 2 ? v[2] : v[3];
}

struct InferSmem {
    Weights w;
    float f[kIn * kRow], h1[kHid * kRow], h2[kHid * kRow];
};

__global__ void __launch_bounds__(kMlpThreads, 2) mlp_infer_kernel(const float* __restrict__ features, int n,
                                                                   const __half* __restrict__ weights,
                                                                   float confidence, int8_t* __restrict__ actions,
                                                                   float* __restrict__ probs) {
    extern __shared__ __align__(16) unsigned char smem[];
    InferSmem& m = *reinterpret_cast<InferSmem*>(smem);
    load_weights(weights, m.w);
    const Block block;
    const int tiles = ceil_div(n, kSampleTile);
    TileFeatures next;
    next.load(features, static_cast<int64_t>(blockIdx.x) * kSampleTile, n);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t first = static_cast<int64_t>(tile) * kSampleTile;
        __syncthreads();  // the weights, or the previous tile's readers
        next.store(m.f);
        __syncthreads();
        next.load(features, first + static_cast<int64_t>(gridDim.x) * kSampleTile, n);
        float h[kBlockRows][4];
        layer<kIn>(m.w.w1, m.w.b1, m.f, block, m.h1, h);
        __syncthreads();
        layer<kHid>(m.w.w2, m.w.b2, m.h1, block, m.h2, h);
        __syncthreads();
        float logit[2][kOut];
        tile_logits(m.w, m.h2, logit);
        const int a = threadIdx.x & 3;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float mx = logit[half][0];
            int best = 0;
#pragma unroll
            for (int q = 1; q < kOut; ++q)
                if (logit[half][q] > mx) {
                    mx = logit[half][q];
                    best = q;
                }
            float e[kOut], sum = 0.0f;
#pragma unroll
            for (int q = 0; q < kOut; ++q) {
                e[q] = __expf(logit[half][q] - mx);
                sum += e[q];
            }
            const int64_t id = first + 2 * (threadIdx.x >> 2) + half;
            if (id >= n) continue;
            if (probs) probs[id * kOut + a] = pick(e, a) / sum;
            if (a == half)
                actions[id] = pick(e, best) / sum >= confidence ? static_cast<int8_t>(best) : static_cast<int8_t>(-1);
        }
    }
}

struct TrainSmem {
    Weights w;
    float w2_out[kHid * kHid];  // W2 output-major
    float f[kIn * kRow], h1[kHid * kRow], h2[kHid * kRow], z2[kHid * kRow];
    float dl[kOut * kRow];
    double loss[kMlpThreads / 32];
};
static_assert(kMlpParams % 4 == 0 && kMlpParams <= 2 * kHid * kRow, "the gradient leaves in 16-byte vectors over h1, h2");

// sum over samples first .. first + 31 of x[i][s] * y[j][s] added to acc[i][j], rows
// row + 8 i of x and col + 8 j of y.
template <int I, int J>
__device__ __forceinline__ void outer_product(const float* __restrict__ x, const float* __restrict__ y, int row,
                                              int col, int first, float acc[I][J]) {
#pragma unroll 1
    for (int s = first; s < first + 32; s += 4) {
        float4 a[I];
#pragma unroll
        for (int i = 0; i < I; ++i) a[i] = *reinterpret_cast<const float4*>(x + (row + 8 * i) * kRow + s);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const float4 b = *reinterpret_cast<const float4*>(y + (col + 8 * j) * kRow + s);
#pragma unroll
            for (int i = 0; i < I; ++i) {
                acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
                acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
                acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
                acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
            }
        }
    }
}

__device__ __forceinline__ float row_sum(const float* __restrict__ row) {
    float v = 0.0f;
#pragma unroll 4
    for (int s = 0; s < kSampleTile; s += 4) {
        const float4 q = *reinterpret_cast<const float4*>(row + s);
        v += q.x;
        v += q.y;
        v += q.z;
        v += q.w;
    }
    return v;
}

__global__ void __launch_bounds__(kMlpThreads, 1) mlp_train_kernel(const float* __restrict__ features,
                                                                   const int* __restrict__ labels,
                                                                   const float* __restrict__ sample_weights, int n,
                                                                   float weight_norm,
                                                                   const __half* __restrict__ weights,
                                                                   float* __restrict__ grad,
                                                                   double* __restrict__ loss) {
    extern __shared__ __align__(16) unsigned char smem[];
    TrainSmem& m = *reinterpret_cast<TrainSmem*>(smem);
    load_weights(weights, m.w);
    for (int i = threadIdx.x; i < kHid * kHid; i += kMlpThreads) m.w2_out[i] = __half2float(weights[kOffW2 + i]);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const Block block;
    // weight gradients: two warps form all of them over a quarter of the tile's samples,
    // a thread rows ty + 8 i and inputs tx + 8 j
    const int tx = t & 7, ty = (t >> 3) & 7, part = t >> 6;
    float d2[8][8] = {}, d1[8][2] = {}, d3 = 0.0f, db = 0.0f;
    double loss_sum = 0.0;
    const int tiles = ceil_div(n, kSampleTile);
    const int a = t & 3;
    // the inputs of the coming tile: features, and labels and weights of the two
    // samples 2 (t >> 2) and 2 (t >> 2) + 1
    TileFeatures next;
    int next_label[2];
    float next_weight[2];
    auto load_next = [&](int64_t first) {
        next.load(features, first, n);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int64_t id = first + 2 * (t >> 2) + half;
            next_label[half] = id < n ? labels[id] : 0;
            next_weight[half] = id < n ? sample_weights[id] * weight_norm : 0.0f;
        }
    };
    load_next(static_cast<int64_t>(blockIdx.x) * kSampleTile);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t first = static_cast<int64_t>(tile) * kSampleTile;
        __syncthreads();  // the weights, or the previous tile's readers
        next.store(m.f);
        const int label[2] = {next_label[0], next_label[1]};
        const float sw[2] = {next_weight[0], next_weight[1]};
        __syncthreads();
        load_next(first + static_cast<int64_t>(gridDim.x) * kSampleTile);
        float h[kBlockRows][4];
        layer<kIn>(m.w.w1, m.w.b1, m.f, block, m.h1, h);
        __syncthreads();
        layer<kHid>(m.w.w2, m.w.b2, m.h1, block, m.h2, h);
        __syncthreads();
        {   // softmax cross-entropy, weighted and normalised by the batch weight
            float logit[2][kOut], dl[2];
            tile_logits(m.w, m.h2, logit);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float mx = fmaxf(fmaxf(logit[half][0], logit[half][1]), fmaxf(logit[half][2], logit[half][3]));
                float e[kOut], sum = 0.0f;
#pragma unroll
                for (int q = 0; q < kOut; ++q) {
                    e[q] = expf(logit[half][q] - mx);
                    sum += e[q];
                }
                dl[half] = sw[half] * (pick(e, a) / sum - (a == label[half] ? 1.0f : 0.0f));
                if (loss && a == half && first + 2 * (t >> 2) + half < n) {
                    const double lp =
                        static_cast<double>(pick(logit[half], label[half]) - mx) - log(static_cast<double>(sum));
                    loss_sum -= static_cast<double>(sw[half]) * lp;
                }
            }
            *reinterpret_cast<float2*>(m.dl + a * kRow + 2 * (t >> 2)) = make_float2(dl[0], dl[1]);
        }
        __syncthreads();
        {   // back through layer 3 and the second ReLU; the gradient of W3
            float z[kBlockRows][4] = {};
#pragma unroll
            for (int q = 0; q < kOut; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(m.dl + q * kRow + block.col0);
                const float vj[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < kBlockRows; ++i) {
                    const float wq = m.w.w3[q * kW3Row + block.row0 + i];
#pragma unroll
                    for (int j = 0; j < 4; ++j) z[i][j] = fmaf(wq, vj[j], z[i][j]);
                }
            }
#pragma unroll
            for (int i = 0; i < kBlockRows; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) z[i][j] = h[i][j] > 0.0f ? z[i][j] : 0.0f;
            store_rows(m.z2, block, z);
            const float* dl = m.dl + (t >> 6) * kRow;
            const float* hr = m.h2 + (t & 63) * kRow;
#pragma unroll 4
            for (int s = 0; s < kSampleTile; s += 4) {
                const float4 x = *reinterpret_cast<const float4*>(dl + s);
                const float4 y = *reinterpret_cast<const float4*>(hr + s);
                d3 = fmaf(x.x, y.x, d3);
                d3 = fmaf(x.y, y.y, d3);
                d3 = fmaf(x.z, y.z, d3);
                d3 = fmaf(x.w, y.w, d3);
            }
        }
        __syncthreads();
        {   // back through layer 2 and the first ReLU (into h2's place); the gradient of W2
            float z[kBlockRows][4] = {};
            block_product<kHid>(m.w2_out, m.z2, block, z);
#pragma unroll
            for (int i = 0; i < kBlockRows; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(m.h1 + (block.row0 + i) * kRow + block.col0);
                z[i][0] = v.x > 0.0f ? z[i][0] : 0.0f;
                z[i][1] = v.y > 0.0f ? z[i][1] : 0.0f;
                z[i][2] = v.z > 0.0f ? z[i][2] : 0.0f;
                z[i][3] = v.w > 0.0f ? z[i][3] : 0.0f;
            }
            store_rows(m.h2, block, z);
            outer_product<8, 8>(m.z2, m.h1, ty, tx, 32 * part, d2);
        }
        __syncthreads();
        // the gradients of W1 and of the biases (b1, b2, b3 by threads 0, 64, 128 on)
        outer_product<8, 2>(m.h2, m.f, ty, tx, 32 * part, d1);
        if (t < 64) db += row_sum(m.h2 + t * kRow);
        else if (t < 128) db += row_sum(m.z2 + (t - 64) * kRow);
        else if (t < 128 + kOut) db += row_sum(m.dl + (t - 128) * kRow);
    }
    __syncthreads();
    // the CTA's gradient in its flat layout over h1 and h2 (the four parts in turn),
    // then one vector reduction each
    float* g = m.h1;
    for (int turn = 0; turn < 4; ++turn) {
        if (part == turn) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float* at = g + kOffW1 + (ty + 8 * i) * kIn + tx + 8 * j;
                    *at = turn ? *at + d1[i][j] : d1[i][j];
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float* at = g + kOffW2 + (ty + 8 * i) * kHid + tx + 8 * j;
                    *at = turn ? *at + d2[i][j] : d2[i][j];
                }
            }
        }
        __syncthreads();
    }
    g[kOffW3 + t] = d3;
    if (t < 64) g[kOffB1 + t] = db;
    else if (t < 128) g[kOffB2 + t - 64] = db;
    else if (t < 128 + kOut) g[kOffB3 + t - 128] = db;
    if (loss) {
#pragma unroll
        for (int o = 16; o; o >>= 1) loss_sum += __shfl_xor_sync(0xffffffffu, loss_sum, o);
        if (lane == 0) m.loss[warp] = loss_sum;
    }
    __syncthreads();
    for (int i = t; i < kMlpParams / 4; i += kMlpThreads) red_add_v4(grad + 4 * i, reinterpret_cast<const float4*>(g)[i]);
    if (loss && t == 0) {
        double total = 0.0;
        for (int w = 0; w < kMlpThreads / 32; ++w) total += m.loss[w];
        atomicAdd(loss, total);
    }
}

// Per-block FP64 sums of the sample weights; the host adds the kMlpWeightSums of
// them in order, so the sum is the same every time.
__global__ void __launch_bounds__(kMlpThreads) mlp_weight_sum_kernel(const float* __restrict__ w, int64_t n,
                                                                     double* __restrict__ out) {
    __shared__ double part[kMlpThreads / 32];
    double v = 0.0;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * kMlpThreads + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * kMlpThreads)
        v += w[i];
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double total = 0.0;
        for (int k = 0; k < kMlpThreads / 32; ++k) total += part[k];
        out[blockIdx.x] = total;
    }
}

// Adam on the fp32 master weights; refreshes the fp16 working copy and clears
// the gradient for the next step.
__global__ void mlp_adam_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                                float* __restrict__ grad, __half* __restrict__ weights, float lr, float c1,
                                float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kMlpParams) return;
    const float g = grad[i];
    const float mi = 0.9f * m[i] + 0.1f * g;
    const float vi = 0.999f * v[i] + 0.001f * g * g;
    m[i] = mi;
    v[i] = vi;
    const float p = master[i] - lr * (mi * c1) / (sqrtf(vi * c2) + 1e-8f);
    master[i] = p;
    weights[i] = __float2half_rn(p);
    grad[i] = 0.0f;
}

__global__ void mlp_to_half_kernel(const float* __restrict__ master, __half* __restrict__ weights) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kMlpParams) weights[i] = __float2half_rn(master[i]);
}

// CTAs of a persistent launch over `n` samples: as many as are resident at once,
// at most one per tile. Also raises the kernel's dynamic shared-memory limit.
template <typename Kernel>
int persistent_grid(Kernel kernel, size_t smem, int n, int* grid) {
    int device = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kMlpThreads, smem) != cudaSuccess || per_sm < 1)
        return GSN_ERR_CUDA;
    const int tiles = ceil_div(n, kSampleTile);
    *grid = tiles < sms * per_sm ? tiles : sms * per_sm;
    return GSN_OK;
}

}  // namespace

int launch_mlp_infer(const float* features, int n, const void* weights_f16, float confidence, int8_t* actions,
                     float* probs, cudaStream_t stream) {
    if (n <= 0) return GSN_OK;
    int grid = 0;
    const int st = persistent_grid(mlp_infer_kernel, sizeof(InferSmem), n, &grid);
    if (st != GSN_OK) return st;
    mlp_infer_kernel<<<grid, kMlpThreads, sizeof(InferSmem), stream>>>(
        features, n, static_cast<const __half*>(weights_f16), confidence, actions, probs);
    return launched(1);
}

int launch_mlp_gradients(const float* features, const int* labels, const float* sample_weights, int n,
                         float weight_norm, const void* weights_f16, float* grad, double* loss, cudaStream_t stream) {
    if (n <= 0) return GSN_OK;
    int grid = 0;
    const int st = persistent_grid(mlp_train_kernel, sizeof(TrainSmem), n, &grid);
    if (st != GSN_OK) return st;
    mlp_train_kernel<<<grid, kMlpThreads, sizeof(TrainSmem), stream>>>(
        features, labels, sample_weights, n, weight_norm, static_cast<const __half*>(weights_f16), grad, loss);
    return launched(1);
}

int launch_mlp_weight_sum(const float* weights, int n, double* sums, cudaStream_t stream) {
    if (n <= 0) return GSN_ERR_INVALID_ARGUMENT;
    mlp_weight_sum_kernel<<<kMlpWeightSums, kMlpThreads, 0, stream>>>(weights, n, sums);
    return launched(1);
}

int launch_mlp_adam(float* master, float* m, float* v, float* grad, void* weights_f16, float lr, float c1, float c2,
                    cudaStream_t stream) {
    mlp_adam_kernel<<<ceil_div(kMlpParams, 256), 256, 0, stream>>>(master, m, v, grad,
                                                                     static_cast<__half*>(weights_f16), lr, c1, c2);
    return launched(1);
}

int launch_mlp_to_half(const float* master, void* weights_f16, cudaStream_t stream) {
    mlp_to_half_kernel<<<ceil_div(kMlpParams, 256), 256, 0, stream>>>(master, static_cast<__half*>(weights_f16));
    return launched(1);
}

}  // namespace gsn
