// Learned density policy: a 16 -> 64 -> 64 -> 4 MLP (ReLU, softmax over
// keep / clone / split / prune) with fp16 working weights and fp32 arithmetic.
//
// Weights, flat (kMlpParams floats): W1[64][16], b1[64], W2[64][64], b2[64],
// W3[4][64], b3[4]. Training keeps an fp32 master copy and Adam moments; the
// forward and backward passes read the fp16 copy (mixed precision).
//
// Both passes are bound by FP32 FMA issue (15,104 multiply-adds per trained
// sample, 5,376 per inferred one), so they run as register-tiled GEMMs: a CTA of
// 256 threads takes tiles of 64 samples, keeps the activations of a tile
// feature-major in shared memory and the weights (widened to fp32 once per CTA)
// beside them, and every thread forms a 4 x 4 block of a layer's outputs, two
// 16-byte shared loads per 16 FMAs. CTAs are persistent, two to three per SM; a
// training CTA holds its share of the weight gradients in registers over all of
// its tiles and adds them to the global fp32 gradient once, in 16-byte vector
// reductions. One thread per sample with its vectors in shared memory (two shared
// loads and a widening per FMA, 5,508 atomics per 128 samples) took 1,620 us per
// fit step and 149 us per inference of 300k samples; four steps and an inference
// went from 7,029 to 1,311 us (FP32 FMA floor 0.53 ms).
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
constexpr int kSampleTile = 64;        // samples per tile
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

// This thread's 4 x 4 block: rows row0 .. row0 + 3 of a layer, samples col0 ..
// col0 + 3. A warp covers 16 rows x 32 samples, so its two 16-byte loads per step
// read 64 and 128 distinct bytes.
struct Block {
    int row0, col0;
    __device__ __forceinline__ Block() {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        row0 = 4 * ((lane >> 3) + 4 * (warp >> 1));
        col0 = 4 * ((lane & 7) + 8 * (warp & 1));
    }
};

// acc[i][j] += sum over k of w[k][row0 + i] * x[k][col0 + j], k ascending.
template <int K>
__device__ __forceinline__ void block_product(const float* __restrict__ w, const float* __restrict__ x, const Block& b,
                                              float acc[4][4]) {
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(w + k * kHid + b.row0);
        const float4 v = *reinterpret_cast<const float4*>(x + k * kRow + b.col0);
        const float ai[4] = {a.x, a.y, a.z, a.w}, vj[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ai[i], vj[j], acc[i][j]);
    }
}

__device__ __forceinline__ void store_rows(float* dst, const Block& b, const float v[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(dst + (b.row0 + i) * kRow + b.col0) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
}

// relu(bias + w x) of one layer into `out` (rows of kRow) and, as this thread's
// block, into h.
template <int K>
__device__ __forceinline__ void layer(const float* w, const float* bias, const float* x, const Block& b, float* out,
                                      float h[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) h[i][j] = bias[b.row0 + i];
    block_product<K>(w, x, b, h);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) h[i][j] = fmaxf(h[i][j], 0.0f);
    store_rows(out, b, h);
}

// The tile's features, feature-major (zeros past n).
__device__ __forceinline__ void load_tile(const float* __restrict__ features, int64_t first, int n, float* f) {
#pragma unroll
    for (int u = 0; u < kSampleTile * kIn / kMlpThreads; ++u) {
        const int i = threadIdx.x + u * kMlpThreads;
        const int s = i / kIn, k = i % kIn;
        f[k * kRow + s] = first + s < n ? features[(first + s) * kIn + k] : 0.0f;
    }
}

// The four logits of this thread's sample: thread t has output a = t & 3 of sample
// t >> 2. Two neighbouring samples' products are formed by the eight threads of the
// pair, each over half of the inputs.
__device__ __forceinline__ void tile_logits(const Weights& w, const float* __restrict__ h2, float logit[kOut]) {
    const int a = threadIdx.x & 3, half = (threadIdx.x >> 2) & 1, pair = threadIdx.x >> 3;
    float p0 = half ? 0.0f : w.b3[a], p1 = p0;
    const float* wr = w.w3 + a * kW3Row + half * (kHid / 2);
    const float* hr = h2 + half * (kHid / 2) * kRow + 2 * pair;
#pragma unroll
    for (int o = 0; o < kHid / 2; o += 4) {
        const float4 q = *reinterpret_cast<const float4*>(wr + o);
        const float qi[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 v = *reinterpret_cast<const float2*>(hr + (o + i) * kRow);
            p0 = fmaf(qi[i], v.x, p0);
            p1 = fmaf(qi[i], v.y, p1);
        }
    }
    p0 += __shfl_xor_sync(0xffffffffu, p0, 4);
    p1 += __shfl_xor_sync(0xffffffffu, p1, 4);
    const float mine = half ? p1 : p0;
    const int quad = threadIdx.x & 28;
#pragma unroll
    for (int q = 0; q < kOut; ++q) logit[q] = __shfl_sync(0xffffffffu, mine, quad | q);
}

struct InferSmem {
    Weights w;
    float f[kIn * kRow], h1[kHid * kRow], h2[kHid * kRow];
};

__global__ void __launch_bounds__(kMlpThreads, 3) mlp_infer_kernel(const float* __restrict__ features, int n,
                                                                   const __half* __restrict__ weights,
                                                                   float confidence, int8_t* __restrict__ actions,
                                                                   float* __restrict__ probs) {
    extern __shared__ __align__(16) unsigned char smem[];
    InferSmem& m = *reinterpret_cast<InferSmem*>(smem);
    load_weights(weights, m.w);
    const Block block;
    const int tiles = ceil_div(n, kSampleTile);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t first = static_cast<int64_t>(tile) * kSampleTile;
        __syncthreads();  // the weights, or the previous tile's readers
        load_tile(features, first, n, m.f);
        __syncthreads();
        float h[4][4];
        layer<kIn>(m.w.w1, m.w.b1, m.f, block, m.h1, h);
        __syncthreads();
        layer<kHid>(m.w.w2, m.w.b2, m.h1, block, m.h2, h);
        __syncthreads();
        float logit[kOut];
        tile_logits(m.w, m.h2, logit);
        float mx = logit[0];
        int best = 0;
#pragma unroll
        for (int a = 1; a < kOut; ++a)
            if (logit[a] > mx) {
                mx = logit[a];
                best = a;
            }
        float e[kOut], sum = 0.0f;
#pragma unroll
        for (int a = 0; a < kOut; ++a) {
            e[a] = __expf(logit[a] - mx);
            sum += e[a];
        }
        const int64_t id = first + (threadIdx.x >> 2);
        const int a = threadIdx.x & 3;
        if (id >= n) continue;
        const float mine = a == 0 ? e[0] : a == 1 ? e[1] : a == 2 ? e[2] : e[3];
        if (probs) probs[id * kOut + a] = mine / sum;
        const float top = best == 0 ? e[0] : best == 1 ? e[1] : best == 2 ? e[2] : e[3];
        if (a == 0) actions[id] = top / sum >= confidence ? static_cast<int8_t>(best) : static_cast<int8_t>(-1);
    }
}

// Element-wise atomic add of four floats (PTX red.global.add.v4.f32, sm_90 and later).
__device__ __forceinline__ void red_add_v4(float* address, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(address), "f"(v.x), "f"(v.y), "f"(v.z),
                 "f"(v.w)
                 : "memory");
}

struct TrainSmem {
    Weights w;
    float w2_out[kHid * kHid];  // W2 output-major
    float f[kIn * kRow], h1[kHid * kRow], h2[kHid * kRow], z2[kHid * kRow];
    float dl[kOut * kRow];
    double loss[kMlpThreads / 32];
};
static_assert(kMlpParams % 4 == 0 && kMlpParams <= 2 * kHid * kRow, "the gradient leaves in 16-byte vectors over h1, h2");

// sum over the tile of x[i][s] * y[j][s] added to acc[i][j], rows row + 16 i of x and
// col + 16 j of y.
template <int I, int J>
__device__ __forceinline__ void outer_product(const float* __restrict__ x, const float* __restrict__ y, int row,
                                              int col, float acc[I][J]) {
#pragma unroll 2
    for (int s = 0; s < kSampleTile; s += 4) {
        float4 a[I], b[J];
#pragma unroll
        for (int i = 0; i < I; ++i) a[i] = *reinterpret_cast<const float4*>(x + (row + 16 * i) * kRow + s);
#pragma unroll
        for (int j = 0; j < J; ++j) b[j] = *reinterpret_cast<const float4*>(y + (col + 16 * j) * kRow + s);
#pragma unroll
        for (int i = 0; i < I; ++i)
#pragma unroll
            for (int j = 0; j < J; ++j) {
                acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
                acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
                acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
                acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
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

__global__ void __launch_bounds__(kMlpThreads, 2) mlp_train_kernel(const float* __restrict__ features,
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
    // weight gradients: rows ty + 16 i, inputs tx + 16 j of W2; inputs tx of W1
    const int tx = (lane & 7) + 8 * (warp & 1), ty = (lane >> 3) + 4 * (warp >> 1);
    float d2[4][4] = {}, d1[4][1] = {}, d3 = 0.0f, db = 0.0f;
    double loss_sum = 0.0;
    const int tiles = ceil_div(n, kSampleTile);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t first = static_cast<int64_t>(tile) * kSampleTile;
        __syncthreads();  // the weights, or the previous tile's readers
        load_tile(features, first, n, m.f);
        const int64_t id = first + (t >> 2);
        const bool live = id < n;
        const int label = live ? labels[id] : 0;
        const float sw = live ? sample_weights[id] * weight_norm : 0.0f;
        __syncthreads();
        float h[4][4];
        layer<kIn>(m.w.w1, m.w.b1, m.f, block, m.h1, h);
        __syncthreads();
        layer<kHid>(m.w.w2, m.w.b2, m.h1, block, m.h2, h);
        __syncthreads();
        {   // softmax cross-entropy, weighted and normalised by the batch weight
            float logit[kOut];
            tile_logits(m.w, m.h2, logit);
            const float mx = fmaxf(fmaxf(logit[0], logit[1]), fmaxf(logit[2], logit[3]));
            float e[kOut], sum = 0.0f;
#pragma unroll
            for (int a = 0; a < kOut; ++a) {
                e[a] = expf(logit[a] - mx);
                sum += e[a];
            }
            const int a = t & 3;
            const float mine = a == 0 ? e[0] : a == 1 ? e[1] : a == 2 ? e[2] : e[3];
            m.dl[a * kRow + (t >> 2)] = sw * (mine / sum - (a == label ? 1.0f : 0.0f));
            if (live && loss && a == 0) {
                const float own = label == 0 ? logit[0] : label == 1 ? logit[1] : label == 2 ? logit[2] : logit[3];
                const double lp = static_cast<double>(own - mx) - log(static_cast<double>(sum));
                loss_sum -= static_cast<double>(sw) * lp;
            }
        }
        __syncthreads();
        {   // back through layer 3 and the second ReLU; the gradient of W3
            float z[4][4] = {};
#pragma unroll
            for (int a = 0; a < kOut; ++a) {
                const float4 q = *reinterpret_cast<const float4*>(m.w.w3 + a * kW3Row + block.row0);
                const float4 v = *reinterpret_cast<const float4*>(m.dl + a * kRow + block.col0);
                const float qi[4] = {q.x, q.y, q.z, q.w}, vj[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) z[i][j] = fmaf(qi[i], vj[j], z[i][j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
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
            float z[4][4] = {};
            block_product<kHid>(m.w2_out, m.z2, block, z);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(m.h1 + (block.row0 + i) * kRow + block.col0);
                z[i][0] = v.x > 0.0f ? z[i][0] : 0.0f;
                z[i][1] = v.y > 0.0f ? z[i][1] : 0.0f;
                z[i][2] = v.z > 0.0f ? z[i][2] : 0.0f;
                z[i][3] = v.w > 0.0f ? z[i][3] : 0.0f;
            }
            store_rows(m.h2, block, z);
            outer_product<4, 4>(m.z2, m.h1, ty, tx, d2);
        }
        __syncthreads();
        // the gradients of W1 and of the biases (b1, b2, b3 by threads 0, 64, 128 on)
        outer_product<4, 1>(m.h2, m.f, ty, tx, d1);
        if (t < 64) db += row_sum(m.h2 + t * kRow);
        else if (t < 128) db += row_sum(m.z2 + (t - 64) * kRow);
        else if (t < 128 + kOut) db += row_sum(m.dl + (t - 128) * kRow);
    }
    __syncthreads();
    // the CTA's gradient in its flat layout over h1 and h2, then one vector reduction each
    float* g = m.h1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        g[kOffW1 + (ty + 16 * i) * kIn + tx] = d1[i][0];
#pragma unroll
        for (int j = 0; j < 4; ++j) g[kOffW2 + (ty + 16 * i) * kHid + tx + 16 * j] = d2[i][j];
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
