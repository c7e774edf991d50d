// Kernels of the learned congestion seed around its convolutions
// (seed_conv.cu): the loss, the last bias gradient, tiles from and to
// channels-last maps, the seed demand, and the optimiser.
#include "kcommon.cuh"
#include "seed.hpp"

#include <algorithm>

namespace igr {

namespace {

// Loss, its gradient and the gradient's channel sums: a block per tile row at a
// time, a thread per pixel and four channels.  Memory bound (outputs and targets
// in, gradient out); rows and channels without loss are not read.  One thread
// per value with 64-bit index divisions, and the last layer's bias gradient in a
// pass of its own, took 127 + 161 us for 16 tiles of 288 x 288 (now 33).
__global__ void __launch_bounds__(256) seed_loss_kernel(int T, int S, int halo, const float *y, const float *tg,
                                                        __nv_bfloat16 *dY, double *sums, float *db, double scale) {
    const int part = threadIdx.x & 3;  // channels 4 part .. 4 part + 3
    double se = 0, ae = 0;
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    for (int row = blockIdx.x; row < T * S; row += gridDim.x) {
        const int yy = row % S;
        const bool inner = yy >= halo && yy < S - halo;
        for (int x = threadIdx.x >> 2; x < S; x += 64) {
            const size_t i = ((size_t)row * S + x) * kSeedOut + part * 4;
            float g[4] = {0.f, 0.f, 0.f, 0.f};
            if (inner && x >= halo && x < S - halo && part * 4 < kSeedLayersOut) {
                const float4 a = *reinterpret_cast<const float4 *>(y + i), b = *reinterpret_cast<const float4 *>(tg + i);
                const float e[4] = {a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w};
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (part * 4 + c < kSeedLayersOut) {
                        se += (double)e[c] * e[c];
                        ae += fabs((double)e[c]);
                        g[c] = (float)(2.0 * e[c] * scale);
                    }
            }
            __nv_bfloat162 h[2] = {__floats2bfloat162_rn(g[0], g[1]), __floats2bfloat162_rn(g[2], g[3])};
            *reinterpret_cast<uint2 *>(dY + i) = *reinterpret_cast<const uint2 *>(h);
            sum[0] += __bfloat162float(h[0].x);
            sum[1] += __bfloat162float(h[0].y);
            sum[2] += __bfloat162float(h[1].x);
            sum[3] += __bfloat162float(h[1].y);
        }
    }
    __shared__ double ws[8][2];
    __shared__ float wb[8][16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        se += __shfl_down_sync(0xffffffffu, se, o);
        ae += __shfl_down_sync(0xffffffffu, ae, o);
        if (o >= 4)
#pragma unroll
            for (int c = 0; c < 4; c++) sum[c] += __shfl_down_sync(0xffffffffu, sum[c], o);
    }
    if (lane == 0) { ws[warp][0] = se; ws[warp][1] = ae; }
    if (lane < 4)
        for (int c = 0; c < 4; c++) wb[warp][lane * 4 + c] = sum[c];
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0;
        for (int w = 0; w < 8; w++) t += ws[w][threadIdx.x];
        atomicAdd(sums + threadIdx.x, t);
    } else if (threadIdx.x >= 32 && threadIdx.x < 32 + kSeedLayersOut) {
        float t = 0;
        for (int w = 0; w < 8; w++) t += wb[w][threadIdx.x - 32];
        atomicAdd(db + threadIdx.x - 32, t);
    }
}

// One block per tile row at a time, a thread per pixel and eight channels.
__global__ void __launch_bounds__(256) gather_tiles_kernel(int T, int S, int halo, const TileRef *tiles,
                                                           const __nv_bfloat16 *features, __nv_bfloat16 *out16,
                                                           const __nv_bfloat16 *targets, float *out32) {
    for (int row = blockIdx.x; row < T * S; row += gridDim.x) {
        const int t = row / S;
        const TileRef tr = tiles[t];
        const int x = tr.x0 - halo + row - t * S;
        const bool in = x >= 0 && x < tr.X;
        const long long src = tr.base + (long long)x * tr.Y * kSeedIn;
        for (int q = threadIdx.x; q < 2 * S; q += 256) {
            const int y = tr.y0 - halo + (q >> 1);
            const bool here = in && y >= 0 && y < tr.Y;
            const long long at = src + (long long)y * kSeedIn + (q & 1) * 8;
            const size_t to = ((size_t)row * S + (q >> 1)) * kSeedIn + (q & 1) * 8;
            uint4 f = make_uint4(0, 0, 0, 0), v = f;
            if (here) f = *reinterpret_cast<const uint4 *>(features + at);
            if (here && targets) v = *reinterpret_cast<const uint4 *>(targets + at);
            *reinterpret_cast<uint4 *>(out16 + to) = f;
            if (targets) {
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                float4 o[2];
                float *e = reinterpret_cast<float *>(o);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    e[2 * c] = __uint_as_float(w[c] << 16);
                    e[2 * c + 1] = __uint_as_float(w[c] & 0xffff0000u);
                }
                reinterpret_cast<float4 *>(out32 + to)[0] = o[0];
                reinterpret_cast<float4 *>(out32 + to)[1] = o[1];
            }
        }
    }
}

__global__ void scatter_prediction_kernel(int T, int S, int halo, const TileRef *tiles, const float *y32, float *pred) {
    const int in = S - 2 * halo;
    const long long n = (long long)T * in * in * 4;  // (tile, cell, 4-channel quarter)
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int part = (int)(q & 3);
        const long long p = q >> 2;
        const int t = (int)(p / ((long long)in * in)), r = (int)(p % ((long long)in * in)), i = r / in, j = r % in;
        const TileRef tr = tiles[t];
        const int x = tr.x0 + i, y = tr.y0 + j;
        if (x >= tr.X || y >= tr.Y) continue;
        const float *src = y32 + (((long long)t * S + i + halo) * S + j + halo) * kSeedOut + part * 4;
        *reinterpret_cast<float4 *>(pred + ((long long)x * tr.Y + y) * kSeedOut + part * 4) =
            *reinterpret_cast<const float4 *>(src);
    }
}

__global__ void seed_demand_kernel(int X, int Y, int L, const float *pred, float alpha, int kind, const float *cap,
                                   float *out) {
    const long long n = (long long)L * X * Y;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(i / ((long long)X * Y));
        const long long c = i - (long long)l * X * Y;
        float v = 8.f * pred[c * kSeedOut + 1 + l];
        if (kind == 1) v -= cap[i];
        out[i] = v > 0.f ? alpha * v : 0.f;
    }
}

__global__ void seed_step_kernel(long long n, float *d, const float *base, float *cur, float frac) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float q = 0.5f * rintf(2.f * frac * base[i]);
        const float c = cur[i];
        if (q != c) {
            d[i] += q - c;
            cur[i] = q;
        }
    }
}

__global__ void seed_overflow_kernel(int X, int Y, int L, const float *pred, const float *cap, float *out) {
    const long long n = (long long)X * Y;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        float o = 0;
        for (int l = 0; l < L; l++) o += fmaxf(0.f, 8.f * pred[c * kSeedOut + 1 + l] - cap[(long long)l * n + c]);
        out[c] = o;
    }
}

__global__ void add_demand_kernel(long long n, float *d, const float *seed, float sign) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        d[i] += sign * seed[i];
}

// Where the gradient sum of parameter i ([tap][ci][co]; a bias: its own place)
// and, for a weight, its working copy in WT ([ci][tap][co]) are.
struct ParamAt {
    int sum, turned;
    bool weight;
};
template <int L = 0>
__device__ __forceinline__ ParamAt param_at(int i) {
    if constexpr (L + 1 < kSeedConvs) {
        constexpr int end = seed_at(L + 1);
        if (i >= end) return param_at<L + 1>(i);
    }
    constexpr int at = seed_at(L), weights = seed_weights(L), cin = seed_cin(L), cout = seed_cout(L);
    ParamAt a;
    const int r = i - at;
    a.weight = r < weights;
    const int co = r / (9 * cin), k = r - co * 9 * cin;
    a.sum = a.weight ? at + k * cout + co : i;
    a.turned = at + (k % cin * 9 + k / cin) * cout + co;
    return a;
}
__device__ __forceinline__ void put_weight(int i, const ParamAt &a, float p, __nv_bfloat16 *W, __nv_bfloat16 *WT) {
    if (!a.weight) return;
    const __nv_bfloat16 b = __float2bfloat16(p);
    W[i] = b;
    WT[a.turned] = b;
}

// All parameters in one launch: 24 launches per step (12 of Adam, six each of
// weights and gradient layouts) took about as long as a convolution.
__global__ void adam_kernel(float *P, float *M, float *V, const float *acc, __nv_bfloat16 *W, __nv_bfloat16 *WT,
                            float lr, float b1, float b2, float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kSeedParams) return;
    const ParamAt a = param_at(i);
    const float gi = acc[a.sum];
    const float mi = b1 * M[i] + (1.f - b1) * gi;
    const float vi = b2 * V[i] + (1.f - b2) * gi * gi;
    M[i] = mi;
    V[i] = vi;
    const float p = P[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    P[i] = p;
    put_weight(i, a, p, W, WT);
}

__global__ void seed_weights_kernel(const float *P, __nv_bfloat16 *W, __nv_bfloat16 *WT) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kSeedParams) put_weight(i, param_at(i), P[i], W, WT);
}

__global__ void seed_grad_layout_kernel(const float *acc, float *G) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kSeedParams) G[i] = acc[param_at(i).sum];
}

constexpr int kParamBlocks = (kSeedParams + 255) / 256;

int blocks_for(long long n) { return (int)std::max<long long>(1, std::min<long long>(148 * 8, (n + 255) / 256)); }

}  // namespace

void launch_seed_loss(int T, int S, int halo, const float *y, const float *target, __nv_bfloat16 *dY, double *sums,
                      float *db, cudaStream_t s) {
    const double count = (double)T * (S - 2 * halo) * (S - 2 * halo) * kSeedLayersOut;
    seed_loss_kernel<<<std::min(T * S, 148 * 8), 256, 0, s>>>(T, S, halo, y, target, dY, sums, db, 1.0 / count);
}

void launch_gather_tiles(int T, int S, int halo, const TileRef *tiles, const __nv_bfloat16 *features,
                         __nv_bfloat16 *out16, const __nv_bfloat16 *targets, float *out32, cudaStream_t s) {
    gather_tiles_kernel<<<std::min(T * S, 148 * 8), 256, 0, s>>>(T, S, halo, tiles, features, out16, targets, out32);
}

void launch_scatter_prediction(int T, int S, int halo, const TileRef *tiles, const float *y32, float *pred,
                               cudaStream_t s) {
    const int in = S - 2 * halo;
    scatter_prediction_kernel<<<blocks_for((long long)T * in * in * 4), 256, 0, s>>>(T, S, halo, tiles, y32, pred);
}

void launch_seed_demand(int X, int Y, int L, const float *pred, float alpha, int kind, const float *cap_ref,
                        float *out_ref, cudaStream_t s) {
    seed_demand_kernel<<<blocks_for((long long)L * X * Y), 256, 0, s>>>(X, Y, L, pred, alpha, kind, cap_ref, out_ref);
}

void launch_seed_step(int64_t n, float *demand, const float *base, float *cur, float frac, cudaStream_t s) {
    seed_step_kernel<<<blocks_for(n), 256, 0, s>>>(n, demand, base, cur, frac);
}

void launch_seed_overflow(int X, int Y, int L, const float *pred, const float *cap_ref, float *out, cudaStream_t s) {
    seed_overflow_kernel<<<blocks_for((long long)X * Y), 256, 0, s>>>(X, Y, L, pred, cap_ref, out);
}

void launch_add_demand(int64_t n, float *demand, const float *seed, float sign, cudaStream_t s) {
    add_demand_kernel<<<blocks_for(n), 256, 0, s>>>(n, demand, seed, sign);
}

void launch_adam(float *P, float *M, float *V, const float *acc, __nv_bfloat16 *W, __nv_bfloat16 *WT, float lr, float b1,
                 float b2, float eps, int t, cudaStream_t s) {
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    adam_kernel<<<kParamBlocks, 256, 0, s>>>(P, M, V, acc, W, WT, lr, b1, b2, eps, c1, c2);
}

void launch_seed_weights(const float *P, __nv_bfloat16 *W, __nv_bfloat16 *WT, cudaStream_t s) {
    seed_weights_kernel<<<kParamBlocks, 256, 0, s>>>(P, W, WT);
}

void launch_seed_grad_layout(const float *acc, float *G, cudaStream_t s) {
    seed_grad_layout_kernel<<<kParamBlocks, 256, 0, s>>>(acc, G);
}

}  // namespace igr
