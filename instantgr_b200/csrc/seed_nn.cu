// Kernels of the learned congestion seed around its convolutions
// (seed_conv.cu): the loss, the last bias gradient, tiles from and to
// channels-last maps, the seed demand, and the optimiser.
#include "kcommon.cuh"
#include "seed.hpp"

#include <algorithm>

namespace igr {

namespace {

__global__ void bias_grad_kernel(int P, int cout, const __nv_bfloat16 *dY, float *db) {
    const int co = blockIdx.x;
    float s = 0;
    for (int p = threadIdx.x + blockIdx.y * blockDim.x; p < P; p += blockDim.x * gridDim.y)
        s += __bfloat162float(dY[(size_t)p * cout + co]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ float w[8];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += w[i];
        atomicAdd(db + co, t);
    }
}

__global__ void seed_loss_kernel(int T, int S, int halo, const float *y, const float *tg, __nv_bfloat16 *dY,
                                 double *sums, double scale) {
    const long long n = (long long)T * S * S * kSeedOut;
    double se = 0, ae = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int ch = (int)(i % kSeedOut);
        const long long p = i / kSeedOut;
        const int x = (int)(p % S), yy = (int)((p / S) % S);
        float g = 0;
        if (ch < kSeedLayersOut && x >= halo && x < S - halo && yy >= halo && yy < S - halo) {
            const float e = y[i] - tg[i];
            se += (double)e * e;
            ae += fabs((double)e);
            g = (float)(2.0 * e * scale);
        }
        dY[i] = __float2bfloat16(g);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        se += __shfl_down_sync(0xffffffffu, se, o);
        ae += __shfl_down_sync(0xffffffffu, ae, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(sums, se);
        atomicAdd(sums + 1, ae);
    }
}

__global__ void gather_tiles_kernel(int T, int S, int halo, const TileRef *tiles, const __nv_bfloat16 *pool,
                                    __nv_bfloat16 *out16, float *out32) {
    // one thread per (tile, pixel, 8-channel half)
    const long long n = (long long)T * S * S * 2;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int h = (int)(q & 1);
        const long long p = q >> 1;
        const int t = (int)(p / ((long long)S * S)), r = (int)(p % ((long long)S * S)), i = r / S, j = r % S;
        const TileRef tr = tiles[t];
        const int x = tr.x0 - halo + i, y = tr.y0 - halo + j;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (x >= 0 && y >= 0 && x < tr.X && y < tr.Y)
            v = *reinterpret_cast<const uint4 *>(pool + tr.base + ((long long)x * tr.Y + y) * kSeedIn + h * 8);
        if (out16) *reinterpret_cast<uint4 *>(out16 + p * kSeedIn + h * 8) = v;
        if (out32) {
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int c = 0; c < 8; c++) out32[p * kSeedIn + h * 8 + c] = __bfloat162float(e[c]);
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

__global__ void adam_kernel(int n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2, float eps,
                            float c1, float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

__global__ void seed_weights_kernel(int cin, int cout, const float *Wm, __nv_bfloat16 *W, __nv_bfloat16 *WT) {
    const int n = cout * 9 * cin;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int co = i / (9 * cin), r = i - co * 9 * cin, tap = r / cin, ci = r - tap * cin;
        const __nv_bfloat16 b = __float2bfloat16(Wm[i]);
        W[i] = b;
        WT[((size_t)ci * 9 + tap) * cout + co] = b;
    }
}

__global__ void seed_grad_layout_kernel(int cin, int cout, const float *dWT, float *dW) {
    const int n = cout * 9 * cin;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int co = i / (9 * cin), r = i - co * 9 * cin;  // r = tap * cin + ci
        dW[i] = dWT[(size_t)r * cout + co];
    }
}

int blocks_for(long long n) { return (int)std::max<long long>(1, std::min<long long>(148 * 8, (n + 255) / 256)); }

}  // namespace

void launch_bias_grad(const ConvSpec &c, int T, const __nv_bfloat16 *dY, float *db, cudaStream_t s) {
    const int P = T * c.hout * c.wout;
    bias_grad_kernel<<<dim3(c.cout, 16), 256, 0, s>>>(P, c.cout, dY, db);
}

void launch_seed_loss(int T, int S, int halo, const float *y, const float *target, __nv_bfloat16 *dY, double *sums,
                      cudaStream_t s) {
    const long long n = (long long)T * S * S * kSeedOut;
    const double count = (double)T * (S - 2 * halo) * (S - 2 * halo) * kSeedLayersOut;
    seed_loss_kernel<<<blocks_for(n), 256, 0, s>>>(T, S, halo, y, target, dY, sums, 1.0 / count);
}

void launch_gather_tiles(int T, int S, int halo, const TileRef *tiles, const __nv_bfloat16 *pool, __nv_bfloat16 *out16,
                         float *out32, cudaStream_t s) {
    gather_tiles_kernel<<<blocks_for((long long)T * S * S * 2), 256, 0, s>>>(T, S, halo, tiles, pool, out16, out32);
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

void launch_adam(int n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2, float eps, int t,
                 cudaStream_t s) {
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    adam_kernel<<<blocks_for(n), 256, 0, s>>>(n, p, g, m, v, lr, b1, b2, eps, c1, c2);
}

void launch_seed_weights(int cin, int cout, const float *Wm, __nv_bfloat16 *W, __nv_bfloat16 *WT, cudaStream_t s) {
    seed_weights_kernel<<<blocks_for((long long)cout * 9 * cin), 256, 0, s>>>(cin, cout, Wm, W, WT);
}

void launch_seed_grad_layout(int cin, int cout, const float *dWT, float *dW, cudaStream_t s) {
    seed_grad_layout_kernel<<<blocks_for((long long)cout * 9 * cin), 256, 0, s>>>(cin, cout, dWT, dW);
}

}  // namespace igr
