// Convolutions of the learned congestion seed and their input gradients as
// implicit GEMMs on the tcgen05 tensor cores.
//
// All of them multiply rows = output pixels by columns = output channels over
// K = taps x input channels.  A tap only shifts which source pixel a row reads,
// so a source tile is brought into shared memory once, with the pixels around
// it, and every tap reads it through a descriptor of another start address: the
// tile lies in planes of 8 channels, 16 bytes a pixel, so that eight pixels in
// a row are a core matrix wherever they start, planes are the leading byte
// offset (K halves) and tile rows the stride byte offset (8-row groups).
// Where the output has twice the source's resolution, a GEMM takes the pixels
// of one parity, whose taps are again shifts of the source; where it has half,
// the tile's even and odd columns lie apart and the row groups skip a row.
//
// A block runs over tiles with three roles: four warps copy source tiles
// (cp.async, three in flight), one thread issues a tile's MMAs, four warps write
// the previous tile's results from TMEM (two stages).  The weights stay in
// shared memory.  What bounds it: the MMAs read their operands from shared
// memory, 6 KB for 128 x 64 x 16, so N = 64 cannot pass a third of the tensor
// peak, and the activations pass through HBM once per layer; the input
// gradients also read the mask and keep the sums of the bias gradients.
// Gathering each tap's operands anew through registers, as the kernel before it
// did, moved nine times the tile.  16 tiles of 288 x 288: forward pass 2.03 ->
// 0.37 ms (135 GFLOP, 365 TFLOP/s), input gradients with the bias gradients
// 2.10 + 0.56 -> 0.47 ms.
//
// The K order of every output is tap by tap and 16 channels at a time.  Every
// wait is bounded (ERR_TIMEOUT in the error word) and the TMEM columns are freed
// on every path.
#include "kcommon.cuh"
#include "seed.hpp"
#include "umma.cuh"
#include "hooks.hpp"
#include "host.hpp"

#include <algorithm>

namespace igr {

namespace {

constexpr unsigned long long kDrainNs = 2000000000ull;

// kSame: same size (its input gradient has the taps turned round); kStride2:
// stride 2; kUp2: nearest x2 first; kStride2T, kUp2T: input gradients of the two
enum Kind { kSame, kStride2, kUp2, kStride2T, kUp2T };

constexpr int pow2_at_least(int v, int from = 32) { return from >= v ? from : pow2_at_least(v, 2 * from); }

template <Kind K, int CIN, int N>
struct Geo {
    static constexpr bool fine = K == kUp2 || K == kStride2T;   // output at twice the tile grid's resolution
    static constexpr bool half = K == kStride2 || K == kUp2T;   // source at twice the tile grid's resolution
    static constexpr int gemms = K == kSame ? 2 : fine ? 4 : 1;  // 128-row GEMMs of a tile
    static constexpr int rows = 16, cols = K == kSame ? 16 : 8;  // tile, in the tile grid's pixels
    // source pixels of a tile, the pitch of their rows and their places in a plane
    static constexpr int srows = K == kStride2 ? 33 : K == kUp2T ? 34 : 18;
    static constexpr int scols = K == kStride2 ? 17 : K == kUp2T || K == kSame ? 18 : 10;
    static constexpr int pitch = half ? (scols + 1) / 2 : scols;
    static constexpr int places = half ? 2 * srows * pitch : srows * scols;
    static constexpr int plane = (places | 1) * 16;  // odd multiple of 16 bytes: the copies meet no bank conflict
    static constexpr int chunks = CIN / 8;
    static constexpr int abytes = (plane * chunks + 127) / 128 * 128;
    static constexpr int bbytes = 9 * CIN * N * 2;
    static constexpr int bufs = 3;
    static constexpr int smem = bufs * abytes + bbytes;
    static constexpr int stage = gemms * N;  // TMEM columns of a tile
    static constexpr int tmem = pow2_at_least(2 * stage);
    static constexpr uint32_t sbo = (half ? 2 : 1) * pitch * 16;
    static __device__ constexpr int place(int a, int b) {  // source pixel (a, b) of the tile
        return half ? (b & 1) * srows * pitch + a * pitch + (b >> 1) : a * pitch + b;
    }
};

struct ConvArgs {
    const __nv_bfloat16 *src, *w;  // [T][sh][sw][CIN]; weights [N][9][CIN]
    int sh, sw, oh, ow;
    int tiles, tx, ty;             // tiles in all, per tile row and per column of an image
    int relu;
    const float *bias;             // forward
    __nv_bfloat16 *out;            // [T][oh][ow][N]
    float *out32;                  // forward, optional
    const __nv_bfloat16 *mask;     // gradient, optional: zero where mask <= 0
    float *db;                     // gradient, optional: sums of out per channel are added
    int *err;
    unsigned long long wait_ns;
    int probe;
};

constexpr int kConvThreads = 288;

template <Kind K, int CIN, int N, bool GRAD, int MINB>
__global__ void __launch_bounds__(kConvThreads, MINB) conv_kernel(const ConvArgs p) {
    using G = Geo<K, CIN, N>;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ __align__(8) uint64_t full[G::bufs], empty[G::bufs], tfull[2], tempty[2];
    __shared__ uint32_t tbase;
    __shared__ volatile int quit;
    __shared__ __align__(16) float sbias[N];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t *sB = sm + G::bufs * G::abytes;
    if (warp == 0) umma::tmem_alloc(&tbase, G::tmem);
    if (tid == 0) {
        quit = 0;
        for (int i = 0; i < G::bufs; i++) {
            umma::mbar_init(&full[i], 128);
            umma::mbar_init(&empty[i]);
        }
        for (int i = 0; i < 2; i++) {
            umma::mbar_init(&tfull[i]);
            umma::mbar_init(&tempty[i], 128);
        }
        umma::mbar_init_fence();
    }
    // weights: a sub-tile of N x 16 per tap and 16 channels
    for (int q = tid; q < 9 * G::chunks * N; q += kConvThreads) {
        const int k8 = q % (9 * G::chunks), n = q / (9 * G::chunks);
        umma::copy16(umma::smem_u32(sB) + (k8 >> 1) * (N * 32) + (n >> 3) * 256 + (k8 & 1) * 128 + (n & 7) * 16,
                     p.w + (size_t)n * 9 * CIN + k8 * 8, true);
    }
    if constexpr (!GRAD)
        for (int n = tid; n < N; n += kConvThreads) sbias[n] = p.bias[n];
    umma::copy_commit();
    umma::copy_wait<0>();
    umma::fence_async_smem();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tbase;
    bool ok = true;
    if (p.probe) {  // test hook: a wait on a phase that nothing completes, before any MMA is issued
        if (tid == 0) ok = umma::mbar_wait(&tfull[0], 0, p.wait_ns);
        ok = __syncthreads_and(ok) != 0;
    }
    const int per_image = p.tx * p.ty;
    const int mine = ok && (int)blockIdx.x < p.tiles ? (p.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    auto tile_at = [&](int it, int &img, int &y0, int &x0) {
        const int t = blockIdx.x + it * gridDim.x;
        img = t / per_image;
        const int r = t - img * per_image;
        y0 = r / p.tx * G::rows;
        x0 = (r - r / p.tx * p.tx) * G::cols;
    };
    if (warp >= 4 && warp < 8) {
        // ---- copies of the source tiles
        const int pt = tid - 128;
        for (int it = 0; it < mine; it++) {
            const int b = it % G::bufs;
            if (it >= G::bufs) ok = umma::mbar_wait(&empty[b], (it / G::bufs - 1) & 1, p.wait_ns, &quit);
            if (!ok) break;
            int img, y0, x0;
            tile_at(it, img, y0, x0);
            const int sy0 = (G::half ? 2 * y0 : y0) - 1, sx0 = (G::half ? 2 * x0 : x0) - 1;
            const __nv_bfloat16 *src = p.src + (size_t)img * p.sh * p.sw * CIN;
            const uint32_t dst = umma::smem_u32(sm) + b * G::abytes;
#pragma unroll 4
            for (int q = pt; q < G::srows * G::scols * G::chunks; q += 128) {
                const int ch = q % G::chunks, px = q / G::chunks, r = px / G::scols, c = px - r * G::scols;
                const int y = sy0 + r, x = sx0 + c;
                const bool in = (unsigned)y < (unsigned)p.sh && (unsigned)x < (unsigned)p.sw;
                umma::copy16(dst + ch * G::plane + G::place(r, c) * 16,
                             src + (in ? ((size_t)y * p.sw + x) * CIN + ch * 8 : 0), in);
            }
            umma::copy_commit();
            if (it > 0) {  // the tile before this one has arrived
                umma::copy_wait<1>();
                umma::fence_async_smem();
                umma::mbar_arrive(&full[(it - 1) % G::bufs]);
            }
        }
        umma::copy_wait<0>();
        umma::fence_async_smem();
        if (ok && mine > 0) umma::mbar_arrive(&full[(mine - 1) % G::bufs]);
    } else if (tid == 256) {
        // ---- MMAs of a tile, per GEMM tap by tap and 16 channels at a time
        constexpr uint32_t idesc = umma::idesc_bf16(128, N);
        const uint64_t db = umma::smem_desc(umma::smem_u32(sB));
        int issued = 0;
        for (int it = 0; it < mine; it++) {
            const int b = it % G::bufs, s = it & 1;
            ok = umma::mbar_wait(&full[b], (it / G::bufs) & 1, p.wait_ns, &quit);
            if (ok && it >= 2) ok = umma::mbar_wait(&tempty[s], ((it >> 1) - 1) & 1, p.wait_ns, &quit);
            if (!ok) break;
            umma::fence_after();
            const uint64_t da = umma::smem_desc(umma::smem_u32(sm) + b * G::abytes, G::plane, G::sbo);
#pragma unroll
            for (int j = 0; j < G::gemms; j++) {
                const uint32_t d = tmem + s * G::stage + j * N;
                bool first = true;
#pragma unroll
                for (int sub = 0; sub < (K == kUp2T ? 4 : 1); sub++)
#pragma unroll
                    for (int tap = 0; tap < 9; tap++) {
                        const int dy = tap / 3, dx = tap % 3, py = j >> 1, px = j & 1;
                        int ay, ax;
                        if (K == kSame) {
                            ay = GRAD ? 2 - dy : dy;
                            ax = (GRAD ? 2 - dx : dx) + 8 * j;
                        } else if (K == kStride2) {
                            ay = dy;
                            ax = dx;
                        } else if (K == kUp2) {
                            ay = 1 + ((py + dy - 1) >> 1);
                            ax = 1 + ((px + dx - 1) >> 1);
                        } else if (K == kStride2T) {
                            if (((py + 1 - dy) & 1) || ((px + 1 - dx) & 1)) continue;  // no such output pixel
                            ay = 1 + (py + 1 - dy) / 2;
                            ax = 1 + (px + 1 - dx) / 2;
                        } else {
                            ay = (sub >> 1) + 2 - dy;
                            ax = (sub & 1) + 2 - dx;
                        }
                        const int at = G::place(ay, ax);
#pragma unroll
                        for (int kc = 0; kc < CIN / 16; kc++) {
                            umma::mma_bf16(d, da + (uint64_t)((2 * kc * G::plane + at * 16) >> 4),
                                           db + (uint64_t)(((tap * (CIN / 16) + kc) * N * 32) >> 4), idesc, !first);
                            first = false;
                        }
                    }
            }
            umma::mma_commit(&empty[b]);
            umma::mma_commit(&tfull[s]);
            issued = it + 1;
        }
        // every issued MMA has completed once the last commit has
        if (issued > 0 && !umma::mbar_wait(&tfull[(issued - 1) & 1], ((issued - 1) >> 1) & 1, kDrainNs)) ok = false;
    } else if (warp < 4) {
        // ---- results: thread = row of the GEMMs = pixel
        const int r = tid >> 3, c = tid & 7;
        float sum[GRAD ? N : 1];
        if constexpr (GRAD)
            for (int n = 0; n < N; n++) sum[n] = 0.f;
        for (int it = 0; it < mine; it++) {
            const int s = it & 1;
            int img, y0, x0;
            tile_at(it, img, y0, x0);
            bool in = false;
            size_t at = 0;
            uint4 m[GRAD ? N / 8 : 1];  // a GEMM's masks, on their way while its MMAs run
            auto pixel = [&](int j) {
                const int y = G::fine ? 2 * (y0 + r) + (j >> 1) : y0 + r;
                const int x = G::fine ? 2 * (x0 + c) + (j & 1) : x0 + c + 8 * j;
                in = y < p.oh && x < p.ow;
                at = in ? (((size_t)img * p.oh + y) * p.ow + x) * N : 0;
                if constexpr (GRAD)
                    if (p.mask)
#pragma unroll
                        for (int i = 0; i < N / 8; i++) m[i] = reinterpret_cast<const uint4 *>(p.mask + at)[i];
            };
            pixel(0);
            ok = umma::mbar_wait(&tfull[s], (it >> 1) & 1, p.wait_ns, &quit);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            umma::fence_after();
#pragma unroll
            for (int j = 0; j < G::gemms; j++) {
                if (j > 0) pixel(j);
#pragma unroll
                for (int n0 = 0; n0 < N; n0 += 16) {
                    uint32_t v[16];
                    umma::tmem_ld(tmem + ((uint32_t)(warp * 32) << 16) + s * G::stage + j * N + n0, v);
                    umma::tmem_wait();
                    uint32_t o[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        float a = __uint_as_float(v[2 * i]), b = __uint_as_float(v[2 * i + 1]);
                        if constexpr (GRAD) {
                            if (p.mask) {
                                const uint4 q = m[n0 / 8 + i / 4];
                                const uint32_t w = i % 4 == 0 ? q.x : i % 4 == 1 ? q.y : i % 4 == 2 ? q.z : q.w;
                                a = __uint_as_float(w << 16) > 0.f ? a : 0.f;
                                b = __uint_as_float(w & 0xffff0000u) > 0.f ? b : 0.f;
                            }
                        } else {
                            a += sbias[n0 + 2 * i];
                            b += sbias[n0 + 2 * i + 1];
                            if (p.relu) {
                                a = fmaxf(a, 0.f);
                                b = fmaxf(b, 0.f);
                            }
                            v[2 * i] = __float_as_uint(a);
                            v[2 * i + 1] = __float_as_uint(b);
                        }
                        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
                        o[i] = *reinterpret_cast<const uint32_t *>(&h);
                        if constexpr (GRAD) {
                            if (in) {
                                sum[n0 + 2 * i] += __bfloat162float(h.x);
                                sum[n0 + 2 * i + 1] += __bfloat162float(h.y);
                            }
                        }
                    }
                    if (in) {
                        umma::store32(p.out + at + n0, o);
                        if constexpr (!GRAD)
                            if (p.out32) {
                                uint32_t h[8];
#pragma unroll
                                for (int i = 0; i < 8; i++) h[i] = v[i];
                                umma::store32(p.out32 + at + n0, h);
#pragma unroll
                                for (int i = 0; i < 8; i++) h[i] = v[8 + i];
                                umma::store32(p.out32 + at + n0 + 8, h);
                            }
                    }
                }
            }
            umma::fence_before();
            umma::mbar_arrive(&tempty[s]);
        }
        if constexpr (GRAD)
            if (p.db && ok)
#pragma unroll
                for (int n = 0; n < N; n++) {
                    float v = sum[n];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                    if (lane == 0 && mine > 0) atomicAdd(p.db + n, v);
                }
    }
    umma::fence_before();
    if (__syncthreads_and(ok) == 0 && tid == 0) set_error(p.err, ERR_TIMEOUT);
    umma::fence_after();
    if (warp == 0) umma::tmem_free(tmem, G::tmem);
}

template <Kind K, int CIN, int N, bool GRAD, int MINB>
void launch(ConvArgs a, int T, int gh, int gw, cudaStream_t s) {
    using G = Geo<K, CIN, N>;
    constexpr int kSmBytes = 228 * 1024, kReserved = 1024;
    // no more blocks on an SM than its 512 TMEM columns serve: a larger
    // allocation keeps further ones off
    constexpr int per_sm = 512 / G::tmem;
    constexpr int floor_bytes = kSmBytes / (per_sm + 1) - kReserved + 16;
    constexpr int smem = G::smem > floor_bytes ? G::smem : floor_bytes;
    static_assert(smem <= 227 * 1024, "a block's shared memory");
    const auto kernel = conv_kernel<K, CIN, N, GRAD, MINB>;
    const KernelShape ks = kernel_setup((const void *)kernel, kConvThreads, smem);
    a.ty = (gh + G::rows - 1) / G::rows;
    a.tx = (gw + G::cols - 1) / G::cols;
    a.tiles = T * a.ty * a.tx;
    a.wait_ns = (unsigned long long)test_hooks().wait_ns.load();
    a.probe = test_hooks().mbar_probe.load();
    const int blocks = std::min(a.tiles, ks.sms * std::min(ks.blocks_per_sm, per_sm));
    kernel<<<blocks, kConvThreads, smem, s>>>(a);
}

[[noreturn]] void no_kernel(const ConvSpec &c) {
    throw Error(ERR_INVALID, "no convolution kernel for " + std::to_string(c.cin) + " -> " + std::to_string(c.cout) +
                                 " channels, mode " + std::to_string(c.mode));
}

}  // namespace

void launch_conv_fwd(const ConvSpec &c, int T, const __nv_bfloat16 *X, const __nv_bfloat16 *W, const float *bias,
                     __nv_bfloat16 *Y, float *Y32, int *err, cudaStream_t s) {
    ConvArgs a{};
    a.src = X; a.w = W; a.sh = c.hin; a.sw = c.win; a.oh = c.hout; a.ow = c.wout;
    a.relu = c.relu; a.bias = bias; a.out = Y; a.out32 = Y32; a.err = err;
    const int key = c.mode * 10000 + c.cin * 100 + c.cout;
    if (key == 1632) launch<kSame, 16, 32, false, 3>(a, T, c.hout, c.wout, s);
    else if (key == 6464) launch<kSame, 64, 64, false, 1>(a, T, c.hout, c.wout, s);
    else if (key == 3216) launch<kSame, 32, 16, false, 2>(a, T, c.hout, c.wout, s);
    else if (key == 13264) launch<kStride2, 32, 64, false, 1>(a, T, c.hout, c.wout, s);
    else if (key == 26432) launch<kUp2, 64, 32, false, 2>(a, T, c.hin, c.win, s);
    else no_kernel(c);
}

void launch_conv_dgrad(const ConvSpec &c, int T, const __nv_bfloat16 *dY, const __nv_bfloat16 *WT,
                       const __nv_bfloat16 *Aprev, __nv_bfloat16 *dXpre, float *db, int *err, cudaStream_t s) {
    ConvArgs a{};
    a.src = dY; a.w = WT; a.sh = c.hout; a.sw = c.wout; a.oh = c.hin; a.ow = c.win;
    a.mask = Aprev; a.out = dXpre; a.db = db; a.err = err;
    const int key = c.mode * 10000 + c.cin * 100 + c.cout;
    if (key == 6464) launch<kSame, 64, 64, true, 1>(a, T, c.hin, c.win, s);
    else if (key == 3216) launch<kSame, 16, 32, true, 2>(a, T, c.hin, c.win, s);
    else if (key == 13264) launch<kStride2T, 64, 32, true, 2>(a, T, c.hout, c.wout, s);
    else if (key == 26432) launch<kUp2T, 32, 64, true, 1>(a, T, c.hin, c.win, s);
    else no_kernel(c);
}

}  // namespace igr
