// Convolutions of the learned congestion seed and their gradients as implicit
// GEMMs on the tcgen05 tensor cores.
//
// The forward convolutions and the input gradients multiply rows = output pixels by columns = output channels over
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
// (cp.async, three in flight), one thread issues a tile's MMAs, eight warps write
// the previous tile's results from TMEM (two stages).  The weights stay in
// shared memory.  What bounds it: the MMAs read their operands from shared
// memory, 6 KB for 128 x 64 x 16, so N = 64 cannot pass a third of the tensor
// peak, and the activations pass through HBM once per layer; the input
// gradients also read the mask and keep the sums of the bias gradients.
// Gathering each tap's operands anew through registers, as the kernel before it
// did, moved nine times the tile.  16 tiles of 288 x 288: forward pass 2.03 ->
// 0.37 ms (135 GFLOP, 350 TFLOP/s by events around each convolution), input
// gradients with the bias gradients 2.10 + 0.56 -> 0.40 ms.  Of the 49 us of a
// 64-channel layer 18 go to the MMAs, 6 to the copies, 5 to the stores and 20 to
// the launch and the hand-over between the roles (measured by leaving each out).
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
    static_assert(K != kStride2 && K != kUp2T || N >= 32, "a group's columns");
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

constexpr int kConvThreads = 416;  // warps 0-7 results, 8-11 copies, 12 MMAs
constexpr int kWgradThreads = 288;

template <Kind K, int CIN, int N, bool GRAD, int MINB>
__global__ void __launch_bounds__(kConvThreads, MINB) conv_kernel(const ConvArgs p) {
    using G = Geo<K, CIN, N>;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ __align__(8) uint64_t full[G::bufs], empty[G::bufs], tfull[2], tempty[2], weights;
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
            umma::mbar_init(&tempty[i], 256);
        }
        umma::mbar_init(&weights, 256);
        umma::mbar_init_fence();
    }
    if constexpr (!GRAD)
        for (int n = tid; n < N; n += kConvThreads) sbias[n] = p.bias[n];
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
    if (warp >= 8 && warp < 12) {
        // ---- copies of the source tiles
        const int pt = tid - 256;
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
    } else if (tid == 384) {
        // ---- MMAs of a tile, per GEMM tap by tap and 16 channels at a time
        constexpr uint32_t idesc = umma::idesc_bf16(128, N);
        const uint64_t db = umma::smem_desc(umma::smem_u32(sB));
        int issued = 0;
        if (mine > 0) ok = umma::mbar_wait(&weights, 0, p.wait_ns, &quit);
        for (int it = 0; it < mine && ok; it++) {
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
    } else if (warp < 8) {
        // ---- weights first: a sub-tile of N x 16 per tap and 16 channels
        for (int q = tid; q < 9 * G::chunks * N; q += 256) {
            const int k8 = q % (9 * G::chunks), n = q / (9 * G::chunks);
            umma::copy16(umma::smem_u32(sB) + (k8 >> 1) * (N * 32) + (n >> 3) * 256 + (k8 & 1) * 128 + (n & 7) * 16,
                         p.w + (size_t)n * 9 * CIN + k8 * 8, true);
        }
        umma::copy_commit();
        umma::copy_wait<0>();
        umma::fence_async_smem();
        umma::mbar_arrive(&weights);
        // ---- results: thread = row of the GEMMs = pixel; the two groups of four warps
        //      share a tile's GEMMs, or the columns of a single one
        constexpr int kCols = G::gemms == 1 ? N / 2 : N;  // columns of a group
        constexpr int kBatch = kCols < 32 ? kCols : 32;   // columns in flight
        const int group = warp >> 2, r = (tid & 127) >> 3, c = tid & 7;
        const int col0 = G::gemms == 1 ? group * kCols : 0;
        float sum[GRAD ? kCols : 1];
        if constexpr (GRAD)
            for (int n = 0; n < kCols; n++) sum[n] = 0.f;
        for (int it = 0; it < mine; it++) {
            const int s = it & 1;
            int img, y0, x0;
            tile_at(it, img, y0, x0);
            bool in = false;
            size_t at = 0;
            uint4 m[GRAD ? kCols / 8 : 1];  // a GEMM's masks, on their way while its MMAs run
            auto pixel = [&](int j) {
                const int y = G::fine ? 2 * (y0 + r) + (j >> 1) : y0 + r;
                const int x = G::fine ? 2 * (x0 + c) + (j & 1) : x0 + c + 8 * j;
                in = y < p.oh && x < p.ow;
                at = in ? (((size_t)img * p.oh + y) * p.ow + x) * N + col0 : 0;
                if constexpr (GRAD) {
                    if (p.mask) {
#pragma unroll
                        for (int i = 0; i < kCols / 8; i++) m[i] = reinterpret_cast<const uint4 *>(p.mask + at)[i];
                    }
                }
            };
            const int j0 = G::gemms == 1 ? 0 : group;
            pixel(j0);
            ok = umma::mbar_wait(&tfull[s], (it >> 1) & 1, p.wait_ns, &quit);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            umma::fence_after();
#pragma unroll
            for (int jj = 0; jj < (G::gemms + 1) / 2; jj++) {
                const int j = j0 + 2 * jj;
                if (jj > 0) pixel(j);
#pragma unroll
                for (int b0 = 0; b0 < kCols; b0 += kBatch) {
                    uint32_t v[kBatch / 16][16];
#pragma unroll
                    for (int k = 0; k < kBatch / 16; k++)
                        umma::tmem_ld(tmem + ((uint32_t)((warp & 3) * 32) << 16) + s * G::stage + j * N + col0 + b0 +
                                          16 * k, v[k]);
                    umma::tmem_wait();
#pragma unroll
                    for (int k = 0; k < kBatch / 16; k++) {
                        const int n0 = b0 + 16 * k;
                        uint32_t o[8];
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            float a = __uint_as_float(v[k][2 * i]), b = __uint_as_float(v[k][2 * i + 1]);
                            if constexpr (GRAD) {
                                if (p.mask) {
                                    const uint4 q = m[n0 / 8 + i / 4];
                                    const uint32_t w = i % 4 == 0 ? q.x : i % 4 == 1 ? q.y : i % 4 == 2 ? q.z : q.w;
                                    a = __uint_as_float(w << 16) > 0.f ? a : 0.f;
                                    b = __uint_as_float(w & 0xffff0000u) > 0.f ? b : 0.f;
                                }
                            } else {
                                const float2 bb = *reinterpret_cast<const float2 *>(&sbias[col0 + n0 + 2 * i]);
                                a += bb.x;
                                b += bb.y;
                                if (p.relu) {
                                    a = fmaxf(a, 0.f);
                                    b = fmaxf(b, 0.f);
                                }
                                v[k][2 * i] = __float_as_uint(a);
                                v[k][2 * i + 1] = __float_as_uint(b);
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
                                    for (int i = 0; i < 8; i++) h[i] = v[k][i];
                                    umma::store32(p.out32 + at + n0, h);
#pragma unroll
                                    for (int i = 0; i < 8; i++) h[i] = v[k][8 + i];
                                    umma::store32(p.out32 + at + n0 + 8, h);
                                }
                        }
                    }
                }
            }
            umma::fence_before();
            umma::mbar_arrive(&tempty[s]);
        }
        if constexpr (GRAD) {
            if (p.db && ok && mine > 0) {
                // sums over the lanes: half of the channels change hands at each step,
                // until lane l has channels l kCols / 32 ..
#pragma unroll
                for (int st = 0; st < 5; st++) {
                    const int o = 16 >> st, half = kCols >> (st + 1);
                    const bool up = lane & o;
#pragma unroll
                    for (int n = 0; n < (kCols >> (st + 1)); n++) {
                        const float give = up ? sum[n] : sum[n + half];
                        sum[n] = (up ? sum[n + half] : sum[n]) + __shfl_xor_sync(0xffffffffu, give, o);
                    }
                }
#pragma unroll
                for (int n = 0; n < kCols / 32; n++) atomicAdd(p.db + col0 + lane * (kCols / 32) + n, sum[n]);
            }
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

// ---------------------------------------------------------------- weight gradients
//
// dW[tap][ci][co] = sum over pixels of X[pixel + tap][ci] dY[pixel][co]: K is the
// pixels, so both operands are MN-major, and the planes of 8 channels serve
// again: 16 pixels of a tile row are the two K groups of an MMA.  A tile lies
// [row][plane][pixel], so that an operand of 128 rows, or of N columns, covers
// several tile rows of channels: A takes 128 / CA rows of its tensor, B the rows
// of the other one that any of them meets under a tap, and one MMA makes the
// products of all these row pairs for one horizontal shift.  The tap of a pair is
// the difference of its rows; pairs further apart are not read out.  All of an
// SM's sums stay in TMEM over its tiles (at most 512 columns) and go to memory
// once, by f32 additions.
//
// wSame: both tensors at one resolution; A is dY, or X where it has more
// channels.  wUp2 (X at half the resolution of dY): A is X, B the pixels of dY of
// one row parity (a block's) and both column parities; nearest upsampling gives
// the taps that read the same X pixel the same product, which is added to each.
// wStride2 (X at twice the resolution of dY): A is dY, B the four parities of X.
// Bound by the operand reads from shared memory (8 KB for 128 x 128 x 16) and
// the copies of the tiles; transposing both operands through registers element
// by element, as the kernel before it did, took 3.62 ms for 16 tiles of 288 x 288
// (now 0.38 ms: 51 and 61 us for the two layers at full resolution, 52 for the
// strided one and for each of the 64-channel layers, 110 for the upsampled one).
enum WKind { wSame, wUp2, wStride2 };

template <WKind K, bool AX, int CA, int CB, int CBALL>
struct WGeo {
    static constexpr int arows = 128 / CA;               // rows of A in an MMA
    static constexpr int rows = K == wStride2 ? 8 : 16;  // tile rows of A
    static constexpr int ach = CA / 8, bch = CB / 8;
    static constexpr int parts = K == wSame ? 1 : K == wUp2 ? 2 : 4;  // parity classes of B
    static constexpr int brows = K == wStride2 ? rows + 1 : rows + 2;
    static constexpr int bcols = K == wStride2 ? 17 : 18;
    static constexpr int apitch = 17, bpitch = bcols | 1;  // odd: the copies meet no bank conflict
    static constexpr int part = brows * bch * bpitch * 16;
    static constexpr int abytes = rows * ach * apitch * 16;
    static constexpr int bytes = (abytes + parts * part + 127) / 128 * 128;
    static constexpr int bufs = K == wUp2 ? 2 : 3;
    static constexpr int smem = bufs * bytes;
    // columns of TMEM: one MMA's N per horizontal shift (and row parity)
    static constexpr int n = K == wSame ? (arows + 2) * CB : 3 * CB;
    static constexpr int shifts = K == wUp2 ? 4 : 3;
    static constexpr int columns = shifts * n + (K == wStride2 ? shifts * 2 * CB : 0);
    static_assert(columns <= 512 && n % 16 == 0 && n <= 256, "the sums of an SM");
};

struct WgradArgs {
    const __nv_bfloat16 *A, *B;  // channels-last; CA and CBALL channels
    int ah, aw, bh, bw;
    int tiles, tx, ty;
    float *dWT;                  // [9][cin][cout]
    int cin, cout;
    int *err;
    unsigned long long wait_ns;
    int probe;
};

__device__ __forceinline__ void add4(float *p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <WKind K, bool AX, int CA, int CB, int CBALL>
__global__ void __launch_bounds__(kWgradThreads, 1) wgrad_kernel(const WgradArgs p) {
    using G = WGeo<K, AX, CA, CB, CBALL>;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ __align__(8) uint64_t full[G::bufs], empty[G::bufs], done;
    __shared__ uint32_t tbase;
    __shared__ volatile int quit;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int half = blockIdx.y;  // wSame: which CB channels of B; wUp2: row parity of dY
    if (warp == 0) umma::tmem_alloc(&tbase, 512);
    if (tid == 0) {
        quit = 0;
        for (int i = 0; i < G::bufs; i++) {
            umma::mbar_init(&full[i], 256);
            umma::mbar_init(&empty[i]);
        }
        umma::mbar_init(&done);
        umma::mbar_init_fence();
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tbase;
    bool ok = true;
    if (p.probe) {  // test hook: a wait on a phase that nothing completes, before any MMA is issued
        if (tid == 0) ok = umma::mbar_wait(&done, 0, p.wait_ns);
        ok = __syncthreads_and(ok) != 0;
    }
    const int per_image = p.tx * p.ty;
    const int mine = ok && (int)blockIdx.x < p.tiles ? (p.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (warp < 8) {
        for (int it = 0; it < mine; it++) {
            const int b = it % G::bufs;
            if (it >= G::bufs) ok = umma::mbar_wait(&empty[b], (it / G::bufs - 1) & 1, p.wait_ns, &quit);
            if (!ok) break;
            const int t = blockIdx.x + it * gridDim.x, img = t / per_image, rem = t - img * per_image;
            const int y0 = rem / p.tx * G::rows, x0 = (rem - rem / p.tx * p.tx) * 16;
            const uint32_t dst = umma::smem_u32(sm) + b * G::bytes;
            const __nv_bfloat16 *A = p.A + (size_t)img * p.ah * p.aw * CA;
#pragma unroll 4
            for (int q = tid; q < G::rows * 16 * G::ach; q += 256) {
                const int ch = q % G::ach, px = q / G::ach, r = px >> 4, c = px & 15;
                const int y = y0 + r, x = x0 + c;
                const bool in = y < p.ah && x < p.aw;
                umma::copy16(dst + ((r * G::ach + ch) * G::apitch + c) * 16,
                             A + (in ? ((size_t)y * p.aw + x) * CA + ch * 8 : 0), in);
            }
            const __nv_bfloat16 *B = p.B + (size_t)img * p.bh * p.bw * CBALL + (K == wSame ? half * CB : 0);
#pragma unroll 4
            for (int q = tid; q < G::parts * G::brows * G::bcols * G::bch; q += 256) {
                const int ch = q % G::bch, px = q / G::bch, part = px / (G::brows * G::bcols);
                const int rc = px - part * (G::brows * G::bcols), r = rc / G::bcols, c = rc - r * G::bcols;
                int y = y0 - 1 + r, x = x0 - 1 + c;
                if (K == wUp2) {  // part: column parity
                    y = 2 * y + half;
                    x = 2 * x + part;
                } else if (K == wStride2) {  // part: row parity, column parity
                    y = 2 * y + (part >> 1);
                    x = 2 * x + (part & 1);
                }
                const bool in = (unsigned)y < (unsigned)p.bh && (unsigned)x < (unsigned)p.bw;
                umma::copy16(dst + G::abytes + part * G::part + ((r * G::bch + ch) * G::bpitch + c) * 16,
                             B + (in ? ((size_t)y * p.bw + x) * CBALL + ch * 8 : 0), in);
            }
            umma::copy_commit();
            if (it > 0) {
                umma::copy_wait<1>();
                umma::fence_async_smem();
                umma::mbar_arrive(&full[(it - 1) % G::bufs]);
            }
        }
        umma::copy_wait<0>();
        umma::fence_async_smem();
        if (ok && mine > 0) umma::mbar_arrive(&full[(mine - 1) % G::bufs]);
    } else if (lane == 0) {
        constexpr uint32_t idesc = umma::idesc_bf16_mn(128, G::n);
        int issued = 0;
        for (int it = 0; it < mine; it++) {
            const int b = it % G::bufs;
            ok = umma::mbar_wait(&full[b], (it / G::bufs) & 1, p.wait_ns, &quit);
            if (!ok) break;
            umma::fence_after();
            const uint32_t base = umma::smem_u32(sm) + b * G::bytes;
            const uint64_t da = umma::smem_desc(base, 128, G::apitch * 16);
            const uint64_t db = umma::smem_desc(base + G::abytes, 128, G::bpitch * 16);
            // start of row r, column c of part q of B
            auto at = [](int q, int r, int c) { return (uint64_t)((q * G::part + (r * G::bch * G::bpitch + c) * 16) >> 4); };
            for (int g = 0; g < G::rows; g += G::arows) {
                const uint64_t a = da + (uint64_t)(g * G::ach * G::apitch);
                const bool acc = it > 0 || g > 0;
                if (K == wSame) {
#pragma unroll
                    for (int e = 0; e < 3; e++)
                        umma::mma_bf16(tmem + e * G::n, a, db + at(0, g, e), idesc, acc);
                } else if (K == wUp2) {
#pragma unroll
                    for (int e = 0; e < 4; e++)  // column parity e >> 1, X column minus dY column - 1 + (e >> 1) + (e & 1)
                        umma::mma_bf16(tmem + e * G::n, a,
                                       db + at(e >> 1, g + 1 - half, 2 - (e >> 1) - (e & 1)), idesc, acc);
                } else {
                    constexpr uint32_t ieven = umma::idesc_bf16_mn(128, 2 * CB);
#pragma unroll
                    for (int dx = 0; dx < 3; dx++) {
                        const int qx = dx == 1 ? 0 : 1, c = dx == 0 ? 0 : 1;
                        umma::mma_bf16(tmem + dx * G::n, a, db + at(2 + qx, g, c), idesc, acc);
                        umma::mma_bf16(tmem + 3 * G::n + dx * 2 * CB, a, db + at(qx, g + 1, c), ieven, acc);
                    }
                }
            }
            umma::mma_commit(&empty[b]);
            issued = it + 1;
        }
        if (issued > 0) {
            umma::mma_commit(&done);
            if (!umma::mbar_wait(&done, 0, kDrainNs)) ok = false;
        }
    }
    umma::fence_before();
    const bool good = __syncthreads_and(ok) != 0;
    umma::fence_after();
    if (good && mine > 0 && warp < 4) {
        const int a = tid / CA, ca = tid % CA;  // row and channel of A
        auto place = [&](int ty, int tx, int cb) {
            const int ci = AX || K == wUp2 ? ca : (K == wSame ? half * CB : 0) + cb;
            const int co = AX || K == wUp2 ? cb : ca;
            return p.dWT + ((size_t)(ty * 3 + tx) * p.cin + ci) * p.cout + co;
        };
        for (int n0 = 0; n0 < G::columns; n0 += 16) {
            uint32_t v[16];
            umma::tmem_ld(tmem + ((uint32_t)(warp * 32) << 16) + n0, v);
            umma::tmem_wait();
            const bool even = K == wStride2 && n0 >= 3 * G::n;
            const int e = even ? (n0 - 3 * G::n) / (2 * CB) : n0 / G::n;
            const int left = even ? n0 - 3 * G::n - e * 2 * CB : n0 - e * G::n;
            const int b = left / CB, cb = left - b * CB;
            // the taps this pair of rows and this shift belong to
            int ty0 = 0, ty1 = -1, tx0 = 0, tx1 = -1;
            if (K == wSame) {
                const int ey = b - a;
                if (ey >= 0 && ey <= 2) ty0 = ty1 = AX ? 2 - ey : ey;
                tx0 = tx1 = AX ? 2 - e : e;
            } else if (K == wUp2) {
                // X pixel minus dY pixel at half resolution: parity 0: -1 (tap 0), 0 (taps 1, 2);
                // parity 1: 0 (taps 0, 1), 1 (tap 2)
                const int oy = a - b + half, ox = -1 + (e >> 1) + (e & 1), px = e >> 1;
                if (half == 0 && oy == -1) ty0 = ty1 = 0;
                if (half == 0 && oy == 0) { ty0 = 1; ty1 = 2; }
                if (half == 1 && oy == 0) { ty0 = 0; ty1 = 1; }
                if (half == 1 && oy == 1) ty0 = ty1 = 2;
                if (px == 0 && ox == -1) tx0 = tx1 = 0;
                if (px == 0 && ox == 0) { tx0 = 1; tx1 = 2; }
                if (px == 1 && ox == 0) { tx0 = 0; tx1 = 1; }
                if (px == 1 && ox == 1) tx0 = tx1 = 2;
            } else {
                if (even) {
                    if (b == a) ty0 = ty1 = 1;
                } else {
                    if (b == a) ty0 = ty1 = 0;
                    if (b == a + 1) ty0 = ty1 = 2;
                }
                tx0 = tx1 = e;
            }
            for (int ty = ty0; ty <= ty1; ty++)
                for (int tx = tx0; tx <= tx1; tx++) {
                    if (AX || K == wUp2) {
                        float *q = place(ty, tx, cb);
#pragma unroll
                        for (int i = 0; i < 16; i += 4)
                            add4(q + i, __uint_as_float(v[i]), __uint_as_float(v[i + 1]), __uint_as_float(v[i + 2]),
                                 __uint_as_float(v[i + 3]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; i++) atomicAdd(place(ty, tx, cb + i), __uint_as_float(v[i]));
                    }
                }
        }
        umma::fence_before();
    } else if (!good && tid == 0) {
        set_error(p.err, ERR_TIMEOUT);
    }
    __syncthreads();
    if (warp == 0) umma::tmem_free(tmem, 512);
}

template <WKind K, bool AX, int CA, int CB, int CBALL>
void launch_wgrad(WgradArgs a, int T, int halves, cudaStream_t s) {
    using G = WGeo<K, AX, CA, CB, CBALL>;
    constexpr int floor_bytes = 228 * 1024 / 2 - 1024 + 16;  // one block holds an SM's TMEM
    constexpr int smem = G::smem > floor_bytes ? G::smem : floor_bytes;
    static_assert(smem <= 227 * 1024, "a block's shared memory");
    const auto kernel = wgrad_kernel<K, AX, CA, CB, CBALL>;
    const KernelShape ks = kernel_setup((const void *)kernel, kWgradThreads, smem);
    a.ty = (a.ah + G::rows - 1) / G::rows;
    a.tx = (a.aw + 15) / 16;
    a.tiles = T * a.ty * a.tx;
    a.wait_ns = (unsigned long long)test_hooks().wait_ns.load();
    a.probe = test_hooks().mbar_probe.load();
    kernel<<<dim3(std::min(a.tiles, ks.sms / halves), halves), kWgradThreads, smem, s>>>(a);
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
    if (key == 1632) launch<kSame, 16, 32, false, 2>(a, T, c.hout, c.wout, s);
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
    else if (key == 3216) launch<kSame, 16, 32, true, 1>(a, T, c.hin, c.win, s);
    else if (key == 13264) launch<kStride2T, 64, 32, true, 1>(a, T, c.hout, c.wout, s);
    else if (key == 26432) launch<kUp2T, 32, 64, true, 1>(a, T, c.hin, c.win, s);
    else no_kernel(c);
}

void launch_conv_wgrad(const ConvSpec &c, int T, const __nv_bfloat16 *X, const __nv_bfloat16 *dY, float *dWT,
                       int *err, cudaStream_t s) {
    WgradArgs a{};
    a.dWT = dWT; a.cin = c.cin; a.cout = c.cout; a.err = err;
    auto of_x = [&](const __nv_bfloat16 *&t, int &h, int &w) { t = X; h = c.hin; w = c.win; };
    auto of_dy = [&](const __nv_bfloat16 *&t, int &h, int &w) { t = dY; h = c.hout; w = c.wout; };
    const int key = c.mode * 10000 + c.cin * 100 + c.cout;
    if (key == 3216 || key == 26432) {  // A is X
        of_x(a.A, a.ah, a.aw);
        of_dy(a.B, a.bh, a.bw);
        if (key == 3216) launch_wgrad<wSame, true, 32, 16, 16>(a, T, 1, s);
        else launch_wgrad<wUp2, true, 64, 32, 32>(a, T, 2, s);
        return;
    }
    of_dy(a.A, a.ah, a.aw);
    of_x(a.B, a.bh, a.bw);
    if (key == 1632) launch_wgrad<wSame, false, 32, 16, 16>(a, T, 1, s);
    else if (key == 6464) launch_wgrad<wSame, false, 64, 32, 64>(a, T, 2, s);
    else if (key == 13264) launch_wgrad<wStride2, false, 64, 32, 32>(a, T, 1, s);
    else no_kernel(c);
}

}  // namespace igr
