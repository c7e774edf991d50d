// Phase-1 conflict shapes and claim lists of the batch colouring, built on the
// device from the flattened trees already resident there.
//
// The shapes of a routing net (net::construct_rsmt, src/database_cuda.hpp:
// 746-820) are its tree nodes as points and, per tree edge, its segments and
// end or corner points; the claims (generate_batches_rsmt_gpu,
// src/database_cuda.hpp:288-434) are the cell, left, right and lower cells of
// every point and every `sparsity`-th cell of every segment.  They depend only
// on the set of tree edges, so they are generated here from the (node,
// parent) pairs of the DFS-ordered trees; the colouring treats points and
// claims as sets, so the order inside a net is free.  Two passes: counts per
// net with their exclusive sums (sums per block, one block over those, then the
// offsets: one block over all nets took 2.9 ms for the 1.4M routing nets of the
// 800k-net design, now 24 µs), then the fill.  The rip-up passes
// use the same kernels for the rerouted nets, with the DAG points given and
// the segments of their trees.
#include "kcommon.cuh"

#include <algorithm>

namespace igr {

namespace {

constexpr int kScanThreads = 1024;

template <class Pt, class Hs, class Vs>
__device__ __forceinline__ void net_shapes(const int *nodes, const int *par, int m, int X, int Y, Pt &&point,
                                           Hs &&hseg, Vs &&vseg) {
    const int XY = X * Y;
    for (int i = 0; i < m; i++) {
        const int p = nodes[i] % XY;
        point(p / Y, p % Y);
    }
    for (int i = 1; i < m; i++) {
        const int j = par[i];
        if (j < 0) continue;
        const int pi = nodes[i] % XY, pj = nodes[j] % XY;
        const int xi = pi / Y, yi = pi % Y, xj = pj / Y, yj = pj % Y;
        const int mnx = min(xi, xj), mxx = max(xi, xj), mny = min(yi, yj), mxy = max(yi, yj);
        if (xi != xj && yi != yj) {
            hseg(mnx, mxx, mny);
            hseg(mnx, mxx, mxy);
            vseg(mny, mxy, mnx);
            vseg(mny, mxy, mxx);
            point(xi, yj);
            point(xj, yi);
        } else if (xi != xj) {
            hseg(mnx, mxx, mny);
            point(mnx, mny);
            point(mxx, mny);
        } else if (yi != yj) {
            vseg(mny, mxy, mnx);
            point(mnx, mny);
            point(mnx, mxy);
        }
    }
}

// claimed cells of a point: the cell, the one below, left and right (in the grid)
__device__ __forceinline__ int point_claims(int x, int y, int X, int Y) {
    return 1 + (y > 0) + (x > 0) + (x + 1 < X);
}

// shape k: routing net ids[k] (k when ids is null); its points are the tree's
// (nodes and edge points) or, when ext_off is given, ext_pts[ext_off[k] ..
// ext_off[k+1]); its segments are always the tree's
struct ShapeSrc {
    const int *tree_off, *tree_nodes, *tree_par, *ids, *ext_off, *ext_pts;
    const long long *ext_at;
    const int *ext_cnt;
    int ext_stride, n, X, Y, sp;
};

template <class Pt, class Hs, class Vs>
__device__ __forceinline__ void shape_of(const ShapeSrc &a, int k, Pt &&point, Hs &&hseg, Vs &&vseg) {
    const int net = a.ids ? a.ids[k] : k;
    const int t = a.tree_off[net], m = a.tree_off[net + 1] - t;
    if (a.ext_off || a.ext_at) {
        const long long q0 = a.ext_at ? a.ext_at[k] : a.ext_off[k];
        const long long q1 = a.ext_at ? q0 + a.ext_cnt[(size_t)k * a.ext_stride] : a.ext_off[k + 1];
        for (long long q = q0; q < q1; q++) point(a.ext_pts[q] / a.Y, a.ext_pts[q] % a.Y);
        net_shapes(a.tree_nodes + t, a.tree_par + t, m, a.X, a.Y, [](int, int) {}, hseg, vseg);
    } else {
        net_shapes(a.tree_nodes + t, a.tree_par + t, m, a.X, a.Y, point, hseg, vseg);
    }
}

// Sum of v over the block (kCountThreads threads), for every thread.
constexpr int kCountThreads = 256;
__device__ long long block_sum(int v) {
    __shared__ long long part[kCountThreads / 32];
    long long x = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = x;
    __syncthreads();
    x = 0;
    for (int i = 0; i < kCountThreads / 32; i++) x += part[i];
    return x;
}

// points and claims of each shape, and their sums over each block
__global__ void __launch_bounds__(kCountThreads) shape_count_kernel(ShapeSrc a, int *pt_cnt, int *claim_cnt,
                                                                   long long *sums) {
    const int k = blockIdx.x * kCountThreads + threadIdx.x;
    const int X = a.X, Y = a.Y, sp = a.sp;
    int np = 0, nc = 0;
    if (k < a.n) {
        shape_of(
            a, k,
            [&](int x, int y) {
                np++;
                nc += point_claims(x, y, X, Y);
            },
            [&](int lo, int hi, int) { nc += (hi - lo) / sp + 1; },
            [&](int lo, int hi, int) { nc += (hi - lo) / sp + 1; });
        pt_cnt[k + 1] = np;
        claim_cnt[k + 1] = nc;
    }
    const long long sp_ = block_sum(np), sc_ = block_sum(nc);
    if (threadIdx.x == 0) {
        sums[2 * blockIdx.x] = sp_;
        sums[2 * blockIdx.x + 1] = sc_;
    }
}

// exclusive sums over the blocks, in place; the totals (64-bit, so that an
// overflow of the 32-bit offsets is seen)
__global__ void __launch_bounds__(kScanThreads) shape_blocks_kernel(int blocks, long long *sums, long long *totals) {
    __shared__ long long part[2][kScanThreads];
    const int t = threadIdx.x;
    const int chunk = (blocks + kScanThreads - 1) / kScanThreads;
    const int lo = min(blocks, t * chunk), hi = min(blocks, lo + chunk);
    long long own[2] = {0, 0};
    for (int i = lo; i < hi; i++)
        for (int f = 0; f < 2; f++) own[f] += sums[2 * i + f];
    for (int f = 0; f < 2; f++) part[f][t] = own[f];
    __syncthreads();
    for (int d = 1; d < kScanThreads; d <<= 1) {
        long long v[2] = {0, 0};
        if (t >= d)
            for (int f = 0; f < 2; f++) v[f] = part[f][t - d];
        __syncthreads();
        for (int f = 0; f < 2; f++) part[f][t] += v[f];
        __syncthreads();
    }
    long long run[2] = {part[0][t] - own[0], part[1][t] - own[1]};
    for (int i = lo; i < hi; i++)
        for (int f = 0; f < 2; f++) {
            const long long v = sums[2 * i + f];
            sums[2 * i + f] = run[f];
            run[f] += v;
        }
    if (t == kScanThreads - 1)
        for (int f = 0; f < 2; f++) totals[f] = part[f][t];
}

// counts to offsets: a[0] = 0, a[k + 1] = sum of the counts of shapes 0..k
__global__ void __launch_bounds__(kCountThreads) shape_offsets_kernel(int n, int *pt_off, int *claim_off,
                                                                      const long long *sums) {
    __shared__ int part[2][kCountThreads / 32];
    const int k = blockIdx.x * kCountThreads + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int v[2] = {k < n ? pt_off[k + 1] : 0, k < n ? claim_off[k + 1] : 0};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int f = 0; f < 2; f++) {
            const int u = __shfl_up_sync(0xffffffffu, v[f], o);
            if (lane >= o) v[f] += u;
        }
    if (lane == 31)
        for (int f = 0; f < 2; f++) part[f][warp] = v[f];
    __syncthreads();
    for (int f = 0; f < 2; f++) {
        long long base = sums[2 * blockIdx.x + f];
        for (int w = 0; w < warp; w++) base += part[f][w];
        int *off = f ? claim_off : pt_off;
        if (k < n) off[k + 1] = (int)(base + v[f]);
        if (k == 0) off[0] = 0;
    }
}

// Sorts a[0..n) (Shell's method, Ciura's gaps) and moves its distinct values
// to the front; returns their number.
__device__ int sort_unique(int *a, int n) {
    constexpr int kGaps[8] = {701, 301, 132, 57, 23, 10, 4, 1};
#pragma unroll 1
    for (int gi = 0; gi < 8; gi++) {
        const int gap = kGaps[gi];
        for (int i = gap; i < n; i++) {
            const int v = a[i];
            int j = i;
            while (j >= gap && a[j - gap] > v) {
                a[j] = a[j - gap];
                j -= gap;
            }
            a[j] = v;
        }
    }
    int m = 0;
    for (int i = 0; i < n; i++)
        if (m == 0 || a[i] != a[m - 1]) a[m++] = a[i];
    return m;
}

// Every repetition of shape k's points and claims, in the order of its tree.
__device__ void fill_shape(const ShapeSrc &a, int k, int *&pt, int *&cl) {
    const int X = a.X, Y = a.Y, sp = a.sp;
    shape_of(
        a, k,
        [&](int x, int y) {
            *pt++ = x * Y + y;
            *cl++ = x * Y + y;
            if (y > 0) *cl++ = x * Y + y - 1;
            if (x > 0) *cl++ = (x - 1) * Y + y;
            if (x + 1 < X) *cl++ = (x + 1) * Y + y;
        },
        [&](int lo, int hi, int y) {
            for (int x = lo; x <= hi; x += sp) *cl++ = x * Y + y;
        },
        [&](int lo, int hi, int x) {
            for (int y = lo; y <= hi; y += sp) *cl++ = x * Y + y;
        });
}

__global__ void shape_fill_kernel(ShapeSrc a, const int *pt_off, const int *claim_off, int *pts, int *claim) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n) return;
    int *pt = pts + pt_off[k], *cl = claim + claim_off[k];
    fill_shape(a, k, pt, cl);
}

// A shape's points and claims, each once, through a hash set in shared memory
// (keys: cell and whether it is a claim); called by whole warps, `tid` of
// `threads`.  A node of a tree is a point once for itself and again for every
// straight edge it ends, and the claims of neighbouring points and of segment
// samples overlap; the colouring only asks whether a cell is claimed and whether
// a point is owned, so each is kept once, in any order.
struct CellSet {
    int *table;
    unsigned mask;
    int *count;  // [2] points, claims
    int *out[2];
    __device__ bool insert(int key) const {
        unsigned h = ((unsigned)key * 0x9E3779B1u >> 9) & mask;
        while (true) {
            const int was = atomicCAS(table + h, -1, key);
            if (was == -1) return true;
            if (was == key) return false;
            h = (h + 1) & mask;
        }
    }
    // adds cell as a point (0) or claim (1) where `have`; whether it is new
    __device__ bool put(bool have, int cell, int which) const {
        const bool fresh = have && insert(2 * cell + which);
        const unsigned m = __ballot_sync(0xffffffffu, fresh);
        if (m) {
            const int lane = threadIdx.x & 31;
            int base = 0;
            if (lane == 0) base = atomicAdd(count + which, __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (fresh) out[which][base + __popc(m & ((1u << lane) - 1))] = cell;
        }
        return fresh;
    }
};

__device__ void unique_shape(const ShapeSrc &a, int k, const CellSet &s, int tid, int threads) {
    const int X = a.X, Y = a.Y, XY = X * Y, sp = a.sp;
    const int net = a.ids ? a.ids[k] : k;
    const int t = a.tree_off[net], m = a.tree_off[net + 1] - t;
    const int *nodes = a.tree_nodes + t, *par = a.tree_par + t;
    auto point = [&](bool have, int cell) {
        const bool fresh = s.put(have, cell, 0);
        if (!__any_sync(0xffffffffu, fresh)) return;
        const int x = cell / Y, y = cell - x * Y;
        s.put(fresh, cell, 1);
        s.put(fresh && y > 0, cell - 1, 1);
        s.put(fresh && x > 0, cell - Y, 1);
        s.put(fresh && x + 1 < X, cell + Y, 1);
    };
    const bool given = a.ext_off || a.ext_at;
    if (given) {
        const long long q0 = a.ext_at ? a.ext_at[k] : a.ext_off[k];
        const int n = (int)(a.ext_at ? a.ext_cnt[(size_t)k * a.ext_stride] : a.ext_off[k + 1] - q0);
        for (int i0 = 0; i0 < n; i0 += threads) {
            const int i = i0 + tid;
            point(i < n, i < n ? a.ext_pts[q0 + i] : 0);
        }
    } else {
        for (int i0 = 0; i0 < m; i0 += threads) {
            const int i = i0 + tid;
            point(i < m, i < m ? nodes[i] % XY : 0);
        }
    }
    for (int i0 = 1; i0 < m; i0 += threads) {
        const int i = i0 + tid;
        const int j = i < m ? par[i] : -1;
        int x0 = 0, x1 = 0, y0 = 0, y1 = 0, ca = 0, cb = 0, nh = 0, nv = 0;
        bool bent = false;
        if (j >= 0) {
            const int pi = nodes[i] % XY, pj = nodes[j] % XY;
            const int xi = pi / Y, yi = pi % Y, xj = pj / Y, yj = pj % Y;
            bent = xi != xj && yi != yj;
            x0 = min(xi, xj); x1 = max(xi, xj); y0 = min(yi, yj); y1 = max(yi, yj);
            ca = xi * Y + yj;
            cb = xj * Y + yi;
            if (xi != xj) nh = (x1 - x0) / sp + 1;
            if (yi != yj) nv = (y1 - y0) / sp + 1;
        }
        if (!given && __any_sync(0xffffffffu, bent)) {  // the ends of straight edges are nodes
            point(bent, ca);
            point(bent, cb);
        }
        // samples: a straight edge's segment, or both legs of both bends
        const int one = nh + nv, all = bent ? 2 * one : one;
        for (int q = 0; __any_sync(0xffffffffu, q < all); q++) {
            const int r = q < one ? q : q - one;
            const int cell = r < nh ? (x0 + r * sp) * Y + (q < one ? y0 : y1)
                                    : (q < one ? x0 : x1) * Y + y0 + (r - nh) * sp;
            s.put(q < all, cell, 1);
        }
    }
}

constexpr int kWarpTable = 1024, kBlockTable = 16384;
// entries of the hash set of a shape of `raw` points and claims
__device__ __forceinline__ int table_size(int raw) {
    int n = 64;
    while (2 * n < 3 * raw) n <<= 1;
    return n;
}

// Distinct points and claims of each shape, moved to the front of its ranges:
// a warp per shape, larger ones listed in big[1 ..] (big[0]: their number).  A
// thread per shape that sorted its lists in memory took 3.7 ms for the 42,915
// rerouted nets of the 800k-net design (now 0.15).
__global__ void __launch_bounds__(256) shape_unique_kernel(ShapeSrc a, const int *pt_off, const int *claim_off,
                                                           int *pts, int *claim, int *pt_n, int *claim_n, int *big) {
    __shared__ int tables[8][kWarpTable];
    __shared__ int counts[8][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = blockIdx.x * 8 + warp; k < a.n; k += gridDim.x * 8) {
        const int p0 = pt_off[k], c0 = claim_off[k];
        const int size = table_size(pt_off[k + 1] - p0 + claim_off[k + 1] - c0);
        if (size > kWarpTable) {
            if (lane == 0) big[1 + atomicAdd(big, 1)] = k;
            continue;
        }
        for (int i = lane; i < size; i += 32) tables[warp][i] = -1;
        if (lane < 2) counts[warp][lane] = 0;
        __syncwarp();
        unique_shape(a, k, CellSet{tables[warp], (unsigned)size - 1, counts[warp], {pts + p0, claim + c0}}, lane, 32);
        __syncwarp();
        if (lane == 0) {
            pt_n[k] = counts[warp][0];
            claim_n[k] = counts[warp][1];
        }
        __syncwarp();
    }
}

// The larger shapes, a block each; those beyond its table by one thread, sorted.
__global__ void __launch_bounds__(256) shape_unique_big_kernel(ShapeSrc a, const int *pt_off, const int *claim_off,
                                                               int *pts, int *claim, int *pt_n, int *claim_n,
                                                               const int *big) {
    extern __shared__ int table[];
    __shared__ int counts[2];
    for (int i = blockIdx.x; i < big[0]; i += gridDim.x) {
        const int k = big[1 + i], p0 = pt_off[k], c0 = claim_off[k];
        const int size = table_size(pt_off[k + 1] - p0 + claim_off[k + 1] - c0);
        __syncthreads();
        if (size > kBlockTable) {
            if (threadIdx.x == 0) {
                int *pt = pts + p0, *cl = claim + c0;
                fill_shape(a, k, pt, cl);
                pt_n[k] = sort_unique(pts + p0, (int)(pt - (pts + p0)));
                claim_n[k] = sort_unique(claim + c0, (int)(cl - (claim + c0)));
            }
            continue;
        }
        for (int j = threadIdx.x; j < size; j += 256) table[j] = -1;
        if (threadIdx.x < 2) counts[threadIdx.x] = 0;
        __syncthreads();
        unique_shape(a, k, CellSet{table, (unsigned)size - 1, counts, {pts + p0, claim + c0}}, threadIdx.x, 256);
        __syncthreads();
        if (threadIdx.x == 0) {
            pt_n[k] = counts[0];
            claim_n[k] = counts[1];
        }
    }
}

}  // namespace

int shape_count_blocks(int n) { return (n + kCountThreads - 1) / kCountThreads; }

void launch_shape_count(const ShapeArgs &a, int *pt_off, int *claim_off, long long *totals, long long *sums,
                        cudaStream_t s) {
    const ShapeSrc src{a.tree_off, a.tree_nodes, a.tree_par, a.ids, a.ext_off, a.ext_pts, a.ext_at,
                       a.ext_cnt, a.ext_stride, a.n, a.X, a.Y, a.sparsity};
    const int blocks = std::max(1, shape_count_blocks(a.n));  // no shapes: the offsets and totals are zero
    shape_count_kernel<<<blocks, kCountThreads, 0, s>>>(src, pt_off, claim_off, sums);
    shape_blocks_kernel<<<1, kScanThreads, 0, s>>>(blocks, sums, totals);
    shape_offsets_kernel<<<blocks, kCountThreads, 0, s>>>(a.n, pt_off, claim_off, sums);
}

void launch_shape_fill(const ShapeArgs &a, const int *pt_off, const int *claim_off, int *pts, int *claim,
                       int *pt_n, int *claim_n, int *big, cudaStream_t s) {
    const ShapeSrc src{a.tree_off, a.tree_nodes, a.tree_par, a.ids, a.ext_off, a.ext_pts, a.ext_at,
                       a.ext_cnt, a.ext_stride, a.n, a.X, a.Y, a.sparsity};
    if (a.n <= 0) return;
    if (!pt_n) {
        shape_fill_kernel<<<(a.n + 255) / 256, 256, 0, s>>>(src, pt_off, claim_off, pts, claim);
        return;
    }
    cudaMemsetAsync(big, 0, sizeof(int), s);
    const KernelShape ks = kernel_setup((const void *)shape_unique_kernel, 256, 0);
    shape_unique_kernel<<<std::min((a.n + 7) / 8, ks.sms * ks.blocks_per_sm), 256, 0, s>>>(
        src, pt_off, claim_off, pts, claim, pt_n, claim_n, big);
    const size_t smem = kBlockTable * sizeof(int);
    const KernelShape kb = kernel_setup((const void *)shape_unique_big_kernel, 256, smem);
    shape_unique_big_kernel<<<std::min(a.n, kb.sms), 256, smem, s>>>(src, pt_off, claim_off, pts, claim, pt_n,
                                                                     claim_n, big);
}

}  // namespace igr
