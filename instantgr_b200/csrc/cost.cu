// Fused congestion-cost refresh: wire cost, via cost and the per-track prefix
// sums of wire cost, in one pass over each track.
//
// Replaces three full-grid kernels of InstantGR (update_wcost_cuda_ispd24,
// update_vcost_ispd24, compute_presum; src/graph.hpp:40-71, :101-104,
// :405-430).  A CTA owns one track (several short ones), a warp 256 consecutive cells: it
// loads capacity and demand, evaluates the cost model for every cell, writes
// vcost (f32), and scans the wire costs in f64 into presum.  The wire cost array
// itself is never written: 20 bytes of DRAM traffic per cell (4+4 read, 4+8
// written) instead of the reference's >= 44.
//
// The prefix sum keeps the exact association of the reference's in-place
// Sklansky scan (at level d, element i with bit d set adds element
// ((i >> d) << d) - 1), so presum is bit-identical to the reference's for the
// same demand.
#include "kcommon.cuh"
#include "host.hpp"

#include <algorithm>
#include <cstdint>
#include <type_traits>

namespace igr {

namespace {

// Cost model of cell i of a track staged in s_cap / s_dem: writes its via cost
// and returns the scan input, the wire cost of edge i-1 (0 for i = 0).
__device__ __forceinline__ double cell_costs(const GridDev &g, const TrackInfo &ti, const float *s_cap,
                                             const float *s_dem, int i, double sc, const int *elen) {
    const int n = ti.len;
    const float c = s_cap[i], d = s_dem[i];
    const double of0 = of_cost(c, d);
    const double bh = fmin(1e12, (of_cost(c, (float)((double)d + 0.5)) - of0) * sc);
    float v;
    double x = 0;
    if (i == 0) {
        v = (float)fmin(1e12, (of_cost(c, (float)((double)d + 1.0)) - of0) * sc);
    } else {
        const float cp = s_cap[i - 1], dp = s_dem[i - 1];
        const double ofp = of_cost(cp, dp);
        const double a1p = fmin(1e12, (of_cost(cp, (float)((double)dp + 1.0)) - ofp) * sc);
        if (i == n - 1) {
            v = (float)a1p;
        } else {
            const double bhp = fmin(1e12, (of_cost(cp, (float)((double)dp + 0.5)) - ofp) * sc);
            v = (float)(bh + bhp);
        }
        // scan input: wire cost of edge i-1 (graph.hpp:44-46)
        float w = (float)a1p;
        w = (float)fma(g.unit_wire, (double)elen[i - 1], (double)w);
        x = (double)w;
    }
    v = (float)((double)v + g.unit_via);
    g.vcost[ti.base + i] = v;
    return x;
}

// of_cost_scaled (graph.hpp:23-27, of_cost_scale = 1) in float: the
// reference's exponent arguments 0.5 * (d - c) and 1.5 * d are formed in
// double from float operands, where both products are exact, and rounded to
// float, which is the correctly rounded float product 0.5f * (d - c) or
// 1.5f * d.  Its test c > 0.001 in double is c >= 0.001f (the least float above
// it), and (float)((double)d + 0.5) and + 1.0 are the float sums (rounding the sum of
// two floats to double first never changes its rounding to float).
//
// float to double by the integer multiplier, for normal floats and, up to an
// error of 2^-127, zero
__device__ __forceinline__ double widen(float f) {
    return __longlong_as_double((long long)((unsigned long long)__float_as_uint(f) * 0x20000000ull + (0x38000000ull << 32)));
}
// A cell's costs of one more unit (rounded to float, its only use) and of half a
// unit (graph.hpp:40-71).  The conversions to double are what the refresh has most
// of on the slowest pipe, so the usual ones go through the multiplier: without
// capacity a cost is 0 or at least 1, so that 2^-127 is rounded away or cancels;
// with capacity the costs have to be well above it.
__device__ __forceinline__ void unit_costs(float c, float d, double sc, float &one, double &half) {
    const bool has_cap = c >= 0.001f;
    const float off = has_cap ? c : 0.f, k = has_cap ? 0.5f : 1.5f;
    const float d5 = d + 0.5f, d1 = d + 1.f;
    const float e0 = has_cap || d > 0.f ? __expf(k * (d - off)) : 0.f;
    const float e5 = has_cap || d5 > 0.f ? __expf(k * (d5 - off)) : 0.f;
    const float e1 = has_cap || d1 > 0.f ? __expf(k * (d1 - off)) : 0.f;
    double w0 = widen(e0), w5 = widen(e5), w1 = widen(e1);
    if ((has_cap && e0 < 0x1p-60f) || !(e1 < INFINITY)) {
        w0 = (double)e0;
        w5 = (double)e5;
        w1 = (double)e1;
    }
    const double h = (w5 - w0) * sc, o = (w1 - w0) * sc;  // min(1e12, .), 1e12 for NaN
    half = h < 1e12 ? h : 1e12;
    one = (float)(o < 1e12 ? o : 1e12);
}

// Cells of a track by thread: a warp has 128 consecutive ones, or 256 in two
// passes, four consecutive ones a lane and pass, so that whole sectors are read and
// written where tracks start on 16 bytes, two levels of the scan are within a lane,
// and the block has one barrier.  Bound by the instructions of the cost model
// (79% of the issue slots; 9 of about 150 per cell go to the slowest pipe,
// exponentials and conversions).  1600 x 1600 cells, 9 layers: 153 us; 840 x 1140:
// 63; as rows of 256 cells with the costs in shared memory and ten barriers a track
// 185 and 81.  (Predicated additions in the scan, end cells apart from the others
// and a path for cells with capacity alone took fewer instructions but 164 to 172 us.)
constexpr int kPassCells = 128;
constexpr int kOnePassCells = 1024;  // tracks of at most this many cells: one pass a warp

// A block has the warps that a track of the longer direction needs; of the other
// direction it takes as many tracks as fit, each with the warps it needs.  (With a
// block per track of either, the others' warps evaluated the cost model for cells that
// are not there: 64 x 4096 cells took 645 us a call, 2000 x 200 136, now 81 and 59;
// 840 x 1140, where that was one of the five warps of every second layer, 92 and 85.)
// Tracks of a block share its barriers, though they need not come to the same number
// of them: a warp without a track, or done with it, leaves the kernel, and a barrier waits
// for the threads still in it.
struct TrackSplit {
    int warps0, warps1;    // per track, of the layers along x and along y
    int tracks0, tracks1;  // per block
    int blocks0, blocks1;  // per layer
};
// this warp's track and its number among the track's warps and the block's
struct TrackWarp {
    TrackInfo ti;
    int tr, warp, slot;
    __device__ __forceinline__ bool leader() const { return warp == 0 && (threadIdx.x & 31) == 0; }
};
// The blocks are in the order of the layers.  False: no track for this warp.  MIXED: some
// tracks take fewer warps than the block has (none does at 1600 x 1600: 167 us a call without
// this, 174 with it; then a block is a track, whose flags are read before anything else).
template <bool MIXED>
__device__ __forceinline__ bool own_track(const GridDev &g, const TrackSplit &sp, TrackWarp &tw) {
    if constexpr (!MIXED) {
        tw.tr = blockIdx.x;
        tw.slot = tw.warp = threadIdx.x >> 5;
        return true;
    }
    const int first = g.DIR ? sp.blocks1 : sp.blocks0, pair = sp.blocks0 + sp.blocks1;
    int l = 0, t = blockIdx.x;  // layer and block of it, two layers at a time
    for (; t >= pair; t -= pair) l += 2;
    if (t >= first) {
        t -= first;
        l++;
    }
    const int dir = layer_dir(g, l);
    const int warps = dir ? sp.warps1 : sp.warps0, tracks = dir ? sp.tracks1 : sp.tracks0;
    tw.slot = tw.warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // shuffled: uniform, for the compiler
    int group = 0;
    for (; tw.warp >= warps; tw.warp -= warps) group++;
    t = t * tracks + group;
    if (group >= tracks || t >= (dir ? g.X : g.Y)) return false;
    tw.tr = (l >> 1) * (g.X + g.Y) + (l & 1) * (g.DIR ? g.X : g.Y) + t;
    tw.ti.l = l;
    tw.ti.t = t;
    tw.ti.dir = dir;
    tw.ti.len = dir ? g.Y : g.X;
    tw.ti.base = (int64_t)l * g.X * g.Y + (int64_t)t * tw.ti.len;
    return true;
}
template <int P>
struct TrackCells {
    float c[P][4], d[P][4];
};

__device__ __forceinline__ void store_sums(double *p, int left, bool vec, const double (&x)[4], double *stage,
                                           int lane) {
    if (vec) {  // lanes past the track's end but for its last cells
        if (left >= 4) {
            asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x[0]), "d"(x[1]), "d"(x[2]), "d"(x[3])
                         : "memory");
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < left) p[j] = x[j];
        }
        return;
    }
    // coalesced through shared memory
#pragma unroll
    for (int j = 0; j < 4; j++) stage[4 * lane + j] = x[j];
    __syncwarp();
    double *row = p - 4 * lane;
    const int n = left + 4 * lane;
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (32 * j + lane < n) row[32 * j + lane] = stage[32 * j + lane];
    __syncwarp();
}

__device__ __forceinline__ double int_to_double(int v) {  // 2^52 + 2^31 + v, less the constant
    return __hiloint2double(0x43300000, v ^ (int)0x80000000) - 4503601774854144.0;
}

// Cost model and Sklansky prefix sums of one track of n cells; every warp of
// the track calls it and n is tallied in g.stats[slot].  (pc, pd): capacity and demand
// of the cell before the warp's first, for lane 0.
//
// Level m of the scan adds element ((i >> m) << m) - 1 to the elements i with bit m
// set: levels 0-1 within a lane, 2-6 between lanes (the source is a lane's last
// element), 7 between the two passes, and 8 on between warps, each of which adds
// up the totals it needs in the order of the levels.
template <int W, int P>
__device__ __forceinline__ void refresh_track(const GridDev &g, const TrackWarp &tw, const TrackCells<P> &t, float pc,
                                              float pd, bool vec, int slot) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ double s_total[W];
    __shared__ double s_stage[W][kPassCells];
    const TrackInfo &ti = tw.ti;
    const int n = ti.len, lane = threadIdx.x & 31, warp = tw.warp;
    const double sc = g.short_cost[ti.l];
    const int *elen = ti.dir ? g.ylen : g.xlen;
    const bool evec = (reinterpret_cast<uintptr_t>(elen) & 15) == 0;
    if (tw.leader()) atomicAdd(&g.stats[slot], (unsigned long long)n);  // refreshed cells, for the roofline
    const bool via_float = (double)(float)g.unit_via == g.unit_via;  // then the float sum is the same
    double x[P][4];
    float left_one = 0.f;  // of the cell before this lane's first
    double left_half = 0.0;
    if (lane == 0) unit_costs(pc, pd, sc, left_one, left_half);
#pragma unroll
    for (int p = 0; p < P; p++) {
        const int i0 = warp * P * kPassCells + p * kPassCells + 4 * lane;
        float one[4];
        double half[4];
#pragma unroll
        for (int j = 0; j < 4; j++) unit_costs(t.c[p][j], t.d[p][j], sc, one[j], half[j]);
        int el[4];
        load4(elen + i0, n - 1 - i0, evec, el);
        const float so = __shfl_sync(kFull, one[3], (lane + 31) & 31);
        const double sh = __shfl_sync(kFull, half[3], (lane + 31) & 31);
        int se = __shfl_up_sync(kFull, el[3], 1);
        if (lane == 0) se = i0 > 0 && i0 < n ? elen[i0 - 1] : 0;
        float po = lane ? so : left_one;
        double ph = lane ? sh : left_half;
        if (lane == 0) {  // the second pass follows the first's last lane
            left_one = so;
            left_half = sh;
        }
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int i = i0 + j;
            const float c = i == 0 ? one[0] : i == n - 1 ? po : (float)(half[j] + ph);
            v[j] = via_float ? c + (float)g.unit_via : (float)((double)c + g.unit_via);
            // scan input: wire cost of edge i-1 (graph.hpp:44-46)
            const float w = (float)fma(g.unit_wire, int_to_double(j ? el[j - 1] : se), (double)po);
            x[p][j] = i > 0 && i < n ? (double)w : 0.0;
            po = one[j];
            ph = half[j];
        }
        store4(g.vcost + ti.base + i0, n - i0, vec, v);
        x[p][1] += x[p][0];
        x[p][3] += x[p][2];
        x[p][2] += x[p][1];
        x[p][3] += x[p][1];
#pragma unroll
        for (int m = 0; m < 5; m++) {
            const double o = __shfl_sync(kFull, x[p][3], (((lane >> m) << m) - 1) & 31);
            if ((lane >> m) & 1)
#pragma unroll
                for (int j = 0; j < 4; j++) x[p][j] += o;
        }
    }
    if constexpr (P > 1) {
        const double o = __shfl_sync(kFull, x[0][3], 31);
#pragma unroll
        for (int j = 0; j < 4; j++) x[1][j] += o;
    }
    if constexpr (W > 1) {
        if (lane == 31) s_total[tw.slot] = x[P - 1][3];
        __syncthreads();
#pragma unroll
        for (int m = 0; (1 << m) < W; m++) {
            if ((warp >> m) & 1) {
                const int last = tw.slot - warp + ((warp >> m) << m) - 1;  // the 2^m warps up to it, added up as a tree
                double o[8];
#pragma unroll
                for (int k = 0; k < 8; k++) o[k] = k < 1 << m ? s_total[last - k] : 0.0;
#pragma unroll
                for (int h = 1; h < 8; h <<= 1)
#pragma unroll
                    for (int k = 0; k < 8; k += 2 * h)
                        if (k + h < 1 << m) o[k] += o[k + h];
#pragma unroll
                for (int p = 0; p < P; p++)
#pragma unroll
                    for (int j = 0; j < 4; j++) x[p][j] += o[0];
            }
        }
    }
#pragma unroll
    for (int p = 0; p < P; p++) {
        const int i0 = warp * P * kPassCells + p * kPassCells + 4 * lane;
        store_sums(g.presum + ti.base + i0, n - i0, vec, x[p], s_stage[tw.slot], lane);
    }
}

// whether a track's arrays can be read and written 16 (sums: 32) bytes at a time
__device__ __forceinline__ bool track_vec(const GridDev &g, const TrackInfo &ti) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(g.cap + ti.base) | reinterpret_cast<uintptr_t>(g.demand + ti.base) |
                        reinterpret_cast<uintptr_t>(g.vcost + ti.base);
    return ((a | reinterpret_cast<uintptr_t>(g.presum + ti.base) >> 1) & 15) == 0;
}

template <int W, int P, bool MIXED>
__global__ void __launch_bounds__(32 * W, 28 / W) cost_refresh_kernel(GridDev g, TrackSplit sp, int only_dirty) {
    chain_begin();
    TrackWarp tw;
    if (!own_track<MIXED>(g, sp, tw)) return;
    if (only_dirty) {
        if (!g.dirty_cost[tw.tr]) return;
    }
    if (!MIXED) tw.ti = decode_track(g, tw.tr);
    const TrackInfo &ti = tw.ti;
    const bool vec = track_vec(g, ti);
    const int n = ti.len, lane = threadIdx.x & 31, first = tw.warp * P * kPassCells;
    const float *cap = g.cap + ti.base, *dem = g.demand + ti.base;
    TrackCells<P> t;
#pragma unroll
    for (int p = 0; p < P; p++) {
        const int i0 = first + p * kPassCells + 4 * lane;
        load4(cap + i0, n - i0, vec, t.c[p]);
        load4(dem + i0, n - i0, vec, t.d[p]);
    }
    const bool before = lane == 0 && first > 0 && first <= n;
    const float pc = before ? cap[first - 1] : 0.f, pd = before ? dem[first - 1] : 0.f;
    refresh_track<W, P>(g, tw, t, pc, pd, vec, 2);
    if (only_dirty) {
        if (W == 1) __syncwarp();  // every lane has seen the flag (warps: refresh_track's barrier)
        if (tw.leader()) g.dirty_cost[tw.tr] = 0;
    }
}

// Copies n floats of a track's capacity and demand into
// shared memory in one loop, so that the loads of both arrays are in flight
// together: 16 bytes per load where the track starts on a 16-byte boundary
// (every track of a grid whose X*Y and track lengths are multiples of 4), else
// one float per load.
__device__ __forceinline__ void stage_track(const float *a, const float *b, float *da, float *db, int n, int tid,
                                            int nthreads) {
    if ((reinterpret_cast<uintptr_t>(b) & 15) == 0) {
        const int n4 = n >> 2;
        const float4 *a4 = reinterpret_cast<const float4 *>(a), *b4 = reinterpret_cast<const float4 *>(b);
        float4 *da4 = reinterpret_cast<float4 *>(da), *db4 = reinterpret_cast<float4 *>(db);
        for (int i = tid; i < n4; i += nthreads) {
            const float4 vb = b4[i];
            da4[i] = a4[i];
            db4[i] = vb;
        }
        for (int i = (n4 << 2) + tid; i < n; i += nthreads) {
            da[i] = a[i];
            db[i] = b[i];
        }
    } else {
        for (int i = tid; i < n; i += nthreads) {
            da[i] = a[i];
            db[i] = b[i];
        }
    }
}

// Tracks of more than 4096 cells (up to the reference's 15,360, main.cpp:28):
// a CTA of kLongThreads per track, the costs evaluated into registers, then
// the reference's in-place Sklansky scan level by level in shared memory
// (graph.hpp:421-428; at level d an element reads an element whose bit d is
// clear, which that level never writes).  The f64 scan array reuses the
// shared memory of the staged capacity and demand.
constexpr int kLongThreads = 1024;
constexpr int kLongMaxE = kMaxTrackCells / kLongThreads;  // 15

__global__ void __launch_bounds__(kLongThreads) cost_refresh_long_kernel(GridDev g, int only_dirty) {
    extern __shared__ __align__(16) unsigned char long_smem[];
    float *s_cap = reinterpret_cast<float *>(long_smem);
    float *s_dem = s_cap + kMaxTrackCells;
    double *s_x = reinterpret_cast<double *>(long_smem);  // after the costs: 8 bytes per cell
    const int tid = threadIdx.x;
    const int tr = blockIdx.x;
    if (only_dirty && !g.dirty_cost[tr]) return;
    {
        const TrackInfo ti = decode_track(g, tr);
        const int n = ti.len;
        stage_track(g.cap + ti.base, g.demand + ti.base, s_cap, s_dem, n, tid, kLongThreads);
        __syncthreads();
        if (tid == 0) {
            if (only_dirty) g.dirty_cost[tr] = 0;
            atomicAdd(&g.stats[2], (unsigned long long)n);
        }
        const double sc = g.short_cost[ti.l];
        const int *elen = ti.dir ? g.ylen : g.xlen;
        double x[kLongMaxE];
#pragma unroll
        for (int r = 0; r < kLongMaxE; r++) {
            const int i = tid + r * kLongThreads;
            x[r] = i < n ? cell_costs(g, ti, s_cap, s_dem, i, sc, elen) : 0.0;
        }
        __syncthreads();  // every read of the staged capacity and demand is done
#pragma unroll
        for (int r = 0; r < kLongMaxE; r++) {
            const int i = tid + r * kLongThreads;
            if (i < n) s_x[i] = x[r];
        }
        __syncthreads();
        for (int d = 0; (1 << d) < n; d++) {
            for (int i = tid; i < n; i += kLongThreads)
                if ((i >> d) & 1) s_x[i] += s_x[((i >> d) << d) - 1];
            __syncthreads();
        }
        for (int i = tid; i < n; i += kLongThreads) g.presum[ti.base + i] = s_x[i];
    }
}

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Batch commit and cost refresh of one track in one pass (phase 1): the wire
// difference array is scanned into demand and stamps (compute_presum_general
// + commit_all_edge, graph.hpp:74-137), the via crossings the tree DP counted
// per cell are added where this batch's wires left no stamp
// (commit_via_demand, graph.hpp:496-543: half a unit on each track edge
// beside the cell, a full unit at the track ends), and the costs and prefix
// sums are rebuilt from the demand in registers.  Tracks with no pending commit
// and clean costs are skipped.  With refresh = 0 the costs are only marked dirty.
template <int W, int P, bool MIXED>
__global__ void __launch_bounds__(32 * W, 28 / W) commit_refresh_kernel(GridDev g, TrackSplit sp, int *vcnt, int stamp,
                                                                          int refresh) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ int s_sum[W];
    __shared__ float s_first[W], s_last[W];
    __shared__ long long s_wl[W];
    chain_begin();
    TrackWarp tw;
    if (!own_track<MIXED>(g, sp, tw)) return;
    const int lane = threadIdx.x & 31, warp = tw.warp, slot = tw.slot, first = warp * P * kPassCells;
    const int tr = tw.tr;
    const bool commit = g.dirty_commit[tr] != 0;
    if (!commit && !(refresh && g.dirty_cost[tr])) return;
    if (!MIXED) tw.ti = decode_track(g, tr);
    const TrackInfo &ti = tw.ti;
    const int n = ti.len;
    const bool vec = track_vec(g, ti);
    float *dem = g.demand + ti.base;
    const float *cap = g.cap + ti.base;
    TrackCells<P> t;
#pragma unroll
    for (int p = 0; p < P; p++) {
        const int i0 = first + p * kPassCells + 4 * lane;
        if (refresh) load4(cap + i0, n - i0, vec, t.c[p]);
        load4(dem + i0, n - i0, vec, t.d[p]);
    }
    float pd = lane == 0 && first > 0 && first <= n ? dem[first - 1] : 0.f;
    const float pc = refresh && lane == 0 && first > 0 && first <= n ? cap[first - 1] : 0.f;
    if (commit) {
        const int *elen = ti.dir ? g.ylen : g.xlen;
        int *pre = g.pre + ti.base, *vc = vcnt + ti.base, *stp = g.stamp + ti.base;
        const bool pvec = ((reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(vc)) & 15) == 0;
        int cnt[P][4], via[P][4], run = 0;
#pragma unroll
        for (int p = 0; p < P; p++) {
            const int i0 = first + p * kPassCells + 4 * lane;
            load4(pre + i0, n - i0, pvec, cnt[p]);
            load4(vc + i0, n - i0, pvec, via[p]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (cnt[p][j] != 0) pre[i0 + j] = 0;
                if (via[p][j] != 0) vc[i0 + j] = 0;
                if (j) cnt[p][j] += cnt[p][j - 1];
            }
            const int sum = cnt[p][3], inc = warp_incl_scan(sum, lane);
#pragma unroll
            for (int j = 0; j < 4; j++) cnt[p][j] += run + inc - sum;
            run += __shfl_sync(kFull, inc, 31);
        }
        if (lane == 0) s_sum[slot] = run;
        __syncthreads();
        int base = 0;
#pragma unroll
        for (int w = 0; w < W; w++) base += w < warp ? s_sum[slot - warp + w] : 0;
        // wires: demand, stamps, wirelength; then the vias of cells without this batch's stamp
        long long wl = 0;
        float own[P][4], prev[P][4];  // a via's part of its own edge and of the one before
#pragma unroll
        for (int p = 0; p < P; p++) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = first + p * kPassCells + 4 * lane + j, k = cnt[p][j] + base;
                const bool wire = i < n - 1 && k > 0;
                if (wire) {
                    t.d[p][j] += (float)k;
                    stp[i] = stamp;
                    wl += (long long)k * elen[i];
                }
                const float c = (float)via[p][j];
                const bool add = via[p][j] != 0 && !wire && stp[i] < stamp;
                own[p][j] = !add || i == n - 1 ? 0.f : i == 0 ? c : 0.5f * c;
                prev[p][j] = !add || i == 0 ? 0.f : i == n - 1 ? c : 0.5f * c;
            }
        }
        if (lane == 0) s_first[slot] = prev[0][0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wl += __shfl_down_sync(kFull, wl, o);
        if (lane == 0) s_wl[slot] = wl;
        __syncthreads();
        const float after = first + P * kPassCells < n ? s_first[slot + 1] : 0.f;  // of the cell after the warp's last
#pragma unroll
        for (int p = 0; p < P; p++) {
            float next = __shfl_down_sync(kFull, prev[p][0], 1);
            const float other = p == P - 1 ? after : __shfl_sync(kFull, prev[P - 1][0], 0);
            if (lane == 31) next = other;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                t.d[p][j] += own[p][j];
                t.d[p][j] += j < 3 ? prev[p][j + 1] : next;
            }
            const int i0 = first + p * kPassCells + 4 * lane;
            store4(dem + i0, n - i0, vec, t.d[p]);
        }
        if (lane == 31) s_last[slot] = t.d[P - 1][3];
        __syncthreads();
        if (lane == 0 && warp > 0) pd = s_last[slot - 1];
        if (tw.leader()) {
            long long sum = 0;
            for (int w = 0; w * P * kPassCells < n; w++) sum += s_wl[slot + w];
            if (sum) atomicAdd(&g.stats[0], (unsigned long long)sum);
            atomicAdd(&g.stats[3], (unsigned long long)n);  // committed cells, for the roofline
            g.dirty_commit[tr] = 0;
            g.dirty_cost[tr] = refresh ? 0 : 1;
        }
    } else {
        __syncthreads();
        if (tw.leader()) g.dirty_cost[tr] = 0;
    }
    if (refresh) refresh_track<W, P>(g, tw, t, pc, pd, vec, 4);
}

template <typename T>
__global__ void ref_to_track_kernel(GridDev g, const T *ref, T *trk) {
    const int64_t n = g.N;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        int l = (int)(k / ((int64_t)g.X * g.Y));
        int rem = (int)(k - (int64_t)l * g.X * g.Y);
        int x = rem / g.Y, y = rem % g.Y;
        trk[cell_at(g, l, x, y)] = ref[k];
    }
}

template <typename T>
__global__ void track_to_ref_kernel(GridDev g, const T *trk, T *ref) {
    const int64_t n = g.N;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        int l = (int)(k / ((int64_t)g.X * g.Y));
        int rem = (int)(k - (int64_t)l * g.X * g.Y);
        int x = rem / g.Y, y = rem % g.Y;
        ref[k] = trk[cell_at(g, l, x, y)];
    }
}

}  // namespace

// A CTA per track (or per few short ones): the hardware block scheduler hands the dirty tracks to
// the SMs as they free up, and a CTA that finds its track clean exits at once
// (a resident grid striding over the tracks balanced the uneven dirty tracks
// worse: 11.9 -> 15.8 ms per route of the 800k-net design; a resident grid
// over a list of the dirty tracks made by a one-CTA pass saved nothing).
//
// Calls f(W, P) with W warps of P passes per track for tracks of maxlen <=
// kMaxFusedTrackCells cells.  One
// pass up to 1024 cells, where the shorter chain counts (a track of 61 cells: 6.8 us
// in place of 9.7), two above, where 13 warps of one pass took 179 us for 153.
template <int P, int W, class F>
static void with_warps(int w, F &&f) {
    if constexpr (W * P * kPassCells >= (P == 1 ? kOnePassCells : kMaxFusedTrackCells)) {
        f(std::integral_constant<int, W>(), std::integral_constant<int, P>());
    } else {
        if (w <= W) f(std::integral_constant<int, W>(), std::integral_constant<int, P>());
        else with_warps<P, W + 1>(w, f);
    }
}
template <class F>
static void with_track_shape(int maxlen, F &&f) {
    if (maxlen <= kOnePassCells) with_warps<1, 1>((maxlen + kPassCells - 1) / kPassCells, f);
    else with_warps<2, kOnePassCells / (2 * kPassCells) + 1>((maxlen + 2 * kPassCells - 1) / (2 * kPassCells), f);
}

// Warps and tracks a block for the tracks of either direction, with W warps of P passes a
// block; returns the number of blocks.
static int split_tracks(const GridDev &g, int W, int P, TrackSplit &sp) {
    auto warps = [&](int len) { return (len + P * kPassCells - 1) / (P * kPassCells); };
    sp.warps0 = warps(g.X);
    sp.warps1 = warps(g.Y);
    sp.tracks0 = W / sp.warps0;
    sp.tracks1 = W / sp.warps1;
    sp.blocks0 = (g.Y + sp.tracks0 - 1) / sp.tracks0;
    sp.blocks1 = (g.X + sp.tracks1 - 1) / sp.tracks1;
    const int odd = g.L / 2, even = g.L - odd;  // layers of the other and of layer 0's direction
    return g.DIR ? even * sp.blocks1 + odd * sp.blocks0 : even * sp.blocks0 + odd * sp.blocks1;
}

void launch_cost_refresh(const GridDev &g, bool only_dirty, cudaStream_t s) {
    const int maxlen = g.X > g.Y ? g.X : g.Y;
    const int od = only_dirty ? 1 : 0;
    if (maxlen <= kMaxFusedTrackCells) {
        with_track_shape(maxlen, [&](auto wc, auto pc) {
            constexpr int W = decltype(wc)::value, P = decltype(pc)::value;
            TrackSplit sp;
            const int blocks = split_tracks(g, W, P, sp);
            launch_chained(sp.warps0 == sp.warps1 ? cost_refresh_kernel<W, P, false> : cost_refresh_kernel<W, P, true>,
                           dim3(blocks), dim3(32 * W), 0, s, g, sp, od);
        });
    } else {
        const size_t smem = (size_t)kMaxTrackCells * 8;
        kernel_setup((const void *)cost_refresh_long_kernel, kLongThreads, smem);
        cost_refresh_long_kernel<<<g.ntracks, kLongThreads, smem, s>>>(g, od);
    }
}

void launch_commit_refresh(const GridDev &g, int *vcnt, int stamp, bool refresh, cudaStream_t s) {
    const int maxlen = g.X > g.Y ? g.X : g.Y;
    if (maxlen > kMaxFusedTrackCells) throw Error(ERR_STATE, "fused batch commit on tracks longer than 4096 cells");
    const int rf = refresh ? 1 : 0;
    with_track_shape(maxlen, [&](auto wc, auto pc) {
        constexpr int W = decltype(wc)::value, P = decltype(pc)::value;
        TrackSplit sp;
        const int blocks = split_tracks(g, W, P, sp);
        launch_chained(sp.warps0 == sp.warps1 ? commit_refresh_kernel<W, P, false> : commit_refresh_kernel<W, P, true>,
                       dim3(blocks), dim3(32 * W), 0, s, g, sp, vcnt, stamp, rf);
    });
}

static int grid_for(int64_t n) {
    int64_t b = (n + 255) / 256;
    if (b > 148 * 32) b = 148 * 32;
    return (int)(b < 1 ? 1 : b);
}

void launch_to_track_layout(const GridDev &g, const float *ref, float *trk, cudaStream_t s) {
    ref_to_track_kernel<float><<<grid_for(g.N), 256, 0, s>>>(g, ref, trk);
}
void launch_to_track_layout_d(const GridDev &g, const double *ref, double *trk, cudaStream_t s) {
    ref_to_track_kernel<double><<<grid_for(g.N), 256, 0, s>>>(g, ref, trk);
}
void launch_to_track_layout_i(const GridDev &g, const int *ref, int *trk, cudaStream_t s) {
    ref_to_track_kernel<int><<<grid_for(g.N), 256, 0, s>>>(g, ref, trk);
}
void launch_from_track_layout_i(const GridDev &g, const int *trk, int *ref, cudaStream_t s) {
    track_to_ref_kernel<int><<<grid_for(g.N), 256, 0, s>>>(g, trk, ref);
}
void launch_from_track_layout_f(const GridDev &g, const float *trk, float *ref, cudaStream_t s) {
    track_to_ref_kernel<float><<<grid_for(g.N), 256, 0, s>>>(g, trk, ref);
}
void launch_from_track_layout_d(const GridDev &g, const double *trk, double *ref, cudaStream_t s) {
    track_to_ref_kernel<double><<<grid_for(g.N), 256, 0, s>>>(g, trk, ref);
}

std::string cuda_error_string(cudaError_t e) { return cudaGetErrorString(e); }

}  // namespace igr
