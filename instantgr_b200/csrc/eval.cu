// Evaluation of a routing result on the device with the rules of the ISPD2024
// evaluator (run/evaluator.cpp:462-633, NVR_DB::read_gr_solution), without
// writing or reading a guide file.
//
// The evaluator reads the guides net by net: a via segment adds one via per
// crossed layer and a via location per layer; a wire marks its cells (both
// ends) with the net and counts one wire on every cell but the last.  At the
// end of a net every via location not yet marked by the same net (by one of
// its wires, or by an earlier via location) adds the stacked-via demand of
// its layer (half a unit on both track edges beside the cell, a full unit at
// the grid boundary).  Per routing layer the cell demand is 2 wires + stacked
// vias (kept in 16 bits as in the evaluator), the overflow loss is
// exp(0.5 * (demand - 2 cap) / 2) where cap > 0.001, else exp(0.5 * 1.5 demand)
// where the demand is positive, and the costs are summed per layer.
//
// Marks only ever compare with the net's own index, so every net is
// independent and all nets run at once.  The segments of a design net are the
// evaluator's guide lines of the route writer, in its order: pin vias from layer
// 0, stacked-pin pairs, then the route records of its routing nets.
//
// A net's lines go into shared memory as two lists, wires (layer, track, start,
// length) and vias (place, layers, position in the net's order), and every via
// asks each wire and each via before it which of its layers they cover: a block
// of 32 threads per net of up to 64 lines, 128 up to 1,024, 512 up to 8,192; the
// latter two put the lines into buckets by track or place first (asking every line,
// they took 0.8 and 3.2 ms on the 800k-net design, now 0.6 and 1.05).  This moves no
// data beyond the lines themselves, where marking every wire cell in a hash set (22M
// inserts on that design) was bound by random accesses to memory: an evaluation of it
// went from 21 to 2.7 ms (with the pins kept on the device and no count read back
// before it; kernels 13.7 -> 2.5 ms), of the 130k-net design from 4.8 to 0.64.
// Nets of more lines, which do not fit shared memory, keep the hash sets
// keyed by (net, layer, x, y): the cells their wires cover, and their via
// locations with the first position in the net's guide order.
#include "kcommon.cuh"

#include <algorithm>

namespace igr {

namespace {

constexpr unsigned long long kEmpty = ~0ull;

__device__ __forceinline__ unsigned long long hash64(unsigned long long k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}

// (net, layer, x, y) as one key: 28 + 4 + 16 + 16 bits
__device__ __forceinline__ unsigned long long cell_key(int net, int z, int x, int y) {
    return ((unsigned long long)net << 36) | ((unsigned long long)z << 32) | ((unsigned long long)x << 16) |
           (unsigned long long)y;
}

// inserts k; returns its slot (every probe sequence ends: the table is never full)
__device__ __forceinline__ unsigned long long set_insert(unsigned long long *keys, unsigned long long mask,
                                                         unsigned long long k) {
    unsigned long long s = hash64(k) & mask;
    for (unsigned long long n = 0; n <= mask; n++, s = (s + 1) & mask) {
        const unsigned long long prev = atomicCAS(keys + s, kEmpty, k);
        if (prev == kEmpty || prev == k) return s;
    }
    return kEmpty;
}

__device__ __forceinline__ bool set_contains(const unsigned long long *keys, unsigned long long mask,
                                             unsigned long long k) {
    unsigned long long s = hash64(k) & mask;
    for (unsigned long long n = 0; n <= mask; n++, s = (s + 1) & mask) {
        const unsigned long long v = keys[s];
        if (v == k) return true;
        if (v == kEmpty) return false;
    }
    return false;
}

// 3-D file-layer position of a route entry, and of a routing layer's cell in the
// track layout (file layer z >= 1 is routing layer z - 1)
__device__ __forceinline__ int64_t cell_at_file(const EvalDev &e, int z, int x, int y) {
    const int l = z - 1;
    const int64_t b = (int64_t)l * e.X * e.Y;
    return (((l & 1) ^ e.DIR) != 0) ? b + (int64_t)x * e.Y + y : b + (int64_t)y * e.X + x;
}

// Calls f(p, q) for every guide line of design net n, in the route writer's
// order, with p <= q (write_guides: pin vias, stacked-pin pairs, records).
template <class F>
__device__ __forceinline__ void for_each_line(const EvalDev &e, int n, F &&f) {
    const int XY = e.X * e.Y;
    for (int64_t i = e.sel_off[n]; i < e.sel_off[n + 1]; i++)
        if (e.sel[i] < XY) f(e.sel[i], e.sel[i] + XY);
    for (int64_t i = e.extra_off[n]; i + 1 < e.extra_off[n + 1]; i += 2) {
        const int a = e.extra[i], b = e.extra[i + 1];
        f(a < b ? a : b, a < b ? b : a);
    }
    for (int s = e.sub_off[n]; s < e.sub_off[n + 1]; s++) {
        const int *r = e.routes + e.route_off[s];
        for (int j = 1; j < r[0]; j += 2) {
            const int a = r[j] + XY, b = r[j + 1] + XY;
            f(a < b ? a : b, a < b ? b : a);
        }
    }
}

// counts per net of the hash class: via locations and wire cells (ends included)
__global__ void eval_count_kernel(EvalDev e, int n_list, const int *list, long long *via_cnt, long long *cell_cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_list) return;
    const int X = e.X, Y = e.Y, XY = X * Y;
    long long vias = 0, cells = 0;
    for_each_line(e, list[i], [&](int p, int q) {
        const int zl = p / XY, zh = q / XY;
        if (zl != zh) {
            vias += zh - zl;
        } else {
            const int xl = p / Y % X, yl = p % Y, xh = q / Y % X, yh = q % Y;
            cells += (xh - xl) + (yh - yl) + 1;
        }
    });
    via_cnt[i] = vias;
    cell_cnt[i] = cells;
}

// most lines of a net of each class but the last
__host__ __device__ constexpr int lines_of(int cls) { return cls == 0 ? 64 : cls == 1 ? 1024 : 8192; }

// upper bound of a net's guide lines: a line per pin, stacked-pin pair and record segment
__global__ void eval_class_kernel(EvalDev e, int *list, int *count) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    int cls = -1;
    if (n < e.n) {
        long long lines = (e.sel_off[n + 1] - e.sel_off[n]) + (e.extra_off[n + 1] - e.extra_off[n]) / 2;
        for (int s = e.sub_off[n]; s < e.sub_off[n + 1]; s++) lines += e.routes[e.route_off[s]] / 2;
        cls = lines <= lines_of(0) ? 0 : lines <= lines_of(1) ? 1 : lines <= lines_of(2) ? 2 : 3;
    }
#pragma unroll
    for (int c = 0; c < kEvalClasses; c++) {
        const unsigned m = __ballot_sync(0xffffffffu, cls == c);
        if (!m) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(count + c, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (cls == c) list[(size_t)c * e.n + at + __popc(m & ((1u << lane) - 1))] = n;
    }
}

// Stacked-via demand of one via location of a net (update_stacked_via_counter,
// evaluator.cpp:636-672): half a unit on both track edges beside the cell, a
// full unit at the grid boundary.
__device__ __forceinline__ void add_stacked(const EvalDev &e, int z, int x, int y) {
    const bool hor = (((z - 1) & 1) ^ e.DIR) == 0;
    const int c = hor ? x : y, last = (hor ? e.X : e.Y) - 1;
    const int64_t at = cell_at_file(e, z, x, y);  // the cell before it along its track is at - 1
    if (c > 0 && c < last) {
        atomicAdd(e.stacked + at - 1, 1);
        atomicAdd(e.stacked + at, 1);
    } else if (c > 0) {
        atomicAdd(e.stacked + at - 1, 2);
    } else if (c < last) {
        atomicAdd(e.stacked + at, 2);
    }
}

// Nets of more than 64 lines: wires in buckets by direction and track, vias by
// place, so that a via asks three buckets.
constexpr int kTracks = 128, kPlaces = 256;  // buckets
__host__ __device__ constexpr bool in_buckets(int lines) { return lines > 64; }
__host__ __device__ constexpr size_t eval_smem(int lines) {
    return (size_t)lines * (sizeof(uint2) + (in_buckets(lines) ? sizeof(uint16_t) : 0));
}
__device__ __forceinline__ int track_bucket(bool hor, unsigned fix) { return (int)(fix & (kTracks / 2 - 1)) * 2 + hor; }
__device__ __forceinline__ int place_bucket(unsigned x, unsigned y) {
    return kTracks + (int)((x * 37 + y) & (kPlaces - 1));
}

// One net at a time: its lines to the lists, wire counts, then the vias.
template <int THREADS, int LINES>
__global__ void __launch_bounds__(THREADS) eval_net_kernel(EvalDev e, const int *list, const int *count, int *queue) {
    extern __shared__ uint2 lists[];  // wires from the front, vias from the back
    __shared__ int s_nw, s_nv, s_next;
    constexpr int kBuckets = in_buckets(LINES) ? kTracks + kPlaces : 1;
    __shared__ int s_end[kBuckets + 1];  // bucket b: entries s_end[b] .. s_end[b + 1] of `order`
    uint16_t *order = reinterpret_cast<uint16_t *>(lists + LINES);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned XY = (unsigned)(e.X * e.Y), Y = (unsigned)e.Y;
    const unsigned rxy = 0xffffffffu / XY, ry = 0xffffffffu / Y;
    const int total = *count;
    unsigned vias[kEvalLayers];
#pragma unroll
    for (int z = 0; z < kEvalLayers; z++) vias[z] = 0;
    for (int turn = 0;; turn++) {
        __syncthreads();
        if (tid == 0) {
            // small nets in fixed turns (a counter would see them all), the others as blocks fall free
            s_next = THREADS == 32 ? blockIdx.x + turn * gridDim.x : atomicAdd(queue, 1);
            s_nw = s_nv = 0;
        }
        __syncthreads();
        if (s_next >= total) break;
        const int n = list[s_next];
        // line t of the net's order from p to q (p <= q)
        auto line = [&](int p, int q, int t) {
            unsigned rp, rq, yl, yh;
            const int zl = (int)div_by((unsigned)p, XY, rxy, rp), zh = (int)div_by((unsigned)q, XY, rxy, rq);
            const int xl = (int)div_by(rp, Y, ry, yl), xh = (int)div_by(rq, Y, ry, yh);
            if (zl != zh) {
                if (rp != rq) set_error(e.err, ERR_STATE);  // a via must be vertical
                const unsigned mask = (1u << zh) - (1u << zl);
                lists[LINES - 1 - atomicAdd(&s_nv, 1)] = make_uint2((unsigned)xl << 16 | yl, (unsigned)t << 16 | mask);
#pragma unroll
                for (int z = 0; z < kEvalLayers; z++) vias[z] += mask >> z & 1;
                return;
            }
            // a wire along its layer: horizontal layers run along x
            const bool hor = zl >= 1 && ((((zl - 1) & 1) ^ e.DIR) == 0);
            if (zl < 1 || (hor && !(xh > xl && yh == yl)) || (!hor && !(yh > yl && xh == xl))) {
                set_error(e.err, ERR_STATE);
                return;
            }
            const unsigned fix = hor ? yl : (unsigned)xl, lo = hor ? (unsigned)xl : yl, len = hor ? xh - xl : yh - yl;
            lists[atomicAdd(&s_nw, 1)] = make_uint2((unsigned)zl << 16 | fix, len << 16 | lo);
        };
        int t0 = 0;
        const int64_t s0 = e.sel_off[n], x0 = e.extra_off[n];
        const int ns = (int)(e.sel_off[n + 1] - s0), ne = (int)((e.extra_off[n + 1] - x0) / 2);
        for (int i = tid; i < ns; i += THREADS) {
            const int p = e.sel[s0 + i];
            if (p < (int)XY) line(p, p + (int)XY, i);
        }
        t0 = ns;
        for (int i = tid; i < ne; i += THREADS) {
            const int a = e.extra[x0 + 2 * i], b = e.extra[x0 + 2 * i + 1];
            line(min(a, b), max(a, b), t0 + i);
        }
        t0 += ne;
        for (int s = e.sub_off[n]; s < e.sub_off[n + 1]; s++) {
            const int *r = e.routes + e.route_off[s];
            const int m = r[0] / 2;  // lines j = 1, 3, .. < r[0]
            for (int i = tid; i < m; i += THREADS) {
                const int a = r[1 + 2 * i] + (int)XY, b = r[2 + 2 * i] + (int)XY;
                line(min(a, b), max(a, b), t0 + i);
            }
            t0 += m;
        }
        __syncthreads();
        const int nw = s_nw, nv = s_nv;
        // wires: one on every cell but the last; short ones a thread each, long ones a warp each
        for (int i = tid; i < nw; i += THREADS) {
            const int z = (int)(lists[i].x >> 16), fix = (int)(lists[i].x & 0xffff), lo = (int)(lists[i].y & 0xffff);
            const int len = (int)(lists[i].y >> 16);
            if (len > 8) continue;
            const bool hor = (((z - 1) & 1) ^ e.DIR) == 0;
            int *w = e.wire + (hor ? cell_at_file(e, z, lo, fix) : cell_at_file(e, z, fix, lo));
            for (int c = 0; c < len; c++) atomicAdd(w + c, 1);
        }
        for (int i = warp; i < nw; i += THREADS / 32) {
            const int len = (int)(lists[i].y >> 16);
            if (len <= 8) continue;
            const int z = (int)(lists[i].x >> 16), fix = (int)(lists[i].x & 0xffff), lo = (int)(lists[i].y & 0xffff);
            const bool hor = (((z - 1) & 1) ^ e.DIR) == 0;
            int *w = e.wire + (hor ? cell_at_file(e, z, lo, fix) : cell_at_file(e, z, fix, lo));
            for (int c = lane; c < len; c += 32) atomicAdd(w + c, 1);
        }
        auto layer_hor = [&](unsigned z) { return (((z - 1) & 1) ^ (unsigned)e.DIR) == 0; };
        auto wire_bucket = [&](uint2 w) { return track_bucket(layer_hor(w.x >> 16), w.x & 0xffff); };
        auto via_bucket = [&](uint2 v) { return place_bucket(v.x >> 16, v.x & 0xffff); };
        if constexpr (in_buckets(LINES)) {
            for (int i = tid; i <= kBuckets; i += THREADS) s_end[i] = 0;
            __syncthreads();
            for (int i = tid; i < nw; i += THREADS) atomicAdd(&s_end[wire_bucket(lists[i])], 1);
            for (int i = tid; i < nv; i += THREADS) atomicAdd(&s_end[via_bucket(lists[LINES - 1 - i])], 1);
            __syncthreads();
            if (warp == 0) {  // counts to ends; filling a bucket then moves its end to its start
                int run = 0;
                for (int b0 = 0; b0 <= kBuckets; b0 += 32) {
                    int v = b0 + lane <= kBuckets ? s_end[b0 + lane] : 0;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int u = __shfl_up_sync(0xffffffffu, v, o);
                        if (lane >= o) v += u;
                    }
                    if (b0 + lane <= kBuckets) s_end[b0 + lane] = run + v;
                    run += __shfl_sync(0xffffffffu, v, 31);
                }
            }
            __syncthreads();
            for (int i = tid; i < nw; i += THREADS) order[atomicSub(&s_end[wire_bucket(lists[i])], 1) - 1] = (uint16_t)i;
            for (int i = tid; i < nv; i += THREADS)
                order[atomicSub(&s_end[via_bucket(lists[LINES - 1 - i])], 1) - 1] = (uint16_t)(LINES - 1 - i);
            __syncthreads();
        }
        // vias: the layers (from 1) that no wire of the net and no earlier via covers there
        for (int i = tid; i < nv; i += THREADS) {
            const uint2 me = lists[LINES - 1 - i];
            const unsigned x = me.x >> 16, y = me.x & 0xffff, t = me.y >> 16;
            unsigned left = me.y & 0xfffe;
            auto by_wire = [&](uint2 w) {
                const unsigned z = w.x >> 16;
                const bool hor = layer_hor(z);
                if ((w.x & 0xffff) == (hor ? y : x) && (hor ? x : y) - (w.y & 0xffff) <= w.y >> 16) left &= ~(1u << z);
            };
            auto by_via = [&](uint2 v) {
                if (v.x == me.x && v.y >> 16 < t) left &= ~v.y;
            };
            if constexpr (in_buckets(LINES)) {
                for (int hor = 0; hor < 2; hor++) {
                    const int b = track_bucket(hor != 0, hor ? y : x);
                    for (int k = s_end[b]; k < s_end[b + 1]; k++) by_wire(lists[order[k]]);
                }
                const int b = place_bucket(x, y);
                for (int k = s_end[b]; k < s_end[b + 1]; k++) by_via(lists[order[k]]);
            } else {
                for (int k = 0; k < nw; k++) by_wire(lists[k]);
                for (int k = 0; k < nv; k++) by_via(lists[LINES - 1 - k]);
            }
            while (left) {
                const int z = __ffs(left) - 1;
                left &= left - 1;
                add_stacked(e, z, (int)x, (int)y);
            }
        }
    }
#pragma unroll
    for (int z = 0; z < kEvalLayers; z++) {
        const unsigned v = __reduce_add_sync(0xffffffffu, vias[z]);
        if (lane == 0 && v) atomicAdd(e.total_vias + z, (unsigned long long)v);
    }
}

// One guide line of design net n at position t of the net's order; its via
// locations go to vloc[at ..].
__device__ __forceinline__ void eval_line(const EvalDev &e, int n, int p, int q, int t, long long at,
                                          unsigned long long *vias) {
    const int X = e.X, Y = e.Y, XY = X * Y;
    const int zl = p / XY, zh = q / XY;
    const int xl = p / Y % X, yl = p % Y, xh = q / Y % X, yh = q % Y;
    if (zl != zh) {
        const bool bad = xl != xh || yl != yh;  // a via must be vertical
        if (bad) set_error(e.err, ERR_STATE);
        for (int z = zl; z < zh; z++) {
            vias[z < kEvalLayers ? z : kEvalLayers - 1]++;
            const unsigned long long k = bad ? cell_key(n, 0, 0, 0) : cell_key(n, z, xl, yl);
            e.vloc[at] = k;
            e.vord[at] = (unsigned)t;
            at++;
            if (bad) continue;
            const unsigned long long s = set_insert(e.vkeys, e.vmask, k);
            if (s == kEmpty) set_error(e.err, ERR_CAPACITY);
            else atomicMin(e.vfirst + s, (unsigned)t);
        }
        return;
    }
    // a wire along its layer: horizontal layers run along x
    const bool hor = zl >= 1 && ((((zl - 1) & 1) ^ e.DIR) == 0);
    if (zl < 1 || (hor && !(xh > xl && yh == yl)) || (!hor && !(yh > yl && xh == xl))) {
        set_error(e.err, ERR_STATE);
        return;
    }
    const int len = hor ? xh - xl : yh - yl;
    for (int c = 0; c <= len; c++) {
        const int x = hor ? xl + c : xl, y = hor ? yl : yl + c;
        if (set_insert(e.wkeys, e.wmask, cell_key(n, zl, x, y)) == kEmpty) set_error(e.err, ERR_CAPACITY);
        if (c < len) atomicAdd(e.wire + cell_at_file(e, zl, x, y), 1);
    }
}

// Hash class: one warp per design net, one lane per guide line: wires mark their cells
// and count wires; vias count per layer and record their locations (in the
// net's order, placed by prefix sums over the lanes)
__global__ void eval_lines_kernel(EvalDev e, int n_list, const int *list, const long long *via_off) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1;
    const int XY = e.X * e.Y;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n_list; i += (gridDim.x * blockDim.x) >> 5) {
        const int n = list[i];
        int tbase = 0;
        long long vbase = via_off[i];
        unsigned long long vias[kEvalLayers];
        for (int z = 0; z < kEvalLayers; z++) vias[z] = 0;
        // a round of up to 32 lines, line `lane` valid when `ok`
        auto round = [&](bool ok, int p, int q) {
            const int nv = ok ? q / XY - p / XY : 0;
            int inc = nv;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (ok) eval_line(e, n, p, q, tbase + __popc(m & lt), vbase + inc - nv, vias);
            tbase += __popc(m);
            vbase += __shfl_sync(0xffffffffu, inc, 31);
        };
        for (int64_t i0 = e.sel_off[n]; i0 < e.sel_off[n + 1]; i0 += 32) {
            const int64_t i = i0 + lane;
            const bool ok = i < e.sel_off[n + 1] && e.sel[i] < XY;
            const int p = ok ? e.sel[i] : 0;
            round(ok, p, p + XY);
        }
        const int64_t x0 = e.extra_off[n];
        const int ne = (int)((e.extra_off[n + 1] - x0) / 2);
        for (int k0 = 0; k0 < ne; k0 += 32) {
            const int k = k0 + lane;
            const bool ok = k < ne;
            const int a = ok ? e.extra[x0 + 2 * k] : 0, b = ok ? e.extra[x0 + 2 * k + 1] : 0;
            round(ok, a < b ? a : b, a < b ? b : a);
        }
        for (int s = e.sub_off[n]; s < e.sub_off[n + 1]; s++) {
            const int *r = e.routes + e.route_off[s];
            const int m = r[0] / 2;  // lines j = 1, 3, .. < r[0]
            for (int k0 = 0; k0 < m; k0 += 32) {
                const int k = k0 + lane;
                const bool ok = k < m;
                const int a = ok ? r[1 + 2 * k] + XY : 0, b = ok ? r[2 + 2 * k] + XY : 0;
                round(ok, a < b ? a : b, a < b ? b : a);
            }
        }
        for (int z = 0; z < kEvalLayers; z++) {
            unsigned long long v = vias[z];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0 && v) atomicAdd(e.total_vias + z, v);
        }
    }
}

// stacked vias of the hash class: the first via location of its key in the
// net's order that no wire of the net covers
__global__ void eval_stacked_kernel(EvalDev e, long long nloc) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nloc) return;
    const unsigned long long k = e.vloc[i];
    const int z = (int)((k >> 32) & 15), x = (int)((k >> 16) & 0xffff), y = (int)(k & 0xffff);
    if (z < 1) return;  // the pin layer is not a routing layer: its demand is not scored
    if (set_contains(e.wkeys, e.wmask, k)) return;
    // the key's slot holds the first position; find it
    unsigned long long s = hash64(k) & e.vmask;
    for (unsigned long long n = 0; n <= e.vmask; n++, s = (s + 1) & e.vmask)
        if (e.vkeys[s] == k) break;
    if (e.vfirst[s] != e.vord[i]) return;
    add_stacked(e, z, x, y);
}

constexpr int kCellThreads = 256;

// per routing layer and block of cells: the overflow loss in a fixed order
// (a fixed tree inside the block) and the wire length; the layer sums are
// then taken over the blocks in order, so the result does not depend on
// scheduling
__global__ void __launch_bounds__(kCellThreads) eval_cells_kernel(EvalDev e, int blocks_per_layer, double *part) {
    __shared__ double s[kCellThreads];
    const int l = blockIdx.x / blocks_per_layer, b = blockIdx.x % blocks_per_layer;
    const int64_t XY = (int64_t)e.X * e.Y;
    const int64_t per = (XY + blocks_per_layer - 1) / blocks_per_layer;
    const int64_t c0 = b * per, c1 = c0 + per < XY ? c0 + per : XY;
    double loss = 0;
    unsigned long long wl = 0;
    const bool hor = ((l & 1) ^ e.DIR) == 0;
    const unsigned along = (unsigned)(hor ? e.X : e.Y);
    for (int64_t c = c0 + threadIdx.x; c < c1; c += kCellThreads) {  // track by track
        const int64_t i = l * XY + c;
        const int w = e.wire[i];
        const unsigned demand = (unsigned)(2 * w + e.stacked[i]) & 0xffffu;  // a 16-bit field in the evaluator
        const double cap = e.cap_d ? e.cap_d[i] : (double)e.cap[i];
        if (cap > 0.001) {
            const double overflow = double(demand) - 2 * cap;
            loss += exp((overflow / 2) * 0.5);
        } else if (cap >= 0 && demand > 0) {
            loss += exp((1.5 * double(demand)) * 0.5);
        }
        if (w) wl += (unsigned long long)w * (unsigned long long)(hor ? e.xlen : e.ylen)[(unsigned)c % along];
    }
    s[threadIdx.x] = loss;
    __syncthreads();
    for (int o = kCellThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = s[0];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wl += __shfl_down_sync(0xffffffffu, wl, o);
    if ((threadIdx.x & 31) == 0 && wl) atomicAdd(e.wl + l, wl);
}

}  // namespace

int eval_blocks_per_layer(int64_t XY) {
    int64_t b = (XY + 4 * kCellThreads - 1) / (4 * kCellThreads);
    return (int)(b < 1 ? 1 : (b > 4096 ? 4096 : b));
}

void launch_eval_nets(const EvalDev &e, int *list, int *count, cudaStream_t s) {
    if (e.n <= 0) return;
    eval_class_kernel<<<(e.n + 255) / 256, 256, 0, s>>>(e, list, count);
    int *queue = count + kEvalClasses;
    auto run = [&](auto kernel, int threads, int cls) {
        const size_t smem = eval_smem(lines_of(cls));
        const KernelShape ks = kernel_setup((const void *)kernel, threads, smem);
        kernel<<<std::min(e.n, ks.sms * ks.blocks_per_sm), threads, smem, s>>>(e, list + (size_t)cls * e.n,
                                                                              count + cls, queue + cls);
    };
    run(eval_net_kernel<512, lines_of(2)>, 512, 2);
    run(eval_net_kernel<128, lines_of(1)>, 128, 1);
    run(eval_net_kernel<32, lines_of(0)>, 32, 0);
}

void launch_eval_count(const EvalDev &e, int n, const int *list, long long *via_cnt, long long *cell_cnt,
                       cudaStream_t s) {
    if (n > 0) eval_count_kernel<<<(n + 255) / 256, 256, 0, s>>>(e, n, list, via_cnt, cell_cnt);
}

void launch_eval_marks(const EvalDev &e, int n, const int *list, const long long *via_off, long long nloc,
                       cudaStream_t s) {
    if (n > 0) {
        const int warps = 8;
        const int blocks = std::min((n + warps - 1) / warps, 148 * 32);
        eval_lines_kernel<<<blocks, 32 * warps, 0, s>>>(e, n, list, via_off);
    }
    if (nloc > 0) eval_stacked_kernel<<<(unsigned)((nloc + 255) / 256), 256, 0, s>>>(e, nloc);
}

void launch_eval_cells(const EvalDev &e, int blocks_per_layer, double *part, cudaStream_t s) {
    eval_cells_kernel<<<blocks_per_layer * e.L, kCellThreads, 0, s>>>(e, blocks_per_layer, part);
}

}  // namespace igr
