// Phase-1 pattern routing: layer-assignment DP over each net's Steiner tree
// with straight and L-shaped edges, then backtrace, route emission and demand
// difference-array updates.
//
// Restates Lshape_route_cuda (src/Lshape_route.hpp:9-153).  The reference runs
// one thread per net with 81-entry f64 tables per node in global memory (928
// bytes of stack per thread), and every tree edge waits on its own gathers.
// Here a warp owns a net, and its edges are processed bottom-up one after
// another (the additions into a parent keep the reference's order), so the
// kernel is bound by the instructions of an edge step in large batches and by
// the step's dependent chain for a long net.  The step therefore spreads over
// 27 lanes, three per layer:
//   (a) the cheapest layer range that contains each layer, as suffix minima
//       over the 45 ranges row by row (three lanes a row) and then minima over
//       the rows (three lanes a layer), in place of one lane per layer that
//       walks up to 25 ranges;
//   (b) for a bent edge the 40 (child layer, parent layer) pairs, whose via
//       and leg costs depend on geometry only and are summed beside (a) by 18
//       lanes, each extending one running sum per starting layer in the
//       reference's order of additions;
//   (c) the running minima of the nine rows of the parent's ranges, three
//       lanes a row.
// The 32 geometry-only costs of an edge (nine legs of the child, nine of the
// parent, seven inner layers of the via columns at both corners) are one load
// per lane, issued an edge ahead.  A node's positions and parent sit in the
// lane of its index.  Nets of at most kNodeTile nodes keep every table in
// shared memory; a larger net keeps its initial tables in global scratch and
// brings a node's table into one of kNodeTile shared slots while the node
// collects its children (a preorder tree needs as many slots as it is deep;
// beyond that the scratch itself is used).  The backtrace resolves the layer
// range of all nodes whose parent is known at once, level by level.
//
// A warp per net with 27 busy lanes replaced a group of 16 or 32 lanes with
// nine busy ones (about 1,000 instructions an edge, now 460 to 540), larger nets
// in global scratch throughout.  Kernel times on a 1600 x 1600 grid, 100,000
// nets of 4.2 nodes on average: 2,559 -> 494 us; on 840 x 1140, 6,000 nets up to
// 200 nodes: 1,521 -> 314 us (the longest net's chain, 7.5 -> 1.5 us an edge);
// 64 nets: 151 -> 36 us.  The launch bound holds the kernel at 128 registers
// (16 warps an SM); the same source with the compiler's own 166 registers, 96 and
// 80 took 1.11, 1.01 and 1.06 of its time on the 100,000 nets.
//
// For the same cost map the chosen layers, routes and demand are bit-identical
// to the reference's: every minimum keeps its first-minimum rule and every sum
// its order, for NaN costs too.
#include "kcommon.cuh"

#include <algorithm>

namespace igr {

namespace {

constexpr int kL = kRouteL;                  // 9 routing layers
constexpr int kR = 45;                       // layer ranges minl <= maxl
constexpr int kNone = 63;                    // "no range": no cost below kInf
// Every table has two more entries, so that lanes whose window ends early load
// and store like the others, without branches: one that is never below kInf to
// read, and one to write to.
constexpr int kEnd = kR, kSink = kR + 1, kTab = kR + 2;
constexpr unsigned kFull = 0xffffffffu;

__host__ __device__ constexpr int tri(int a, int b) { return a * 9 - a * (a - 1) / 2 + (b - a); }

// Choices of an edge per layer l, for the backtrace: bits 0-5 the child's
// cheapest range containing l (tri index, 0 when none has a cost below kInf),
// bits 8-11 the child layer chosen for parent layer l of a bend (15: none),
// bit 15 whether the child's range 0 (layer 0 only) costs less than kInf.
constexpr int kFinite0 = 1 << 15;

template <int T>
struct NetSmem {
    // range tables: of node i (small nets) or of slot i; once an edge is done,
    // its child's table holds the edge's nine costs per parent layer instead
    double dist[T * kTab];
    // geometry-only costs of the current and the next edge (2 x 32), the 45
    // sums of (b) and the 45 minima of (a); first of all the via columns of
    // the nodes (8 per node)
    double work[64 + kTab + kTab];
    double costc[kL + 1];
    unsigned short choice[T * kL];
    unsigned char sa[kTab];
};

// offset of cell (l, x, y): a grid has fewer than 2^32 cells, as its positions fit an int
__device__ __forceinline__ unsigned cell32(const GridDev &g, int l, int x, int y) {
    return (unsigned)l * (unsigned)(g.X * g.Y) + (unsigned)(layer_dir(g, l) ? x * g.Y + y : y * g.X + x);
}

// atomic_add_unit_demand_wire_segment (graph.hpp:105-117), K = 1.  The wire runs
// along one axis, so both ends of its demand are at (xa, ya) and (xb, yb).
__device__ __forceinline__ void add_wire(const GridDev &g, const int *layer_first, int l, int xa, int xb, int ya,
                                         int yb, int stamp) {
    const unsigned cb = cell32(g, l, xb, yb);
    atomicAdd(&g.pre[cell32(g, l, xa, ya)], 1);
    atomicAdd(&g.pre[cb], -((xa == xb) + (ya == yb)));
    g.stamp[cb] = stamp;
    g.dirty_commit[track_of(g, l, xa, ya, layer_first)] = 1;
}

// Via crossings of a via span [lo, hi) at (x, y) for the fused batch commit.
__device__ __forceinline__ void count_vias(const GridDev &g, int *vcnt, const int *layer_first, int lo, int hi, int x,
                                           int y) {
    for (int l = lo; l < hi; l++) {
        atomicAdd(&vcnt[cell32(g, l, x, y)], 1);
        g.dirty_commit[track_of(g, l, x, y, layer_first)] = 1;
    }
}

// A node's position in one word: layer in bits 28-31, x in 14-27, y in 0-13
// (a grid side is at most kMaxTrackCells < 2^14).
struct PosDecoder {
    unsigned XY, Y, rxy, ry;
    __device__ unsigned operator()(int v) const {
        unsigned r, y;
        const unsigned l = div_by((unsigned)v, XY, rxy, r), x = div_by(r, Y, ry, y);
        return l << 28 | x << 14 | y;
    }
};
__device__ __forceinline__ int pos_x(unsigned p) { return (p >> 14) & 0x3fff; }
__device__ __forceinline__ int pos_y(unsigned p) { return p & 0x3fff; }

// What a lane does in an edge step; constant over the kernel.
struct LaneRole {
    int q, sub;          // lane = 9 sub + q; what lanes 27-31 (sub 3) find is not used
    int rb;              // tri(q, m) = rb + m
    // this lane's window: entries of a table in (a1) (read and written, the last
    // range end first) and (a2), parent layers and ranges in (c)
    int row_in[3], row_out[3], row_arg, col[3], diag[3], out[3];
    int via0, viad, leg0, legd;  // (b1): first place of a sum and the step to the next, the same for its leg
    int c0, c1;                  // (b2): the two child layers of this lane
    // gather: lanes 0-8 child leg on layer q, 9-17 parent leg on layer q, 18-24
    // via column at (x, py) and 25-31 at (px, y), layers 1..7
    bool wire, second, dir;
    unsigned base;
    int sx, sy;
};

// Issues the loads of this lane's share of an edge's geometry-only costs.
__device__ __forceinline__ void load_edge(const GridDev &g, const LaneRole &r, unsigned cp, unsigned pp, double &a,
                                          double &b, float &f) {
    const int x = pos_x(cp), y = pos_y(cp), px = pos_x(pp), py = pos_y(pp);
    const bool bent = x != px && y != py;
    a = b = 0.0;
    f = 0.f;
    if (r.wire) {
        // bent: both legs on every layer; straight: the wire on the layers of its direction
        if (bent || (!r.second && (r.dir ? x == px : y == py))) {
            const int fx = r.second ? px : x, fy = r.second ? py : y;
            const int x0 = r.dir ? fx : min(x, px), x1 = r.dir ? fx : max(x, px);
            const int y0 = r.dir ? min(y, py) : fy, y1 = r.dir ? max(y, py) : fy;
            // presum[IDX(l, xmax, ymax)] - presum[IDX(l, xmin, ymin)]  (graph.hpp:19-21)
            a = g.presum[r.base + (unsigned)(x1 * r.sx + y1 * r.sy)];
            b = g.presum[r.base + (unsigned)(x0 * r.sx + y0 * r.sy)];
        }
    } else if (bent) {
        const int vx = r.second ? px : x, vy = r.second ? y : py;
        f = g.vcost[r.base + (unsigned)(vx * r.sx + vy * r.sy)];
    }
}

// One edge step: the child's table nd into the parent's table pd; nd[0..8]
// receive the edge's cost per parent layer (Lshape_route.hpp:33-97).
template <int T>
__device__ __forceinline__ void edge_step(NetSmem<T> &sm, const LaneRole &r, int lane, const double *ring, unsigned cp,
                                          unsigned pp, double *nd, double *pd, unsigned short *choice) {
    double *gc = sm.work + 64, *sv = sm.work + 64 + kTab;
    const int x = pos_x(cp), y = pos_y(cp), px = pos_x(pp), py = pos_y(pp);
    const bool bent = x != px && y != py;
    const int q = r.q, sub = r.sub;
    const int ch0 = nd[0] < kInf ? kFinite0 | 15 << 8 : 15 << 8;
    // (a1) rows: for range start q, the first of the cheapest ends mx >= l, l in this lane's window
    {
        double v[3], cur = kInf;
        int va[3], arg = kNone;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double c = nd[r.row_in[j]];
            const bool take = c <= cur & c < kInf;
            cur = take ? c : cur;
            arg = take ? r.row_arg - j : arg;
            v[j] = cur;
            va[j] = arg;
        }
        const double t0 = __shfl_sync(kFull, cur, q), t1 = __shfl_sync(kFull, cur, 9 + q);
        const int a0 = __shfl_sync(kFull, arg, q), a1 = __shfl_sync(kFull, arg, 9 + q);
        const bool second = sub == 2 & t1 <= t0;
        const double in = sub == 0 ? kInf : second ? t1 : t0;
        const int ia = sub == 0 ? kNone : second ? a1 : a0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const bool own = v[j] <= in;
            sv[r.row_out[j]] = own ? v[j] : in;
            sm.sa[r.row_out[j]] = (unsigned char)(own ? va[j] : ia);
        }
    }
    // (b1) bent: via costs between the layers of the corner plus the parent's leg,
    //      for lower layer q; lanes of one table take q as the child's layer, of
    //      the other as the parent's (sums past the top layer are not stored)
    if (bent && sub < 2) {
        const double *vc = ring + 18 + 7 * sub - 1 + q;  // vc[k]: layer q + k
        const double *leg = ring + r.leg0;
        double *to = gc + r.via0;
        double s = 0;
#pragma unroll
        for (int k = 1; k <= 7; k += 2) {
            const double sum = s + leg[r.legd * (k >> 1)];
            if (q + k <= 8) to[r.viad * (k >> 1)] = sum;
            s += vc[k];
            s += vc[k + 1];
        }
    }
    __syncwarp();
    // (a2) layers: the cheapest row for layer q, rows in this lane's window, then over the windows
    double mcc = kInf;
    int cf = kNone;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const double c = sv[r.col[j]];
        const int ca = sm.sa[r.col[j]];
        const bool take = c < mcc;
        mcc = take ? c : mcc;
        cf = take ? ca : cf;
    }
    {
        const double m1 = __shfl_down_sync(kFull, mcc, 9), m2 = __shfl_down_sync(kFull, mcc, 18);
        const int c1 = __shfl_down_sync(kFull, cf, 9), c2 = __shfl_down_sync(kFull, cf, 18);
        const bool t1 = m1 < mcc;
        mcc = t1 ? m1 : mcc;
        cf = t1 ? c1 : cf;
        const bool t2 = m2 < mcc;
        mcc = t2 ? m2 : mcc;
        cf = t2 ? c2 : cf;
    }
    // lanes 0-8 hold the minima from here on
    int ch = ch0 | (cf == kNone ? 0 : cf);
    double d = mcc + ring[q];
    if (!bent) {
        if (!(r.dir ? x == px : y == py)) d = kInf;
    } else {
        if (lane < kL) sm.costc[q] = d;
        __syncwarp();
        // (b2) parent layer q: the first of the cheapest child layers of opposite parity
        const double d0 = sm.costc[r.c0] + gc[q * 5 + sub], d1 = sm.costc[r.c1] + gc[q * 5 + min(sub + 3, 4)];
        const bool take0 = d0 < kInf;
        d = take0 ? d0 : kInf;
        int bc = take0 ? r.c0 : 15;
        const bool take1 = d1 < d;
        d = take1 ? d1 : d;
        bc = take1 ? r.c1 : bc;
        const double b1 = __shfl_down_sync(kFull, d, 9), b2 = __shfl_down_sync(kFull, d, 18);
        const int c1 = __shfl_down_sync(kFull, bc, 9), c2 = __shfl_down_sync(kFull, bc, 18);
        const bool t1 = b1 < d | (b1 == d & c1 < bc);
        d = t1 ? b1 : d;
        bc = t1 ? c1 : bc;
        const bool t2 = b2 < d | (b2 == d & c2 < bc);
        d = t2 ? b2 : d;
        bc = t2 ? c2 : bc;
        ch = (ch & ~(15 << 8)) | bc << 8;
    }
    if (lane < kL) {
        nd[q] = d;
        choice[q] = (unsigned short)ch;
    }
    const bool nan = __any_sync(kFull, lane < kL && d != d);
    __syncwarp();
    // (c) range minima with the reference's <= rule, accumulated into the parent
    if (!nan) {
        double m[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            m[j] = nd[r.diag[j]];
            if (j > 0) m[j] = m[j - 1] <= m[j] ? m[j - 1] : m[j];
        }
        const double t0 = __shfl_sync(kFull, m[2], q), t1 = __shfl_sync(kFull, m[2], 9 + q);
        const double in = sub == 2 & t1 < t0 ? t1 : t0;
#pragma unroll
        for (int j = 0; j < 3; j++) pd[r.out[j]] += sub != 0 & in <= m[j] ? in : m[j];
    } else if (lane < kL) {  // a NaN starts the running minimum anew: row by row as the reference
        double row = nd[q];
        for (int mx = q; mx < kL; mx++) {
            const double dg = nd[mx];
            if (mx > q && !(row <= dg)) row = dg;
            pd[r.rb + mx] += row;
        }
    }
}

template <int T>
__global__ void __launch_bounds__(128, 4) pattern_route_kernel(GridDev g, TreeBatchDev b, int stamp) {
    extern __shared__ unsigned char smem_raw[];
    chain_begin();
    if (b.gate && (b.gate->status != 0 || b.gate->big_nodes > (unsigned long long)b.scratch_nodes)) return;
    static_assert(T * 8 + 2 * kL <= 64 + 2 * kTab && 32 % T == 0 && T >= 5, "via columns fit the work area, blocks the slots");
    NetSmem<T> &sm = reinterpret_cast<NetSmem<T> *>(smem_raw)[threadIdx.x >> 5];
    __shared__ int layer_first[kL + 1];
    __shared__ unsigned char s_range[kR];  // range t: minl << 4 | maxl
    if (threadIdx.x == 0) {
        int f = 0;
        for (int l = 0; l < g.L; l++) { layer_first[l] = f; f += layer_dir(g, l) ? g.X : g.Y; }
        layer_first[g.L] = f;
        for (int a = 0, t = 0; a < kL; a++)
            for (int c = a; c < kL; c++, t++) s_range[t] = (unsigned char)(a << 4 | c);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int X = g.X, Y = g.Y, XY = X * Y;
    const PosDecoder pack_pos{(unsigned)XY, (unsigned)Y, 0xffffffffu / (unsigned)XY, 0xffffffffu / (unsigned)Y};
    LaneRole r;
    r.q = lane % 9;
    r.sub = lane / 9;
    r.rb = r.q * 9 - r.q * (r.q - 1) / 2 - r.q;
    r.row_arg = r.rb + 8 - 3 * r.sub;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int end = 8 - 3 * r.sub - j, lay = r.q + 3 * r.sub + j, start = 3 * r.sub + j;
        r.row_in[j] = end >= r.q ? r.rb + end : kEnd;
        r.row_out[j] = end >= r.q ? r.rb + end : kSink;
        r.col[j] = start <= r.q ? tri(start, r.q) : kEnd;
        r.diag[j] = min(lay, kL - 1);
        r.out[j] = lay < kL ? r.rb + lay : kSink;
    }
    r.wire = lane < 18;
    r.second = r.wire ? lane >= 9 : lane >= 25;
    {
        const int l = r.wire ? r.q : (r.second ? lane - 24 : lane - 17);
        r.dir = layer_dir(g, l) != 0;
        r.base = (unsigned)l * (unsigned)XY;
        r.sx = r.dir ? Y : 1;
        r.sy = r.dir ? 1 : X;
        // the column at (x, py) (table 0) belongs to child layers that run along y
        const bool child = r.sub == (layer_dir(g, r.q) ? 0 : 1);  // q is the child's layer in (b1)
        r.via0 = child ? (r.q + 1) * 5 + (r.q >> 1) : r.q * 5 + ((r.q + 1) >> 1);
        r.viad = child ? 10 : 1;
        r.leg0 = 9 + (child ? r.q + 1 : r.q);
        r.legd = child ? 2 : 0;
        r.c0 = ((r.q & 1) ^ 1) + 2 * r.sub;
        r.c1 = r.sub < 2 && r.c0 + 6 < kL ? r.c0 + 6 : kL;  // kL: none
    }
    for (int i = lane; i < T; i += 32) sm.dist[i * kTab + kEnd] = kInf;
    if (lane == 0) {
        sm.work[64 + kTab + kEnd] = kInf;
        sm.costc[kL] = __longlong_as_double(0x7ff0000000000000LL);
    }

    // the first net of a warp by its index, the following ones from the queue,
    // asked for a net ahead
    const int warps = gridDim.x * (blockDim.x >> 5);
    int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int net = 0, nb = 0, n = 0;
    auto net_info = [&](int kk) {
        if (kk < b.n) {
            net = b.net_ids[b.order ? b.order[kk] : kk];
            nb = b.node_off[net];
            n = b.node_off[net + 1] - nb;
        }
    };
    net_info(k);
    while (k < b.n) {
        int knext = 0;
        if (lane == 0) knext = warps + atomicAdd(b.queue, 1);
        const int *nodes = b.nodes + nb;
        const int *par = b.par + nb;
        const int this_net = net, nn = n;
        const bool small = nn <= T;
        double *gdist = nullptr;
        unsigned short *gchoice = nullptr;
        int *glr = nullptr;
        int bad = 0;
        if (!small) {
            const int64_t so = b.scratch_off[this_net];
            if (so < 0 || so + nn > b.scratch_nodes) {
                bad = so < 0 ? ERR_STATE : ERR_CAPACITY;
            } else {
                gdist = b.scratch + so * kPatternScratchD;
                int *ib =
                    reinterpret_cast<int *>(b.scratch + b.scratch_nodes * kPatternScratchD) + so * kPatternScratchI;
                gchoice = reinterpret_cast<unsigned short *>(ib + (int64_t)nn * 8);
                glr = ib + (int64_t)nn * (8 + (kR + 1) / 2);
            }
        }
        // a block of 32 nodes: positions, parents and their parents' positions, a node per lane
        unsigned npos = 0, nppos = 0;
        int npar = -1, blk = 0;
        auto load_block = [&](int base) {
            blk = base;
            const int i = base + lane;
            npos = nppos = 0;
            npar = -1;
            if (i < nn) {
                npos = pack_pos(nodes[i]);
                npar = par[i];
            }
            nppos = __shfl_sync(kFull, npos, npar & 31);
            if (base > 0 && i < nn && npar >= 0 && npar < base) nppos = pack_pos(nodes[npar]);
        };
        // ---- 1. via-stack cost of every node and layer range (Lshape_route.hpp:22-32),
        //         T nodes at a time from their via columns, every load of which is in flight at once
        for (int base = 0; base < nn && !bad; base += 32) {
            load_block(base);
            // a parent that does not come before its node ends the net
            const bool wrong = base + lane > 0 && base + lane < nn && (npar < 0 || npar >= base + lane);
            if (__any_sync(kFull, wrong)) bad = ERR_STATE;
            for (int h = 0; h < 32 && base + h < nn; h += T) {
                const int cnt = min(T, nn - base - h);
                constexpr int kLoads = (T * 8 + 31) / 32;
                float c[kLoads];
#pragma unroll
                for (int u = 0; u < kLoads; u++) {
                    const int p = lane + 32 * u;
                    const unsigned pos = __shfl_sync(kFull, npos, (h + (p >> 3)) & 31);
                    c[u] = 0.f;
                    if (p < cnt * 8) c[u] = g.vcost[cell32(g, p & 7, pos_x(pos), pos_y(pos))];
                }
#pragma unroll
                for (int u = 0; u < kLoads; u++)
                    if (lane + 32 * u < cnt * 8) sm.work[lane + 32 * u] = (double)c[u];
                __syncwarp();
                double *out = small ? sm.dist : gdist + (int64_t)(base + h) * kR;
                const int stride = small ? kTab : kR;
                for (int t0 = 0; t0 < cnt * kL; t0 += 32) {
                    const int t = t0 + lane, i = t / kL, mn = t - i * kL;
                    const int l = (int)(__shfl_sync(kFull, npos, (h + i) & 31) >> 28);
                    if (t < cnt * kL) {
                        const double *cc = sm.work + i * 8 - 1;
                        double *row = out + i * stride + (mn * 9 - mn * (mn - 1) / 2 - mn);
                        const int lo = l < kL ? l : -1;  // a pin's layer lies in the range
                        const bool off = l < kL && mn > l;
                        double acc = 0;
#pragma unroll
                        for (int j = 0; j < kL; j++) {
                            const int mx = mn + j;
                            if (mx < kL) row[mx] = (off || mx < lo) ? kInf : acc;
                            acc = acc + cc[mx + 1];
                        }
                    }
                }
                __syncwarp();
            }
        }
        if (bad) {
            if (lane == 0) set_error(g.err, bad);
            k = __shfl_sync(kFull, knext, 0);
            net_info(k);
            continue;
        }
        // ---- 2. bottom-up over tree edges
        double ga = 0, gb = 0;
        float gf = 0;
        unsigned ncp = 0, npp = 0;  // the next edge's child and parent: positions, tables
        int np = 0, ct = 0, pt = 0;
        int owner = lane < T ? -1 : -2;  // large nets: node whose table is in slot `lane`
        unsigned fresh = 0;              // bit 0, 1: the child's, the parent's table is on its way to its slot
        double val[4];
        // slot of node v's table: its own, a free one, or one whose table goes back to the scratch
        // (never one of the nodes at work: i, pi and v's fellow w)
        auto slot_of = [&](int v, int i, int pi, int w, unsigned bit, double *to) {
            const unsigned has = __ballot_sync(kFull, owner == v);
            if (has) return __ffs(has) - 1;
            unsigned can = __ballot_sync(kFull, owner == -1);
            if (!can) {
                can = __ballot_sync(kFull, owner >= 0 && owner != i && owner != pi && owner != w);
                const int sl = __ffs(can) - 1, u = __shfl_sync(kFull, owner, sl);
                gdist[(int64_t)u * kR + lane] = sm.dist[sl * kTab + lane];
                if (lane + 32 < kR) gdist[(int64_t)u * kR + lane + 32] = sm.dist[sl * kTab + lane + 32];
            }
            const int sl = __ffs(can) - 1;
            if (lane == sl) owner = v;
            to[0] = gdist[(int64_t)v * kR + lane];
            to[1] = lane + 32 < kR ? gdist[(int64_t)v * kR + lane + 32] : 0.0;
            fresh |= bit;
            return sl;
        };
        auto fill = [&](int sl, const double *from) {
            sm.dist[sl * kTab + lane] = from[0];
            if (lane + 32 < kR) sm.dist[sl * kTab + lane + 32] = from[1];
        };
        // edge i's nodes, tables and gathers, while edge i + 1 (child c, parent p) is at work
        auto next_edge = [&](int i, int c, int p) {
            if (i < blk) load_block(blk - 32);
            ncp = __shfl_sync(kFull, npos, i & 31);
            npp = __shfl_sync(kFull, nppos, i & 31);
            np = __shfl_sync(kFull, npar, i & 31);
            load_edge(g, r, ncp, npp, ga, gb, gf);
            if (small) {
                ct = i;
                pt = np;
            } else {
                fresh = 0;
                ct = slot_of(i, c, p, np, 1, val);
                pt = slot_of(np, c, p, i, 2, val + 2);
            }
        };
        auto store_edge = [&](int i) { sm.work[(i & 1) * 32 + lane] = r.wire ? ga - gb : (double)gf; };
        if (nn > 1) {
            next_edge(nn - 1, -3, -3);
            store_edge(nn - 1);
        }
        for (int i = nn - 1; i >= 1; i--) {
            if (fresh & 1) fill(ct, val);
            if (fresh & 2) fill(pt, val + 2);
            __syncwarp();
            const unsigned cp = ncp, pp = npp;
            const int pi = np;
            double *nd = sm.dist + ct * kTab, *pd = sm.dist + pt * kTab;
            unsigned short *choice = sm.choice + (small ? i : 0) * kL;
            if (i > 1) next_edge(i - 1, i, pi);
            edge_step<T>(sm, r, lane, sm.work + (i & 1) * 32, cp, pp, nd, pd, choice);
            if (i > 1) store_edge(i - 1);
            if (!small) {
                if (owner == i) owner = -1;  // the child's table is done
                if (lane < kL) {
                    gdist[(int64_t)i * kR + lane] = nd[lane];
                    gchoice[(int64_t)i * kL + lane] = choice[lane];
                }
            }
        }
        __syncwarp();
        const double *root = sm.dist;
        if (!small) {
            const unsigned has = __ballot_sync(kFull, owner == 0);
            root = has ? sm.dist + (__ffs(has) - 1) * kTab : gdist;
        }
        // the next net's record while this one's route is written
        k = __shfl_sync(kFull, knext, 0);
        net_info(k);
        // ---- 3. root range: first minimum in (minl, maxl) order (Lshape_route.hpp:99-105)
        const double inf = __longlong_as_double(0x7ff0000000000000LL);
        const double ra = root[lane], rb = lane + 32 < kR ? root[lane + 32] : inf;
        double bv = ra < inf ? ra : inf;
        if (rb < bv) bv = rb;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(kFull, bv, o);
            if (ov < bv) bv = ov;
        }
        const unsigned at0 = __ballot_sync(kFull, ra == bv), at1 = __ballot_sync(kFull, lane + 32 < kR && rb == bv);
        const int bi = at0 ? __ffs(at0) - 1 : at1 ? __ffs(at1) + 31 : 0;
        const bool root_ok = root[bi] < kInf;
        // ---- 4. backtrace, route emission and demand (Lshape_route.hpp:99-152),
        //      32 nodes at a time: the nodes whose parent's range is known take
        //      theirs from their code, until all have one; the first node
        //      without a finite range ends the route.  The segments of a node
        //      (its via stack, then the straight wire or the leg, corner via and
        //      leg of a bend) get their positions in the record from a prefix
        //      sum over the nodes, in the reference's order, and the demand of
        //      each segment that fits the record is applied.
        int *rec = b.routes + b.route_off[this_net];
        const int cap = b.route_cap[this_net];
        const int smax = cap >= 1 ? (cap - 1) / 2 : 0;  // segments that fit the record
        int carry = 0;  // segments of the nodes before this block
        bool stopped = false;
        int nvias = 0;
        for (int base = 0; base < nn && !stopped; base += 32) {
            if (blk != base) load_block(base);
            const int i = base + lane;
            const bool have = i < nn;
            const int x = pos_x(npos), y = pos_y(npos), px = pos_x(nppos), py = pos_y(nppos);
            const bool straight = px == x || py == y;
            // range of the node, -1 until its parent's is known; child and parent layer of its edge
            int lr = have ? -1 : 0, plr = -1, curl = 0, parl = 0;
            bool ok = root_ok;
            if (i == 0) lr = bi;
            else if (have && npar < base) plr = glr[npar];
            while (true) {
                if (lr < 0 && plr >= 0) {
                    // the cheapest parent layer of the parent's range, by the rule of the range
                    // minima, then the child layer and the child's range chosen for it
                    const double *dg = small ? sm.dist + i * kTab : gdist + (int64_t)i * kR;
                    const unsigned short *ch = small ? sm.choice + i * kL : gchoice + (int64_t)i * kL;
                    int p = s_range[plr] >> 4;
                    double row = dg[p];
                    for (int m = p + 1, end = s_range[plr] & 15; m <= end; m++) {
                        const double c = dg[m];
                        if (!(row <= c)) { row = c; p = m; }
                    }
                    int c = ch[p] >> 8 & 15;
                    if (straight) c = (layer_dir(g, p) ? x == px : y == py) ? p : 15;
                    lr = 0;
                    if (c < kL) {
                        lr = ch[c] & 63;
                        curl = c;
                        parl = p;
                    }
                    ok = lr != 0 || (ch[0] & kFinite0);
                }
                const int got = __shfl_sync(kFull, lr, npar & 31);
                if (lr < 0 && npar >= base) plr = got;
                if (!__any_sync(kFull, lr < 0)) break;
            }
            if (!small) {
                if (have) glr[i] = lr;
                __syncwarp();
            }
            const unsigned bad = __ballot_sync(kFull, have && !ok);
            stopped = bad != 0;
            const bool out = have && (!stopped || lane < __ffs(bad) - 1);
            const int mn = s_range[lr] >> 4, mx = s_range[lr] & 15;
            const int cnt = out ? (mn < mx) + (i == 0 ? 0 : straight ? 1 : 3) : 0;
            int inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(kFull, inc, o);
                if (lane >= o) inc += t;
            }
            int sidx = carry + inc - cnt;  // index of this node's next segment
            carry += __shfl_sync(kFull, inc, 31);
            if (!out || sidx >= smax) continue;
            // up to four segments: the via stack; the straight wire, or the leg beside the
            // child, the corner's via and the leg beside the parent
            const int minx = min(x, px), maxx = max(x, px), miny = min(y, py), maxy = max(y, py);
            const bool alongy = layer_dir(g, curl) != 0;
            const int vx = alongy ? x : px, vy = alongy ? py : y;  // the corner of a bend
            const int here = x * Y + y, there = px * Y + py, corner = vx * Y + vy;
#pragma unroll 1
            for (int w = 0; w < 4; w++) {
                if (w == 0 ? mn >= mx : i == 0 || (straight && w > 1)) continue;
                if (sidx >= smax) break;
                int pa, pc;
                if (w == 0) {
                    pa = mn * XY + here;
                    pc = mx * XY + here;
                } else if (straight) {
                    pa = curl * XY + minx * Y + miny;
                    pc = curl * XY + maxx * Y + maxy;
                } else {
                    pa = w == 1 ? curl * XY + here : (w == 2 ? curl : parl) * XY + corner;
                    pc = w == 3 ? parl * XY + there : (w == 1 ? curl : parl) * XY + corner;
                }
                rec[1 + 2 * sidx] = pa;
                rec[2 + 2 * sidx] = pc;
                sidx++;
                if (w & 1) {
                    const bool ay = straight ? x == px : alongy == (w == 1);  // this wire runs along y
                    const int fx = w == 1 ? x : px, fy = w == 1 ? y : py;
                    add_wire(g, layer_first, w == 1 ? curl : parl, ay ? fx : minx, ay ? fx : maxx, ay ? miny : fy,
                             ay ? maxy : fy, stamp);
                } else if (b.vcnt) {
                    const int lo = w == 0 ? mn : min(curl, parl), hi = w == 0 ? mx : max(curl, parl);
                    count_vias(g, b.vcnt, layer_first, lo, hi, w == 0 ? x : vx, w == 0 ? y : vy);
                    nvias += hi - lo;
                }
            }
        }
        __syncwarp();
        if (b.vcnt) nvias = __reduce_add_sync(kFull, nvias);
        if (lane == 0) {
            // the reference meets whichever comes first: a record overflow at a node
            // before the stop ends the walk there; otherwise the state error at the stop
            if (carry > smax) set_error(g.err, ERR_CAPACITY);
            else if (stopped) set_error(g.err, ERR_STATE);
            rec[0] = 1 + 2 * min(carry, smax);
            if (nvias) atomicAdd(&g.stats[1], (unsigned long long)nvias);
        }
        __syncwarp();
    }
}

}  // namespace

void launch_pattern_route(const GridDev &g, const TreeBatchDev &b, int stamp, cudaStream_t s) {
    if (b.n <= 0) return;
    constexpr int kThreads = 128, kWarps = kThreads / 32;
    using Smem = NetSmem<kPatternNodeTile>;
    const void *kernel = (const void *)pattern_route_kernel<kPatternNodeTile>;
    const size_t smem = sizeof(Smem) * kWarps;
    const KernelShape ks = kernel_setup(kernel, kThreads, smem);
    const int blocks = std::min((b.n + kWarps - 1) / kWarps, ks.sms * ks.blocks_per_sm);
    launch_chained(pattern_route_kernel<kPatternNodeTile>, dim3(blocks), dim3(kThreads), smem, s, g, b, stamp);
}

}  // namespace igr
