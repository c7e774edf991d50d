// Detour DAGs of the rerouted nets, built on the device: a warp per net.
//
// The construction is the host builder's (dag_build.cpp), which restates
// net::generate_detours_reconstruct (src/database_cuda.hpp:1429-2086) with
// construct_segments = false; that file lists the steps and the reference's
// quirks, all kept here in the same order of node creation:
//   root by leaf-peeling BFS (:826-856); congestion regions, stems and trunk
//   ranges by a DFS from the root (:1494-1637); DAG nodes by a second DFS
//   (mirrors placed by the stem displacement rule :1734-1772, L and Z shapes,
//   long edges split at 50/150 GCells :1671-1724); renumbering so that parents
//   come first, with each node's depth its longest distance from the root
//   (:2027-2085).
// The recursions become explicit stacks and the growing containers become
// slices of a work area.  A net whose DAG does not fit its slices reports so and
// is built again with larger ones.  A finished DAG reserves its ranges of the
// node, edge and point pools with one atomic add each and is written there; a
// DAG that finds a pool full is built again once the pools have grown.  A second
// kernel gathers the DAGs of each colour batch into the batch-local arrays of
// the DAG router.
//
// The construction is a chain of dependent steps, so its time is that of the
// chain's memory accesses times the number of nets an SM can have in flight.  A
// warp's work area is 16-bit entries in shared memory (15 KB: 14 nets an SM, or
// 79 KB for the few larger nets).  One lane makes the graph; everything the graph
// only looks up is prepared by all lanes beforehand (decoded positions, the
// congestion of every tree edge, the order of every bend's Z shapes), and what
// follows from it is done by all lanes afterwards (sorting the points, parent
// lists, depths, writing).  A thread per net with its work area in global memory
// kept 2.2 of 32 lanes active: 31 + 8 ms for the 84,000 DAGs of the three rip-up
// passes of the 800k-net design (its small and its larger nets), now 7.8 + 2.2.
// Nets that outgrow both classes (and their 16-bit entries) have their work areas
// in global memory.
#include "kcommon.cuh"

#include <algorithm>
#include <type_traits>

namespace igr {

namespace {

enum : int { kOk = 0, kTooLarge = 1, kMalformed = 2, kPoolFull = 3 };

// in-place ascending heap sort of a[0..n)
template <typename V>
__device__ void heap_sort(V *a, int n) {
    auto sift = [&](int i, int m) {
        while (true) {
            int l = 2 * i + 1;
            if (l >= m) return;
            if (l + 1 < m && a[l + 1] > a[l]) l++;
            if (a[l] <= a[i]) return;
            const V t = a[i]; a[i] = a[l]; a[l] = t;
            i = l;
        }
    };
    for (int i = n / 2 - 1; i >= 0; i--) sift(i, n);
    for (int m = n - 1; m > 0; m--) {
        const V t = a[0]; a[0] = a[m]; a[m] = t;
        sift(0, m);
    }
}

// Entries of a work area: tree nodes, stems (of both directions), mirror nodes,
// DAG nodes, links, conflict points before deduplication.
template <int TC, int SC, int MC, int NC, int EC, int PC>
struct WarpCaps {
    static constexpr int tc = TC, sc = SC, mc = MC, nc = NC, ec = EC, pc = PC;
};
using SmallCaps = WarpCaps<32, 256, 256, 256, 512, 1024>;
using LargeCaps = WarpCaps<128, 1024, 1024, 1536, 3072, 6144>;
using LastCaps = WarpCaps<2048, 32768, 16384, 16384, 32768, 65536>;

// Positions are packed: layer, x, y.  Narrow: 4, 14 and 14 bits (grids of up to
// kDagNarrowSide a side); wide: 8, 28 and 28.
__device__ __forceinline__ int at_l(unsigned p) { return (int)(p >> 28); }
__device__ __forceinline__ int at_x(unsigned p) { return (p >> 14) & 0x3fff; }
__device__ __forceinline__ int at_y(unsigned p) { return p & 0x3fff; }
__device__ __forceinline__ unsigned cell_of(unsigned p) { return p & 0xfffffff; }
using Pos64 = unsigned long long;
__device__ __forceinline__ int at_l(Pos64 p) { return (int)(p >> 56); }
__device__ __forceinline__ int at_x(Pos64 p) { return (int)(p >> 28) & 0xfffffff; }
__device__ __forceinline__ int at_y(Pos64 p) { return (int)p & 0xfffffff; }
__device__ __forceinline__ Pos64 cell_of(Pos64 p) { return p & 0xffffffffffffffull; }
template <class P>
__device__ __forceinline__ P at(int l, int x, int y) {
    constexpr int side = sizeof(P) == 8 ? 28 : 14;
    return (P)l << 2 * side | (P)x << side | (P)y;
}

// Work area of a warp: tree, graph, and what only the construction (`pre`) or
// only the renumbering (`post`) needs.
template <class CAPS, bool WIDE>
struct WarpArea {
    using C = CAPS;
    using P = std::conditional_t<WIDE, Pos64, unsigned>;
    using I = std::conditional_t<WIDE, int, int16_t>;
    using U = std::conditional_t<WIDE, int, uint16_t>;
    int nn, nl, np, nmu, nsu[2], bad;  // nodes, links, points, mirrors and stems so far; status
    P tp[C::tc];                   // tree positions
    P node[C::nc];                 // DAG positions
    U ao[C::tc + 1], nb[2 * C::tc];  // adjacency
    I tpar[C::tc];                 // parent under the chosen root
    uint8_t cong[2 * C::tc];       // per neighbour: 0, or congestion 1 / 2, + 4 when along y
    uint8_t zk[C::tc][2][10];      // per node with a bent edge and leg: Z shapes k in order, 0: none
    U child_pre[C::nc], pn[C::nc];  // links as parent and as child
    U lc[C::ec], lp[C::ec], lrank[C::ec];  // links: child, parent * 10 + slot, number among the child's
    union {
        struct {
            I region[2][C::tc], rlo[2][C::tc], rhi[2][C::tc], shead[2][C::tc];
            I rid[2][C::tc], mlo[2][C::tc], mstep[2][C::tc], mskip[2][C::tc], mcnt[2][C::tc];
            I sval[2][C::sc / 2], snext[2][C::sc / 2], ss[C::sc];
            I qn[3 * C::tc + 4], qf[3 * C::tc + 4];
            I mx[2][C::tc], mp[2][C::tc], mq[2][C::tc], pe[C::tc], pp[C::tc], ppn[C::tc], ps[C::tc];
            I pl_own[2][C::tc], pl_cnt[2][C::tc], nm_off[2][C::tc], nm_cnt[2][C::tc];
            I mpool[C::mc];
            uint8_t seen[C::tc];
            P pts[C::pc];
        } pre;
        struct {
            U poff[C::nc + 1], pcode[C::ec], visit[C::nc], ord[C::nc], stn[C::nc], stq[C::nc], newid[C::nc];
            int dep[C::nc], cn[C::nc];
        } post;
    };
};

// Z-shape candidate k of leg pi between parent position (ppx, ppy) and (cx, cy)
// with mz steps; false when it leaves the grid or meets an end
__device__ __forceinline__ bool z_mids(int k, int pi, int mz, int ppx, int ppy, int cx, int cy, int X, int Y, int &x1,
                                       int &y1, int &x2, int &y2) {
    x1 = pi ? ppx : (ppx * k + cx * (mz - k)) / mz;
    y1 = pi ? (ppy * k + cy * (mz - k)) / mz : ppy;
    x2 = pi ? cx : (ppx * k + cx * (mz - k)) / mz;
    y2 = pi ? (ppy * k + cy * (mz - k)) / mz : cy;
    if (x1 < 0 || y1 < 0 || x1 >= X || y1 >= Y) return false;
    if (x1 == ppx && y1 == ppy) return false;
    if (x1 == cx && y1 == cy) return false;
    if (x2 < 0 || y2 < 0 || x2 >= X || y2 >= Y) return false;
    if (x2 == cx && y2 == cy) return false;
    if (x2 == ppx && y2 == ppy) return false;
    return true;
}

// The construction by one lane over the prepared work area.  Warps are at
// different places of it, so its code has to stay small: inlined into the bodies
// of unrolled loops the steps missed the instruction cache 11.5 of 18.5 cycles an
// instruction; the ones used in many places are functions, their state is in the
// work area, and loops over the two directions stay loops: 1.92 -> 1.63 ms for 16,638 DAGs.
template <class A>
__device__ __noinline__ int dag_create(A &w, int l, int x, int y) {
    const int n = w.nn;
    if (n >= A::C::nc) {
        w.bad = w.bad ? w.bad : kTooLarge;
        return 0;
    }
    w.node[n] = at<typename A::P>(l, x, y);
    w.child_pre[n] = 0;
    w.pn[n] = 0;
    w.nn = n + 1;
    return n;
}

// a link; long ones get one or two intermediate nodes (connect_node, :1671-1724)
template <class A>
__device__ __noinline__ void dag_connect(A &w, int p, int ch, int slot) {
    using C = typename A::C;
    using U = typename A::U;
    if (w.bad) return;
    const int ax = at_x(w.node[p]), ay = at_y(w.node[p]), bx = at_x(w.node[ch]), by = at_y(w.node[ch]);
    const int len = abs(ax - bx) + abs(ay - by);
    int m1 = -1, m2 = -1;
    if (len >= 150) {
        if (ax != bx && ay != by) {
            w.bad = kMalformed;  // a detour DAG edge that is not straight
            return;
        }
        const bool h = ay == by;
        m1 = dag_create(w, 9, h ? ax * 2 / 3 + bx / 3 : ax, h ? ay : ay * 2 / 3 + by / 3);
        m2 = dag_create(w, 9, h ? ax * 1 / 3 + bx * 2 / 3 : ax, h ? ay : ay * 1 / 3 + by * 2 / 3);
    } else if (len >= 50) {
        m1 = dag_create(w, 9, (ax + bx) / 2, (ay + by) / 2);
    }
#pragma unroll 1
    while (!w.bad) {
        const int to = m1 >= 0 ? m1 : ch, nl = w.nl, np = w.np;
        if (nl >= C::ec || np + 2 > C::pc) {
            w.bad = kTooLarge;
            return;
        }
        w.pre.pts[np] = cell_of(w.node[to]);
        w.pre.pts[np + 1] = cell_of(w.node[p]);
        w.np = np + 2;
        w.lc[nl] = (U)to;
        w.lp[nl] = (U)(p * 10 + slot);
        w.lrank[nl] = w.pn[to]++;
        w.nl = nl + 1;
        w.child_pre[p]++;
        if (m1 < 0) return;
        p = m1;
        slot = 0;
        m1 = m2;
        m2 = -1;
    }
}

// union-find root with path compression; a chain that meets -1 gives -1
// and every entry on it becomes -1, as the recursive form does
template <class A>
__device__ __noinline__ int dag_region(A &w, int x, int dir, int T) {
    using I = typename A::I;
    if (x < 0) return -1;
    I *r = w.pre.region[dir];
    int y = x, res, steps = 0;
    while (true) {
        const int ry = r[y];
        if (ry == -1) { res = -1; break; }
        if (ry == y) { res = y; break; }
        y = ry;
        if (++steps > T) {
            w.bad = kMalformed;
            return -1;
        }
    }
    y = x;
    while (r[y] != -1 && r[y] != y) {
        const int nx = r[y];
        r[y] = (I)res;
        y = nx;
    }
    return res;
}

template <class A>
__device__ __noinline__ void dag_stem(A &w, int dir, int node, int v) {
    using I = typename A::I;
    const int n = w.nsu[dir];
    if (n >= A::C::sc / 2) {
        w.bad = w.bad ? w.bad : kTooLarge;
        return;
    }
    I &h = w.pre.shead[dir][node];
    w.pre.sval[dir][n] = (I)v;
    w.pre.snext[dir][n] = h;
    h = (I)n;
    w.nsu[dir] = n + 1;
}

template <class A>
struct LaneBuilder {
    using C = typename A::C;
    using P = typename A::P;
    using I = typename A::I;
    using U = typename A::U;
    A &w;
    int T, X, Y;
    float ratio;
    int num_tracks, zs, sel;
    int root = -1;

    __device__ int deg(int x) const { return w.ao[x + 1] - w.ao[x]; }
    __device__ int create(int l, int x, int y) { return dag_create(w, l, x, y); }
    __device__ void connect(int p, int ch, int slot) { dag_connect(w, p, ch, slot); }
    __device__ int region_of(int x, int dir) { return dag_region(w, x, dir, T); }
    __device__ void stem_push(int dir, int node, int v) { dag_stem(w, dir, node, v); }

    // appends a copy of src's stems to dst's (the multiset is what matters)
    __device__ void stem_copy(int dir, int dst, int src) {
        for (int i = w.pre.shead[dir][src]; i != -1 && !w.bad; i = w.pre.snext[dir][i])
            stem_push(dir, dst, w.pre.sval[dir][i]);
    }

    __device__ void range_merge(int dir, int dst, int lo, int hi) {
        I &a = w.pre.rlo[dir][dst], &b = w.pre.rhi[dir][dst];
        a = (I)min((int)a, lo);
        b = (I)max((int)b, hi);
    }

    // leaf-peeling BFS; the root is the last node taken from the queue
    __device__ int select_root() {
        int head = 0, tail = 0, last = -1;
        const int qcap = 3 * C::tc + 4;
        for (int i = 0; i < T; i++) {
            w.pre.seen[i] = 0;
            if (deg(i) == 1) {
                w.pre.qn[tail] = (I)i;
                w.pre.qf[tail] = -1;
                tail++;
            }
        }
        while (head < tail) {
            const int f = w.pre.qn[head], from = w.pre.qf[head];
            head++;
            last = f;
            if (w.pre.seen[f]) continue;
            w.pre.seen[f] = 1;
            for (int q = w.ao[f]; q < w.ao[f + 1]; q++) {
                const int j = w.nb[q];
                if (j == from) continue;
                if (tail >= qcap) {
                    w.bad = kMalformed;
                    return -1;
                }
                w.pre.qn[tail] = (I)j;
                w.pre.qf[tail] = (I)f;
                tail++;
            }
        }
        return last;
    }

    // region bookkeeping of direction `dir` for tree edge (x, e) of congestion
    // `cg` before the DFS descends into e (:1494-1637)
    __device__ void mark_edge(int x, int e, int cg, int dir) {
        const int cong = cg & 3;
        if (!cong || cg >> 2 != dir) return;
        I *r = w.pre.region[dir];
        if (cong == 1) {
            int target;
            if (x != root) {
                if (r[x] == -1) r[x] = (I)x;
                target = region_of(x, dir);
            } else {
                if (r[e] == -1) r[e] = (I)e;
                target = region_of(e, dir);
            }
            if (target < 0) {  // cannot happen for a tree: the entry was just set
                w.bad = kMalformed;
                return;
            }
            r[e] = (I)target;
            if (x != root) stem_copy(dir, target, e);
            range_merge(dir, target, w.pre.rlo[dir][e], w.pre.rhi[dir][e]);
        } else {
            if (x != root && r[x] == -1) r[x] = (I)x;
            if (r[e] == -1) r[e] = (I)e;
        }
    }

    // stems across region borders once all children of x are done
    __device__ void mark_post(int x, int par, int dir) {
        const int cx = at_x(w.tp[x]), cy = at_y(w.tp[x]);
        const int xr = region_of(x, dir);
        for (int q = w.ao[x]; q < w.ao[x + 1] && !w.bad; q++) {
            const int e = w.nb[q];
            if (e == par) continue;
            const int er = region_of(e, dir);
            if (xr == er) continue;
            const int ex = at_x(w.tp[e]), ey = at_y(w.tp[e]);
#pragma unroll 1
            for (int end = 0; end < 2; end++) {  // e's position for x's region, x's for e's
                const int rg = end ? er : xr;
                if (rg < 0) continue;
                const int along = end ? (dir ? cy : cx) : (dir ? ey : ex);
                stem_push(dir, rg, end ? (dir ? cx : cy) : (dir ? ex : ey));
                range_merge(dir, rg, along, along);
            }
        }
    }

    // regions, stems and ranges of direction `dir`; the two share nothing but
    // the parents, which both write alike
    __device__ void mark_all(int dir) {
        for (int x = 0; x < T && !w.bad; x++) {
            const P v = w.tp[x];
            w.tpar[x] = -1;
            w.pre.region[dir][x] = -1;
            w.pre.shead[dir][x] = -1;
            if (at_l(v) < 9) stem_push(dir, x, dir ? at_x(v) : at_y(v));
            w.pre.rlo[dir][x] = w.pre.rhi[dir][x] = (I)(dir ? at_y(v) : at_x(v));
        }
        I *mx = w.pre.mx[dir], *mp = w.pre.mp[dir], *mq = w.pre.mq[dir];
        int top = 1;
        mx[0] = (I)root; mp[0] = -1; mq[0] = (I)w.ao[root];
        while (top > 0 && !w.bad) {
            const int f = top - 1;
            const int x = mx[f], q = mq[f];
            if (q < w.ao[x + 1]) {
                mq[f] = (I)(q + 1);
                const int e = w.nb[q];
                if (e == mp[f]) continue;
                mark_edge(x, e, w.cong[q], dir);
                if (top >= C::tc) {  // deeper than the tree has nodes: not a tree
                    w.bad = kMalformed;
                    return;
                }
                w.tpar[e] = (I)x;
                mx[top] = (I)e; mp[top] = (I)x; mq[top] = (I)w.ao[e];
                top++;
            } else {
                mark_post(x, mp[f], dir);
                top--;
            }
        }
    }

    // mirror positions of region root t (get_mirror_places, :1734-1772): every
    // mstep-th from mlo on, without the mskip-th, t's own; ss: room for the stems
    __device__ void mirror_places(int t, int dir, I *ss) {
        const int cx = at_x(w.tp[t]), cy = at_y(w.tp[t]);
        const int trunk = w.pre.rhi[dir][t] - w.pre.rlo[dir][t];
        const int maxd = (int)__fmul_rn(ratio, (float)trunk);
        const int orig = dir ? cx : cy;
        // The displacement D(q) = sum of |stem - q| over the region's stems is
        // walked incrementally over its sorted stems:
        //   D(q-1) = D(q) + n - 2 #{s < q},  D(q+1) = D(q) + 2 #{s <= q} - n,
        // which gives exactly the sums the reference recomputes at every step.
        int n = 0, od = 0, lt = 0;  // stems, D(orig), #{s < orig}
        for (int i = w.pre.shead[dir][t]; i != -1; i = w.pre.snext[dir][i]) {
            const int v = w.pre.sval[dir][i];
            od += abs(v - orig);
            lt += v < orig;
            if (n < 64) {  // short lists are kept sorted as they come
                int j = n;
                while (j > 0 && ss[j - 1] > v) { ss[j] = ss[j - 1]; j--; }
                ss[j] = (I)v;
            } else {
                ss[n] = (I)v;
            }
            n++;
        }
        if (n > 64) heap_sort(ss, n);
        int lo = orig, hi = orig;
        const int bound = dir ? X : Y;
        // D is linear between stems, so both walks go from stem to stem.
        {   // lo: down while D(lo - 1) - od <= maxd (it holds at lo: maxd >= 0)
            int D = od, below = lt;  // below = #{s < lo}
            while (lo > 0) {
                const int slope = n - 2 * below, k = lo - (below > 0 ? ss[below - 1] : 0);
                const int m = slope <= 0 ? k : min(k, (maxd + od - D) / slope);
                lo -= m;
                D += slope * m;
                if (m < k) break;
                while (below > 0 && ss[below - 1] >= lo) below--;
            }
        }
        {   // hi: up while D(hi - 1) - od <= maxd (hi - 1: kept from :1750)
            int D = od + n - 2 * lt;  // D(hi - 1)
            int le = 0;               // #{s <= hi - 1}
            while (le < n && ss[le] < hi) le++;
            while (hi + 1 < bound && D - od <= maxd) {
                const int slope = 2 * le - n, room = bound - 1 - hi;
                const int k = le < n ? min(ss[le] - hi + 1, room) : room;
                const int m = slope <= 0 ? k : min(k, (maxd + od - D) / slope + 1);
                hi += m;
                D += slope * m;
                while (le < n && ss[le] < hi) le++;
            }
        }
        // the smallest step >= 1 with fewer than num_tracks tracks at step + 1
        // (falling in the step; it fails up to span / (num_tracks + 2) and holds
        // from span / num_tracks + 1 on)
        const int span = hi - lo;
        int d0 = max(2, span / (num_tracks + 2) + 1), d1 = max(2, span / num_tracks + 1);
        while (d0 < d1) {
            const int d = (d0 + d1) / 2;
            if ((orig - lo) / d + (hi - orig) / d >= num_tracks) d0 = d + 1;
            else d1 = d;
        }
        const int step = d0 - 1;
        const int before = (orig - lo) / step, after = (hi - orig) / step;
        w.pre.mlo[dir][t] = (I)(orig - before * step);
        w.pre.mstep[dir][t] = (I)step;
        w.pre.mskip[dir][t] = (I)before;
        w.pre.mcnt[dir][t] = (I)(before + after);
    }

    // DAG nodes of tree node x (one call of the reference's recursive DFS)
    __device__ int visit(int x, int par, int par_node, int slot) {
        const P v = w.tp[x];
        const int cl = at_l(v), cx = at_x(v), cy = at_y(v);
        const int me = create(cl, cx, cy);
#pragma unroll 1
        for (int dir = 0; dir < 2; dir++) {
            w.pre.pl_own[dir][x] = w.pre.pl_cnt[dir][x] = 0;
            w.pre.nm_off[dir][x] = w.pre.nm_cnt[dir][x] = 0;
        }
        if (par != -1) {  // every call but the root's receives the parent's places
#pragma unroll 1
            for (int dir = 0; dir < 2 && !w.bad; dir++) {
                const int rid = w.pre.rid[dir][x];
                if (rid < 0) continue;
                const int own = x == rid ? x : w.pre.pl_own[dir][par];  // whose places
                const int pcnt = x == rid ? w.pre.mcnt[dir][x] : w.pre.pl_cnt[dir][par];
                w.pre.pl_own[dir][x] = (I)own;
                w.pre.pl_cnt[dir][x] = (I)pcnt;
                const int moff = w.pre.nm_off[dir][par], mcnt = w.pre.nm_cnt[dir][par];
                if (rid != x && pcnt != mcnt) {  // mirror count mismatch
                    w.bad = kMalformed;
                    return me;
                }
                if (w.nmu + pcnt > C::mc) {
                    w.bad = kTooLarge;
                    return me;
                }
                const int noff = w.nmu;
                w.nmu += pcnt;
                w.pre.nm_off[dir][x] = (I)noff;
                w.pre.nm_cnt[dir][x] = (I)pcnt;
                const int lo = w.pre.mlo[dir][own], step = w.pre.mstep[dir][own], skip = w.pre.mskip[dir][own];
                for (int m = 0; m < pcnt && !w.bad; m++) {
                    const int place = lo + step * (m + (m >= skip));
                    const int nx = dir ? place : cx, ny = dir ? cy : place;
                    int nm;
                    if (rid != x) {
                        nm = create(9, nx, ny);
                        connect(w.pre.mpool[moff + m], nm, slot);
                    } else {
                        const int pxx = at_x(w.node[par_node]), pyy = at_y(w.node[par_node]);
                        if (nx != pxx && ny != pyy) {
                            const int t0 = create(9, pxx, ny);
                            connect(par_node, t0, slot);
                            const int t1 = create(9, nx, pyy);
                            connect(par_node, t1, slot);
                            nm = create(9, nx, ny);
                            connect(t0, nm, 0);
                            connect(t1, nm, 0);
                        } else {
                            nm = create(9, nx, ny);
                            connect(par_node, nm, slot);
                        }
                    }
                    w.pre.mpool[noff + m] = (I)nm;
                }
            }
        }
        if (w.bad) return me;
        if (par_node != -1) {
            const int ppx = at_x(w.node[par_node]), ppy = at_y(w.node[par_node]);
            if (ppx != cx && ppy != cy) {
#pragma unroll 1
                for (int pi = 0; pi <= 1; pi++) {
                    const int corner = create(9, pi ? cx : ppx, pi ? ppy : cy);
                    connect(par_node, corner, slot);
                    connect(corner, me, 0);
                }
#pragma unroll 1
                for (int pi = 0; pi <= 1 && !w.bad; pi++) {
                    const int mz = min(zs, pi ? abs(ppy - cy) : abs(ppx - cx));
                    for (int ii = 0; ii < sel && !w.bad; ii++) {
                        const int k = w.zk[x][pi][ii];
                        if (k == 0) continue;  // not a Z shape
                        int x1, y1, x2, y2;
                        z_mids(k, pi, mz, ppx, ppy, cx, cy, X, Y, x1, y1, x2, y2);
                        const int p1 = create(9, x1, y1);
                        connect(par_node, p1, slot);
                        if (w.np >= C::pc) {
                            w.bad = kTooLarge;
                            return me;
                        }
                        w.pre.pts[w.np++] = at<P>(0, (x1 + x2) / 2, (y1 + y2) / 2);
                        const int p2 = create(9, x2, y2);
                        connect(p1, p2, 0);
                        connect(p2, me, 0);
                    }
                }
            }
#pragma unroll 1
            for (int dir = 0; dir < 2 && !w.bad; dir++) {
                const int rid = w.pre.rid[dir][x], prid = w.pre.rid[dir][par];
                if (prid >= 0 && rid != prid) {
                    const int moff = w.pre.nm_off[dir][par], mcnt = w.pre.nm_cnt[dir][par];
                    for (int m = 0; m < mcnt && !w.bad; m++) {
                        const int pm = w.pre.mpool[moff + m];
                        const int mx0 = at_x(w.node[pm]), my0 = at_y(w.node[pm]);
                        if (mx0 != cx && my0 != cy) {
#pragma unroll 1
                            for (int pi = 0; pi <= 1; pi++) {
                                const int ni = create(9, pi ? cx : mx0, pi ? my0 : cy);
                                connect(pm, ni, slot);
                                connect(ni, me, 0);
                            }
                        } else {
                            connect(pm, me, slot);
                        }
                    }
                }
            }
            if (ppx == cx || ppy == cy) connect(par_node, me, slot);
        }
#pragma unroll 1
        for (int dir = 0; dir < 2 && !w.bad; dir++) {
            if (w.pre.rid[dir][x] >= 0 && x != root && cl < 9) {
                const int moff = w.pre.nm_off[dir][x], mcnt = w.pre.nm_cnt[dir][x];
                for (int m = 0; m < mcnt && !w.bad; m++) {
                    const int dup = create(cl, cx, cy);
                    connect(w.pre.mpool[moff + m], dup, deg(x) - 1);
                }
            }
        }
        return me;
    }

    __device__ void dfs_all() {
        int top = 1;
        w.pre.pe[0] = (I)root; w.pre.pp[0] = -1; w.pre.ppn[0] = -1; w.pre.ps[0] = -1;
        while (top > 0 && !w.bad) {
            top--;
            const int x = w.pre.pe[top], par = w.pre.pp[top], par_node = w.pre.ppn[top], slot = w.pre.ps[top];
            const int me = visit(x, par, par_node, slot);
            if (w.bad) return;
            int cnt = 0;
            for (int q = w.ao[x]; q < w.ao[x + 1]; q++) cnt += w.nb[q] != par;
            if (top + cnt > C::tc) {  // each tree node is pending once: not a tree
                w.bad = kMalformed;
                return;
            }
            // children in adjacency order: pushed last to first
            for (int q = w.ao[x + 1] - 1; q >= w.ao[x]; q--) {
                const int e = w.nb[q];
                if (e == par) continue;
                cnt--;
                w.pre.pe[top] = (I)e; w.pre.pp[top] = (I)x; w.pre.ppn[top] = (I)me;
                w.pre.ps[top] = (I)cnt;
                top++;
            }
        }
    }

    // order in which all links to a node's children are done (:2027-2085)
    __device__ void order() {
        auto &q = w.post;
        int otop = 0;
        for (int i = 0; i < w.nn; i++) {
            if (w.child_pre[i] != 0) continue;
            if (otop >= w.nn) { w.bad = kMalformed; return; }
            q.ord[otop++] = (U)i;
            q.stn[0] = (U)i; q.stq[0] = q.poff[i];
            int stop = 1;
            while (stop > 0) {
                const int f = stop - 1, at = q.stq[f];
                if (at >= q.poff[q.stn[f] + 1]) { stop--; continue; }
                q.stq[f] = (U)(at + 1);
                const int p = q.pcode[at] / 10;
                if (p >= w.nn) { w.bad = kMalformed; return; }
                const int seen = q.visit[p] + 1;
                q.visit[p] = (U)seen;
                if (seen == w.child_pre[p]) {
                    if (otop >= w.nn || stop >= w.nn) { w.bad = kMalformed; return; }
                    q.ord[otop++] = (U)p;
                    q.stn[stop] = (U)p; q.stq[stop] = q.poff[p];
                    stop++;
                }
            }
        }
        if (otop != w.nn) w.bad = kMalformed;  // not acyclic
    }
};

__device__ __forceinline__ int warp_prefix(int x, int lane) {  // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += u;
    }
    return x;
}

// ascending sort of a[0..n) by one warp; every exchange puts the smaller value
// first, so that entries past n (which count as largest) are never touched
template <class P>
__device__ void warp_sort(P *a, int n, int lane) {
    for (int size = 1; 1 << (size - 1) < n; size++) {
        for (int half = size - 1; half >= 0; half--) {  // (exponents)
            const int span = 1 << half;
            const bool mirror = half == size - 1;
            for (int t = lane; t < (n + 1) / 2 + span; t += 32) {
                const int r = t & (span - 1), base = (t - r) * 2;
                const int lo = base + r, hi = mirror ? base + 2 * span - 1 - r : lo + span;
                if (hi < n) {
                    const P u = a[lo], v = a[hi];
                    if (u > v) {
                        a[lo] = v;
                        a[hi] = u;
                    }
                }
            }
            __syncwarp();
        }
    }
}

template <class A>
__device__ void build_one(const DagBuildArgs &a, A &w, int k, int lane) {
    using C = typename A::C;
    using P = typename A::P;
    using I = typename A::I;
    using U = typename A::U;
    constexpr unsigned kFull = 0xffffffffu;
    const int XY = a.X * a.Y, Y = a.Y;
    const int id = a.ids[k];
    const int b = a.tree_off[id], T = a.tree_off[id + 1] - b;
    LaneBuilder<A> B{w, T, a.X, a.Y};
    const bool few = a.mode == 0 || a.mode == 1;
    B.ratio = few ? 0.1f : 0.15f;
    B.num_tracks = few ? 6 : 9;
    B.zs = few ? 7 : 10;
    B.sel = few ? 2 : 10;
    int bad = T > C::tc ? kTooLarge : T < 2 ? kMalformed : kOk;
    // ---- the tree: positions, neighbours, congestion of the edges
    if (!bad) {
        const int q0 = a.adj_off[b], nq = a.adj_off[b + T] - q0;
        bool wrong = false;
        if (nq > 2 * C::tc) {
            bad = kTooLarge;
        } else {
            for (int i = lane; i < T; i += 32) {
                const int v = a.pos[b + i], l = v / XY, r = v - l * XY, x = r / Y;
                w.tp[i] = at<P>(l, x, r - x * Y);
            }
            for (int i = lane; i <= T; i += 32) w.ao[i] = (U)(a.adj_off[b + i] - q0);
            for (int i = lane; i < nq; i += 32) {
                const int j = a.adj[q0 + i];
                wrong |= j < 0 || j >= T;
                w.nb[i] = (U)j;
            }
        }
        if (__any_sync(kFull, wrong)) bad = kMalformed;
        __syncwarp();
    }
    if (!bad) {
        auto ys = [&](int x, int y) { return __ldg(a.ysum + (size_t)x * Y + y); };
        auto xs = [&](int x, int y) { return __ldg(a.xsum + (size_t)x * Y + y); };
        for (int x = lane; x < T; x += 32) {
            const int cx = at_x(w.tp[x]), cy = at_y(w.tp[x]);
            for (int q = w.ao[x]; q < w.ao[x + 1]; q++) {
                const P e = w.tp[w.nb[q]];
                const int ex = at_x(e), ey = at_y(e);
                const int x0 = min(ex, cx), x1 = max(ex, cx), y0 = min(ey, cy), y1 = max(ey, cy);
                int cg = 0;
                if (ex == cx) {
                    if (__fsub_rn(ys(cx, y1), ys(cx, y0)) > 0) cg = 4 + 1;
                } else if (ey == cy) {
                    if (__fsub_rn(xs(x1, cy), xs(x0, cy)) > 0) cg = 1;
                } else {
                    const float a0 = ys(cx, y1), a1 = ys(cx, y0), b0 = ys(ex, y1), b1 = ys(ex, y0);
                    const float c0 = xs(x1, cy), c1 = xs(x0, cy), d0 = xs(x1, ey), d1 = xs(x0, ey);
                    if (__fsub_rn(a0, a1) > 0 || __fsub_rn(b0, b1) > 0) cg = 4 + 2;
                    else if (__fsub_rn(c0, c1) > 0 || __fsub_rn(d0, d1) > 0) cg = 2;
                }
                w.cong[q] = (uint8_t)cg;
            }
        }
        __syncwarp();
        if (lane == 0) {
            w.nn = w.nl = w.np = w.nmu = w.nsu[0] = w.nsu[1] = w.bad = 0;
            B.root = B.select_root();
            if (B.root < 0 && !w.bad) w.bad = kMalformed;  // a tree without leaves
        }
        __syncwarp();
        B.root = __shfl_sync(kFull, B.root, 0);
        if (lane < 2 && !w.bad) B.mark_all(lane);  // a lane per direction
        __syncwarp();
        bad = w.bad;
        __syncwarp();
    }
    // ---- regions and mirror places, a lane per tree node and direction
    if (!bad) {
        int used = 0;  // stems given room
        for (int i0 = 0; i0 < 2 * T; i0 += 32) {
            const int i = i0 + lane, dir = i & 1, x = i >> 1;
            bool places = false;
            int n = 0;
            if (i < 2 * T) {
                int y = x, steps = 0;
                while (y >= 0 && w.pre.region[dir][y] != y && steps <= T) {
                    y = w.pre.region[dir][y];
                    steps++;
                }
                if (steps > T) w.bad = kMalformed;
                w.pre.rid[dir][x] = (I)y;
                places = y == x && x != B.root;
            }
            if (places)
                for (int j = w.pre.shead[dir][x]; j != -1; j = w.pre.snext[dir][j]) n++;
            const int at = warp_prefix(n, lane);
            if (places) B.mirror_places(x, dir, w.pre.ss + used + at - n);
            used += __shfl_sync(kFull, at, 31);
        }
        __syncwarp();
        bad = w.bad;
        __syncwarp();
    }
    // ---- Z shapes of every bent edge, a lane per leg and candidate: ascending
    //      (overflow, k) over the first mz - 1 candidates, those that do not fit (0, 0)
    if (!bad) {
        auto ys = [&](int x, int y) { return __ldg(a.ysum + (size_t)x * Y + y); };
        const int pi = lane >= 9, k = lane - 9 * pi + 1;
        for (int x = 0; x < T; x++) {
            if (w.tpar[x] < 0) continue;  // the root
            const P c = w.tp[x], p = w.tp[w.tpar[x]];
            const int cx = at_x(c), cy = at_y(c), ppx = at_x(p), ppy = at_y(p);
            if (cx == ppx || cy == ppy) continue;
            const int mz = min(B.zs, pi ? abs(ppy - cy) : abs(ppx - cx));
            float rv = 0.f;
            int rk = 0, x1, y1, x2, y2;
            const bool cand = lane < 18 && k < mz;
            if (cand && z_mids(k, pi, mz, ppx, ppy, cx, cy, a.X, Y, x1, y1, x2, y2)) {
                const float u0 = ys(max(x1, x2), max(y1, y2)), u1 = ys(min(x1, x2), min(y1, y2));
                const float v0 = ys(max(x1, ppx), max(y1, ppy)), v1 = ys(min(x1, ppx), min(y1, ppy));
                const float w0 = ys(max(cx, x2), max(cy, y2)), w1 = ys(min(cx, x2), min(cy, y2));
                int of = 0;  // int += float: the sum is taken in float and truncated
                of = (int)__fadd_rn((float)of, __fsub_rn(u0, u1));
                of = (int)__fadd_rn((float)of, __fsub_rn(v0, v1));
                of = (int)__fadd_rn((float)of, __fsub_rn(w0, w1));
                rv = (float)of;
                rk = k;
            }
            int rank = 0;
#pragma unroll
            for (int j = 0; j < 9; j++) {
                const float ov = __shfl_sync(kFull, rv, 9 * pi + j);
                const int ok = __shfl_sync(kFull, rk, 9 * pi + j);
                const bool before = ov < rv || (ov == rv && (ok < rk || (ok == rk && j + 1 < k)));
                rank += j + 1 < mz && j + 1 != k && before;
            }
            if (cand) w.zk[x][pi][rank] = (uint8_t)rk;
            // past the candidates: none
            if (lane < 20) {
                const int leg = lane >= 10, at = lane - 10 * leg;
                const int legz = min(B.zs, leg ? abs(ppy - cy) : abs(ppx - cx));
                if (at >= max(legz - 1, 0)) w.zk[x][leg][at] = 0;
            }
        }
        __syncwarp();
        if (lane == 0) B.dfs_all();
        __syncwarp();
        bad = w.bad;
        __syncwarp();
    }
    const int nn = bad ? 0 : w.nn, nl = bad ? 0 : w.nl, np = bad ? 0 : w.np;
    // ---- conflict points, each once, ascending
    int npu = 0;
    if (!bad) {
        P *pts = w.pre.pts;
        warp_sort(pts, np, lane);
        for (int i0 = 0; i0 < np; i0 += 32) {
            const int i = i0 + lane;
            const P v = i < np ? pts[i] : 0;
            const bool keep = i < np && (i == 0 || pts[i - 1] != v);
            // (entries before i0 have moved down, but the last one read equals the last one kept)
            const unsigned m = __ballot_sync(kFull, keep);
            __syncwarp();
            if (keep) pts[npu + __popc(m & ((1u << lane) - 1))] = v;
            npu += __popc(m);
            __syncwarp();
        }
    }
    // ---- place the DAG: node, edge and point ranges reserved in the pools
    // (their order varies from run to run; every reader goes through the
    // per-DAG offsets, so results do not)
    long long no = 0, eo = 0, po = 0;
    if (!bad) {
        if (lane == 0) {
            no = (long long)atomicAdd(a.used + 0, (unsigned long long)nn);
            eo = (long long)atomicAdd(a.used + 1, (unsigned long long)nl);
            po = (long long)atomicAdd(a.used + 2, (unsigned long long)npu);
        }
        no = __shfl_sync(kFull, no, 0);
        eo = __shfl_sync(kFull, eo, 0);
        po = __shfl_sync(kFull, po, 0);
        if (no + nn > a.cap_nodes || eo + nl > a.cap_edges || po + npu > a.cap_points) bad = kPoolFull;
    }
    // ---- parents-first renumbering (:2027-2085)
    int D = 0, S = 0, mc = 0;
    if (!bad) {
        for (int i = lane; i < npu; i += 32) a.out_points[po + i] = at_x(w.pre.pts[i]) * Y + at_y(w.pre.pts[i]);
        __syncwarp();
        auto &q = w.post;
        int run = 0;  // parent lists by child, in the order of the links
        for (int i0 = 0; i0 < nn; i0 += 32) {
            const int i = i0 + lane, c = i < nn ? w.pn[i] : 0;
            const int x = warp_prefix(c, lane);
            if (i < nn) {
                q.poff[i] = (U)(run + x - c);
                q.visit[i] = 0;
            }
            run += __shfl_sync(kFull, x, 31);
        }
        if (lane == 0) q.poff[nn] = (U)run;
        __syncwarp();
        for (int l = lane; l < nl; l += 32) q.pcode[q.poff[w.lc[l]] + w.lrank[l]] = w.lp[l];
        __syncwarp();
        if (lane == 0) B.order();
        __syncwarp();
        bad = w.bad;
        __syncwarp();
    }
    if (!bad) {
        auto &q = w.post;
        for (int i = lane; i < nn; i += 32) {
            const int kk = nn - 1 - i;  // the node ordered i-th gets this number
            q.newid[q.ord[i]] = (U)kk;
            q.dep[kk] = 0;
            q.cn[kk] = 0;
        }
        __syncwarp();
        // parent slots in the new numbering, by node; longest distances from the
        // root by relaxation, 32 nodes at a time (parents come first)
        int run = 0;
        for (int i0 = 0; i0 < nn; i0 += 32) {
            const int kk = i0 + lane;
            const int old = kk < nn ? q.ord[nn - 1 - kk] : 0, c = kk < nn ? w.pn[old] : 0;
            const int x = warp_prefix(c, lane);
            const int e0 = run + x - c;
            for (int j = 0; j < c; j++) {
                const int code = q.pcode[q.poff[old] + j], sp = q.newid[code / 10], sl = code % 10;
                a.out_par[eo + e0 + j] = sp;
                a.out_child_idx[eo + e0 + j] = sl;
                atomicMax(&q.cn[sp], sl + 1);
            }
            if (kk < nn) {
                const P v = w.node[old];
                a.out_nodes[no + kk] = at_l(v) * XY + at_x(v) * Y + at_y(v);
                a.out_par_num[no + kk] = c;
            }
            run += __shfl_sync(kFull, x, 31);
        }
        __syncwarp();
        for (int i0 = 0; i0 < nn; i0 += 32) {
            const int kk = i0 + lane, old = kk < nn ? q.ord[nn - 1 - kk] : 0;
            const int q0 = kk < nn ? q.poff[old] : 0, q1 = kk < nn ? q.poff[old + 1] : 0;
            int d = 0;
            while (true) {
                int m = d;
                for (int j = q0; j < q1; j++) m = max(m, q.dep[q.newid[q.pcode[j] / 10]] + 1);
                __syncwarp();
                if (m != d) q.dep[kk] = m;
                __syncwarp();
                const bool moved = m != d;
                d = m;
                if (!__any_sync(kFull, moved)) break;
            }
        }
        for (int i = lane; i < nn; i += 32) {
            const int d = q.dep[i], c = q.cn[i];
            a.out_depth[no + i] = d;
            a.out_child_num[no + i] = c;
            D = max(D, d + 1);
            S += c;
            mc = max(mc, c);
        }
        D = __reduce_max_sync(kFull, D);
        S = __reduce_add_sync(kFull, S);
        mc = __reduce_max_sync(kFull, mc);
    }
    if (lane == 0) {
        int *sz = a.sizes + (size_t)k * kDagSizeFields;
        sz[0] = bad ? 0 : nn;
        sz[1] = bad ? 0 : nl;
        sz[2] = bad ? 0 : npu;
        sz[3] = D;
        sz[4] = S;
        sz[5] = mc;
        sz[6] = bad;
        a.node_at[k] = no;
        a.edge_at[k] = eo;
        a.point_at[k] = po;
    }
    __syncwarp();
}

// WARPS nets at a time per block, the nets of the list as warps fall free; the
// work areas in shared memory, or one a block in a.work
template <class A, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) dag_build_kernel(DagBuildArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    A &w = reinterpret_cast<A *>(a.work ? a.work : (void *)smem)[blockIdx.x * (a.work != nullptr) + (threadIdx.x >> 5)];
    const int lane = threadIdx.x & 31;
    while (true) {
        int i = 0;
        if (lane == 0) i = atomicAdd(a.queue, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= a.n_list) return;
        build_one(a, w, a.list ? a.list[i] : i, lane);
    }
}

// A warp per net of the batch layout: copies its DAG from the per-net arrays
// into the batch-local arrays of the DAG router (the layout the host builds in
// the reference-order path: nodes, parent CSR with child slots and edge children,
// child-slot offsets, per-depth node lists).  Copies, so bound by memory; a
// thread per net took 1.58 ms for 42,915 DAGs, this takes 0.10.
constexpr int kGatherWarps = 4, kGatherDepths = 1024;
__global__ void __launch_bounds__(32 * kGatherWarps) dag_gather_kernel(DagGatherArgs a) {
    __shared__ int at_depth[kGatherWarps][kGatherDepths];
    constexpr unsigned kFull = 0xffffffffu;
    const int j = blockIdx.x * kGatherWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= a.n) return;
    const int *d = a.desc + (size_t)j * kDagDescFields;
    const int k = d[0], base = d[1], ebl = d[2], sl0 = d[3], lvb = d[4], jl = d[5], b = d[6];
    const int *bi = a.batch + (size_t)b * kDagBatchFields;  // nb, eb, pb, lb, nnb, nets
    const long long no = a.node_at[k], eo = a.edge_at[k];
    const int *sz = a.sizes + (size_t)k * kDagSizeFields;
    const int m = sz[0], ne = sz[1], D = sz[3];
    const int nb0 = bi[0] + base, eb0 = bi[1] + ebl, pb0 = bi[2] + base, lb0 = bi[3] + lvb, nnb0 = bi[4] + jl;
    if (jl == 0 && lane == 0) {
        a.par_off[bi[2]] = 0;
        a.child_off[bi[2]] = 0;
        a.net_node_off[bi[4]] = 0;
        a.net_level_off[bi[4]] = 0;
    }
    for (int e = lane; e < ne; e += 32) {
        a.par[eb0 + e] = base + a.src_par[eo + e];
        a.child_slot[eb0 + e] = a.src_child_idx[eo + e];
    }
    int *cnt = at_depth[threadIdx.x >> 5];
    const bool few = D <= kGatherDepths;
    if (few)
        for (int i = lane; i < D; i += 32) cnt[i] = 0;
    __syncwarp();
    int e0 = 0, s0 = sl0;
    for (int v0 = 0; v0 < m; v0 += 32) {
        const int v = v0 + lane;
        const bool in = v < m;
        const int pn = in ? a.src_par_num[no + v] : 0, cn = in ? a.src_child_num[no + v] : 0;
        const int ep = warp_prefix(pn, lane), sp = warp_prefix(cn, lane);
        if (in) {
            a.nodes[nb0 + v] = a.src_nodes[no + v];
            a.par_off[pb0 + v + 1] = ebl + e0 + ep;
            a.child_off[pb0 + v + 1] = s0 + sp;
            for (int q = ep - pn; q < ep; q++) a.edge_child[eb0 + e0 + q] = base + v;
            if (few) atomicAdd(&cnt[a.src_depth[no + v]], 1);
        }
        e0 += __shfl_sync(kFull, ep, 31);
        s0 += __shfl_sync(kFull, sp, 31);
    }
    __syncwarp();
    // per-depth lists: level_off[d] = first position of depth d, nodes of one
    // depth in node order
    if (few) {
        int pos = base;
        for (int i0 = 0; i0 < D; i0 += 32) {
            const int i = i0 + lane, c = i < D ? cnt[i] : 0, p = warp_prefix(c, lane);
            if (i < D) {
                a.level_off[lb0 + i] = pos + p - c;
                cnt[i] = pos + p - c;
            }
            pos += __shfl_sync(kFull, p, 31);
        }
        __syncwarp();
        for (int v0 = 0; v0 < m; v0 += 32) {
            const int v = v0 + lane, dep = v < m ? a.src_depth[no + v] : -1;
            const unsigned same = __match_any_sync(kFull, dep);
            int at = 0;
            if (v < m) at = cnt[dep] + __popc(same & ((1u << lane) - 1));
            __syncwarp();
            if (v < m) {
                a.level_nodes[bi[0] + at] = base + v;
                if ((same >> lane) == 1) cnt[dep] = at + 1;  // the last of its depth
            }
            __syncwarp();
        }
    } else {
        int pos = base;
        for (int dd = 0; dd < D; dd++) {
            if (lane == 0) a.level_off[lb0 + dd] = pos;
            for (int v0 = 0; v0 < m; v0 += 32) {
                const int v = v0 + lane;
                const unsigned at = __ballot_sync(kFull, v < m && a.src_depth[no + v] == dd);
                if (at >> lane & 1) a.level_nodes[bi[0] + pos + __popc(at & ((1u << lane) - 1))] = base + v;
                pos += __popc(at);
            }
        }
    }
    if (lane == 0) {
        a.level_off[lb0 + D] = base + m;
        a.net_node_off[nnb0 + 1] = base + m;
        a.net_ids[bi[5] + jl] = a.ids[k];
        a.net_level_off[nnb0 + 1] = lvb + D + 1;
    }
}

}  // namespace

size_t dag_work_bytes() { return sizeof(WarpArea<LastCaps, true>); }

void launch_dag_build(const DagBuildArgs &a, int cls, int builders, cudaStream_t s) {
    if (a.n_list <= 0) return;
    const bool wide = a.X > kDagNarrowSide || a.Y > kDagNarrowSide;
    cudaMemsetAsync(a.queue, 0, sizeof(int), s);
    auto run = [&](auto kernel, int warps, size_t area) {
        const size_t smem = area * warps;
        const KernelShape ks = kernel_setup((const void *)kernel, 32 * warps, smem);
        kernel<<<std::min((a.n_list + warps - 1) / warps, ks.sms * ks.blocks_per_sm), 32 * warps, smem, s>>>(a);
    };
    if (cls == 0 && !wide) run(dag_build_kernel<WarpArea<SmallCaps, false>, 2>, 2, sizeof(WarpArea<SmallCaps, false>));
    if (cls == 0 && wide) run(dag_build_kernel<WarpArea<SmallCaps, true>, 2>, 2, sizeof(WarpArea<SmallCaps, true>));
    if (cls == 1 && !wide) run(dag_build_kernel<WarpArea<LargeCaps, false>, 1>, 1, sizeof(WarpArea<LargeCaps, false>));
    if (cls == 1 && wide) run(dag_build_kernel<WarpArea<LargeCaps, true>, 1>, 1, sizeof(WarpArea<LargeCaps, true>));
    if (cls == 2) dag_build_kernel<WarpArea<LastCaps, true>, 1><<<std::min(builders, a.n_list), 32, 0, s>>>(a);
}

void launch_dag_gather(const DagGatherArgs &a, cudaStream_t s) {
    if (a.n <= 0) return;
    dag_gather_kernel<<<(a.n + kGatherWarps - 1) / kGatherWarps, 32 * kGatherWarps, 0, s>>>(a);
}

}  // namespace igr
