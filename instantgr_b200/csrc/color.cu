// Batch colouring: greedy independent sets of spatially disjoint nets.
//
// Semantics of generate_batches_rsmt_gpu (src/database_cuda.hpp:288-434,
// :437-631): nets are ranked by their position in the colouring order (higher
// rank wins a cell by atomicMax); in every round each unassigned, unblocked
// net claims the 4-neighbourhood of its conflict points and every
// `sparsity`-th cell of its tree segments; a net joins the batch when it still
// owns all of its points; nets whose points are owned by a net that joined are
// blocked for this batch and release their cells.  At most 30 rounds per
// batch; a batch with no new member ends the colouring.
//
// The reference is nondeterministic (a claiming thread re-reads the cell right
// after its atomicMax while others are still writing, and returns early).
// Here claiming and committing are separate phases separated by grid barriers,
// so the batches depend only on the input.
//
// A cell of the map holds the round, the rank of its claimer and, once the
// claimer has joined, a member bit above both.  A claim of a later round
// therefore replaces every older one but a member's, so that a blocked net need
// not look for the cells it still holds to give them back (660M reads on the
// 800k-net design), a lost net sees from the map alone whether a member owns one
// of its points, and, since members' cells do not change any more, it claims for
// the next round in the same phase: two grid barriers a round.  The owners are
// those of the round-by-round release: a net joins only when no candidate of a
// higher rank claims its points, candidates only drop out, and so no later claim
// ever meets a member's cell with a higher rank.  Above all that a cell holds the
// batch's generation, so that the map need not be cleared between batches and the
// nets left over claim for the next batch in the phase that lists them (300 nets:
// 512 -> 502 us a run, 40k: 4.75 -> 4.62 ms).  The 800k-net design's four
// colourings went from 17.4 + 7.5 + 4.5 + 4.0 to 14.9 + 5.3 + 3.1 + 2.7 ms, most
// of it in the rip-up passes through a warp per net of short lists; what bounds
// them now is the chain of dependent reads of a phase and the atomics of the claims.
//
// Work layout: the cells a net claims are precomputed once (claim lists, CSR
// per shape) and gathered per rank into one 16-byte header; a group of 8 lanes
// handles one net (a warp, when there are few).  Each round walks only the nets it
// concerns: the candidates (commit) and the nets that lost a point; the lists
// are rebuilt every phase with one global atomic per block (appends are staged
// in shared memory).  The whole colouring is one persistent cooperative
// kernel; the last rounds of a batch, which have few candidates, run in one
// block with block barriers.  Every grid barrier gives up after two seconds
// and reports ERR_TIMEOUT instead of waiting forever.
//
// Optionally (ColorDev::rev set) the round-0 map of every batch is kept up to
// date instead of being cleared and re-claimed by every net without a batch:
// the claimers of each cell are grouped by cell once; after a batch, each cell
// whose round-0 owner joined gets as new owner its highest claimer still
// without a batch (one warp per such cell, assigned claimers dropped from the
// list), which is the max the re-claim would give, since every other cell's
// owner is still without a batch and still the highest of a smaller set.
#include "gridsync.cuh"
#include "hooks.hpp"
#include "host.hpp"

namespace igr {

namespace {

constexpr int kThreads = 1024;
constexpr int kG = 8;                          // lanes per net of long lists
constexpr int kGroups = kThreads / kG;         // groups per block
constexpr int kBuf = 4096;                     // staged list entries per block
// rounds with at most this many candidates run in block 0 alone (two nets per
// group and phase at most)
constexpr int kBlockRounds = 2 * kGroups;

// flags (ints): [0..1] and [14..15] lost counts (by round parity, of even and odd
// batches), [2] batches, [4..5] barrier counter, [6] error, [8] rounds run, [9..10]
// candidate counts (by round parity), [11..12] nets left after a batch (by batch
// parity), [13] cells to recompute.  A counter is zeroed a barrier before it is used
// and a barrier after it was last read.
__device__ __forceinline__ int lost_counts(int batch) { return batch & 1 ? 14 : 0; }
enum : int { F_NB = 2, F_BAR = 4, F_ERR = 6, F_ROUNDS = 8, F_CAND = 9, F_LEFT = 11, F_DIRTY = 13 };

constexpr int kMaxRounds = 30;
// Lists that take the groups of the grid at most this many steps are listed and
// claim in one phase; longer ones are listed by a thread per net first, since the
// claims of a step would wait for its nets' batches to be read.
constexpr int kLeftSteps = 4;
// A map value, from the top bit down: generation of the batch, member, epoch, rank.
// The epoch is the round, unless ranks leave it too few bits: then the claims that
// are not members' are cleared from time to time.  A claim of a later generation
// is above everything of the ones before, so the map is cleared only when the
// generations run out, and the nets that a batch left claim for the next one while
// they are listed.
struct Values {
    int base, member;  // of the batch's generation: least value, least value of a member
    int bits;          // of the rank
    __device__ __forceinline__ int epoch(int e) const { return base + (e << bits); }  // | rank: a claim
};
__device__ __forceinline__ Values batch_values(const ColorDev &c, int gen) {
    const int base = gen << (c.rank_bits + c.epoch_bits + 1);
    return {base, base + (1 << (c.rank_bits + c.epoch_bits)), c.rank_bits};
}

// memory operations of this thread, summed into c.ops at the end (roofline
// accounting): claimed cells, points checked for commit, points checked for
// blocking, cells checked when a net joins, list entries scanned
struct Ops {
    unsigned long long claims = 0, points = 0, bpoints = 0, releases = 0, scans = 0;
};

struct Stage {
    int buf[kBuf];
    int n, base;
};

// Stages `k` of every lane with `want` set; called by all 32 lanes of a warp.
__device__ __forceinline__ void stage(Stage &st, bool want, int k, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, want);
    if (!m) return;
    int base = 0;
    if (lane == 0) base = atomicAdd(&st.n, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (want) st.buf[base + __popc(m & ((1u << lane) - 1))] = k;
}

// Appends the staged entries to list[*count ...]; every thread of the block calls it.
__device__ __forceinline__ void flush(Stage &st, int *list, int *count) {
    __syncthreads();
    const int m = st.n;
    if (threadIdx.x == 0 && m > 0) st.base = atomicAdd(count, m);
    __syncthreads();
    if (m > 0) {
        const int b = st.base;
        for (int i = threadIdx.x; i < m; i += blockDim.x) list[b + i] = st.buf[i];
    }
    if (threadIdx.x == 0) st.n = 0;
    __syncthreads();
}

// exclusive prefix of v over the block's threads (all threads call it); *total
// receives the block's sum
__device__ int block_exclusive(int v, int *total) {
    __shared__ int warp_sum[kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int t = lane < kThreads / 32 ? warp_sum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < kThreads / 32) warp_sum[lane] = t;  // inclusive over warps
    }
    __syncthreads();
    const int before = (wid ? warp_sum[wid - 1] : 0) + x - v;
    *total = warp_sum[kThreads / 32 - 1];
    __syncthreads();
    return before;
}

// map and batch change during the kernel: read them from L2
__device__ __forceinline__ int owner(const ColorDev &c, int cell) { return __ldcg(c.map + cell); }

// The three phases of a round.  A group of G lanes takes a net; blocks blk,
// blk+nblk, ... of the workers, group j of a block list entry j.  Lists that
// leave warps without a net are walked with a warp per net (a net of 300 claims
// takes three steps in place of ten), longer ones with kG lanes.
template <typename F8, typename F32>
__device__ __forceinline__ void by_length(int n, int nblk, F8 &&f8, F32 &&f32) {
    if (n <= nblk * (kThreads / 32)) f32();
    else f8();
}

// A group's walk over a list: entry and header of the net at hand.  On long lists
// (AHEAD) the header of the next net and the entry after it are on their way, so
// that the chain of reads of a step begins at the net's points (800k nets: 97.2 ->
// 96.2 ms a run, 130k: 4.41 -> 4.38; short lists, of a step or two, only lose by it).
template <bool AHEAD>
struct Walk {
    int k = -1, k1 = -1, k2 = -1;
    int4 h, h1;
    static __device__ __forceinline__ int entry(const int *list, int n, int idx) { return idx < n ? list[idx] : -1; }
    static __device__ __forceinline__ int4 header(const ColorDev &c, int k) {
        return k >= 0 ? c.hdr[k] : make_int4(0, 0, 0, 0);
    }
    __device__ __forceinline__ Walk(const ColorDev &c, const int *list, int n, int idx, int step) {
        if constexpr (AHEAD) {
            k = entry(list, n, idx);
            k1 = entry(list, n, idx + step);
            h = header(c, k);
        }
    }
    // to be called at the start of the step at idx, and next() at its end
    __device__ __forceinline__ void at(const ColorDev &c, const int *list, int n, int idx, int step) {
        if constexpr (AHEAD) {
            h1 = header(c, k1);
            k2 = entry(list, n, idx + 2 * step);
        } else {
            k = entry(list, n, idx);
            h = header(c, k);
        }
    }
    __device__ __forceinline__ void next() {
        if constexpr (AHEAD) {
            k = k1;
            h = h1;
            k1 = k2;
        }
    }
};

// Candidates claim their cells, four cells in flight per lane.  (Reading a cell
// before the atomic, though most cells have a higher owner already, made the
// claims 1.4 times slower: the atomics are not waited for, the reads are.)
template <int G>
__device__ __forceinline__ void claim_cells(const ColorDev &c, int4 h, int gl, int v) {
    for (int i = h.x + gl; i < h.y; i += 4 * G) {
        int cl[4];
#pragma unroll
        for (int u = 0; u < 4; u++) cl[u] = i + u * G < h.y ? __ldg(c.claim + i + u * G) : -1;
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (cl[u] >= 0) atomicMax(c.map + cl[u], v);
    }
}
template <int G>
__device__ __forceinline__ void claim_nets(const ColorDev &c, const int *list, int n, int value, int blk, int nblk,
                                           Ops &ops) {
    constexpr int kPer = kThreads / G;
    const int gl = threadIdx.x % G, first = blk * kPer + threadIdx.x / G;
    Walk<G == kG> w(c, list, n, first, nblk * kPer);
    for (int idx = first; idx < n; idx += nblk * kPer, w.next()) {
        w.at(c, list, n, idx, nblk * kPer);
        if (gl == 0) ops.claims += w.h.y - w.h.x;
        claim_cells<G>(c, w.h, gl, value | w.k);
    }
}
// round 0 of a batch
__device__ __forceinline__ void claim_phase(const ColorDev &c, const int *list, int n, int value, int blk, int nblk,
                                            Ops &ops) {
    by_length(n, nblk, [&] { claim_nets<kG>(c, list, n, value, blk, nblk, ops); },
              [&] { claim_nets<32>(c, list, n, value, blk, nblk, ops); });
}

// The nets of `list` still without a batch go to `left` and claim for round 0 of
// the next batch.
template <int G>
__device__ __forceinline__ void left_nets(const ColorDev &c, Stage &st, const int *list, int n, int *left, int *left_cnt,
                                          int value, int blk, int nblk, Ops &ops) {
    constexpr int kPer = kThreads / G;
    const int lane = threadIdx.x & 31, gl = lane % G;
    int it = 0;
    for (int b0 = blk * kPer; b0 < n; b0 += nblk * kPer, it++) {
        const int idx = b0 + threadIdx.x / G;
        const int k = idx < n ? list[idx] : -1;
        const bool stays = k >= 0 && __ldcg(c.batch + k) == -1;
        if (k >= 0 && gl == 0) ops.scans++;
        if (stays) {
            const int4 h = c.hdr[k];
            if (gl == 0) ops.claims += h.y - h.x;
            claim_cells<G>(c, h, gl, value | k);
        }
        stage(st, stays && gl == 0, k, lane);
        if ((it + 1) % (kBuf / kPer) == 0) flush(st, left, left_cnt);
    }
    flush(st, left, left_cnt);
}
__device__ __forceinline__ void left_phase(const ColorDev &c, Stage &st, const int *list, int n, int *left,
                                           int *left_cnt, int value, int blk, int nblk, Ops &ops) {
    by_length(n, nblk, [&] { left_nets<kG>(c, st, list, n, left, left_cnt, value, blk, nblk, ops); },
              [&] { left_nets<32>(c, st, list, n, left, left_cnt, value, blk, nblk, ops); });
}

// Candidates owning all their points join batch `cur` and mark the cells they
// own; the others go to the lost list.  (Four points in flight per lane made
// this and the next phase 1.1 times slower, stopping at the first foreign point,
// G points at a time, 1.4 times: fewer reads, but a longer chain of them.)  Block-uniform loop (staging and flushes).
template <int G>
__device__ __forceinline__ void commit_nets(const ColorDev &c, Stage &st, const int *list, int n, const Values &vs,
                                            int epoch, int cur, int *lost_cnt, int blk, int nblk, Ops &ops) {
    constexpr int kPer = kThreads / G;
    const int lane = threadIdx.x & 31, grp = lane / G, gl = lane % G;
    int it = 0;
    Walk<G == kG> w(c, list, n, blk * kPer + threadIdx.x / G, nblk * kPer);
    for (int b0 = blk * kPer; b0 < n; b0 += nblk * kPer, it++, w.next()) {
        const int idx = b0 + threadIdx.x / G;
        const bool valid = idx < n;
        w.at(c, list, n, idx, nblk * kPer);
        const int k = w.k;
        const int4 h = w.h;
        const int v = vs.epoch(epoch) | k, own = v + (vs.member - vs.base);
        bool ok = true;
        if (valid) {
            if (gl == 0) ops.points += h.w - h.z;
            for (int i = h.z + gl; i < h.w; i += 2 * G) {
                const int p0 = __ldg(c.pts + i);
                const int p1 = i + G < h.w ? __ldg(c.pts + i + G) : -1;
                const int o0 = owner(c, p0);
                const int o1 = p1 >= 0 ? owner(c, p1) : v;
                ok &= (o0 == v) & (o1 == v);
            }
        }
        const unsigned bad = (__ballot_sync(0xffffffffu, !ok) >> (grp * G)) & (0xffffffffu >> (32 - G));
        if (valid && bad == 0) {
            if (gl == 0) {
                c.batch[k] = cur;
                ops.releases += h.y - h.x;
            }
            for (int i = h.x + gl; i < h.y; i += 4 * G) {
                int cl[4], ow[4];
#pragma unroll
                for (int u = 0; u < 4; u++) cl[u] = i + u * G < h.y ? __ldg(c.claim + i + u * G) : -1;
#pragma unroll
                for (int u = 0; u < 4; u++) ow[u] = cl[u] >= 0 ? owner(c, cl[u]) : -1;
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (ow[u] == v) c.map[cl[u]] = own;
            }
        }
        stage(st, valid && bad != 0 && gl == 0, k, lane);
        if ((it + 1) % (kBuf / kPer) == 0) flush(st, c.lost, lost_cnt);
    }
    flush(st, c.lost, lost_cnt);
}
__device__ __forceinline__ void commit_phase(const ColorDev &c, Stage &st, const int *list, int n, const Values &vs,
                                             int epoch, int cur, int *lost_cnt, int blk, int nblk, Ops &ops) {
    by_length(n, nblk, [&] { commit_nets<kG>(c, st, list, n, vs, epoch, cur, lost_cnt, blk, nblk, ops); },
              [&] { commit_nets<32>(c, st, list, n, vs, epoch, cur, lost_cnt, blk, nblk, ops); });
}

// Lost nets with a point owned by a member are blocked for this batch; the
// others stay candidates and claim their cells for the next round, `epoch`.
template <int G>
__device__ __forceinline__ void next_nets(const ColorDev &c, Stage &st, int n, const Values &vs, int epoch,
                                          int *cand_cnt, int blk, int nblk, Ops &ops) {
    constexpr int kPer = kThreads / G;
    const int lane = threadIdx.x & 31, grp = lane / G, gl = lane % G;
    int it = 0;
    Walk<G == kG> w(c, c.lost, n, blk * kPer + threadIdx.x / G, nblk * kPer);
    for (int b0 = blk * kPer; b0 < n; b0 += nblk * kPer, it++, w.next()) {
        const int idx = b0 + threadIdx.x / G;
        const bool valid = idx < n;
        w.at(c, c.lost, n, idx, nblk * kPer);
        const int k = w.k;
        const int4 h = w.h;
        bool hit = false;
        if (valid) {
            if (gl == 0) ops.bpoints += h.w - h.z;
            for (int i = h.z + gl; i < h.w; i += 2 * G) {
                const int p0 = __ldg(c.pts + i);
                const int p1 = i + G < h.w ? __ldg(c.pts + i + G) : -1;
                const int o0 = owner(c, p0);
                const int o1 = p1 >= 0 ? owner(c, p1) : -1;
                hit |= (o0 >= vs.member) | (o1 >= vs.member);
            }
        }
        const bool blocked = ((__ballot_sync(0xffffffffu, hit) >> (grp * G)) & (0xffffffffu >> (32 - G))) != 0;
        if (valid && !blocked) {
            if (gl == 0) ops.claims += h.y - h.x;
            claim_cells<G>(c, h, gl, vs.epoch(epoch) | k);
        }
        stage(st, valid && !blocked && gl == 0, k, lane);
        if ((it + 1) % (kBuf / kPer) == 0) flush(st, c.cand, cand_cnt);
    }
    flush(st, c.cand, cand_cnt);
}
__device__ __forceinline__ void next_phase(const ColorDev &c, Stage &st, int n, const Values &vs, int epoch,
                                           int *cand_cnt, int blk, int nblk, Ops &ops) {
    by_length(n, nblk, [&] { next_nets<kG>(c, st, n, vs, epoch, cand_cnt, blk, nblk, ops); },
              [&] { next_nets<32>(c, st, n, vs, epoch, cand_cnt, blk, nblk, ops); });
}

// Rounds `round`.. of batch `cur` in this block alone, over the nc candidates
// in c.cand, which have claimed in that round.  Every thread of the block calls it.
__device__ void block_rounds(const ColorDev &c, Stage &st, const Values &vs, int round, int nc, int cur,
                             int *rounds_ctr, Ops &ops) {
    __shared__ int s_lost, s_cand;
    while (true) {
        if (threadIdx.x == 0) {
            s_lost = 0;
            s_cand = 0;
            (*rounds_ctr)++;
        }
        __syncthreads();
        commit_phase(c, st, c.cand, nc, vs, round, cur, &s_lost, 0, 1, ops);
        const int nl = s_lost;  // flush ends with a block barrier
        if (nl == nc || round + 1 >= kMaxRounds) break;
        round++;
        next_phase(c, st, nl, vs, round, &s_cand, 0, 1, ops);
        nc = s_cand;
        __syncthreads();  // every thread has read the counters before they are reset
        if (nc == 0) break;
    }
}

// Per batch: every net without a batch claims (atomicMax), candidates owning
// all their points join, lost nets are blocked or claim again.  Two grid
// barriers per round; the last rounds of a batch, with few candidates, run in
// block 0 alone.  The lists are unordered: every phase is order-independent.
__global__ void __launch_bounds__(kThreads, 1) coloring_kernel(ColorDev c, int max_batches) {
    __shared__ Stage st;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nth = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    const int XY = c.X * c.Y;
    int *flags = c.flags;
    volatile int *vflags = c.flags;
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(c.flags + F_BAR);
    int *err = c.flags + F_ERR;
    unsigned long long epoch_of_bar = 0;
    Ops ops;
    auto sum_ops = [&]() {
        if (!c.ops) return;
        unsigned long long v[5] = {ops.claims, ops.points, ops.bpoints, ops.releases, ops.scans};
#pragma unroll
        for (int j = 0; j < 5; j++) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_down_sync(0xffffffffu, v[j], o);
            if (lane == 0 && v[j]) atomicAdd(c.ops + j, v[j]);
        }
    };
    if (threadIdx.x == 0) st.n = 0;
    int *act = c.active, *act2 = c.active2;
    for (int k = tid; k < c.n; k += nth) {
        const int sh = c.perm ? c.perm[k] : k;
        const int c0 = c.claim_off[sh], p0 = c.pt_off[sh];
        c.hdr[k] = make_int4(c0, c.claim_n ? c0 + c.claim_n[sh] : c.claim_off[sh + 1], p0,
                             c.pt_n ? p0 + c.pt_n[sh] : c.pt_off[sh + 1]);
        act[k] = k;
    }
    const bool inc = c.rev != nullptr;
    for (int i = tid; i < XY; i += nth) {
        c.map[i] = -1;
        if (inc) c.rev_cnt[i] = 0;
    }
    if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
    if (inc) {
        // claimers of every cell (ranks), grouped by cell: counts, an exclusive
        // scan over the cells (a chunk per block), then the entries
        for (int k = tid; k < c.n; k += nth) {
            const int4 h = c.hdr[k];
            for (int i = h.x; i < h.y; i++) atomicAdd(c.rev_cnt + __ldg(c.claim + i), 1);
        }
        if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
        const int chunk = (XY + gridDim.x - 1) / gridDim.x;
        const int lo = min(XY, blockIdx.x * chunk), hi = min(XY, lo + chunk);
        const int per = (hi - lo + kThreads - 1) / kThreads;
        const int a0 = min(hi, lo + threadIdx.x * per), a1 = min(hi, a0 + per);
        int mine = 0, total = 0;
        for (int i = a0; i < a1; i++) mine += c.rev_cnt[i];
        int run = block_exclusive(mine, &total);
        if (threadIdx.x == 0) c.part[blockIdx.x] = total;
        if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
        if (tid == 0) {
            int acc = 0;
            for (int b = 0; b < (int)gridDim.x; b++) {
                const int t = c.part[b];
                c.part[b] = acc;
                acc += t;
            }
        }
        if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
        run += c.part[blockIdx.x];
        for (int i = a0; i < a1; i++) {
            c.rev_off[i] = run;
            run += c.rev_cnt[i];
            c.rev_cnt[i] = 0;
        }
        if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
        for (int k = tid; k < c.n; k += nth) {
            const int4 h = c.hdr[k];
            for (int i = h.x; i < h.y; i++) {
                const int cell = __ldg(c.claim + i);
                c.rev[c.rev_off[cell] + atomicAdd(c.rev_cnt + cell, 1)] = k;
            }
        }
        if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
    }
    int na = c.n, gen = 0;
    const int gens = inc ? 1 : 1 << (30 - c.rank_bits - c.epoch_bits);
    bool claimed = false;  // the nets without a batch have claimed for round 0
    for (int cur = 0; cur < max_batches; cur++) {
        const Values vs = batch_values(c, gen);
        const int f_lost = lost_counts(cur);
        const int *cand = act;  // round 0: every net without a batch
        int nc = na, epoch = 0;
        // with the round-0 map kept up to date, round 0 of a later batch starts
        // from it (its counters were reset before the last barrier)
        if (!claimed && !(inc && cur > 0)) {
            claim_phase(c, cand, nc, vs.base, blockIdx.x, gridDim.x, ops);
            if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
        }
        if (inc && cur == 0)  // the first round-0 map, whether or not its owners have joined yet
            for (int i = tid; i < XY; i += nth) {
                const int v = __ldcg(c.map + i);
                c.snap[i] = v >= vs.member ? v - vs.member : v;
            }
        for (int round = 0;; epoch++) {
            if (tid == 0) {
                flags[F_ROUNDS]++;
                flags[F_CAND + ((round + 1) & 1)] = 0;
            }
            commit_phase(c, st, cand, nc, vs, epoch, cur, flags + f_lost + (round & 1), blockIdx.x, gridDim.x, ops);
            if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
            if (tid == 0 && round == 0) {  // the next batch's counters
                flags[F_LEFT + ((cur + 1) & 1)] = 0;
                flags[lost_counts(cur + 1)] = 0;
            }
            const int nl = vflags[f_lost + (round & 1)];
            if (nl == nc || round + 1 >= kMaxRounds) break;  // no net joined, or the last round
            round++;
            if ((epoch + 1) >> c.epoch_bits) {  // out of epochs: clear all claims but the members'
                for (int i = tid; i < XY; i += nth)
                    if (__ldcg(c.map + i) < vs.member) c.map[i] = -1;
                epoch = -1;
                if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
            }
            if (tid == 0) flags[f_lost + (round & 1)] = 0;
            next_phase(c, st, nl, vs, epoch + 1, flags + F_CAND + (round & 1), blockIdx.x, gridDim.x, ops);
            if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
            cand = c.cand;
            nc = vflags[F_CAND + (round & 1)];
            if (nc == 0) break;
            // the tail counts its rounds as epochs
            if (nc <= kBlockRounds && epoch + 1 == round && !(kMaxRounds >> c.epoch_bits)) {
                if (blockIdx.x == 0) block_rounds(c, st, vs, round, nc, cur, flags + F_ROUNDS, ops);
                if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
                break;
            }
        }
        // nets still without a batch stay active and claim for the next batch; out
        // of generations, the map is cleared instead, or, when the round-0 map is
        // kept, the cells whose round-0 owner joined this batch are marked for
        // recomputation
        const bool fresh = gen + 1 < gens;
        gen = fresh ? gen + 1 : 0;
        claimed = fresh && na <= kLeftSteps * (int)gridDim.x * kGroups;
        if (!inc && !fresh)
            for (int i = tid; i < XY; i += nth) c.map[i] = -1;
        if (claimed)
            left_phase(c, st, act, na, act2, flags + F_LEFT + (cur & 1), batch_values(c, gen).base, blockIdx.x,
                       gridDim.x, ops);
        int it = 0;
        for (int b0 = blockIdx.x * kThreads; b0 < na && !claimed; b0 += nth, it++) {
            const int i = b0 + threadIdx.x;
            const int k = i < na ? act[i] : -1;
            const int bk = k >= 0 ? __ldcg(c.batch + k) : -2;
            if (k >= 0) ops.scans++;
            if (inc && bk == cur) {
                const int4 h = c.hdr[k];
                ops.releases += h.y - h.x;
                for (int q = h.x; q < h.y; q++) {
                    const int cell = __ldg(c.claim + q);
                    if (c.snap[cell] == k) {
                        c.snap[cell] = -1;
                        c.dirty[atomicAdd(flags + F_DIRTY, 1)] = cell;
                    }
                }
            }
            stage(st, bk == -1, k, lane);
            if ((it + 1) % (kBuf / kThreads) == 0) flush(st, act2, flags + F_LEFT + (cur & 1));
        }
        flush(st, act2, flags + F_LEFT + (cur & 1));
        if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
        na = vflags[F_LEFT + (cur & 1)];
        int *t = act; act = act2; act2 = t;
        if (na == 0) {
            if (tid == 0) flags[F_NB] = cur + 1;
            sum_ops();
            return;
        }
        if (inc) {
            // new round-0 owner of every marked cell: its highest claimer
            // still without a batch (claimers with a batch leave the list)
            // one warp per marked cell: 32 claimers per step, compacted in place
            // (a step writes only below the entries it has read)
            const int nd = vflags[F_DIRTY];
            for (int i = tid >> 5; i < nd; i += nth >> 5) {
                const int cell = c.dirty[i];
                const int base = c.rev_off[cell], len = c.rev_cnt[cell];
                int best = -1, w = 0;
                for (int q0 = 0; q0 < len; q0 += 32) {
                    const int q = q0 + lane;
                    const int k = q < len ? c.rev[base + q] : -1;
                    const bool live = k >= 0 && __ldcg(c.batch + k) == -1;
                    const unsigned m = __ballot_sync(0xffffffffu, live);
                    if (live) {
                        c.rev[base + w + __popc(m & ((1u << lane) - 1))] = k;
                        best = max(best, k);
                    }
                    w += __popc(m);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
                if (lane == 0) {
                    ops.scans += len;
                    c.rev_cnt[cell] = w;
                    c.snap[cell] = best;
                }
            }
            if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
            for (int i = tid; i < XY; i += nth) c.map[i] = c.snap[i];
            if (tid == 0) flags[F_DIRTY] = 0;
            if (!grid_sync(bar, err, epoch_of_bar, c.wait_ns, c.phantom)) return;
        }
    }
    if (tid == 0) flags[F_NB] = max_batches;
    sum_ops();
}

}  // namespace

void build_claims(int nshapes, const int *pt_off, const int *pts, const int *h_off, const int *hseg,
                  const int *v_off, const int *vseg, int X, int Y, int sparsity, std::vector<int> &off,
                  std::vector<int> &cells, int threads) {
    static const int dx[4] = {0, 0, -1, 1}, dy[4] = {0, -1, 0, 0};
    // cells of shape k in claim order; emit(cell) is called for each
    auto walk = [&](int k, auto &&emit) {
        for (int i = pt_off[k]; i < pt_off[k + 1]; i++) {
            const int x = pts[i] / Y, y = pts[i] % Y;
            for (int j = 0; j < 4; j++) {
                const int nx = x + dx[j], ny = y + dy[j];
                if (nx >= 0 && nx < X && ny >= 0 && ny < Y) emit(nx * Y + ny);
            }
        }
        for (int i = h_off[k]; i < h_off[k + 1]; i++) {
            const int s0 = hseg[2 * i], e0 = hseg[2 * i + 1], y = s0 % Y;
            for (int x = s0 / Y; x <= e0 / Y; x += sparsity) emit(x * Y + y);
        }
        for (int i = v_off[k]; i < v_off[k + 1]; i++) {
            const int s0 = vseg[2 * i], e0 = vseg[2 * i + 1], x = s0 / Y;
            for (int y = s0 % Y; y <= e0 % Y; y += sparsity) emit(x * Y + y);
        }
    };
    off.assign(nshapes + 1, 0);
    parallel_for(nshapes, threads, [&](int b, int e) {
        for (int k = b; k < e; k++) {
            int n = 0;
            walk(k, [&](int) { n++; });
            off[k + 1] = n;
        }
    });
    for (int k = 0; k < nshapes; k++) off[k + 1] += off[k];
    cells.resize(off[nshapes]);
    parallel_for(nshapes, threads, [&](int b, int e) {
        for (int k = b; k < e; k++) {
            int *o = cells.data() + off[k];
            walk(k, [&](int c) { *o++ = c; });
        }
    });
}

int run_coloring(ColorDev &c, int max_batch, cudaStream_t s) {
    (void)max_batch;
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, coloring_kernel, kThreads, 0);
    int blocks = sms * (per < 1 ? per : 1);
    if (blocks < 1) blocks = 1;
    c.wait_ns = (unsigned long long)test_hooks().wait_ns.load();
    c.phantom = (unsigned)test_hooks().barrier_phantom.load();
    for (c.rank_bits = 1; c.rank_bits < 29 && (c.n >> c.rank_bits) != 0;) c.rank_bits++;
    c.epoch_bits = std::min(5, 30 - c.rank_bits);
    cudaMemsetAsync(c.flags, 0, 16 * sizeof(int), s);
    cudaMemsetAsync(c.batch, 0xff, sizeof(int) * (size_t)c.n, s);
    int max_batches = c.n + 1;
    void *args[] = {&c, &max_batches};
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)coloring_kernel, dim3(blocks), dim3(kThreads), args, 0, s);
    if (e != cudaSuccess) return -1;
    int h[16];
    if (cudaMemcpyAsync(h, c.flags, sizeof h, cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
    if (h[F_ERR] != 0) return -2;
    c.rounds = h[F_ROUNDS];
    return h[F_NB];
}

}  // namespace igr
