// Phase-1 tree DP for callers that cannot allocate device memory.
//
// The tree DP keeps the layer tables of nets with more than kPatternNodeTile
// nodes in global scratch, and every launch needs a work counter, a per-net
// scratch offset and a net-id list.  igr_pattern_route gets these from
// cudaMalloc'd staging buffers.  Some callers cannot let a library allocate:
// a host that hands the GPU's memory to its own pool allocator and forbids
// other allocations, a real-time loop where a cudaMalloc (which can
// synchronise the device) would stall the other streams, or a process that
// runs close to the memory limit and must know its footprint up front.  For
// them this file holds the scratch in one fixed array in the library's own
// device image, so a call allocates nothing.
//
// Layout of the array (byte offsets, each part 256-byte aligned):
//   [0, 256)           StaticHeader (status, counters, scratch node count)
//   [256, ...)         net ids, those kept in scratch first (int32)
//   [..., ...)         scratch offset per net (int64, -1 for nets kept on chip)
//   [..., capacity)    layer tables of the nets kept in scratch (doubles)
// The header is cleared at the start of every call; the rest is rewritten by
// every call before it is read.
//
// A call is one checking kernel and the DP: the DP reads the checks' outcome
// from the header itself and does nothing when one failed, so the host waits
// once, at the end.  The nets kept in scratch (the long ones) come first in
// the DP's queue, so that none of them starts when the others are done.  A
// scan over the nets in one block, a second checking kernel and a wait before
// the DP took 182 + 15 us of kernels for 100,000 nets (now 18 us), and the
// caller's order left the long nets' chains to the end (0.37 of 1.0 ms).
#include "kcommon.cuh"
#include "router.hpp"

#include <mutex>
#include <string>

namespace igr {

namespace {

// One array per device that loads the library, held until the process exits.
static __device__ __align__(256) unsigned char g_pattern_scratch[kStaticScratchBytes];

struct StaticHeader {
    int queue;       // work counter of the DP launch
    int bad_net;     // a net that failed validation
    int big, little; // nets listed so far from the front (kept in scratch) and from the back
    PatternGate gate;
};

enum : int { kBadOffsets = 1, kBadNode = 2, kBadParent = 4, kBadRecord = 8 };

constexpr size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

// Validation of a net's offsets, node positions, preorder parents and record
// bounds, its place in the list of net ids and, for a net of more than `tile`
// nodes, its scratch (places and scratch in any order: the routes do not depend
// on either), one thread per net.
__global__ void __launch_bounds__(256)
static_prep_kernel(int n, const int *node_off, long long total_nodes, int tile, const int *nodes, const int *par,
                   const int64_t *route_off, const int *route_cap, long long routes_len, long long cells,
                   StaticHeader *h, int *ids, long long *so) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    int bad = 0, cnt = 0;
    if (k < n) {
        const int a = node_off[k], b = node_off[k + 1];
        cnt = b - a;
        if (a < 0 || cnt < 1 || b > total_nodes || (k == 0 && a != 0) || (k == n - 1 && b != total_nodes)) {
            bad = kBadOffsets;
        } else {
            const long long ro = route_off[k];
            const int rc = route_cap[k];
            if (ro < 0 || rc < 1 || ro + rc > routes_len) bad |= kBadRecord;
            for (int i = a; i < b; i++) {
                const int loc = i - a;
                if (nodes[i] < 0 || nodes[i] >= cells) bad |= kBadNode;
                if (loc == 0 ? par[i] != -1 : (par[i] < 0 || par[i] >= loc)) bad |= kBadParent;
            }
        }
        if (bad) {
            atomicOr(&h->gate.status, bad);
            atomicExch(&h->bad_net, k);
        }
    }
    const bool big = k < n && cnt > tile;
    const unsigned mb = __ballot_sync(0xffffffffu, big), ml = __ballot_sync(0xffffffffu, k < n && !big);
    // nodes of the warp's nets kept in scratch, up to and with this one
    long long sum = big ? cnt : 0;
    if (mb) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += t;
        }
    }
    int b0 = 0, l0 = 0;
    long long s0 = 0;
    if (lane == 31) {
        if (mb) {
            b0 = atomicAdd(&h->big, __popc(mb));
            s0 = (long long)atomicAdd(&h->gate.big_nodes, (unsigned long long)sum);
        }
        if (ml) l0 = atomicAdd(&h->little, __popc(ml));
    }
    b0 = __shfl_sync(0xffffffffu, b0, 31);
    l0 = __shfl_sync(0xffffffffu, l0, 31);
    s0 = __shfl_sync(0xffffffffu, s0, 31);
    if (k >= n) return;
    const unsigned below = (1u << lane) - 1;
    ids[big ? b0 + __popc(mb & below) : n - 1 - (l0 + __popc(ml & below))] = k;
    so[k] = big ? s0 + sum - cnt : -1;
}

std::mutex g_setup_mu;
unsigned char *g_scratch_ptr[kStaticMaxDevices] = {};

// Device address of g_pattern_scratch on the current device, looked up once
// per device.  In host code the symbol names a host-side shadow, never the
// device memory, so it is not handed to a kernel itself.
unsigned char *static_scratch_ptr() {
    int dev = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev < 0 || dev >= kStaticMaxDevices) throw Error(ERR_INVALID, "device ordinal beyond the static scratch table");
    std::lock_guard<std::mutex> lock(g_setup_mu);
    if (!g_scratch_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_pattern_scratch);
        if (e != cudaSuccess || !p)
            throw Error(ERR_CUDA, std::string("cudaGetSymbolAddress of the static scratch: ") + cudaGetErrorString(e));
        g_scratch_ptr[dev] = static_cast<unsigned char *>(p);
    }
    return g_scratch_ptr[dev];
}

}  // namespace

void pattern_route_static(const GridDev &g, int n, const int *node_off, int64_t total_nodes, const int *nodes,
                          const int *par, const int64_t *route_off, const int *route_cap, int *routes,
                          int64_t routes_len, int stamp, cudaStream_t s) {
    if (n < 0 || total_nodes < 0 || routes_len < 0) throw Error(ERR_INVALID, "negative size");
    if (n > kStaticMaxNets)
        throw Error(ERR_CAPACITY, "batch of " + std::to_string(n) + " nets exceeds the static-scratch limit of " +
                                      std::to_string(kStaticMaxNets) + " nets per call");
    if (n == 0) return;
    if (!node_off || !nodes || !par || !route_off || !route_cap || !routes) throw Error(ERR_INVALID, "null pointer");
    unsigned char *base = static_scratch_ptr();
    const size_t off_ids = 256;
    const size_t off_so = align256(off_ids + sizeof(int) * (size_t)n);
    const size_t off_tab = align256(off_so + sizeof(long long) * (size_t)n);
    auto *h = reinterpret_cast<StaticHeader *>(base);
    auto *ids = reinterpret_cast<int *>(base + off_ids);
    auto *so = reinterpret_cast<long long *>(base + off_so);
    // nodes whose tables fit behind the lists
    const int64_t room = off_tab < kStaticScratchBytes ? (int64_t)((kStaticScratchBytes - off_tab) / sizeof(double)) : 0;
    int64_t max_big = room * 2 / (2 * kPatternScratchD + kPatternScratchI);
    while (max_big > 0 && pattern_scratch_doubles(max_big) > room) max_big--;
    cuda_check(cudaMemsetAsync(h, 0, sizeof(StaticHeader), s), "memset");
    const long long cells = (long long)(g.L + 1) * g.X * g.Y;
    static_prep_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, node_off, total_nodes, kPatternNodeTile, nodes, par,
                                                       route_off, route_cap, routes_len, cells, h, ids, so);
    TreeBatchDev tb{ids, node_off, nodes, par, route_off, route_cap, routes,
                    reinterpret_cast<double *>(base + off_tab), reinterpret_cast<const int64_t *>(so),
                    max_big, n};
    tb.queue = &h->queue;
    tb.gate = &h->gate;
    launch_pattern_route(g, tb, stamp, s);
    cuda_check(cudaGetLastError(), "launch");
    StaticHeader hh{};
    cuda_check(cudaMemcpyAsync(&hh, h, sizeof hh, cudaMemcpyDeviceToHost, s), "D2H");
    cuda_check(cudaStreamSynchronize(s), "sync");
    const int status = hh.gate.status;
    const int64_t big_nodes = (int64_t)hh.gate.big_nodes;
    if (status & kBadOffsets)
        throw Error(ERR_INVALID, "node_off must start at 0, end at total_nodes and give every tree a node (near net " +
                                     std::to_string(hh.bad_net) + ")");
    if (status & kBadRecord)
        throw Error(ERR_INVALID, "route record of net " + std::to_string(hh.bad_net) + " lies outside routes");
    if (status & kBadNode)
        throw Error(ERR_INVALID, "node position out of range (net " + std::to_string(hh.bad_net) + ")");
    if (status & kBadParent)
        throw Error(ERR_STATE, "tree nodes must be in preorder with par[i] < i (net " + std::to_string(hh.bad_net) + ")");
    const size_t need = off_tab + sizeof(double) * (size_t)pattern_scratch_doubles(big_nodes);
    if (need > kStaticScratchBytes)
        throw Error(ERR_CAPACITY, "batch needs " + std::to_string(need) + " bytes of scratch (" +
                                      std::to_string(big_nodes) + " nodes in nets of more than " +
                                      std::to_string(kPatternNodeTile) + " nodes); the static scratch holds " +
                                      std::to_string(kStaticScratchBytes) + " bytes");
}

}  // namespace igr
