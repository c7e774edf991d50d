// Copies between device memory and the caller's pageable memory through
// page-locked chunks, by several host threads.
//
// A plain copy to pageable memory runs at the speed of one driver thread, which
// also takes the page faults of a fresh array: 34 MB of demand in 10 ms, 82 MB
// in 21 ms.  Here each of up to 16 threads takes a chunk at a time: DMA into its
// own page-locked chunk, then a memcpy to its place, so that the faults and
// copies of the chunks overlap.  A prediction of 1600 x 1600 GCells (164 MB of
// features rounded to BF16 on the way up, 164 MB down, 16 cores) went from 95 ms
// to 11; with 8 threads 13, with 4 threads 20.  Below kMinBytes the threads cost
// more than they save.
#include <sched.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "router.hpp"

namespace igr {

namespace {

constexpr size_t kChunk = (size_t)1 << 20;
constexpr size_t kMinBytes = (size_t)4 << 20;
constexpr int kMaxThreads = 16;

// Cores this process may run on (the machine's number of them says nothing about that).
int usable_cores() {
    cpu_set_t set;
    if (sched_getaffinity(0, sizeof set, &set) != 0) return hw_threads();
    return std::max(1, CPU_COUNT(&set));
}

// The caller's CUDA context, for its workers.  It need not be the primary one of its
// device, which cudaSetDevice would take: events of that one are refused on a stream of
// another.
class CallerContext {
    int (*set_)(void *) = nullptr;
    void *ctx_ = nullptr;

    template <typename F>
    static void entry(const char *name, F &f) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        cuda_check(cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q), name);
        if (q != cudaDriverEntryPointSuccess || !p) throw Error(ERR_CUDA, std::string("no driver entry point ") + name);
        f = reinterpret_cast<F>(p);
    }

public:
    CallerContext() {
        int (*get)(void **);
        entry("cuCtxGetCurrent", get);
        entry("cuCtxSetCurrent", set_);
        int rc = get(&ctx_);
        if (rc == 0 && !ctx_) {  // a thread that has not used CUDA yet: its device's primary context
            int dev = 0;
            cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
            cuda_check(cudaSetDevice(dev), "cudaSetDevice");
            rc = get(&ctx_);
        }
        if (rc != 0) throw Error(ERR_CUDA, "cuCtxGetCurrent");
    }
    void take() const {
        if (set_(ctx_) != 0) throw Error(ERR_CUDA, "cuCtxSetCurrent");
    }
};

// fn(worker) on `n` threads (the caller's among them), each in the caller's
// context; the first exception is rethrown once all have returned
template <typename F>
void run_workers(int n, F &&fn) {
    const CallerContext caller;
    std::mutex mu;
    std::exception_ptr err;
    auto work = [&](int w) {
        try {
            if (w > 0) caller.take();
            fn(w);
        } catch (...) {
            std::lock_guard<std::mutex> lock(mu);
            if (!err) err = std::current_exception();
        }
    };
    std::vector<std::thread> ts;
    ts.reserve((size_t)n);  // no exception may leave this function past a running thread
    for (int w = 1; w < n; w++) {
        try {
            ts.emplace_back(work, w);
        } catch (const std::exception &) {
            break;  // fewer threads than asked for: the others take the chunks
        }
    }
    work(0);
    for (auto &t : ts) t.join();
    if (err) std::rethrow_exception(err);
}

// a worker's page-locked chunk (a plain one where page-locked memory has run out:
// copies of it are staged by the driver) and the event of its last copy
struct Slot {
    PinnedBuf<unsigned char> buf;
    std::vector<unsigned char> plain;
    unsigned char *p = nullptr;
    cudaEvent_t ev = nullptr;
    Slot() {
        try {
            buf.alloc(kChunk);
            p = buf.p;
        } catch (const Error &) {
            (void)cudaGetLastError();
            plain.resize(kChunk);
            p = plain.data();
        }
        cuda_check(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "event");
    }
    ~Slot() {
        if (ev) cudaEventDestroy(ev);
    }
};

// Chunks of `items` items of `size` device bytes each, handed to the workers;
// each(slot, first, count) issues a chunk's copies on `s`.
template <typename F>
void by_chunks(size_t items, size_t size, cudaStream_t s, F &&each) {
    const size_t per = kChunk / size, chunks = (items + per - 1) / per;
    const int n = (int)std::min<size_t>({(size_t)kMaxThreads, (size_t)usable_cores(), chunks});
    std::atomic<size_t> next{0};
    std::atomic<bool> stop{false};
    run_workers(n, [&](int) {
        Slot slot;
        // a chunk whose copy may still run is not given back
        struct Drain {
            cudaStream_t s;
            ~Drain() { cudaStreamSynchronize(s); }
        } drain{s};
        try {
            while (!stop) {
                const size_t c = next.fetch_add(1);
                if (c >= chunks) break;
                each(slot, c * per, std::min(per, items - c * per));
            }
        } catch (...) {
            stop = true;
            throw;
        }
    });
}

// Whether a copy to or from p is best left to the driver.  Page-locked or registered
// memory needs no staging: through the chunks everything would move twice (34 MB of
// demand in 1.29 ms, directly in 0.67).  What is not plain host memory at all is the
// driver's to judge.  And where there is no second core, its own staging is faster than
// a thread that waits for each chunk (34 MB into an array in use: 2.2 ms, in chunks by
// as many threads as the machine has cores 3.7; with two cores and two threads 1.7).
bool direct(const void *p) {
    if (usable_cores() < 2) return true;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

// float -> BF16, to nearest even, NaN to the canonical one (as __float2bfloat16)
inline uint16_t bf16_bits(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    const uint32_t r = (u + 0x7fffu + ((u >> 16) & 1u)) >> 16;
    return (u & 0x7fffffffu) > 0x7f800000u ? 0x7fff : (uint16_t)r;
}

}  // namespace

void copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    if (bytes < kMinBytes || direct(dst)) {
        cuda_check(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), "D2H");
        cuda_check(cudaStreamSynchronize(s), "sync");
        return;
    }
    by_chunks(bytes, 1, s, [&](Slot &slot, size_t at, size_t n) {
        cuda_check(cudaMemcpyAsync(slot.p, static_cast<const char *>(src) + at, n, cudaMemcpyDeviceToHost, s), "D2H");
        cuda_check(cudaEventRecord(slot.ev, s), "event");
        cuda_check(cudaEventSynchronize(slot.ev), "D2H");
        std::memcpy(static_cast<char *>(dst) + at, slot.p, n);
    });
}

void copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    if (bytes < kMinBytes || direct(src)) {
        cuda_check(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s), "H2D");
        return;
    }
    by_chunks(bytes, 1, s, [&](Slot &slot, size_t at, size_t n) {
        cuda_check(cudaEventSynchronize(slot.ev), "H2D");  // the slot's last copy (none yet: returns at once)
        std::memcpy(slot.p, static_cast<const char *>(src) + at, n);
        cuda_check(cudaMemcpyAsync(static_cast<char *>(dst) + at, slot.p, n, cudaMemcpyHostToDevice, s), "H2D");
        cuda_check(cudaEventRecord(slot.ev, s), "event");
    });
}

void convert_to_bf16(const float *src, size_t n, __nv_bfloat16 *out) {
    auto *o = reinterpret_cast<uint16_t *>(out);
    for (size_t i = 0; i < n; i++) o[i] = bf16_bits(src[i]);
}

void copy_to_device_bf16(__nv_bfloat16 *dst, const float *src, size_t n, cudaStream_t s) {
    if (n * 2 < kMinBytes / 4) {
        std::vector<__nv_bfloat16> v(n);
        convert_to_bf16(src, n, v.data());
        cuda_check(cudaMemcpyAsync(dst, v.data(), n * 2, cudaMemcpyHostToDevice, s), "H2D");
        cuda_check(cudaStreamSynchronize(s), "H2D");
        return;
    }
    by_chunks(n, 2, s, [&](Slot &slot, size_t at, size_t m) {
        cuda_check(cudaEventSynchronize(slot.ev), "H2D");
        convert_to_bf16(src + at, m, reinterpret_cast<__nv_bfloat16 *>(slot.p));
        cuda_check(cudaMemcpyAsync(dst + at, slot.p, m * 2, cudaMemcpyHostToDevice, s), "H2D");
        cuda_check(cudaEventRecord(slot.ev, s), "event");
    });
}

}  // namespace igr
