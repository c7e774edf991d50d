// tcgen05 (5th-generation tensor core) building blocks for sm_100a: shared
// memory matrix descriptors, the instruction descriptor of a BF16 x BF16 ->
// F32 MMA, TMEM allocation, MMA issue and commit, bounded mbarrier waits and
// TMEM loads.  Operand tiles use the canonical layouts without swizzle: core
// matrices of 8 x 16 bytes (128 contiguous bytes).  K-major: 8 rows of 8 K
// elements each, the two K halves of a K = 16 step apart by the leading byte
// offset, groups of 8 rows by the stride byte offset.  MN-major: 8 K rows of 8
// elements along M or N each, groups of 8 K apart by the leading byte offset,
// groups of 8 elements along M or N by the stride byte offset.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace igr {
namespace umma {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lead, uint32_t stride) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFF);  // start address
    d |= (uint64_t)(lead >> 4) << 16;                // leading byte offset
    d |= (uint64_t)(stride >> 4) << 32;              // stride byte offset
    d |= (uint64_t)1 << 46;                          // descriptor version of sm_100
    return d;                                        // base offset 0, no swizzle
}
// a sub-tile of 16 K columns and 128 (or fewer) rows, end to end: per group of 8 rows
// the core matrices of its two K halves, 128 bytes apart, groups 256
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) { return smem_desc(saddr, 128, 256); }

// kind::f16 instruction descriptor: F32 accumulator, BF16 A and B, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// the same with both operands MN-major (the sum runs over the core matrices' rows)
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int M, int N) {
    return idesc_bf16(M, N) | (1u << 15) | (1u << 16);
}

// one warp: allocate `cols` TMEM columns (power of two >= 32), address into *dst
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, int cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, int cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, int arrivals = 1) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// waits for the phase of `parity` to complete; gives up after `limit_ns`
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, unsigned long long limit_ns) {
    const uint32_t a = smem_u32(bar);
    const unsigned long long t0 = now_ns();
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if (now_ns() - t0 > limit_ns) return false;
    }
}

// The same for one of several roles of a block that wait on one another: gives
// up also once another role has (`*quit`), and tells them when its own limit
// runs out.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, unsigned long long limit_ns,
                                          volatile int *quit) {
    const uint32_t a = smem_u32(bar);
    unsigned long long t0 = 0;
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if (*quit) return false;
        const unsigned long long t = now_ns();
        if (!t0) t0 = t;
        if (t - t0 > limit_ns) {
            *quit = 1;
            return false;
        }
    }
}

// 16-byte asynchronous copy to shared memory; zeros when !valid (src is then not read)
__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// D[tmem] (+)= A * B^T for one K = 16 step; issued by one thread
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n" ::"r"(tmem),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
        : "memory");
}
// arrives on `bar` once every MMA issued so far by this thread has completed
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 16 consecutive f32 columns of this thread's TMEM lane (warp w reads lanes 32 (w % 4) on),
// to be waited for with tmem_wait
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                 "[%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32-byte global store (32-byte aligned address)
__device__ __forceinline__ void store32(void *p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

}  // namespace umma
}  // namespace igr
