// Inline-PTX helpers for the 5th-generation tensor cores (sm_103a): shared
// memory matrix descriptors, tcgen05.mma / commit / ld, mbarriers with bounded
// waits, and the swizzled operand layouts of the fast tensor-core kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sdbe {
namespace tc5 {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// Layout field (bits 61-63) of a shared-memory descriptor.
constexpr uint32_t kNoSwizzle = 0, kSwizzle128 = 2, kSwizzle64 = 4, kSwizzle32 = 6;

// Shared-memory matrix descriptor: start address, leading / stride byte
// offsets (16-byte units), descriptor version 1 (bit 46), layout.
__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
    return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) |
           (static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) |
           (static_cast<uint64_t>(layout) << 61);
}

// Instruction descriptor of kind::f16: FP32 accumulator, FP16 A and B, both K-major.
__host__ __device__ constexpr uint32_t idesc_f16(int m, int n) {
    return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u));
}

// The same, issued by one elected lane of a converged warp (the lowest active
// lane, the same one every time).
__device__ __forceinline__ void mma_f16_elect(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u));
}

// The barrier completes when every tcgen05 operation this thread issued so far has.
__device__ __forceinline__ void commit(uint64_t *mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
                 : "memory");
}

// commit() by the elected lane of a converged warp (the lane that issued the MMAs).
__device__ __forceinline__ void commit_elect(uint64_t *mbar) {
    asm volatile(
        "{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(mbar))
        : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t *mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t *mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_n(uint64_t *mbar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(n) : "memory");
}

// 2 TMEM columns of this thread's lane, no wait.
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
}

// 8 TMEM columns of this thread's lane, no wait.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// One try_wait on the phase with parity `parity`: the thread may sleep in it
// until the phase completes, for at most `hint_ns`.
__device__ __forceinline__ uint32_t mbar_try(uint64_t *mbar, uint32_t parity, uint32_t hint_ns) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(mbar)), "r"(parity & 1u), "r"(hint_ns)
        : "memory");
    return done;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// One try_wait without a time hint: returns at once when the phase has
// completed (the common case in a pipelined consumer, about 20 cycles).
__device__ __forceinline__ uint32_t mbar_poll(uint64_t *mbar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(mbar)), "r"(parity & 1u)
        : "memory");
    return done;
}

// Bounded wait for the phase with parity `parity`: a quick poll first, then
// sleeps in try_wait rather than spinning (so waiting warps take no issue
// slots from working ones) and gives up after `limit_ns` of global time;
// false on time-out.
__device__ __forceinline__ bool mbar_wait(uint64_t *mbar, uint32_t parity, uint64_t limit_ns = 1000000000ull) {
    if (mbar_poll(mbar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        if (mbar_try(mbar, parity, 100000u)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

__device__ __forceinline__ bool flag_set(const int *flag) { return *reinterpret_cast<const volatile int *>(flag) != 0; }
// mbar_wait by a whole warp that raises `flag` (shared memory) on time-out; once
// it is raised, waits return at once.  Lanes poll for themselves and may see the
// phase complete at different times, so the warp votes (and joins again after
// the slow way): the instructions behind a wait are often .sync.aligned.
// Returns whether this lane saw the phase complete.
__device__ __forceinline__ bool wait_or_flag(uint64_t *mbar, uint32_t parity, int *flag) {
    if (__all_sync(0xffffffffu, mbar_poll(mbar, parity))) return true;
    const bool done = !flag_set(flag) && mbar_wait(mbar, parity);
    if (!done) *reinterpret_cast<volatile int *>(flag) = 1;
    __syncwarp();
    return done;
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// 16 bytes global -> shared, not through L1.
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Bulk copy global -> shared of `bytes` (multiple of 16), completing on mbar.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *mbar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(mbar))
        : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Generic-proxy shared-memory writes made visible to the tensor cores (async proxy).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 TMEM columns of this thread's lane (taddr = base | lane quarter << 16 | column), no wait.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// Waits for this thread's TMEM loads, then ties the N registers of each of
// a and b to an empty asm after the wait so that no use moves above it.
template <int N>
__device__ __forceinline__ void tmem_wait(uint32_t *a, uint32_t *b) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; i += 4) {
        asm volatile("" : "+r"(a[i]), "+r"(a[i + 1]), "+r"(a[i + 2]), "+r"(a[i + 3]));
        asm volatile("" : "+r"(b[i]), "+r"(b[i + 1]), "+r"(b[i + 2]), "+r"(b[i + 3]));
    }
}

// The same for one array of N registers.
template <int N>
__device__ __forceinline__ void tmem_wait1(uint32_t *a) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; i += 4) asm volatile("" : "+r"(a[i]), "+r"(a[i + 1]), "+r"(a[i + 2]), "+r"(a[i + 3]));
}

// Byte offset of the complex element (row, kc) of a K-major FP16 operand whose
// rows hold (re, im) pairs, in the 128-byte swizzle (rows of 32 complex
// values: 16-byte chunk c of row r stored at chunk c ^ (r % 8); 8-row atoms of
// 1024 bytes) and in the 64-byte swizzle (rows of 16 complex values: chunk c
// at c ^ ((r % 8) / 2); 8-row atoms of 512 bytes).  Atoms must be aligned to
// their size.
__device__ __forceinline__ uint32_t sw128_off(int row, int kc) {
    return static_cast<uint32_t>((row >> 3) * 1024 + (row & 7) * 128 + ((((kc >> 2) ^ (row & 7)) & 7) << 4) +
                                 (kc & 3) * 4);
}
__device__ __forceinline__ uint32_t sw64_off(int row, int kc) {
    return static_cast<uint32_t>((row >> 3) * 512 + (row & 7) * 64 + ((((kc >> 2) ^ ((row & 7) >> 1)) & 3) << 4) +
                                 (kc & 3) * 4);
}

// Tensor memory of `cols` columns (a power of two, 32 to 512), by one whole
// warp; the base address lands in shared memory at dst.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}

// 32 registers to or from 32 columns of this thread's lane (taddr as in tmem_ld16), no wait.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"f"(r[0]),
        "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]), "f"(r[9]), "f"(r[10]),
        "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ldf16(uint32_t taddr, float *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]),
          "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
        : "r"(taddr)
        : "memory");
}
#define SDBE_RIN(r) \
    "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), \
    "f"(r[8]), "f"(r[9]), "f"(r[10]), "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]), \
    "f"(r[16]), "f"(r[17]), "f"(r[18]), "f"(r[19]), "f"(r[20]), "f"(r[21]), "f"(r[22]), "f"(r[23]), \
    "f"(r[24]), "f"(r[25]), "f"(r[26]), "f"(r[27]), "f"(r[28]), "f"(r[29]), "f"(r[30]), "f"(r[31])
#define SDBE_ROUT(r) \
    "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), \
    "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]), \
    "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23]), \
    "=f"(r[24]), "=f"(r[25]), "=f"(r[26]), "=f"(r[27]), "=f"(r[28]), "=f"(r[29]), "=f"(r[30]), "=f"(r[31])
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,"
        "%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::SDBE_RIN(r),
        "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : SDBE_ROUT(r)
        : "r"(taddr)
        : "memory");
}
#undef SDBE_RIN
#undef SDBE_ROUT
// N complex values of this thread (N a multiple of 8) set aside in 2 N
// columns of its lane, and taken back by the same thread.
template <int N>
__device__ __forceinline__ void tmem_park(uint32_t taddr, const float2 *v) {
    float r[2 * N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[2 * i] = v[i].x;
        r[2 * i + 1] = v[i].y;
    }
#pragma unroll
    for (int i = 0; i + 16 <= N; i += 16) tmem_st32(taddr + 2 * i, r + 2 * i);
    if constexpr (N % 16 == 8) tmem_st16(taddr + 2 * (N - 8), r + 2 * (N - 8));
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void tmem_unpark(uint32_t taddr, float2 *v) {
    float r[2 * N];
#pragma unroll
    for (int i = 0; i + 16 <= N; i += 16) tmem_ld32(taddr + 2 * i, r + 2 * i);
    if constexpr (N % 16 == 8) tmem_ldf16(taddr + 2 * (N - 8), r + 2 * (N - 8));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) {
        asm volatile("" : "+f"(r[2 * i]), "+f"(r[2 * i + 1]));  // no use moves above the wait
        v[i] = make_float2(r[2 * i], r[2 * i + 1]);
    }
}

// (a, b) -> the FP16 pair rn(a), rn(b) as a 32-bit word.
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %2, %1;" : "=r"(r) : "f"(a), "f"(b));
    return r;
}

}  // namespace tc5
}  // namespace sdbe
