// Inline-PTX wrappers for the fifth-generation tensor core path (tcgen05.mma with accumulators in
// tensor memory) and the mbarrier waits around it, shared by the kernels that use it.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace smelt {

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait on an mbarrier phase: try_wait suspends the thread in hardware for up to the hinted
// time (a spinning warp would take issue slots from the warp that shares its scheduler), the
// loop gives up after about a second and reports failure instead of waiting forever: a try that fails takes
// 4.0 us, with the hint of one as without a hint (256 to 1024 tries in a row, a warp alone or 24).
__device__ __forceinline__ bool mbar_poll_bounded(uint64_t* bar, uint32_t parity) {
#pragma unroll 1
    for (uint32_t i = 0; i < (1u << 18); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity), "r"(1000u)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// Waits for a phase; gives up after about a second, or as soon as another role has.
__device__ __forceinline__ bool wait_alive(uint64_t* bar, uint32_t parity, volatile uint32_t* dead) {
#pragma unroll 1
    for (uint32_t i = 0; i < (1u << 18); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity), "r"(1000u)
            : "memory");
        if (ok) return true;
        if (*dead) return false;
    }
    *dead = 1u;
    return false;
}
// The same with as little code as it takes, for kernels whose roles compete for the instruction cache: without the instruction's time
// hint, with which the compiler makes a timed loop around every wait (the 16-bit product, whose waits are few, is 1 % faster with it).  2^18
// tries are a second here too.
// bar, dead: addresses of shared memory.
__device__ __forceinline__ bool wait_alive_short(uint32_t bar, uint32_t parity, uint32_t dead) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 n, d;\n\t"
        "mov.u32 n, 262144;\n"
        "again_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra through_%=;\n\t"
        "ld.volatile.shared.u32 d, [%3];\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 q, d, 0;\n\t"
        "@q bra through_%=;\n\t"
        "setp.ne.u32 q, n, 0;\n\t"
        "@q bra again_%=;\n\t"
        "mov.u32 d, 1;\n\t"
        "st.volatile.shared.u32 [%3], d;\n"
        "through_%=:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(dead)
        : "memory");
    return ok != 0;
}
// A shared-memory address that stays in a register: left to itself the compiler makes it again from the CTA's number at every use.
__device__ __forceinline__ uint32_t kept(uint32_t address) {
    uint32_t a;
    asm volatile("mov.u32 %0, %1;" : "=r"(a) : "r"(address));
    return a;
}
// A box of a 2-D tensor map, x the inner coordinate (a multiple of 16 bytes).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y),
                 "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d_at(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void arrive_at(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void arrive_expect_at(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand tile, rows of 64 fp16 = 128 bytes, 128-byte swizzle: eight rows form a
// 1024-byte atom, atoms follow one another along the rows (stride 1024 bytes).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// D[128 x N] (+)= A[128 x 64] . B[N x 64]^T from shared memory as four steps of 16 columns (32 bytes in the descriptors' address fields).
// A whole warp calls it, one lane issues: the operands stay in the uniform registers that the instruction reads.
__device__ __forceinline__ void umma_f16_block(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
        "add.u64 a1, %1, 2;\n\tadd.u64 a2, %1, 4;\n\tadd.u64 a3, %1, 6;\n\t"
        "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The lane that issued, too (elect.sync chooses the same one every time).
__device__ __forceinline__ void commit_elected(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
// A value that is the same in all lanes, where the compiler can see it: what follows from it stays in uniform registers.
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t t, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                   "=r"(v[14]), "=r"(v[15])
                 : "r"(t)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_ld16(uint32_t (&v)[16]) {  // the loads behind v have arrived
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]),
                   "+r"(v[14]), "+r"(v[15])::"memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t cols) {  // one warp, converged; cols a power of two, 32..512
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// A row-major matrix of `width`-byte elements read in boxes of box_rows rows x 128 bytes, 128-byte swizzle; beyond its edges: zeros
// (affine_line.cu).
bool encode_rows(CUtensorMap* map, CUtensorMapDataType type, int width, const void* base, long rows, long cols, int box_rows);

}  // namespace smelt
