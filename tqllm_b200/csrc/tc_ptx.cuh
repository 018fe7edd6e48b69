// Inline-PTX helpers for the sm_100a kernels: mbarriers with bounded waits, bulk (TMA) copies, cp.async, tcgen05
// (tensor-memory allocation, MMA issue, commit, loads) and the shared-memory matrix descriptor.
#pragma once
#include <stdint.h>

namespace b2 {
namespace tc {

constexpr uint32_t WAIT_LIMIT = 1u << 18;   // tries before a wait gives up; a try that fails took 2.0 us on a B200 (tests/test_gpu_bounded_wait.py): half a second

__device__ __forceinline__ uint32_t saddr(const void * p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One try at a phase of a barrier: the hardware suspends the thread until the phase completes, or for a time of its own choice (an
// explicit limit costs an operand at every wait: 1 % of the decode-sized products)
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// One phase of a barrier, one thread; false = gave up after WAIT_LIMIT tries
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
#pragma unroll 1
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i)
        if (bar_try(bar, parity)) return true;
    return false;
}
// The same for a whole converged warp, all lanes on one barrier
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
#pragma unroll 1
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i)
        if (__all_sync(0xffffffffu, bar_try(bar, parity))) return true;
    return false;
}
// TMA gather: rows y0..y3, 64 16-bit columns from x (a multiple of 8), of the mapped matrix (box of one row) -> four consecutive
// 128-byte rows at dst, 128-byte swizzled, completion on an mbarrier
__device__ __forceinline__ void tma_gather4(uint32_t dst, const void * map, int x, int y0, int y1, int y2, int y3, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(bar) : "memory");
}
// TMA box of a mapped 3-D array from (x, y, z), completion on an mbarrier (what lies outside the array arrives as zeros)
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void * map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// one lane of a converged warp, the same every time
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok));
    return ok != 0;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// tensor memory: one warp allocates `cols` columns (a power of two >= 32) and writes the base address to shared memory
__device__ __forceinline__ void tmem_alloc(uint32_t slot_saddr, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_saddr), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

// shared-memory matrix descriptor, the 128-byte swizzled K-major form: a row's 64 16-bit values are 128 contiguous bytes whose
// 16-byte pieces are XORed with the row's low three bits; eight rows (1024 bytes, aligned so) form an atom, sbo = bytes between
// atoms. Split in halves: the low half carries the address, the high half is a constant (sbo 1024, fixed bit 46, swizzle).
constexpr uint32_t SW128_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t sw128_desc_lo(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
// instruction descriptor: fp32 accumulator, K-major A and B, M x N; ab_format: 0 = E4M3 (kind::f8f6f4) / fp16 (kind::f16),
// 1 = bf16 (kind::f16)
__device__ __forceinline__ uint32_t idesc(uint32_t m, uint32_t n, uint32_t ab_format) {
    return (1u << 4) | (ab_format << 7) | (ab_format << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// Products with A (128 x 16 per product, fp16) in tensor memory (row in lane, two values of K per column) and B (N x 16 each) in
// shared memory, fp32 sums in tensor memory: one 64-column step is four of them, even ones into d0 (added to what is there when
// acc0), odd ones into d1 (acc1); the two may be the same. Then `bar` gets one arrival when every product issued so far has
// completed, and `bar2` too when it is not 0. Called by a whole converged warp; one elected lane issues. One statement with
// predicates: as separate calls inside a branch each product cost the warp 48 cycles, the commit 60.
#define B2_MMA(D, A, B, P) " @pe tcgen05.mma.cta_group::1.kind::f16 [" D "], [" A "], " B ", id, " P ";\n"
#define B2_MMA_STEP(BLO, A0, A1, A2, A3, P0, P1, P2)                                                                                  \
    " mov.b64 db, {" BLO ", bh};\n" B2_MMA("%0", A0, "db", P0) " add.u32 t, " BLO ", 2;\n mov.b64 db, {t, bh};\n" B2_MMA("%1", A1, "db", P1)  \
    " add.u32 t, " BLO ", 4;\n mov.b64 db, {t, bh};\n" B2_MMA("%0", A2, "db", P2) " add.u32 t, " BLO ", 6;\n mov.b64 db, {t, bh};\n" B2_MMA("%1", A3, "db", P2)
#define B2_MMA_HEAD                                                                                                                  \
    "{\n .reg .pred pe, p0, p1, pt, pb, pc;\n .reg .b64 db;\n .reg .b32 t, a1, a2, a3, a4, a5, a6, a7, id, bh;\n"                        \
    " elect.sync _|pe, 0xffffffff;\n setp.ne.b32 p0, %5, 0;\n setp.ne.b32 p1, %6, 0;\n setp.eq.b32 pt, 0, 0;\n setp.ne.and.b32 pb, %8, 0, pe;\n" \
    " mov.b32 id, %4;\n mov.b32 bh, %9;\n add.u32 a1, %2, 8;\n add.u32 a2, %2, 16;\n add.u32 a3, %2, 24;\n"
#define B2_MMA_TAIL                                                                                                                  \
    " @pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n"                                               \
    " @pb tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%8];\n}"
__device__ __forceinline__ void mma_step(uint32_t d0, uint32_t d1, uint32_t a, uint32_t b_lo, uint32_t id, uint32_t acc0, uint32_t acc1, uint32_t bar, uint32_t bar2) {
    asm volatile(B2_MMA_HEAD B2_MMA_STEP("%3", "%2", "a1", "a2", "a3", "p0", "p1", "pt") B2_MMA_TAIL
                 ::"r"(d0), "r"(d1), "r"(a), "r"(b_lo), "r"(id), "r"(acc0), "r"(acc1), "r"(bar), "r"(bar2), "r"(SW128_DESC_HI) : "memory");
}
// two steps whose A operands follow each other (32 columns each) and whose B operands start at b_lo and b_lo2
__device__ __forceinline__ void mma_unit(uint32_t d0, uint32_t d1, uint32_t a, uint32_t b_lo, uint32_t id, uint32_t acc0, uint32_t acc1, uint32_t bar, uint32_t bar2,
                                         uint32_t b_lo2) {
    asm volatile(B2_MMA_HEAD " add.u32 a4, %2, 32;\n add.u32 a5, %2, 40;\n add.u32 a6, %2, 48;\n add.u32 a7, %2, 56;\n"
                 B2_MMA_STEP("%3", "%2", "a1", "a2", "a3", "p0", "p1", "pt") B2_MMA_STEP("%10", "a4", "a5", "a6", "a7", "pt", "pt", "pt") B2_MMA_TAIL
                 ::"r"(d0), "r"(d1), "r"(a), "r"(b_lo), "r"(id), "r"(acc0), "r"(acc1), "r"(bar), "r"(bar2), "r"(SW128_DESC_HI), "r"(b_lo2) : "memory");
}
// the barrier gets one arrival when every MMA this thread issued before has completed
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 16 consecutive fp32 columns of this thread's lane (lane = 32 * (warp & 3) + lane id)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
// a warp's 16 rows x 32 columns from the registers of an m16n8-style fragment: register 4 i + 2 r + c of lane 4 g + t is column
// 8 i + 2 t + c of row g + 8 r; taddr's lane is the first of the 16 (a multiple of 16 inside the warp's quarter)
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
                   "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

}  // namespace tc
}  // namespace b2
