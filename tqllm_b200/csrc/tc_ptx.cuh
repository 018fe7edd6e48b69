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
// TMA box of a mapped matrix from (x, y), completion on an mbarrier (what lies outside arrives as zeros)
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void * map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// TMA box of a mapped 3-D array from (x, y, z), completion on an mbarrier (what lies outside the array arrives as zeros)
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void * map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// the same with a policy (first_out_policy)
__device__ __forceinline__ void tma_load_3d_first_out(uint32_t dst, const void * map, int x, int y, int z, uint32_t bar, uint64_t policy) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void * map, int x, int y, int z, int w, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}
// a tensor map that copies will need soon
__device__ __forceinline__ void prefetch_map(const void * map) { asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory"); }
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
// the same for rows of 32 bytes (sixteen 16-bit values), 32-byte swizzle: eight rows are 256 bytes
constexpr uint32_t SW32_DESC_HI = (256u >> 4) | (1u << 14) | (6u << 29);
// instruction descriptor: fp32 accumulator, K-major A and B, M x N; ab_format: 0 = E4M3 (kind::f8f6f4) / fp16 (kind::f16),
// 1 = bf16 (kind::f16)
__device__ __forceinline__ uint32_t idesc(uint32_t m, uint32_t n, uint32_t ab_format) {
    return (1u << 4) | (ab_format << 7) | (ab_format << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// One product with A (128 x 16, fp16) in tensor memory (row in lane, two values of K per column) and B (N x 16) in shared memory,
// fp32 sums in tensor memory, added to what is there when acc != 0. The thread with `lead` set issues it: the loop around it can
// then be walked by the whole converged warp, whose addresses the compiler keeps in uniform registers.
template <uint32_t DESC_HI = SW128_DESC_HI>
__device__ __forceinline__ void mma_f16(bool lead, uint32_t d, uint32_t a, uint32_t b_lo, uint32_t id, uint32_t acc) {
    asm volatile("{\n .reg .pred p, q;\n .reg .b64 db;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %6, 0;\n mov.b64 db, {%2, %5};\n"
                 " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n}" ::"r"(d), "r"(a), "r"(b_lo), "r"(id), "r"(acc), "r"(DESC_HI), "r"(uint32_t(lead)) : "memory");
}
// a 64-column step: four products, even ones into d0 (added when acc0), odd ones into d1 (acc1); the two may be the same
__device__ __forceinline__ void mma_step(bool lead, uint32_t d0, uint32_t d1, uint32_t a, uint32_t b_lo, uint32_t id, uint32_t acc0, uint32_t acc1) {
    mma_f16(lead, d0, a, b_lo, id, acc0);
    mma_f16(lead, d1, a + 8, b_lo + 2, id, acc1);
    mma_f16(lead, d0, a + 16, b_lo + 4, id, 1);
    mma_f16(lead, d1, a + 24, b_lo + 6, id, 1);
}
// the barrier gets one arrival when every MMA this thread issued before has completed
__device__ __forceinline__ void mma_commit(bool lead, uint32_t bar) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar), "r"(uint32_t(lead)) : "memory");
}
// 16 consecutive fp32 columns of this thread's lane (lane = 32 * (warp & 3) + lane id)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
// 16 consecutive columns of this thread's lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
                   "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
// 16 rows x 8 columns, as the first four registers of the next one
__device__ __forceinline__ void tmem_st_16x256b_x1(uint32_t taddr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
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
