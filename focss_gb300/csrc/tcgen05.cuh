// tcgen05.cuh -- thin wrappers over the fifth-generation tensor-core, mbarrier
// and bulk-copy instructions, shared by the kernels that issue them (cnn.cu,
// triplet.cu, ldbp.cu).
#pragma once

#include <cuda.h>  // CUtensorMap
#include <cuda_runtime.h>
#include <stdint.h>

namespace fg {
namespace tcg {

constexpr long long kWaitCap = 1ll << 22;  // mbarrier polls before giving up

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---------------------------------------------------------------- mbarriers
__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// Waits for the phase of parity `parity` of `bar`, at most kWaitCap polls.
// Gives up early when *abort is set, and sets it when the polls run out.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity, volatile int* abort) {
    const uint32_t a = smem_addr(bar);
    for (long long it = 0; it < kWaitCap; ++it) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if (abort && *abort) return false;
    }
    if (abort) *abort = 1;
    return false;
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
// Shared-memory writes of this thread become visible to the asynchronous proxy
// (tensor core and copy engine).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// ---------------------------------------------------------------- copies
// `bytes` (a multiple of 16) global -> shared, completing on `bar`; both
// addresses on 16-byte boundaries.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// TMA tensor copy of one box at (x, y, z) of a 3-D tensor map into shared
// memory, completing on `bar` (x * element size must be a multiple of 16 bytes).
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
        : "memory");
}

// ---------------------------------------------------------------- tensor core
// Shared-memory matrix descriptor: start address, LBO and SBO in 16-byte
// units, the descriptor version 1 at bit 46, base offset 0, no swizzling.
// K-major operand: core matrices of 8 rows x 16 bytes (rows 16 bytes apart),
// LBO = byte stride between core matrices along K, SBO = along M or N.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}
// The same for a K-major operand in the 32-byte swizzled layout: rows of 32
// bytes, 8-row groups 256 bytes apart, swizzling mode 6 at bit 61 (16-byte
// chunks swapped where address bit 7 is set; it follows the absolute address,
// so a start at any 32-byte row needs no base offset).  LBO is not used.
__device__ __forceinline__ uint64_t smem_desc_sw32(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
}
// An MN-major operand in the 64-byte swizzled layout: rows of 32 elements (64
// bytes), one per k, 8-row groups 512 bytes apart, 32-element groups along M or
// N `lbo` bytes apart; mode 4 (16-byte chunks XORed with address bits 7 and 8,
// again of the absolute address).
__device__ __forceinline__ uint64_t smem_desc_sw64_mn(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) |
           (1ull << 46) | (4ull << 61);
}
// D (tensor memory) = A B (+ D when `accumulate`), kind::f16, one CTA.
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate));
}
// The same issued by a whole converged warp, executed by its elected lane:
// the descriptors stay in uniform registers, where a divergent single thread
// moves all of them there again for every MMA (~105 cycles per MMA issued,
// ~70 from a converged warp).
__device__ __forceinline__ void mma_f16_warp(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p, e;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate));
}
__device__ __forceinline__ void mma_commit_warp(unsigned long long* bar) {
    asm volatile(
        "{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_addr(bar))
        : "memory");
}
// mbar_wait by every lane of a converged warp, one answer for all.
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long* bar, uint32_t parity, volatile int* abort) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort));
}
// Arrives on `bar` once every tcgen05 operation this thread issued so far completes.
__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// Tensor-memory allocation of `cols` columns (a power of two >= 32) by one
// whole warp; the address lands in *base.
__device__ __forceinline__ void tmem_alloc(uint32_t* base, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(base)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(cols));
}

// tcgen05.ld of 16 columns without the wait; wait_ld then waits for every
// load in flight and ties these registers to the wait, so that no use of
// them can be scheduled before it.
__device__ __forceinline__ void ld_x16_async(uint32_t taddr, uint32_t (&u)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
          "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(taddr));
}
__device__ __forceinline__ void wait_ld(uint32_t (&u)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]),
                   "+r"(u[8]), "+r"(u[9]), "+r"(u[10]), "+r"(u[11]), "+r"(u[12]), "+r"(u[13]), "+r"(u[14]), "+r"(u[15])
                 :
                 : "memory");
}

__device__ __forceinline__ void ld_x8_async(uint32_t taddr, uint32_t (&u)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(taddr));
}
// Waits for every load in flight; ties four sets of eight registers to it.
__device__ __forceinline__ void wait_ld8(uint32_t (&a)[8], uint32_t (&b)[8], uint32_t (&c)[8], uint32_t (&d)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7])
                 :
                 : "memory");
    asm volatile(""
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7]),
                   "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7])
                 :
                 : "memory");
}

}  // namespace tcg
}  // namespace fg
