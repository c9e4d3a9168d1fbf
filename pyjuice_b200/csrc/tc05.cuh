// tcgen05 helpers shared by the tensor-memory kernels: shared-memory operand descriptors
// (no swizzle, K-major canonical layout: 8-row x 16-byte core matrices), the instruction
// descriptor of kind::f16 with BF16 operands and FP32 accumulation, mbarriers with bounded
// waits, tensor-memory allocation and loads.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace pcb {
namespace tc05 {

constexpr int kSpinLimit = 1 << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle (descriptor version 1): lbo = bytes between
// core matrices adjacent along K, sbo = bytes between 8-row groups.
__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

// Instruction descriptor: D f32, A and B bf16, both K-major, M = 128, N.
template <int N>
__device__ __forceinline__ constexpr uint32_t idesc_kk() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* m, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(m)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* m, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(m)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase of the given parity to complete, at most kSpinLimit polls.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* m, uint32_t parity) {
    for (int i = 0; i < kSpinLimit; ++i)
        if (mbar_try_wait(m, parity)) return true;
    return false;
}

// Bytes that the barrier's current phase still waits for (and the one arrival)
__device__ __forceinline__ void mbar_expect_tx(uint64_t* m, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
}

// Untiled bulk copy of this GPU's memory to shared memory (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(mbar))
        : "memory");
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// An allocation waits, without a limit, until the SM has so many of its 512 columns free. So no CTA
// that holds columns may wait for one that could be kept from allocating:
// * A CTA that is started early must not hold columns that a CTA of the grid before it still
//   wants. So the kernels allocate after their wait for that grid (pdl_wait), all but
//   lse_tmem_kernel, whose launches lose 1 to 2 us by it when two of its CTAs start on an SM. It has 256
//   columns and at least 77 KB of shared memory, of which an SM has 228 (a CTA takes 1 KB more than
//   it asks for): two beside nothing else that allocates, or one beside one of lse_tc05.cu's kernels
//   (at least 80 KB, up to 128 columns) or of sum_pflows_tc05.cu's (102 KB, up to 128). The persistent
//   form (512 columns) asks for 152 KB, so never beside it; sum_pflows_lanes_kernel (up to 256 columns,
//   two beside it) lets its successor start only after it has allocated.
// * The CTAs of a cluster wait for one another with their columns held: those of lse_tmem_kernel
//   and sum_pflows_tc05_kernel, which fit together as above.
// (All early, with every successor held back behind the allocation: 0.5 to 2 us a launch. Shared
// memory that keeps any CTAs of more than 512 columns apart: takes the L1 that the parameter flows
// need, 291 -> 331 us for 200 regions of 256 x 256.)
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}

// 16 consecutive FP32 columns of this thread's accumulator row (warp w reads lanes
// 32 (w % 4) .. + 31).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// generic-proxy writes to shared memory visible to the tensor cores (async proxy)
__device__ __forceinline__ void fence_smem_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

}  // namespace tc05
}  // namespace pcb
