// The fifth-generation tensor core: operand descriptors, MMA issue, completion, tensor-memory loads and stores.
//
// One warp of a block issues the MMAs, by one of its lanes (in latent_attention_tc.cu that lane runs the loop, elsewhere the warp); the accumulators (and, for `mma_ts`, the A operand) live in tensor
// memory, which one warp of the block allocates and frees.  Operands in shared memory are K-major tiles of
// rows of 128 bytes under the 128-byte swizzle that TMA writes (tma.cuh).
#pragma once

#include "tma.cuh"

namespace frb_tc {

using frb_tma::smem_addr;

// Shared-memory operand descriptor: start address in 16-byte units; leading byte offset 1 (not used by a
// swizzled K-major tile); groups of 8 rows 1024 bytes apart (stride byte offset); descriptor version 1 of
// this architecture; 128-byte swizzle.  16 further elements along K are 32 bytes: add 2 to the descriptor.
__device__ __forceinline__ uint64_t tile_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// Instruction descriptor: float32 accumulators, bfloat16 operands, both K-major, D = M x N.
__device__ __forceinline__ uint32_t instr_desc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem]^T
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

// D[tmem] = D 2^-SHIFT + A[tmem] * B[smem]^T (SHIFT up to 15)
template <int SHIFT>
__device__ __forceinline__ void mma_ts_scaled(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, %4;\n\t}"
        ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc), "n"(SHIFT) : "memory");
}

// True in one lane of a converged warp.  A loop that issues MMAs is run by a whole warp, and only the instructions themselves by this
// lane: their operands are then in uniform registers, where a loop of one lane would have to move each of them there every time.
__device__ __forceinline__ bool elect_one() {
    uint32_t mine;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(mine));
    return mine != 0;
}

// A wait of a whole warp: either all of its lanes go on or none.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* failed) {
    return __all_sync(0xffffffffu, frb_tma::bar_wait(bar, parity, failed));
}

// The waits of a warp for two barriers, both looked at before either is waited for.
__device__ __forceinline__ bool warp_wait_both(uint64_t* bar0, uint32_t parity0, uint64_t* bar1, uint32_t parity1, volatile int* failed) {
    const bool first = frb_tma::bar_try(smem_addr(bar0), parity0), second = frb_tma::bar_try(smem_addr(bar1), parity1);
    if (__all_sync(0xffffffffu, first && second)) return true;
    return warp_wait(bar0, parity0, failed) && warp_wait(bar1, parity1, failed);
}

// The barrier gets one arrival when every MMA that this thread has issued so far has finished.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// 16 columns of this warp's 32 lanes of tensor memory; the values are there after tmem_wait_ld().
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One warp of the block allocates `columns` (a power of two, at least 32) of tensor memory and leaves their
// address in *slot (shared memory); the same warp frees them before the block ends.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(columns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_free(uint32_t address, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

}  // namespace frb_tc
