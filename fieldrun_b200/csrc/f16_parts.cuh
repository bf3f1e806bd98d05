// Float32 operands for the tensor cores (tcgen05, kind f16) as two float16 parts each, hi = float16(v) and lo = float16(2^11 (v - hi)), of
// entries that a power of two has brought below 2^15: 22 bits of every entry down to 2^-14.
#pragma once

#include <cuda_fp16.h>

#include "attention_tc.cuh"

using namespace frb_at;

__device__ __forceinline__ uint32_t half2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }

// The parts of four entries times their row's scale; lo is 2^11 times what hi leaves, so that it is no smaller than hi.
#define PART_LO 2048.f
__device__ __forceinline__ void split_two(uint64_t v, uint32_t& hi, uint32_t& lo) {
    float a, b;
    halves_of(v, a, b);
    const __half2 h = __floats2half2_rn(a, b);
    hi = half2_bits(h);
    // 2^11 v - 2^11 hi: both exact, and so is what is left
    halves_of(mul_pairs(v, pair_of(PART_LO, PART_LO)), a, b);
    asm("{\n\t.reg .f16 l, h, m;\n\tmov.b32 {l, h}, %2;\n\tmov.b16 m, 0xE800;\n\t"
        "fma.rn.f32.f16 %0, l, m, %0;\n\tfma.rn.f32.f16 %1, h, m, %1;\n\t}" : "+f"(a), "+f"(b) : "r"(hi));
    lo = half2_bits(__floats2half2_rn(a, b));
}

__device__ __forceinline__ void split_four(float4 v, float scale, uint32_t& hi0, uint32_t& hi1, uint32_t& lo0, uint32_t& lo1) {
    const uint64_t s = pair_of(scale, scale);
    split_two(mul_pairs(pair_of(v.x, v.y), s), hi0, lo0);
    split_two(mul_pairs(pair_of(v.z, v.w), s), hi1, lo1);
}

// `sums` = the products of an operand in tensor memory (its parts at a_hi and a_lo) with one in shared memory, KSTEPS runs of sixteen
// entries; b_at(k): the place of run k from the second operand's start, in units of 16 bytes.  One lane.
template <int KSTEPS, typename At>
__device__ __forceinline__ void products_of_parts(uint32_t sums, uint32_t a_hi, uint32_t a_lo, uint64_t b_hi, uint64_t b_lo, uint32_t idesc, At b_at) {
#pragma unroll
    for (int k = 0; k < KSTEPS; ++k) frb_tc::mma_ts(sums, a_lo + 8 * k, b_hi + b_at(k), idesc, k != 0);
#pragma unroll
    for (int k = 0; k < KSTEPS; ++k) frb_tc::mma_ts(sums, a_hi + 8 * k, b_lo + b_at(k), idesc, 1);
    frb_tc::mma_ts_scaled<11>(sums, a_hi, b_hi, idesc);
#pragma unroll
    for (int k = 1; k < KSTEPS; ++k) frb_tc::mma_ts(sums, a_hi + 8 * k, b_hi + b_at(k), idesc, 1);
}
