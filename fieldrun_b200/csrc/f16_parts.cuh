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

__device__ __forceinline__ float power_of_two(int exponent) { return __uint_as_float((uint32_t)(exponent + 127) << 23); }

__device__ __forceinline__ void copy_bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(frb_tma::smem_addr(dst)), "l"(src), "r"(bytes), "r"(frb_tma::smem_addr(bar)) : "memory");
}

// The place of entry `c` of row `r` in pieces [64 rows][64 entries] of rows of 128 bytes, 128-byte swizzle, in float16 entries.
__device__ __forceinline__ int piece_place(int r, int c) { return (c >> 6) * (64 * 64) + r * 64 + (((c >> 3 & 7) ^ (r & 7)) << 3) + (c & 7); }

// An N-major operand of such pieces, the rows along the inner size: a run of sixteen of it is 128 on in units of 16 bytes.
__device__ __forceinline__ uint64_t desc_n_major(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(64 * 128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// N entries of a lane times its scale, as parts, to N / 2 columns of tensor memory each.
template <int N>
__device__ __forceinline__ void store_parts(const float (&x)[N], float scale, uint32_t to_hi, uint32_t to_lo) {
    static_assert(N % 32 == 0, "entries of a store");
#pragma unroll
    for (int n = 0; n < N; n += 32) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) split_two(mul_pairs(pair_of(x[n + 2 * i], x[n + 2 * i + 1]), pair_of(scale, scale)), hi[i], lo[i]);
        frb_tc::tmem_st16(to_hi + n / 2, hi);
        frb_tc::tmem_st16(to_lo + n / 2, lo);
    }
}

// N columns of tensor memory, there after tmem_wait_ld().
template <int N>
__device__ __forceinline__ void load_columns(uint32_t from, uint32_t (&v)[N / 16][16]) {
#pragma unroll
    for (int i = 0; i < N / 16; ++i) frb_tc::tmem_ld16(from + 16 * i, v[i]);
}

// The exponent of the power of two that brings `top` to [2^14, 2^15); of a smaller one than 2^-100 as if it were that, of a NaN too.
__device__ __forceinline__ int parts_exponent(float top) {
    return 14 + 127 - (int)(__float_as_uint(fminf(fmaxf(top, 7.888609052210118e-31f), 3.402823466e38f)) >> 23);
}

// Parts of one scale hold the digits of entries down to 2^-29 of the largest; smaller ones are off by up to 2^-51 of it, and with them the
// sums that they alone make.  Whether that counts is seen at the sums: in units of the scales, products of parts below 2^15 whose errors
// are up to 2^-21 each.  A warp's row of 32 sums with one of PARTS_LEAST units or more is off by 2^-31 of it a product, at most 2^-24 with 128.
#define PARTS_LEAST 1024.f

__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The unit of the warp's columns: the largest of what takes their scales off, a column of zeros aside.
__device__ __forceinline__ float warp_unit(float top, int exponent) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, top > 0.f ? __float_as_uint(power_of_two(-exponent)) : 0u));
}

// The first of the warp's rows with an entry that is not zero; N: none.
template <int N>
__device__ __forceinline__ int first_row(const float (&u)[N]) {
    if (__any_sync(0xffffffffu, u[0] != 0.f)) return 0;
    int first = N;
#pragma unroll
    for (int t = N - 1; t > 0; --t)
        if (__any_sync(0xffffffffu, u[t] != 0.f)) first = t;
    return first;
}
