// Float32 products on mma.sync: each operand as two TF32 parts, hi = the entry rounded to TF32 and lo = what is left, of
// either sign.  hi hi + hi lo + lo hi keeps 22 bits of every product (with hi cut instead of rounded, lo lo, which is left out, would
// be four times as large and always of one sign).  The tensor cores' adder cuts off instead of rounding, which over a long sum costs
// more than the parts do: sums are kept short there and added in float32 registers, rounded.
#pragma once

#include "common.cuh"

struct Tf32Parts {
    uint32_t hi, lo;
};

// The tensor cores read the upper 19 bits of an operand.  Three full-rate instructions; with the conversion instruction (lo rounded as
// well) the chunks of gla_chunks.cu took 525 us instead of 492.  A NaN stays one in lo.
__device__ __forceinline__ Tf32Parts tf32_parts(float v) {
    Tf32Parts p;
    p.hi = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;                 // half of the last place that is kept, then cut
    p.lo = __float_as_uint(v - __uint_as_float(p.hi));
    return p;
}

// C (16 x 8) += A (16 x 8) B (8 x 8).  With g = lane / 4 and t = lane % 4: a[0] = A(g, t), a[1] = A(g + 8, t), a[2] = A(g, t + 4),
// a[3] = A(g + 8, t + 4), b[0] = B(t, g), b[1] = B(t + 4, g), c[0..1] = C(g, 2 t ..), c[2..3] = C(g + 8, 2 t ..).  The order of
// the inner index is the caller's: here entries 2 t and 2 t + 1 of a run of eight take the places t and t + 4.
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The products of M row tiles with NN column tiles, added on the tensor cores.  The three products of a tile's parts depend on one
// another through its accumulators: one part of all tiles after the other leaves every product M NN places to finish.
template <int M, int NN>
__device__ __forceinline__ void mma_tiles(float (&c)[M][NN][4], const Tf32Parts (&a)[M][4], const Tf32Parts (&b)[NN][2]) {
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int m = 0; m < M; ++m) mma_tf32(c[m][n], a[m][0].lo, a[m][1].lo, a[m][2].lo, a[m][3].lo, b[n][0].hi, b[n][1].hi);
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int m = 0; m < M; ++m) mma_tf32(c[m][n], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[n][0].lo, b[n][1].lo);
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int m = 0; m < M; ++m) mma_tf32(c[m][n], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[n][0].hi, b[n][1].hi);
}

// The same with the small products (hi lo and lo hi) in sums of their own: a third as many cuts of the large sums.
template <int M, int NN>
__device__ __forceinline__ void mma_tiles_apart(float (&large)[M][NN][4], float (&small)[M][NN][4], const Tf32Parts (&a)[M][4],
                                                const Tf32Parts (&b)[NN][2]) {
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int m = 0; m < M; ++m) mma_tf32(small[m][n], a[m][0].lo, a[m][1].lo, a[m][2].lo, a[m][3].lo, b[n][0].hi, b[n][1].hi);
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int m = 0; m < M; ++m) mma_tf32(large[m][n], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[n][0].hi, b[n][1].hi);
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int m = 0; m < M; ++m) mma_tf32(small[m][n], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[n][0].lo, b[n][1].lo);
}

// The products of RUNS runs of eight entries from zero, the small ones of all runs before the large ones: RUNS cuts of the large sum.
template <int M, int NN, int RUNS>
__device__ __forceinline__ void mma_runs(float (&t)[M][NN][4], const Tf32Parts (&a)[RUNS][M][4], const Tf32Parts (&b)[RUNS][NN][2]) {
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int n = 0; n < NN; ++n) t[m][n][0] = t[m][n][1] = t[m][n][2] = t[m][n][3] = 0.f;
#pragma unroll
    for (int r = 0; r < RUNS; ++r) {
#pragma unroll
        for (int n = 0; n < NN; ++n)
#pragma unroll
            for (int m = 0; m < M; ++m) mma_tf32(t[m][n], a[r][m][0].lo, a[r][m][1].lo, a[r][m][2].lo, a[r][m][3].lo, b[r][n][0].hi, b[r][n][1].hi);
#pragma unroll
        for (int n = 0; n < NN; ++n)
#pragma unroll
            for (int m = 0; m < M; ++m) mma_tf32(t[m][n], a[r][m][0].hi, a[r][m][1].hi, a[r][m][2].hi, a[r][m][3].hi, b[r][n][0].lo, b[r][n][1].lo);
    }
#pragma unroll
    for (int r = 0; r < RUNS; ++r)
#pragma unroll
        for (int n = 0; n < NN; ++n)
#pragma unroll
            for (int m = 0; m < M; ++m) mma_tf32(t[m][n], a[r][m][0].hi, a[r][m][1].hi, a[r][m][2].hi, a[r][m][3].hi, b[r][n][0].hi, b[r][n][1].hi);
}

// C += A B over RUNS runs of eight entries, NP of the NN column tiles at a time (for their registers' sake), every 8 RUNS entries' sum added
// in float32 registers; load_b(b, r, n) brings tile n's operands of run r.  Four prompts of 2,048 tokens, error against 64-bit sums of the
// outputs and time, all sums on the tensor cores | this way | token by token: state_space_chunks 8.1e-7, 643 us | 1.4e-7, 680 | 1.3e-7,
// delta_chunks 4.2e-7, 579 | 1.9e-7, 590 | 1.4e-7, gla_chunks 7.2e-7, 486 | 3.8e-7, 497 | 9.9e-7.
template <int NP, int M, int NN, int RUNS, typename LoadB>
__device__ __forceinline__ void add_runs(float (&c)[M][NN][4], const Tf32Parts (&a)[RUNS][M][4], LoadB load_b) {
#pragma unroll
    for (int n = 0; n < NN; n += NP) {
        Tf32Parts b[RUNS][NP][2];
#pragma unroll
        for (int r = 0; r < RUNS; ++r)
#pragma unroll
            for (int i = 0; i < NP; ++i) load_b(b[r][i], r, n + i);
        float t[M][NP][4];
        mma_runs(t, a, b);
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int i = 0; i < NP; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[m][n + i][e] += t[m][i][e];
    }
}

// Operands from shared memory.  `at` is the address of the fragment's first entry; rows of the inner index lie along the row
// (stride = 8 modulo 32 floats: no bank conflicts) or down the column (stride = 4 modulo 16).
__device__ __forceinline__ void a_along(Tf32Parts (&a)[4], const float* at, int stride, int lane) {
    const float2 x = *(const float2*)(at + (lane >> 2) * stride + 2 * (lane & 3));
    const float2 y = *(const float2*)(at + ((lane >> 2) + 8) * stride + 2 * (lane & 3));
    a[0] = tf32_parts(x.x);
    a[1] = tf32_parts(y.x);
    a[2] = tf32_parts(x.y);
    a[3] = tf32_parts(y.y);
}
__device__ __forceinline__ void a_down(Tf32Parts (&a)[4], const float* at, int stride, int lane) {
    const float* x = at + 2 * (lane & 3) * stride + (lane >> 2);
    a[0] = tf32_parts(x[0]);
    a[1] = tf32_parts(x[8]);
    a[2] = tf32_parts(x[stride]);
    a[3] = tf32_parts(x[stride + 8]);
}
__device__ __forceinline__ void b_along(Tf32Parts (&b)[2], const float* at, int stride, int lane) {
    const float2 x = *(const float2*)(at + (lane >> 2) * stride + 2 * (lane & 3));
    b[0] = tf32_parts(x.x);
    b[1] = tf32_parts(x.y);
}
__device__ __forceinline__ void b_down(Tf32Parts (&b)[2], const float* at, int stride, int lane) {
    const float* x = at + 2 * (lane & 3) * stride + (lane >> 2);
    b[0] = tf32_parts(x[0]);
    b[1] = tf32_parts(x[stride]);
}

// An infinity has no parts: its lo is a NaN, and so is every product it meets; entries next to the largest float32 round to one.
// A caller looks at its finished sums and adds those that are not finite again, entry by entry from the operands themselves.
__device__ __forceinline__ bool is_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

template <int M, int NN>
__device__ __forceinline__ bool all_finite(const float (&c)[M][NN][4]) {
    float sum = 0.f;                                                     // becomes a NaN at the first that is not
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int n = 0; n < NN; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum = fmaf(c[m][n][e], 0.f, sum);
    return sum == 0.f;
}

// sum_k a[k] b[k] f[k] (without `f`: all one), the entries of a and b so far apart.
static __device__ __noinline__ float sum_entry_by_entry(const float* a, size_t a_stride, const float* b, size_t b_stride, const float* f, int count) {
    float sum = 0.f;
    for (int k = 0; k < count; ++k) sum = fmaf(f ? a[k * a_stride] * f[k] : a[k * a_stride], b[k * b_stride], sum);
    return sum;
}

__device__ __forceinline__ void copy16_async(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }
