// z / (1 + exp(-z)) of several z in float32.
#pragma once

#include "common.cuh"

// Below 80 the divisor and its reciprocal are far from the ends of float32: there an approximate reciprocal serves, and the quotient's
// residual, which fma() has exactly, corrects it (Markstein, IBM Journal of Research and Development 34, 1990).  That alone does not
// promise the division's bits; a test has them at a million z of each of nine sizes and both signs.  (The residual's sign is that way
// round so that minus zero stays what it is.)  A division's own branch lets no other work in between: with one for each z the state
// space's launch 3 was bound by these, at 196 us.
template <int N>
__device__ __forceinline__ void silu_of(float (&z)[N]) {
    float top = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) top = fmaxf(top, fabsf(z[i]));
    if (top < 80.f) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float d = 1.0f + expf(-z[i]);
            float r;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
            const float q = z[i] * r;
            z[i] = fmaf(-fmaf(q, d, -z[i]), r, q);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) z[i] = z[i] / (1.0f + expf(-z[i]));
    }
}
