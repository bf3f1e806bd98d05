// The state-space scan of scans.cu for prompts, in chunks of 128 tokens that run side by side.  Per head, with one decay a token
// and B, C shared by the heads of a group:
//
//     S <- a_t S + B_t (dt_t x_t)^T,   y_t = S^T C_t + D x_t,   a_t = exp(-exp(A_log) dt_t)          (S is [N, vdim])
//
// With w(j, i) the product of the decays of tokens j + 1 .. i of a chunk:
//   1. per chunk and group the products C_i . B_j of its pairs j <= i, for all heads of the group;
//   2. per chunk, 128 columns of the group's heads at a time: the chunk's own contribution U = sum_j B_j (w(j, end) dt_j x_j)^T;
//   3. along the chunks: the state at each chunk's start over U's place, and the sequence's new state;
//   4. per chunk and head: y_i = w(start, i) (S^T C_i) + sum_(j <= i) w(j, i) (C_i . B_j) (dt_j x_j), then D x and the gate.
// A weight is the exponential of a sum of logarithms that has its tokens' alone, or a product of such factors: never a quotient, and no
// difference of two sums either, which behind one strong decay would have lost the digits of the mild ones.  The sums run over up to 16
// tokens inside a block, 112 between blocks and 127 to the chunk's end: a rounding of their logarithms, which are large only where the
// weight is small.
//
// Everything is float32; the products run on tensor cores with each operand as two TF32 parts (tf32_parts.cuh), over inner sizes
// of at most 256 entries, added in float32 registers every 16 (launches 1 and 2: every 8).  Four prompts of 2,048 tokens, 64 heads of
// 128 x 64 in 8 groups: 0.68 ms (about 0.05 + 0.19 + 0.06 + 0.38 for the launches in turn; scans.cu token by token 1.21 ms).  What bounds
// them: launch 4 issues on half of the cycles, a third of its instructions the operands' parts, and keeps the tensor cores busy for
// 39 %.
#include "tf32_parts.cuh"

#define SC_TOKENS 128
#define SC_BLOCK 16
#define SC_BLOCKS (SC_TOKENS / SC_BLOCK)
#define SC_THREADS 256
#define SC_COLUMNS 128        // columns of U a block of launch 2 takes
#define SC_LC (64 + 8)        // rows of 64 entries of the inner size, read along
#define SC_SLICE 64           // value columns a block of launch 4 takes

struct StateSpaceChunks {
    const float* proj;       // [T, proj_stride]: z of channel j at z_offset + j, dt of head h at dt_offset + h
    const float* xbc;        // [T, xbc_stride]: x of head h at h * vdim, B of group g at b_offset + g * N, C at c_offset + g * N
    const float *dt_bias, *a_log, *d;            // [heads]
    const int *seq_slot, *seq_start, *cu_q_len, *chunk_seq, *chunk_begin, *chunk_end, *seq_chunk0;
    float* state;            // [slots][2][copy_floats], this part's [heads][N][vdim] at state_offset
    long long copy_floats, state_offset;
    float* out;              // [T, heads * vdim]
    float* states;           // [chunks][heads][N][vdim]
    float* decays;           // [chunks][heads]
    float* pairs;            // [chunks][groups][SC_TOKENS][SC_TOKENS]
    int proj_stride, z_offset, dt_offset, xbc_stride, b_offset, c_offset, heads, vdim, N, groups;
};

__device__ __forceinline__ float sc_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// `count` rows of WIDTH floats on their way into rows `ld` apart; zeros in the rows up to `most`.
template <int WIDTH>
__device__ __forceinline__ void sc_copy_rows(float* to, int ld, const float* from, int stride, int count, int most) {
#pragma unroll 4
    for (int i = threadIdx.x; i < most * (WIDTH / 4); i += SC_THREADS) {
        const int t = i / (WIDTH / 4), u = i % (WIDTH / 4);
        if (t < count) copy16_async(to + t * ld + 4 * u, from + (size_t)t * stride + 4 * u);
        else *(float4*)(to + t * ld + 4 * u) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Launch 1.  grid (chunk, group).  A warp takes row tiles a and 7 - a (the same number of earlier tokens for every a) and every
// other eight columns.
__global__ void __launch_bounds__(SC_THREADS, 2) state_space_pairs_kernel(StateSpaceChunks p) {
    extern __shared__ float4 sc_smem[];
    float* c_s = (float*)sc_smem;                   // [SC_TOKENS][SC_LC]
    float* b_s = c_s + SC_TOKENS * SC_LC;           // [SC_TOKENS][SC_LC]
    const int item = blockIdx.x, g = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item];
    const float* rows = p.xbc + ((size_t)p.cu_q_len[b] + p.chunk_begin[item]) * p.xbc_stride;
    const int tiles[2] = {warp & 3, 7 - (warp & 3)}, odd = warp >> 2;
    float acc[2][SC_BLOCKS][4] = {};
    for (int n0 = 0; n0 < p.N; n0 += 64) {
        __syncthreads();
        sc_copy_rows<64>(c_s, SC_LC, rows + p.c_offset + g * p.N + n0, p.xbc_stride, count, SC_TOKENS);
        sc_copy_rows<64>(b_s, SC_LC, rows + p.b_offset + g * p.N + n0, p.xbc_stride, count, SC_TOKENS);
        copies_commit();
        copies_wait<0>();
        __syncthreads();
#pragma unroll 2
        for (int k = 0; k < 64; k += 8) {
            Tf32Parts a[2][1][1][4], bb[1][1][2];
#pragma unroll
            for (int m = 0; m < 2; ++m) a_along(a[m][0][0], c_s + tiles[m] * SC_BLOCK * SC_LC + k, SC_LC, lane);
#pragma unroll
            for (int n = 0; n < SC_BLOCKS; ++n) {                        // n: the 16 columns of block n, this warp's half of them
                if (n > tiles[0] && n > tiles[1]) break;
                b_along(bb[0][0], b_s + (n * SC_BLOCK + 8 * odd) * SC_LC + k, SC_LC, lane);
#pragma unroll
                for (int m = 0; m < 2; ++m)
                    if (n <= tiles[m]) {
                        float t[1][1][4];
                        mma_runs(t, a[m], bb);
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[m][n][e] += t[0][0][e];
                    }
            }
        }
    }
    if (!all_finite(acc)) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < SC_BLOCKS; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = tiles[m] * SC_BLOCK + (lane >> 2) + 8 * (e >> 1), j = n * SC_BLOCK + 8 * odd + 2 * (lane & 3) + (e & 1);
                    if (j <= i && i < count && !is_finite(acc[m][n][e]))
                        acc[m][n][e] = sum_entry_by_entry(rows + (size_t)i * p.xbc_stride + p.c_offset + g * p.N, 1,
                                                          rows + (size_t)j * p.xbc_stride + p.b_offset + g * p.N, 1, nullptr, p.N);
                }
    }
    float* out = p.pairs + ((size_t)item * p.groups + g) * SC_TOKENS * SC_TOKENS;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < SC_BLOCKS; ++n)
            if (n <= tiles[m]) {
                float* to = out + (tiles[m] * SC_BLOCK + (lane >> 2)) * SC_TOKENS + n * SC_BLOCK + 8 * odd + 2 * (lane & 3);
                *(float2*)to = make_float2(acc[m][n][0], acc[m][n][1]);
                *(float2*)(to + 8 * SC_TOKENS) = make_float2(acc[m][n][2], acc[m][n][3]);
            }
}

// Launch 2.  grid (chunk, tile of 128 columns of the heads' values).  A warp takes 32 rows (64 with N = 64: two warps a row tile
// less) by 64 columns of U.
template <int N>
__global__ void __launch_bounds__(SC_THREADS, 2) state_space_states_kernel(StateSpaceChunks p) {
    constexpr int LB = N + 4, LX = SC_COLUMNS + 4, PART = 32;            // tokens of a part; two parts in turn
    extern __shared__ float4 sc_smem[];
    __shared__ float factor[2][SC_TOKENS], warp_sums[2][SC_TOKENS / 32];
    float* parts = (float*)sc_smem;                 // [2]: B [PART][LB], x [PART][LX]
    const int item = blockIdx.x, column0 = blockIdx.y * SC_COLUMNS, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item];
    const size_t row0 = (size_t)p.cu_q_len[b] + p.chunk_begin[item];
    const float* rows = p.xbc + row0 * p.xbc_stride;
    const int heads_here = p.vdim >= SC_COLUMNS ? 1 : 2, head0 = column0 / p.vdim, g = head0 / (p.heads / p.groups);

    auto copy_part = [&](int part) {
        float* b_s = parts + (part & 1) * PART * (LB + LX);
        const float* at = rows + (size_t)(part * PART) * p.xbc_stride;
        const int left = count - part * PART;
        sc_copy_rows<N>(b_s, LB, at + p.b_offset + g * N, p.xbc_stride, left, PART);
        sc_copy_rows<SC_COLUMNS>(b_s + PART * LB, LX, at + column0, p.xbc_stride, left, PART);
        copies_commit();
    };
    copy_part(0);

    // a thread a (head, token): the step times the decays behind it, to the chunk's end
    {
        const int hh = tid / SC_TOKENS, t = tid % SC_TOKENS, h = head0 + hh;
        const bool in = hh < heads_here && t < count;
        const float step = in ? sc_softplus(p.proj[(row0 + t) * p.proj_stride + p.dt_offset + h] + p.dt_bias[h]) : 0.f;
        const float la = in ? -expf(p.a_log[h]) * step : 0.f;
        float sum = la;                              // of this token and those behind it in the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float other = __shfl_down_sync(0xffffffffu, sum, o);
            if (lane + o < 32) sum += other;
        }
        float tail = __shfl_down_sync(0xffffffffu, sum, 1);
        if (lane == 31) tail = 0.f;
        if (lane == 0) warp_sums[hh][warp % (SC_TOKENS / 32)] = sum;
        __syncthreads();
        for (int w = t / 32 + 1; w < SC_TOKENS / 32; ++w) tail += warp_sums[hh][w];
        factor[hh][t] = step * expf(tail);
        if (t == 0 && hh < heads_here && column0 % p.vdim == 0) p.decays[(size_t)item * p.heads + h] = expf(la + tail);
    }

    constexpr int ROW_TILES = N / 32;                // 4 or 2 runs of 32 rows
    const int c0 = warp % ROW_TILES * 32, wide = SC_COLUMNS / (SC_THREADS / 32 / ROW_TILES), v0 = warp / ROW_TILES * wide;
    constexpr int NT = SC_COLUMNS / (SC_THREADS / 32 / ROW_TILES) / 8;
    float acc[2][NT][4] = {};
    for (int part = 0; part * PART < count; ++part) {
        const float* b_s = parts + (part & 1) * PART * (LB + LX);
        float* x_s = parts + (part & 1) * PART * (LB + LX) + PART * LB;
        copies_wait<0>();
        __syncthreads();                             // this part is there, and nobody reads the other one any more
        if ((part + 1) * PART < count) copy_part(part + 1);
#pragma unroll
        for (int i = tid; i < PART * SC_COLUMNS / 4; i += SC_THREADS) {
            const int t = i / (SC_COLUMNS / 4), u = i % (SC_COLUMNS / 4);
            const float f = factor[heads_here == 2 ? 4 * u / SC_SLICE : 0][part * PART + t];
            float4* at = (float4*)(x_s + t * LX + 4 * u);
            float4 x = *at;
            x.x *= f; x.y *= f; x.z *= f; x.w *= f;
            *at = x;
        }
        __syncthreads();
#pragma unroll 2
        for (int j = 0; j < PART; j += 8) {
            Tf32Parts a[1][2][4];
#pragma unroll
            for (int m = 0; m < 2; ++m) a_down(a[0][m], b_s + j * LB + c0 + 16 * m, LB, lane);
            add_runs<2>(acc, a, [&](Tf32Parts (&b)[2], int, int n) { b_down(b, x_s + j * LX + v0 + 8 * n, LX, lane); });
        }
    }
    if (!all_finite(acc)) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!is_finite(acc[m][n][e])) {
                        const int column = v0 + 8 * n + 2 * (lane & 3) + (e & 1);
                        acc[m][n][e] = sum_entry_by_entry(rows + p.b_offset + g * N + c0 + 16 * m + (lane >> 2) + 8 * (e >> 1), p.xbc_stride,
                                                          rows + column0 + column, p.xbc_stride, factor[heads_here == 2 ? column / SC_SLICE : 0],
                                                          count);
                    }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int column = column0 + v0 + 8 * n, h = column / p.vdim;
        float* out = p.states + ((size_t)item * p.heads + h) * N * p.vdim + column - h * p.vdim + 2 * (lane & 3);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            float* to = out + (size_t)(c0 + 16 * m + (lane >> 2)) * p.vdim;
            *(float2*)to = make_float2(acc[m][n][0], acc[m][n][1]);
            *(float2*)(to + 8 * (size_t)p.vdim) = make_float2(acc[m][n][2], acc[m][n][3]);
        }
    }
}

// Launch 3.  grid (sequence, head, runs of 1,024 state elements): bound by reading and writing U's place once.
__global__ void __launch_bounds__(256) state_space_chain_kernel(StateSpaceChunks p) {
    const int b = blockIdx.x, h = blockIdx.y, e = (blockIdx.z * 256 + threadIdx.x) * 4, elements = p.N * p.vdim;
    if (e >= elements) return;
    const int first = p.seq_chunk0[b], last = p.seq_chunk0[b + 1], start = p.seq_start[b], n = p.cu_q_len[b + 1] - p.cu_q_len[b];
    float* kept = p.state + (size_t)p.seq_slot[b] * 2 * p.copy_floats + p.state_offset + (size_t)h * elements + e;
    float4 S = *(const float4*)(kept + (start & 1) * p.copy_floats);
    for (int s0 = first; s0 < last; s0 += 8) {                  // eight chunks' loads on their way at once
        float4 u[8];
        float decay[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (s0 + i < last) {
                const size_t at = (size_t)(s0 + i) * p.heads + h;
                u[i] = *(const float4*)(p.states + at * elements + e);
                decay[i] = p.decays[at];
            }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (s0 + i < last) {
                *(float4*)(p.states + ((size_t)(s0 + i) * p.heads + h) * elements + e) = S;
                S.x = fmaf(decay[i], S.x, u[i].x);
                S.y = fmaf(decay[i], S.y, u[i].y);
                S.z = fmaf(decay[i], S.z, u[i].z);
                S.w = fmaf(decay[i], S.w, u[i].w);
            }
    }
    *(float4*)(kept + ((start + n) & 1) * p.copy_floats) = S;
}

// w(j, i) of a chunk's pairs.
struct ChunkWeights {
    float to[SC_TOKENS], from[SC_TOKENS], start[SC_TOKENS];              // from its block's start, to its block's end, from the chunk's start
    float between[SC_BLOCKS][SC_BLOCKS];                                 // the whole blocks between two
    __align__(16) float own[SC_TOKENS][SC_BLOCK + 8];                    // with the tokens of its block; zero for later ones

    __device__ __forceinline__ float of(int j, int i) const {
        const int bi = i / SC_BLOCK, bj = j / SC_BLOCK;
        return bj < bi ? to[i] * (between[bi][bj] * from[j]) : own[i][j % SC_BLOCK];
    }
};

// A token's output from the state at the chunk's start and the tokens up to it: sum_n C_n S_n w(start, i) + sum_(j <= i) w(j, i) pair_j x_j.
static __device__ __noinline__ float output_entry_by_entry(const ChunkWeights& w, int i, const float* c, const float* state, int vdim, int N,
                                                           const float* pairs, const float* x, int ld) {
    float sum = sum_entry_by_entry(c, 1, state, vdim, nullptr, N) * w.start[i];
    for (int j = 0; j <= i; ++j) sum = fmaf(pairs[j] * w.of(j, i), x[j * ld], sum);
    return sum;
}

// Launch 4.  grid (chunk, head, slice of 64 value columns).  A warp takes row tiles a and 7 - a by 32 columns.
__global__ void __launch_bounds__(SC_THREADS, 2) state_space_outputs_kernel(StateSpaceChunks p) {
    constexpr int LV = SC_SLICE + 4;
    extern __shared__ float4 sc_smem[];
    __shared__ float step_s[SC_TOKENS], log_s[SC_TOKENS], block_log[SC_BLOCKS];
    __shared__ ChunkWeights weights;
    constexpr int PART = 32, LP = PART + 8;         // state rows of a part; two parts in turn
    float* parts = (float*)sc_smem;                 // [2]: C [SC_TOKENS][LP], S [PART][LV]
    float* x_s = parts + 2 * (SC_TOKENS * LP + PART * LV);               // [SC_TOKENS][LV]
    const int item = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, column0 = blockIdx.z * SC_SLICE;
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item], g = h / (p.heads / p.groups);
    const size_t row0 = (size_t)p.cu_q_len[b] + p.chunk_begin[item];
    const float* rows = p.xbc + row0 * p.xbc_stride;
    const float* state = p.states + ((size_t)item * p.heads + h) * p.N * p.vdim + column0;
    auto copy_part = [&](int part) {
        float* c_s = parts + (part & 1) * (SC_TOKENS * LP + PART * LV);
        sc_copy_rows<PART>(c_s, LP, rows + p.c_offset + g * p.N + part * PART, p.xbc_stride, count, SC_TOKENS);
        sc_copy_rows<SC_SLICE>(c_s + SC_TOKENS * LP, LV, state + (size_t)(part * PART) * p.vdim, p.vdim, PART, PART);
        copies_commit();
    };
    copy_part(0);

    // a token a thread: its step; the logarithms of the decays from its block's start (with its own) and to its block's end
    if (tid < SC_TOKENS) {
        const bool in = tid < count;
        const float step = in ? sc_softplus(p.proj[(row0 + tid) * p.proj_stride + p.dt_offset + h] + p.dt_bias[h]) : 0.f;
        const float la = in ? -expf(p.a_log[h]) * step : 0.f;
        float before = la, behind = la;
#pragma unroll
        for (int o = 1; o < SC_BLOCK; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, before, o, SC_BLOCK), down = __shfl_down_sync(0xffffffffu, behind, o, SC_BLOCK);
            if (tid % SC_BLOCK >= o) before += up;
            if (tid % SC_BLOCK + o < SC_BLOCK) behind += down;
        }
        float tail = __shfl_down_sync(0xffffffffu, behind, 1, SC_BLOCK);
        if (tid % SC_BLOCK == SC_BLOCK - 1) { tail = 0.f; block_log[tid / SC_BLOCK] = before; }
        step_s[tid] = step;
        log_s[tid] = la;
        weights.to[tid] = expf(before);
        weights.from[tid] = expf(tail);
    }
    __syncthreads();
    if (tid < SC_TOKENS) {                           // a token's weights in its block: the sums begin anew for each, at the token itself
        const int i = tid % SC_BLOCK;
        float sum = 0.f, row[SC_BLOCK];
#pragma unroll
        for (int j = SC_BLOCK - 1; j >= 0; --j) {
            row[j] = j <= i ? expf(sum) : 0.f;
            if (j <= i) sum += log_s[tid - i + j];
        }
#pragma unroll
        for (int j = 0; j < SC_BLOCK; j += 4) *(float4*)&weights.own[tid][j] = make_float4(row[j], row[j + 1], row[j + 2], row[j + 3]);
    } else {
        const int t = tid - SC_TOKENS;
        float sum = 0.f;
        for (int m = 0; m < t / SC_BLOCK; ++m) sum += block_log[m];
        weights.start[t] = expf(sum) * weights.to[t];
        if (t < SC_BLOCKS * SC_BLOCKS) {
            const int i = t / SC_BLOCKS, j = t % SC_BLOCKS;
            sum = 0.f;
            for (int m = j + 1; m < i; ++m) sum += block_log[m];
            weights.between[i][j] = expf(sum);
        }
    }

    const int tiles[2] = {warp & 3, 7 - (warp & 3)}, v0 = (warp >> 2) * 32;
    float acc[2][4][4] = {};
    const int last = p.N / PART - 1;
    for (int part = 0; part <= last; ++part) {
        copies_wait<0>();
        __syncthreads();                             // this part is there, and nobody reads the other one any more
        if (part < last) {
            copy_part(part + 1);
        } else {                                     // behind the last part: the values
            sc_copy_rows<SC_SLICE>(x_s, LV, rows + h * p.vdim + column0, p.xbc_stride, count, SC_TOKENS);
            copies_commit();
        }
        const float* c_s = parts + (part & 1) * (SC_TOKENS * LP + PART * LV);
        const float* s_s = c_s + SC_TOKENS * LP;
#pragma unroll 1
        for (int k = 0; k < PART; k += 16) {
            Tf32Parts a[2][2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int m = 0; m < 2; ++m) a_along(a[r][m], c_s + tiles[m] * SC_BLOCK * LP + k + 8 * r, LP, lane);
            add_runs<2>(acc, a, [&](Tf32Parts (&b)[2], int r, int n) { b_down(b, s_s + (k + 8 * r) * LV + v0 + 8 * n, LV, lane); });
        }
    }
    copies_wait<0>();
    __syncthreads();
    for (int i = tid; i < SC_TOKENS * SC_SLICE / 4; i += SC_THREADS) {
        const int t = i / (SC_SLICE / 4), u = i % (SC_SLICE / 4);
        const float f = step_s[t];
        float4* at = (float4*)(x_s + t * LV + 4 * u);
        float4 x = *at;
        x.x *= f; x.y *= f; x.z *= f; x.w *= f;
        *at = x;
    }
    __syncthreads();
    const float* pairs = p.pairs + ((size_t)item * p.groups + g) * SC_TOKENS * SC_TOKENS;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int bi = tiles[m], i0 = bi * SC_BLOCK + (lane >> 2), i1 = i0 + 8;
        const float e0 = weights.start[i0], e1 = weights.start[i1];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            acc[m][n][0] *= e0;
            acc[m][n][1] *= e0;
            acc[m][n][2] *= e1;
            acc[m][n][3] *= e1;
        }
        const float* at = pairs + i0 * SC_TOKENS + 2 * (lane & 3);
        const float f0 = weights.to[i0], f1 = weights.to[i1];
        const int end = (bi + 1) * SC_BLOCK;
        float2 x_next[2], y_next[2];                 // the pairs of a block's 16 columns, asked for a block ahead
#pragma unroll
        for (int q = 0; q < 2; ++q) { x_next[q] = *(const float2*)(at + 8 * q); y_next[q] = *(const float2*)(at + 8 * SC_TOKENS + 8 * q); }
        for (int block0 = 0; block0 < end; block0 += SC_BLOCK) {
          const float2 xs[2] = {x_next[0], x_next[1]}, ys[2] = {y_next[0], y_next[1]};
          if (block0 + SC_BLOCK < end)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                x_next[q] = *(const float2*)(at + block0 + SC_BLOCK + 8 * q);
                y_next[q] = *(const float2*)(at + 8 * SC_TOKENS + block0 + SC_BLOCK + 8 * q);
            }
          Tf32Parts a[2][1][4];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int j = block0 + 8 * q + 2 * (lane & 3), bj = block0 / SC_BLOCK;
            const float2 x = xs[q], y = ys[q];
            float x0, x1, y0, y1;
            if (bj < bi) {
                const float both = weights.between[bi][bj], u = both * weights.from[j], v = both * weights.from[j + 1];
                x0 = x.x * (f0 * u); x1 = x.y * (f0 * v); y0 = y.x * (f1 * u); y1 = y.y * (f1 * v);
            } else {
                const float2 wx = *(const float2*)&weights.own[i0][j - block0], wy = *(const float2*)&weights.own[i1][j - block0];
                x0 = j <= i0 ? x.x * wx.x : 0.f;
                x1 = j + 1 <= i0 ? x.y * wx.y : 0.f;
                y0 = j <= i1 ? y.x * wy.x : 0.f;
                y1 = j + 1 <= i1 ? y.y * wy.y : 0.f;
            }
            a[q][0][0] = tf32_parts(x0);
            a[q][0][1] = tf32_parts(y0);
            a[q][0][2] = tf32_parts(x1);
            a[q][0][3] = tf32_parts(y1);
          }
          add_runs<4>(reinterpret_cast<float (&)[1][4][4]>(acc[m]), a,
                                  [&](Tf32Parts (&b)[2], int q, int n) { b_down(b, x_s + (block0 + 8 * q) * LV + v0 + 8 * n, LV, lane); });
        }
    }
    // a token's output has the tokens up to it alone: where an infinity or a NaN of the block behind it came in with a weight of zero, the
    // output is added again
    if (!all_finite(acc)) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = tiles[m] * SC_BLOCK + 8 * (e >> 1) + (lane >> 2), v = v0 + 8 * n + 2 * (lane & 3) + (e & 1);
                    if (t < count && !is_finite(acc[m][n][e]))
                        acc[m][n][e] = output_entry_by_entry(weights, t, rows + (size_t)t * p.xbc_stride + p.c_offset + g * p.N, state + v, p.vdim,
                                                             p.N, pairs + t * SC_TOKENS, x_s + v, LV);
                }
    }
    const float dskip = p.d[h];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int t = tiles[m] * SC_BLOCK + 8 * half + (lane >> 2);
            if (t >= count) continue;
            const int v = h * p.vdim + column0 + v0 + 2 * (lane & 3);
            const float* x = rows + (size_t)t * p.xbc_stride + v;
            const float* z = p.proj + (row0 + t) * p.proj_stride + p.z_offset + v;
            float* out = p.out + (row0 + t) * ((size_t)p.heads * p.vdim) + v;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const float2 xv = *(const float2*)(x + 8 * n), zv = *(const float2*)(z + 8 * n);
                const float y0 = fmaf(dskip, xv.x, acc[m][n][2 * half]), y1 = fmaf(dskip, xv.y, acc[m][n][2 * half + 1]);
                *(float2*)(out + 8 * n) = make_float2(y0 * (zv.x / (1.0f + expf(-zv.x))), y1 * (zv.y / (1.0f + expf(-zv.y))));
            }
        }
}

// ----------------------------------------------------------------------------- host side

// Chunks of at most 128 tokens: chunk_seq/begin/end and, per sequence, its first chunk (one entry more at the end).  scratch:
// num_chunks * (heads * N * vdim + groups * 128 * 128 + heads) floats.
FRB_API int frb_state_space_chunks(const float* proj, int proj_stride, int z_offset, int dt_offset, const float* xbc, int xbc_stride,
                                   int b_offset, int c_offset, const float* dt_bias, const float* a_log, const float* d, const int* seq_slot,
                                   const int* seq_start, const int* cu_q_len, float* state, long long copy_floats, long long state_offset,
                                   float* out, int num_seqs, int heads, int vdim, int N, int groups, const int* chunk_seq,
                                   const int* chunk_begin, const int* chunk_end, const int* seq_chunk0, int num_chunks, float* scratch,
                                   cudaStream_t stream) {
    if (num_seqs == 0 || num_chunks == 0) return 0;
    FRB_CHECK_ARG((N == 64 || N == 128) && (vdim == 64 || vdim == 128) && groups >= 1 && heads % groups == 0 &&
                      heads / groups * vdim % SC_COLUMNS == 0 && heads <= 65535, "state-space chunks: %d heads of %d x %d in %d groups", heads, N,
                  vdim, groups);
    FRB_CHECK_ARG(((xbc_stride | b_offset | c_offset) & 3) == 0 && ((proj_stride | z_offset) & 1) == 0 && ((copy_floats | state_offset) & 3) == 0 &&
                      (((uintptr_t)xbc | (uintptr_t)state | (uintptr_t)scratch | (uintptr_t)out) & 15) == 0 && ((uintptr_t)proj & 7) == 0,
                  "state-space chunks: rows of %d entries are not in steps of 16 bytes", xbc_stride);
    StateSpaceChunks p;
    p.proj = proj; p.xbc = xbc; p.dt_bias = dt_bias; p.a_log = a_log; p.d = d; p.seq_slot = seq_slot; p.seq_start = seq_start;
    p.cu_q_len = cu_q_len; p.chunk_seq = chunk_seq; p.chunk_begin = chunk_begin; p.chunk_end = chunk_end; p.seq_chunk0 = seq_chunk0;
    p.state = state; p.copy_floats = copy_floats; p.state_offset = state_offset; p.out = out;
    p.states = scratch;
    p.pairs = scratch + (size_t)num_chunks * heads * N * vdim;
    p.decays = p.pairs + (size_t)num_chunks * groups * SC_TOKENS * SC_TOKENS;
    p.proj_stride = proj_stride; p.z_offset = z_offset; p.dt_offset = dt_offset; p.xbc_stride = xbc_stride; p.b_offset = b_offset;
    p.c_offset = c_offset; p.heads = heads; p.vdim = vdim; p.N = N; p.groups = groups;
    const size_t pairs_smem = 2 * SC_TOKENS * SC_LC * sizeof(float);
    const size_t states_smem = 2 * 32 * (N + 4 + SC_COLUMNS + 4) * sizeof(float);
    const size_t outputs_smem = (2 * (SC_TOKENS * (32 + 8) + 32 * (SC_SLICE + 4)) + SC_TOKENS * (SC_SLICE + 4)) * sizeof(float);
    cudaFuncSetAttribute(state_space_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pairs_smem);
    cudaFuncSetAttribute(state_space_outputs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)outputs_smem);
    state_space_pairs_kernel<<<dim3(num_chunks, groups), SC_THREADS, pairs_smem, stream>>>(p);
    const dim3 states_grid(num_chunks, heads * vdim / SC_COLUMNS);
    if (N == 128) {
        cudaFuncSetAttribute(state_space_states_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)states_smem);
        state_space_states_kernel<128><<<states_grid, SC_THREADS, states_smem, stream>>>(p);
    } else {
        cudaFuncSetAttribute(state_space_states_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)states_smem);
        state_space_states_kernel<64><<<states_grid, SC_THREADS, states_smem, stream>>>(p);
    }
    state_space_chain_kernel<<<dim3(num_seqs, heads, (N * vdim + 1023) / 1024), 256, 0, stream>>>(p);
    state_space_outputs_kernel<<<dim3(num_chunks, heads, vdim / SC_SLICE), SC_THREADS, outputs_smem, stream>>>(p);
    FRB_RETURN_LAUNCH("state_space_chunks");
}
