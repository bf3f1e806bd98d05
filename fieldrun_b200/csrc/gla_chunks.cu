// Gated linear attention for prompts in chunks of 64 tokens that run side by side: the recurrence of gla.cu,
//
//     S_t = diag(alpha_t) S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t,   alpha_t = exp(log sigmoid(A2 a1_t + b) / tau),
//
// written as matrix products.  With w(j, i) the product of the decays of tokens j + 1 .. i of a chunk (channel by channel):
//   1. each chunk alone: alpha, and the chunk's own contribution U = sum_j (w(j, end) k_j) v_j^T with the product D of its decays;
//   2. along the chunks: the state at each chunk's start, S <- D S + U, over U's place, and the sequence's new state;
//   3. each chunk: o_i = (w(start, i) q_i) S + sum_(j <= i) (sum_c q_ic w_c(j, i) k_jc) v_j, then the head's norm and gate.
// A weight w is never split into a quotient of two products (which leave float32 where decays are strong): a chunk is four blocks
// of 16 tokens; between two blocks w(j, i) = w(j, end of j's block) * (whole blocks between) * w(start of i's block, i), factors of
// at most one each; within a block the 136 pairs run as the recurrence does, w k_j multiplied by one decay after the other.
//
// Everything is float32; the products run on tensor cores with each operand as two TF32 parts (tf32_parts.cuh), over inner
// sizes of at most 192 entries, added in float32 registers every 16.  Four prompts of 2,048 tokens, 16 heads of 128 x 128: 0.48 ms
// (181 + 42 + 254 us for the launches in turn; with the rank's products one token at a time and a division's own branch in each gate 191
// and 262; gla.cu 1.66 ms in segments of 128, whose 500 instructions a warp and token run one after the other).  What bounds them: the
// instructions around the products (58 and 48 % of the issue slots; a decay's two exponentials and a logarithm, the parts, the block's own
// pairs), with two blocks an SM to hide the rows' way in; with q, k and v loaded where they are used 0.68 ms.
#include "pairs.cuh"
#include "silu.cuh"
#include "tf32_parts.cuh"

#define GC_TOKENS 64
#define GC_BLOCK 16
#define GC_THREADS 256
#define GC_LA1 (GC_TOKENS + 4)      // tokens of one of the rank's entries in shared memory

struct GlaChunks {
    const float* proj;       // [T, P]: q | k | v | g | a1 at the offsets below
    const void* a2;          // [heads * dim, rank], WT
    const float* a2_bias;    // [heads * dim]
    const float* norm_w;     // [vdim]
    float* state;            // [slots, 2, heads, dim, vdim]
    const int *seq_slot, *seq_start, *cu_q_len;
    const int *chunk_seq, *chunk_begin, *chunk_end, *seq_chunk0;
    float* states;           // [chunks, heads, dim, vdim]: U, then the state at the chunk's start
    float* decays;           // [chunks, heads, dim]: D
    float* alpha;            // [T, heads * dim]
    void* out;               // [T, heads * vdim], OutT
    float inv_tau, q_scale, eps;
    int P, off_q, off_k, off_v, off_g, off_a, heads, rank;
};

// `count` rows of WIDTH floats, `from` and `stride` apart, on their way to `to` (rows `ld` apart); zeros in the rows up to 64.
template <int WIDTH>
__device__ __forceinline__ void gc_copy_rows(float* to, int ld, const float* from, int stride, int count) {
#pragma unroll 4
    for (int i = threadIdx.x; i < GC_TOKENS * WIDTH / 4; i += GC_THREADS) {
        const int t = i / (WIDTH / 4), u = i % (WIDTH / 4);
        if (t < count) copy16_async(to + t * ld + 4 * u, from + (size_t)t * stride + 4 * u);
        else *(float4*)(to + t * ld + 4 * u) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__device__ __forceinline__ float gc_log_sigmoid(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

// Launch 1.  grid (chunk, head).  A thread has one key channel and 64 DIM / 256 neighbouring tokens for what is made channel by
// channel; then the warps take tiles of 32 x 32 of U.
template <int DIM, int VDIM, typename WT>
__global__ void __launch_bounds__(GC_THREADS, 2) gla_chunk_states_kernel(GlaChunks p) {
    constexpr int GROUPS = GC_THREADS / DIM, TOKENS = GC_TOKENS / GROUPS, LK = DIM + 4, LV = VDIM + 4;
    extern __shared__ float4 gc_smem[];
    __shared__ float totals[GROUPS][DIM];
    const int rank = p.rank, la2 = rank + 4;
    float* k_s = (float*)gc_smem;                   // [GC_TOKENS][LK]
    float* v_s = k_s + GC_TOKENS * LK;              // [GC_TOKENS][LV]
    float* a1_s = v_s + GC_TOKENS * LV;             // [rank][GC_LA1]
    float* a2_s = a1_s + GC_LA1 * rank;             // [DIM][la2]
    const int item = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item];
    const size_t row0 = (size_t)p.cu_q_len[b] + p.chunk_begin[item];
    const float* rows = p.proj + row0 * p.P;

    const WT* a2 = (const WT*)p.a2 + (size_t)h * DIM * rank;
    for (int r = lane; r < rank; r += 32) {
        for (int t = warp; t < GC_TOKENS; t += GC_THREADS / 32) a1_s[r * GC_LA1 + t] = t < count ? rows[(size_t)t * p.P + p.off_a + r] : 0.f;
#pragma unroll 8
        for (int c = warp; c < DIM; c += GC_THREADS / 32) a2_s[c * la2 + r] = to_f32<WT>(a2[c * rank + r]);
    }
    gc_copy_rows<DIM>(k_s, LK, rows + p.off_k + h * DIM, p.P, count);
    gc_copy_rows<VDIM>(v_s, LV, rows + p.off_v + h * VDIM, p.P, count);
    copies_commit();
    __syncthreads();

    const int d = tid % DIM, group = tid / DIM, t0 = group * TOKENS;
    const float bias = p.a2_bias[h * DIM + d];
    float la[TOKENS], total = 0.f;
    float* alpha = p.alpha + (row0 * p.heads + h) * DIM + d;
#pragma unroll
    for (int tg = 0; tg < TOKENS; tg += 8) {
        // two tokens at a time (the same multiply-adds, half the instructions)
        uint64_t pairs[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pairs[i] = pair_of(bias, bias);
#pragma unroll 1
        for (int r = 0; r < rank; r += 4) {
            const float4 w = *(const float4*)(a2_s + d * la2 + r);
            const float each[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2* x = (const ulonglong2*)(a1_s + (r + q) * GC_LA1 + t0 + tg);
                const ulonglong2 x0 = x[0], x1 = x[1];
                const uint64_t ww = pair_of(each[q], each[q]);
                pairs[0] = fma_pairs(ww, x0.x, pairs[0]);
                pairs[1] = fma_pairs(ww, x0.y, pairs[1]);
                pairs[2] = fma_pairs(ww, x1.x, pairs[2]);
                pairs[3] = fma_pairs(ww, x1.y, pairs[3]);
            }
        }
        float z[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) halves_of(pairs[i], z[2 * i], z[2 * i + 1]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = t0 + tg + i;
            la[tg + i] = t < count ? gc_log_sigmoid(z[i]) * p.inv_tau : 0.f;
            if (t < count) alpha[(size_t)t * p.heads * DIM] = expf(la[tg + i]);
            total += la[tg + i];
        }
    }
    totals[group][d] = total;
    copies_wait<0>();
    __syncthreads();
    float tail = 0.f;                               // logarithm of the decays behind a token, to the chunk's end
#pragma unroll
    for (int g = GROUPS - 1; g > 0; --g) if (g > group) tail += totals[g][d];
    if (group == 0) p.decays[((size_t)item * p.heads + h) * DIM + d] = expf(total + tail);
#pragma unroll
    for (int i = TOKENS - 1; i >= 0; --i) {
        const int t = t0 + i;
        k_s[t * LK + d] *= expf(tail);
        tail += la[i];
    }
    __syncthreads();

    constexpr int TILES = (DIM / 32) * (VDIM / 32);
    float* out = p.states + ((size_t)item * p.heads + h) * DIM * VDIM;
    for (int tile = warp; tile < TILES; tile += GC_THREADS / 32) {
        const int c0 = tile / (VDIM / 32) * 32, v0 = tile % (VDIM / 32) * 32;
        float acc[2][4][4] = {};
#pragma unroll 1
        for (int j = 0; j < GC_TOKENS; j += 16) {
            Tf32Parts a[2][2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int m = 0; m < 2; ++m) a_down(a[r][m], k_s + (j + 8 * r) * LK + c0 + 16 * m, LK, lane);
            add_runs<2>(acc, a, [&](Tf32Parts (&b)[2], int r, int n) { b_down(b, v_s + (j + 8 * r) * LV + v0 + 8 * n, LV, lane); });
        }
        if (!all_finite(acc)) {
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (!is_finite(acc[m][n][e]))
                            acc[m][n][e] = sum_entry_by_entry(k_s + c0 + 16 * m + (lane >> 2) + 8 * (e >> 1), LK,
                                                              v_s + v0 + 8 * n + 2 * (lane & 3) + (e & 1), LV, nullptr, GC_TOKENS);
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                float* to = out + (size_t)(c0 + 16 * m + (lane >> 2)) * VDIM + v0 + 8 * n + 2 * (lane & 3);
                *(float2*)to = make_float2(acc[m][n][0], acc[m][n][1]);
                *(float2*)(to + 8 * VDIM) = make_float2(acc[m][n][2], acc[m][n][3]);
            }
    }
}

// Launch 2.  grid (sequence, head, runs of 1,024 state elements): bound by reading and writing U's place once.
__global__ void __launch_bounds__(256)
gla_chunk_scan_kernel(GlaChunks p, int dim, int vdim) {
    const int b = blockIdx.x, h = blockIdx.y, e = (blockIdx.z * 256 + threadIdx.x) * 4, elements = dim * vdim;
    if (e >= elements) return;
    const int d = e / vdim, first = p.seq_chunk0[b], last = p.seq_chunk0[b + 1];
    const int start = p.seq_start[b], n = p.cu_q_len[b + 1] - p.cu_q_len[b];
    float* kept = p.state + ((size_t)p.seq_slot[b] * 2 * p.heads + h) * elements + e;
    float4 S = *(const float4*)(kept + (size_t)(start & 1) * p.heads * elements);
    for (int s0 = first; s0 < last; s0 += 8) {                  // eight chunks' loads on their way at once
        float4 u[8];
        float decay[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (s0 + i < last) {
                const size_t at = (size_t)(s0 + i) * p.heads + h;
                u[i] = *(const float4*)(p.states + at * elements + e);
                decay[i] = p.decays[at * dim + d];
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
    *(float4*)(kept + (size_t)((start + n) & 1) * p.heads * elements) = S;
}

// Launch 3.  grid (chunk, head).  Shared memory is shared out in turn, so that two blocks fit an SM: the region of the keys
// later holds rows 64 .. of the state and then the matrix of the pairs' weights, the region of the values first rows 0 .. 63 of
// the state.
template <int DIM, int VDIM, typename OutT>
__global__ void __launch_bounds__(GC_THREADS, 2) gla_chunk_outputs_kernel(GlaChunks p) {
    constexpr int LQ = DIM + 8, LV = VDIM + 4, LA = GC_TOKENS + 8, BLOCKS = GC_TOKENS / GC_BLOCK;
    constexpr int SLABS = DIM / 32, SLAB = 32 * LV;
    extern __shared__ float4 gc_smem[];
    __shared__ float block_decay[BLOCKS][DIM], square_sums[VDIM / 32][GC_TOKENS];
    float* q_s = (float*)gc_smem;                                        // [GC_TOKENS][LQ]
    float* k_s = q_s + GC_TOKENS * LQ;                                   // [GC_TOKENS][LQ], [2][SLAB], [GC_TOKENS][LA]
    constexpr int KEYS = GC_TOKENS * LQ > 2 * SLAB ? GC_TOKENS * LQ : 2 * SLAB;
    float* v_s = k_s + KEYS;                                             // [2][SLAB], [GC_TOKENS][LV]
    const int item = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item];
    const size_t row0 = (size_t)p.cu_q_len[b] + p.chunk_begin[item];
    const float* rows = p.proj + row0 * p.P;
    const float* state = p.states + ((size_t)item * p.heads + h) * DIM * VDIM;
    auto copy_slab = [&](float* to, int slab) {
        for (int i = tid; i < 32 * VDIM / 4; i += GC_THREADS) {
            const int r = i / (VDIM / 4), u = i % (VDIM / 4);
            copy16_async(to + r * LV + 4 * u, state + (size_t)(32 * slab + r) * VDIM + 4 * u);
        }
    };
    gc_copy_rows<DIM>(q_s, LQ, rows + p.off_q + h * DIM, p.P, count);
    gc_copy_rows<DIM>(k_s, LQ, rows + p.off_k + h * DIM, p.P, count);
    copies_commit();
    copy_slab(v_s, 0);
    copy_slab(v_s + SLAB, 1);
    copies_commit();

    // A warp takes a block of 16 tokens and 64 channels, two a lane: queries and keys get their decays to the block's edges in
    // place, and the block's own pairs, whose sums over the channels end in `own`: own[j] of lane 2 i (and 2 i + 1) is the
    // weight of token j for token i.
    const int block = warp >> 1, side = warp & 1;
    float own[GC_BLOCK];
#pragma unroll
    for (int j = 0; j < GC_BLOCK; ++j) own[j] = 0.f;
    const int c = 64 * side + 2 * lane, t0 = block * GC_BLOCK;
    const float* alpha_at = p.alpha + ((row0 + t0) * p.heads + h) * DIM + c;
    float2 alpha[GC_BLOCK];
#pragma unroll
    for (int i = 0; i < GC_BLOCK; ++i)
        alpha[i] = 64 * side < DIM && t0 + i < count ? *(const float2*)(alpha_at + (size_t)i * p.heads * DIM) : make_float2(1.f, 1.f);
    copies_wait<1>();
    __syncthreads();
    if (64 * side < DIM) {
        float2 q[GC_BLOCK], w = make_float2(1.f, 1.f);
#pragma unroll
        for (int i = 0; i < GC_BLOCK; ++i) q[i] = *(const float2*)(q_s + (t0 + i) * LQ + c);
#pragma unroll
        for (int i = 0; i < GC_BLOCK; ++i) {
            q[i].x *= p.q_scale;
            q[i].y *= p.q_scale;
            w.x *= alpha[i].x;
            w.y *= alpha[i].y;
            *(float2*)(q_s + (t0 + i) * LQ + c) = make_float2(q[i].x * w.x, q[i].y * w.y);
        }
        *(float2*)&block_decay[block][c] = w;
        w = make_float2(1.f, 1.f);
#pragma unroll
        for (int j = GC_BLOCK - 1; j >= 0; --j) {
            const float2 k = *(const float2*)(k_s + (t0 + j) * LQ + c);
            *(float2*)(k_s + (t0 + j) * LQ + c) = make_float2(k.x * w.x, k.y * w.y);
            w.x *= alpha[j].x;
            w.y *= alpha[j].y;
            float pair[GC_BLOCK];
            float2 decayed = k;
#pragma unroll
            for (int i = 0; i < GC_BLOCK; ++i) {
                if (i < j) { pair[i] = 0.f; continue; }
                if (i > j) { decayed.x *= alpha[i].x; decayed.y *= alpha[i].y; }
                pair[i] = q[i].x * decayed.x + q[i].y * decayed.y;
            }
            // sixteen sums over 32 lanes: half of them to the lane across, four times, then the two lanes left
#pragma unroll
            for (int n = 8; n > 0; n >>= 1) {
                const bool upper = (lane & (2 * n)) != 0;
#pragma unroll
                for (int i = 0; i < n; ++i) {
                    const float keep = upper ? pair[i + n] : pair[i], send = upper ? pair[i] : pair[i + n];
                    pair[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
                }
            }
            own[j] = pair[0] + __shfl_xor_sync(0xffffffffu, pair[0], 1);
        }
    }
    __syncthreads();

    // pairs of different blocks, units of 16 x 8: (1, 0), (2, 0), (2, 1), (3, 0), (3, 1), (3, 2), two units each
    constexpr int UNITS = BLOCKS * (BLOCKS - 1);
    float across[2][4] = {};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int unit = warp + 8 * u;
        if (unit >= UNITS) break;
        const int pair = unit >> 1, bi = pair == 0 ? 1 : pair < 3 ? 2 : 3, bj = pair - bi * (bi - 1) / 2;
#pragma unroll 2
        for (int k0 = 0; k0 < DIM; k0 += 8) {
            float2 x = *(const float2*)(q_s + (bi * GC_BLOCK + (lane >> 2)) * LQ + k0 + 2 * (lane & 3));
            float2 y = *(const float2*)(q_s + (bi * GC_BLOCK + (lane >> 2) + 8) * LQ + k0 + 2 * (lane & 3));
            for (int m = bj + 1; m < bi; ++m) {                          // the whole blocks between
                const float2 w = *(const float2*)&block_decay[m][k0 + 2 * (lane & 3)];
                x.x *= w.x; x.y *= w.y; y.x *= w.x; y.y *= w.y;
            }
            const Tf32Parts a[1][1][4] = {{{tf32_parts(x.x), tf32_parts(y.x), tf32_parts(x.y), tf32_parts(y.y)}}};
            Tf32Parts bb[1][1][2];
            b_along(bb[0][0], k_s + (bj * GC_BLOCK + 8 * (unit & 1)) * LQ + k0, LQ, lane);
            float t[1][1][4];
            mma_runs(t, a, bb);
#pragma unroll
            for (int e = 0; e < 4; ++e) across[u][e] += t[0][0][e];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (!is_finite(across[u][e])) {
                const float* q = q_s + (bi * GC_BLOCK + (lane >> 2) + 8 * (e >> 1)) * LQ;
                const float* k = k_s + (bj * GC_BLOCK + 8 * (unit & 1) + 2 * (lane & 3) + (e & 1)) * LQ;
                float sum = 0.f;
#pragma unroll 1
                for (int c = 0; c < DIM; ++c) {
                    float x = q[c];
                    for (int m = bj + 1; m < bi; ++m) x *= block_decay[m][c];
                    sum = fmaf(x, k[c], sum);
                }
                across[u][e] = sum;
            }
        __syncwarp();
    }
    __syncthreads();                                                     // the keys are read
    if (SLABS > 2) copy_slab(k_s, 2);
    copies_commit();
    if (SLABS > 3) copy_slab(k_s + SLAB, 3);
    copies_commit();
    {                                                                    // queries: the decays from the chunk's start
        const int channel = tid % DIM;
        float w = block_decay[0][channel];
#pragma unroll
        for (int m = 1; m < BLOCKS; ++m) {
#pragma unroll
            for (int t = m * GC_BLOCK + tid / DIM; t < (m + 1) * GC_BLOCK; t += GC_THREADS / DIM) q_s[t * LQ + channel] *= w;
            w *= block_decay[m][channel];
        }
    }

    // a warp's outputs: row tiles {0, 3} or {1, 2} (each pair looks at the same number of earlier tokens) by 32 value columns
    constexpr int COLUMNS = VDIM / 32;
    const int v0 = warp % COLUMNS * 32, pick = warp / COLUMNS;           // VDIM 64: warps 4 .. 7 have nothing to do
    const bool works = pick < 2;
    const int tiles[2] = {pick == 0 ? 0 : 1, pick == 0 ? 3 : 2};
    float acc[2][4][4] = {};
    auto with_state = [&](const float* slab, int c0) {
        if (works)
#pragma unroll 1
            for (int k0 = 0; k0 < 32; k0 += 16) {
                Tf32Parts a[2][2][4];
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int m = 0; m < 2; ++m) a_along(a[r][m], q_s + tiles[m] * 16 * LQ + c0 + k0 + 8 * r, LQ, lane);
                add_runs<2>(acc, a, [&](Tf32Parts (&b)[2], int r, int n) { b_down(b, slab + (k0 + 8 * r) * LV + v0 + 8 * n, LV, lane); });
            }
    };
    copies_wait<2>();
    __syncthreads();
    with_state(v_s, 0);
    with_state(v_s + SLAB, 32);
    __syncthreads();
    gc_copy_rows<VDIM>(v_s, LV, rows + p.off_v + h * VDIM, p.P, count);
    copies_commit();
    if (SLABS > 2) {
        copies_wait<1>();
        __syncthreads();
        with_state(k_s, 64);
        with_state(k_s + SLAB, 96);
        __syncthreads();
    }
    float* a_s = k_s;                                                    // [GC_TOKENS][LA]
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int unit = warp + 8 * u;
        if (unit >= UNITS) break;
        const int pair = unit >> 1, bi = pair == 0 ? 1 : pair < 3 ? 2 : 3, bj = pair - bi * (bi - 1) / 2;
        float* to = a_s + (bi * GC_BLOCK + (lane >> 2)) * LA + bj * GC_BLOCK + 8 * (unit & 1) + 2 * (lane & 3);
        *(float2*)to = make_float2(across[u][0], across[u][1]);
        *(float2*)(to + 8 * LA) = make_float2(across[u][2], across[u][3]);
    }
    float* own_at = a_s + (block * GC_BLOCK + (lane >> 1)) * LA + block * GC_BLOCK;
    if (side == 0 && (lane & 1) == 0)
#pragma unroll
        for (int j = 0; j < GC_BLOCK; ++j) own_at[j] = own[j];
    __syncthreads();
    if (DIM > 64 && side == 1 && (lane & 1) == 0)
#pragma unroll
        for (int j = 0; j < GC_BLOCK; ++j) own_at[j] += own[j];
    copies_wait<0>();
    __syncthreads();
    if (works)
#pragma unroll
        for (int m = 0; m < 2; ++m)
            for (int j = 0; j < (tiles[m] + 1) * GC_BLOCK; j += 16) {
                Tf32Parts a[2][1][4];
#pragma unroll
                for (int r = 0; r < 2; ++r) a_along(a[r][0], a_s + tiles[m] * 16 * LA + j + 8 * r, LA, lane);
                add_runs<4>(reinterpret_cast<float (&)[1][4][4]>(acc[m]), a,
                                        [&](Tf32Parts (&b)[2], int r, int n) { b_down(b, v_s + (j + 8 * r) * LV + v0 + 8 * n, LV, lane); });
            }

    // a token's output has the tokens up to it alone: where an infinity or a NaN of the block behind it came in with a weight of zero, the
    // output is added again
    if (works && !all_finite(acc))
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!is_finite(acc[m][n][e])) {
                        const int t = tiles[m] * 16 + 8 * (e >> 1) + (lane >> 2), v = v0 + 8 * n + 2 * (lane & 3) + (e & 1);
                        acc[m][n][e] = sum_entry_by_entry(q_s + t * LQ, 1, state + v, VDIM, nullptr, DIM) +
                                       sum_entry_by_entry(a_s + t * LA, 1, v_s + v, LV, nullptr, t + 1);
                    }

    // the head's root mean square over the warps' columns, weight and gate
    if (works)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float ss = 0.f;
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    ss = fmaf(acc[m][n][2 * half], acc[m][n][2 * half], ss);
                    ss = fmaf(acc[m][n][2 * half + 1], acc[m][n][2 * half + 1], ss);
                }
                ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                ss += __shfl_xor_sync(0xffffffffu, ss, 2);
                if ((lane & 3) == 0) square_sums[v0 / 32][tiles[m] * 16 + 8 * half + (lane >> 2)] = ss;
            }
    __syncthreads();
    if (works)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = tiles[m] * 16 + 8 * half + (lane >> 2);
                if (t >= count) continue;
                float ss = 0.f;
#pragma unroll
                for (int w = 0; w < COLUMNS; ++w) ss += square_sums[w][t];
                const float rinv = 1.0f / sqrtf(ss / (float)VDIM + p.eps);
                const float* gate = rows + (size_t)t * p.P + p.off_g + h * VDIM;
                OutT* out = (OutT*)p.out + ((row0 + t) * p.heads + h) * VDIM;
                float gates[8];
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const float2 g = *(const float2*)(gate + v0 + 8 * n + 2 * (lane & 3));
                    gates[2 * n] = g.x;
                    gates[2 * n + 1] = g.y;
                }
                silu_of(gates);
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const int v = v0 + 8 * n + 2 * (lane & 3);
                    out[v] = from_f32<OutT>(acc[m][n][2 * half] * rinv * p.norm_w[v] * gates[2 * n]);
                    out[v + 1] = from_f32<OutT>(acc[m][n][2 * half + 1] * rinv * p.norm_w[v + 1] * gates[2 * n + 1]);
                }
            }
}

// ----------------------------------------------------------------------------- host side

// Chunks of at most 64 tokens: chunk_seq/begin/end and, per sequence, its first chunk (one entry more at the end).  scratch:
// num_chunks * heads * dim * (vdim + 1) + num_tokens * heads * dim floats.
FRB_API int frb_gla_chunks(const float* proj, int P, int off_q, int off_k, int off_v, int off_g, int off_a, const void* a2, int dtype,
                           const float* a2_bias, const float* norm_w, float* state, const int* seq_slot, const int* seq_start,
                           const int* cu_q_len, void* out, int num_seqs, int heads, int dim, int vdim, int rank, float tau, float q_scale,
                           float eps, const int* chunk_seq, const int* chunk_begin, const int* chunk_end, const int* seq_chunk0,
                           int num_chunks, float* scratch, cudaStream_t stream) {
    if (num_seqs == 0 || num_chunks == 0) return 0;
    FRB_CHECK_ARG((dim == 64 || dim == 128) && (vdim == 64 || vdim == 128), "gla chunks: %d x %d per head", dim, vdim);
    FRB_CHECK_ARG(rank >= 4 && rank <= 64 && rank % 4 == 0 && heads >= 1 && heads <= 65535 && tau > 0.f, "gla chunks: %d heads, rank %d", heads, rank);
    FRB_CHECK_ARG(((P | off_q | off_k | off_v | off_g | off_a) & 3) == 0 && ((uintptr_t)proj & 15) == 0 && ((uintptr_t)scratch & 15) == 0 &&
                      ((uintptr_t)state & 15) == 0, "gla chunks: rows of %d entries are not in steps of 16 bytes", P);
    GlaChunks p;
    p.proj = proj; p.a2 = a2; p.a2_bias = a2_bias; p.norm_w = norm_w; p.state = state; p.seq_slot = seq_slot; p.seq_start = seq_start;
    p.cu_q_len = cu_q_len; p.chunk_seq = chunk_seq; p.chunk_begin = chunk_begin; p.chunk_end = chunk_end; p.seq_chunk0 = seq_chunk0;
    const size_t per_chunk = (size_t)heads * dim * vdim;
    p.states = scratch;
    p.decays = scratch + num_chunks * per_chunk;
    p.alpha = p.decays + (size_t)num_chunks * heads * dim;
    p.out = out; p.inv_tau = 1.0f / tau; p.q_scale = q_scale; p.eps = eps; p.P = P;
    p.off_q = off_q; p.off_k = off_k; p.off_v = off_v; p.off_g = off_g; p.off_a = off_a; p.heads = heads; p.rank = rank;
#define FRB_GLA_CHUNKS(DIM, VDIM)                                                                                                    \
    do {                                                                                                                             \
        const size_t one = (size_t)(GC_TOKENS * (DIM + 4 + VDIM + 4) + GC_LA1 * rank + DIM * (rank + 4)) * sizeof(float);            \
        const size_t slabs = 2 * 32 * (VDIM + 4), rows_q = GC_TOKENS * (DIM + 8);                                                    \
        const size_t three = (rows_q + (rows_q > slabs ? rows_q : slabs) + slabs) * sizeof(float);                                   \
        cudaFuncSetAttribute(gla_chunk_states_kernel<DIM, VDIM, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)one);          \
        cudaFuncSetAttribute(gla_chunk_outputs_kernel<DIM, VDIM, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)three);       \
        gla_chunk_states_kernel<DIM, VDIM, T><<<dim3(num_chunks, heads), GC_THREADS, one, stream>>>(p);                              \
        gla_chunk_scan_kernel<<<dim3(num_seqs, heads, (dim * vdim + 1023) / 1024), 256, 0, stream>>>(p, dim, vdim);                  \
        gla_chunk_outputs_kernel<DIM, VDIM, T><<<dim3(num_chunks, heads), GC_THREADS, three, stream>>>(p);                           \
    } while (0)
    FRB_DISPATCH_DTYPE(dtype, T, {
        if (dim == 128 && vdim == 128) FRB_GLA_CHUNKS(128, 128);
        else if (dim == 128) FRB_GLA_CHUNKS(128, 64);
        else if (vdim == 128) FRB_GLA_CHUNKS(64, 128);
        else FRB_GLA_CHUNKS(64, 64);
    });
#undef FRB_GLA_CHUNKS
    FRB_RETURN_LAUNCH("gla_chunks");
}
