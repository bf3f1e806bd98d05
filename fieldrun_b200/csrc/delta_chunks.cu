// The gated delta rule of delta_rule.cu for prompts, in chunks of 64 tokens.  Per head (q and k unit vectors, q also times
// dim^(-1/2); beta and one decay g a token):
//
//     u_i = beta_i (v_i - g_i S_(i-1)^T k_i),   S_i = g_i S_(i-1) + k_i u_i^T,   o_i = S_i^T q_i.
//
// With S the state at a chunk's start and w(j, i) the product of the decays of its tokens j + 1 .. i (w(i): from the chunk's start):
//     (I + M) u = beta v - beta w k^T S,   M_ij = beta_i w(j, i) (k_i . k_j) for j < i,
//     o_i = w(i) S^T q_i + sum_(j <= i) w(j, i) (q_i . k_j) u_j,   S <- w(end) S + sum_j w(j, end) k_j u_j^T.
//   1. every chunk and head side by side: M and the pairs' weights for o; then (I + M) X = [beta w k | beta v] by substitution, a
//      thread a column, in float32: W and U' with u = U' - W S.  (The entries of (I + M)^(-1) are at most one: each is what is left
//      of a unit of v_j under steps that shorten, times beta k_i.)
//   2. along the chunks of a sequence, a block a (sequence, head, 64 value columns) that keeps the state in registers: u = U' - W S,
//      o, and the new state.
//   3. the head's root mean square, weight and gate.
// A weight is the exponential of a sum of logarithms that has its tokens' alone, or a product of such factors: never a quotient, and no
// difference of two sums either, which behind one strong decay would have lost the digits of the mild ones.  The sums run over up to 16
// tokens inside a block and up to 48 between blocks: a rounding of their logarithms, which are large only where the weight is small.
//
// Everything is float32; the products run on tensor cores with each operand as two TF32 parts (tf32_parts.cuh), over inner sizes of
// at most 128 entries, added in float32 registers every 16; so is a chunk's new state to the decayed old one.  Four prompts of 2,048
// tokens, 16 heads of 128 x 128 over 4 key heads: 0.59 ms (0.19 + 0.36 + 0.04 for the launches in turn; delta_rule.cu token by
// token 1.38 ms).  Launch 1 issues on 57 % of the cycles (with the values' loads each waited for in turn: 0.37 ms).  Launch 2 is bound
// by the tensor cores and by the barriers of its three phases: a chunk takes 11.7 us where its products alone take 5.
#include "tf32_parts.cuh"

#define DC_TOKENS 64
#define DC_BLOCK 16
#define DC_BLOCKS (DC_TOKENS / DC_BLOCK)
#define DC_SLICE 64           // value columns a block of launch 2 keeps
#define DC_LM (DC_TOKENS + 8)

struct DeltaChunks {
    const float* conv;       // [T, conv_stride]: q at q_off (kv_heads * dim), k at k_off, v at v_off (heads * vdim)
    const float* proj;       // [T, proj_stride]: beta's logit of head h at b_off + h, the decay's at a_off + h, the gate at g_off (heads * vdim)
    const float *a_log, *dt_bias, *norm;
    const int *seq_slot, *seq_start, *cu_q_len, *chunk_seq, *chunk_begin, *chunk_end, *seq_chunk0;
    float* state;            // [slots][2][copy_floats], this part's [heads][dim][vdim] at state_offset
    long long copy_floats, state_offset;
    void* out;               // [T, heads * vdim], OutT
    float* raw;              // [T, heads * vdim]: o before its norm
    float* w;                // [chunks][heads][DC_TOKENS][dim]
    float* u;                // [chunks][heads][DC_TOKENS][vdim]
    float* pairs;            // [chunks][heads][DC_TOKENS][DC_TOKENS]: the weights of o
    float* q_factor;         // [chunks][heads][DC_TOKENS]: w(i) and the query's norm
    float* k_factor;         // [chunks][heads][DC_TOKENS]: w(j, end) and the key's norm
    float* decays;           // [chunks][heads]: w(end)
    int conv_stride, q_off, k_off, v_off, proj_stride, b_off, a_off, g_off, heads, kv_heads;
    float eps;
};

__device__ __forceinline__ float dc_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// `count` rows of WIDTH floats on their way into rows `ld` apart; zeros in the rows up to 64.
template <int WIDTH, int THREADS>
__device__ __forceinline__ void dc_copy_rows(float* to, int ld, const float* from, int stride, int count) {
#pragma unroll 4
    for (int i = threadIdx.x; i < DC_TOKENS * (WIDTH / 4); i += THREADS) {
        const int t = i / (WIDTH / 4), u = i % (WIDTH / 4);
        if (t < count) copy16_async(to + t * ld + 4 * u, from + (size_t)t * stride + 4 * u);
        else *(float4*)(to + t * ld + 4 * u) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Launch 1.  grid (chunk, head).
template <int DIM, int VDIM>
__global__ void __launch_bounds__(256, 2) delta_chunk_solve_kernel(DeltaChunks p) {
    constexpr int LQ = DIM + 8, LS = DC_TOKENS + 4;
    extern __shared__ float4 dc_smem[];
    __shared__ float beta_s[DC_TOKENS], log_s[DC_TOKENS], to_s[DC_TOKENS], from_s[DC_TOKENS], start_s[DC_TOKENS], q_inv[DC_TOKENS], k_inv[DC_TOKENS];
    __shared__ float block_log[DC_BLOCKS], between[DC_BLOCKS][DC_BLOCKS];
    __shared__ __align__(16) float own[DC_TOKENS][DC_BLOCK + 4];         // w(j, i) of the tokens j of i's block; zero for later ones
    float* q_s = (float*)dc_smem;                   // [DC_TOKENS][LQ]
    float* k_s = q_s + DC_TOKENS * LQ;              // [DC_TOKENS][LQ]
    float* m_s = k_s + DC_TOKENS * LQ;              // [DC_TOKENS][LS]: M, column by column
    const int item = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item], kvh = h / (p.heads / p.kv_heads);
    const size_t row0 = (size_t)p.cu_q_len[b] + p.chunk_begin[item], at = (size_t)item * p.heads + h;
    const float* rows = p.conv + row0 * p.conv_stride;
    dc_copy_rows<DIM, 256>(q_s, LQ, rows + p.q_off + kvh * DIM, p.conv_stride, count);
    dc_copy_rows<DIM, 256>(k_s, LQ, rows + p.k_off + kvh * DIM, p.conv_stride, count);
    copies_commit();

    // a token a thread: beta; the logarithms of the decays from its block's start (with its own) and to its block's end
    if (tid < DC_TOKENS) {
        const float* logits = p.proj + (row0 + min(tid, count - 1)) * p.proj_stride + h;
        const bool in = tid < count;
        beta_s[tid] = in ? 1.0f / (1.0f + expf(-logits[p.b_off])) : 0.f;
        const float la = in ? -expf(p.a_log[h]) * dc_softplus(logits[p.a_off] + p.dt_bias[h]) : 0.f;
        float before = la, behind = la;
#pragma unroll
        for (int o = 1; o < DC_BLOCK; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, before, o, DC_BLOCK), down = __shfl_down_sync(0xffffffffu, behind, o, DC_BLOCK);
            if (tid % DC_BLOCK >= o) before += up;
            if (tid % DC_BLOCK + o < DC_BLOCK) behind += down;
        }
        float tail = __shfl_down_sync(0xffffffffu, behind, 1, DC_BLOCK);
        if (tid % DC_BLOCK == DC_BLOCK - 1) { tail = 0.f; block_log[tid / DC_BLOCK] = before; }
        log_s[tid] = la;
        to_s[tid] = expf(before);
        from_s[tid] = expf(tail);
    }
    copies_wait<0>();
    __syncthreads();
    for (int t = warp; t < DC_TOKENS; t += 8) {
        float qq = 0.f, kk = 0.f;
#pragma unroll
        for (int d = 0; d < DIM; d += 32) {
            const float x = q_s[t * LQ + d + lane], y = k_s[t * LQ + d + lane];
            qq = fmaf(x, x, qq);
            kk = fmaf(y, y, kk);
        }
        qq = warp_sum(qq);
        kk = warp_sum(kk);
        if (lane == 0) {
            q_inv[t] = 1.0f / sqrtf((float)DIM) / sqrtf(qq + 1e-6f);
            k_inv[t] = 1.0f / sqrtf(kk + 1e-6f);
        }
    }
    if (tid < DC_BLOCKS * DC_BLOCKS) {               // the whole blocks between two
        const int i = tid / DC_BLOCKS, j = tid % DC_BLOCKS;
        float sum = 0.f;
        for (int m = j + 1; m < i; ++m) sum += block_log[m];
        between[i][j] = expf(sum);
    } else if (tid >= 64 && tid < 64 + DC_TOKENS) {  // a token's weights in its block: the sums begin anew for each, at the token itself
        const int t = tid - 64, i = t % DC_BLOCK;
        float sum = 0.f, row[DC_BLOCK];
#pragma unroll
        for (int j = DC_BLOCK - 1; j >= 0; --j) {
            row[j] = j <= i ? expf(sum) : 0.f;
            if (j <= i) sum += log_s[t - i + j];
        }
#pragma unroll
        for (int j = 0; j < DC_BLOCK; j += 4) *(float4*)&own[t][j] = make_float4(row[j], row[j + 1], row[j + 2], row[j + 3]);
    } else if (tid >= 128 && tid < 128 + DC_TOKENS) {
        const int t = tid - 128;
        float sum = 0.f;
        for (int m = 0; m < t / DC_BLOCK; ++m) sum += block_log[m];
        start_s[t] = expf(sum) * to_s[t];
    }
    // the chunk's factors for launch 2: a token's decays to the chunk's end
    float rest = 0.f;
    if (tid < DC_TOKENS)
        for (int m = tid / DC_BLOCK + 1; m < DC_BLOCKS; ++m) rest += block_log[m];
    __syncthreads();
    if (tid < DC_TOKENS) {
        p.q_factor[at * DC_TOKENS + tid] = start_s[tid] * q_inv[tid];
        p.k_factor[at * DC_TOKENS + tid] = from_s[tid] * expf(rest) * k_inv[tid];
        if (tid == DC_TOKENS - 1) p.decays[at] = start_s[tid];
    }

    // warps 0 .. 3 the products of keys with keys, 4 .. 7 of queries with keys: row tiles a and 3 - a, every other eight columns
    const bool keys = warp < 4;
    const int tiles[2] = {warp & 1, 3 - (warp & 1)}, odd = warp >> 1 & 1;
    const float* left = keys ? k_s : q_s;
    float acc[2][DC_BLOCKS][4] = {};
#pragma unroll 1
    for (int c = 0; c < DIM; c += 16) {
        Tf32Parts a[2][2][1][4], bb[2][1][2];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r) a_along(a[m][r][0], left + tiles[m] * DC_BLOCK * LQ + c + 8 * r, LQ, lane);
#pragma unroll
        for (int n = 0; n < DC_BLOCKS; ++n) {
#pragma unroll
            for (int r = 0; r < 2; ++r) b_along(bb[r][0], k_s + (n * DC_BLOCK + 8 * odd) * LQ + c + 8 * r, LQ, lane);
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
    float* pairs = p.pairs + at * DC_TOKENS * DC_TOKENS;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < DC_BLOCKS; ++n)
            if (n <= tiles[m])
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = tiles[m] * DC_BLOCK + (lane >> 2) + 8 * (e >> 1), j = n * DC_BLOCK + 8 * odd + 2 * (lane & 3) + (e & 1);
                    const bool seen = keys ? j < i : j <= i;
                    const float w = n < tiles[m] ? to_s[i] * between[tiles[m]][n] * from_s[j] : own[i][j % DC_BLOCK];
                    if (seen && !is_finite(acc[m][n][e])) acc[m][n][e] = sum_entry_by_entry(left + i * LQ, 1, k_s + j * LQ, 1, nullptr, DIM);
                    const float value = seen ? acc[m][n][e] * w * k_inv[j] * (keys ? beta_s[i] * k_inv[i] : q_inv[i]) : 0.f;
                    if (keys) m_s[j * LS + i] = value;
                    else pairs[i * DC_TOKENS + j] = value;
                }
    __syncthreads();

    // substitution: a thread a column of [beta w k | beta v], its 64 entries in registers
    if (tid < DIM + VDIM) {
        const bool key = tid < DIM;
        const float* v = rows + p.v_off + h * VDIM + tid - DIM;
        float x[DC_TOKENS];
        if (key) {
#pragma unroll
            for (int i = 0; i < DC_TOKENS; ++i) x[i] = beta_s[i] * start_s[i] * k_inv[i] * k_s[i * LQ + tid];
        } else {                                     // all of the column's loads on their way before the first is used
#pragma unroll
            for (int i = 0; i < DC_TOKENS; ++i) x[i] = v[(size_t)min(i, count - 1) * p.conv_stride];
#pragma unroll
            for (int i = 0; i < DC_TOKENS; ++i) x[i] = i < count ? x[i] * beta_s[i] : 0.f;
        }
        float* to = key ? p.w + at * DC_TOKENS * DIM + tid : p.u + at * DC_TOKENS * VDIM + tid - DIM;
        const int width = key ? DIM : VDIM;
        // an entry once it is final leaves every later one: those do not depend on one another
#pragma unroll
        for (int i = 0; i < DC_TOKENS; ++i) {
            const float* m = m_s + i * LS;
            const float done = x[i];
            to[(size_t)i * width] = done;
#pragma unroll
            for (int j = (i + 1) & ~3; j < DC_TOKENS; j += 4) {
                const float4 w = *(const float4*)(m + j);
                if (j > i) x[j] = fmaf(-w.x, done, x[j]);
                if (j + 1 > i) x[j + 1] = fmaf(-w.y, done, x[j + 1]);
                if (j + 2 > i) x[j + 2] = fmaf(-w.z, done, x[j + 2]);
                if (j + 3 > i) x[j + 3] = fmaf(-w.w, done, x[j + 3]);
            }
        }
    }
}

// Launch 2.  grid (sequence, head, slice of 64 value columns), 16 warps.  W and the queries are free once u is there, the pairs' weights
// and the keys once the new state is: each time the next chunk's are asked for.
template <int DIM>
__global__ void __launch_bounds__(512, 1) delta_chunk_chain_kernel(DeltaChunks p, int vdim) {
    constexpr int THREADS = 512, LQ = DIM + 8, LK = DIM + 4, LV = DC_SLICE + 4, MT = DIM / 64;
    extern __shared__ float4 dc_smem[];
    __shared__ float q_factor[2][DC_TOKENS], k_factor[2][DC_TOKENS];
    float* w_s = (float*)dc_smem;                   // [DC_TOKENS][LQ]
    float* q_s = w_s + DC_TOKENS * LQ;              // [DC_TOKENS][LQ]
    float* k_s = q_s + DC_TOKENS * LQ;              // [DC_TOKENS][LK]
    float* a_s = k_s + DC_TOKENS * LK;              // [DC_TOKENS][DC_LM]
    float* s_s = a_s + DC_TOKENS * DC_LM;           // [DIM][LV]: the state at the chunk's start
    float* u_s = s_s + DIM * LV;                    // [DC_TOKENS][LV]
    const int b = blockIdx.x, h = blockIdx.y, column0 = blockIdx.z * DC_SLICE, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g8 = lane >> 2, t4 = lane & 3, kvh = h / (p.heads / p.kv_heads);
    const int first = p.seq_chunk0[b], last = p.seq_chunk0[b + 1], start = p.seq_start[b], n_tok = p.cu_q_len[b + 1] - p.cu_q_len[b];
    const size_t seq_row0 = p.cu_q_len[b];
    float* kept = p.state + (size_t)p.seq_slot[b] * 2 * p.copy_floats + p.state_offset + (size_t)h * DIM * vdim + column0;

    auto copy_first = [&](int item) {               // W, queries, their factors
        const int count = p.chunk_end[item] - p.chunk_begin[item];
        const size_t at = (size_t)item * p.heads + h;
        dc_copy_rows<DIM, THREADS>(w_s, LQ, p.w + at * DC_TOKENS * DIM, DIM, DC_TOKENS);
        dc_copy_rows<DIM, THREADS>(q_s, LQ, p.conv + (seq_row0 + p.chunk_begin[item]) * p.conv_stride + p.q_off + kvh * DIM, p.conv_stride, count);
        if (tid < DC_TOKENS / 4) copy16_async(q_factor[item & 1] + 4 * tid, p.q_factor + at * DC_TOKENS + 4 * tid);
        copies_commit();
    };
    auto copy_second = [&](int item) {              // the pairs' weights, keys, their factors
        const int count = p.chunk_end[item] - p.chunk_begin[item];
        const size_t at = (size_t)item * p.heads + h;
        dc_copy_rows<DC_TOKENS, THREADS>(a_s, DC_LM, p.pairs + at * DC_TOKENS * DC_TOKENS, DC_TOKENS, DC_TOKENS);
        dc_copy_rows<DIM, THREADS>(k_s, LK, p.conv + (seq_row0 + p.chunk_begin[item]) * p.conv_stride + p.k_off + kvh * DIM, p.conv_stride, count);
        if (tid < DC_TOKENS / 4) copy16_async(k_factor[item & 1] + 4 * tid, p.k_factor + at * DC_TOKENS + 4 * tid);
        copies_commit();
    };
    if (first < last) {
        copy_first(first);
        copy_second(first);
    }

    // the state: MT row tiles by two column tiles a warp
    const int c0 = (warp & 3) * 16 * MT, s0 = (warp >> 2) * 16;
    float S[MT][2][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int c = c0 + 16 * m + g8, v = s0 + 8 * n + 2 * t4;
            const float* from = kept + (start & 1) * p.copy_floats + (size_t)c * vdim + v;
            const float2 x = *(const float2*)from, y = *(const float2*)(from + 8 * (size_t)vdim);
            S[m][n][0] = x.x; S[m][n][1] = x.y; S[m][n][2] = y.x; S[m][n][3] = y.y;
            *(float2*)(s_s + c * LV + v) = x;
            *(float2*)(s_s + (c + 8) * LV + v) = y;
        }
    // phase 1: warps 0 .. 7 W S, warps 8 .. 15 q S, 16 rows by 32 columns each
    const int tile = warp & 3, v0 = (warp >> 2 & 1) * 32;
    const bool makes_u = warp < 8;
    for (int item = first; item < last; ++item) {
        const size_t at = (size_t)item * p.heads + h;
        float acc[1][4][4] = {}, ahead[4][4];
        if (makes_u) {
            const float* from = p.u + (at * DC_TOKENS + tile * 16 + g8) * vdim + column0 + v0 + 2 * t4;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const float2 x = *(const float2*)(from + 8 * n), y = *(const float2*)(from + 8 * (size_t)vdim + 8 * n);
                ahead[n][0] = x.x; ahead[n][1] = x.y; ahead[n][2] = y.x; ahead[n][3] = y.y;
            }
        }
        const float decay = p.decays[at];
        copies_wait<1>();
        __syncthreads();                             // W and q are there, and so is the state
        const float* left = (makes_u ? w_s : q_s) + tile * 16 * LQ;
#pragma unroll 2
        for (int c = 0; c < DIM; c += 16) {
            Tf32Parts a[2][1][4];
#pragma unroll
            for (int r = 0; r < 2; ++r) a_along(a[r][0], left + c + 8 * r, LQ, lane);
            add_runs<4>(acc, a, [&](Tf32Parts (&b)[2], int r, int n) { b_down(b, s_s + (c + 8 * r) * LV + v0 + 8 * n, LV, lane); });
        }
        if (!all_finite(acc)) {
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!is_finite(acc[0][n][e]))
                        acc[0][n][e] = sum_entry_by_entry(left + (g8 + 8 * (e >> 1)) * LQ, 1, s_s + v0 + 8 * n + 2 * t4 + (e & 1), LV, nullptr, DIM);
        }
        if (makes_u) {
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                float* to = u_s + (tile * 16 + g8) * LV + v0 + 8 * n + 2 * t4;
                *(float2*)to = make_float2(ahead[n][0] - acc[0][n][0], ahead[n][1] - acc[0][n][1]);
                *(float2*)(to + 8 * LV) = make_float2(ahead[n][2] - acc[0][n][2], ahead[n][3] - acc[0][n][3]);
            }
        } else {
            const float f0 = q_factor[item & 1][tile * 16 + g8], f1 = q_factor[item & 1][tile * 16 + g8 + 8];
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                acc[0][n][0] *= f0;
                acc[0][n][1] *= f0;
                acc[0][n][2] *= f1;
                acc[0][n][3] *= f1;
            }
        }
        copies_wait<0>();
        __syncthreads();                             // u, the pairs' weights and the keys are there; nobody reads W, q and the state any more
        if (item + 1 < last) copy_first(item + 1);
        if (!makes_u) {
            float with_pairs[1][4][4];
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) with_pairs[0][n][e] = acc[0][n][e];
            for (int j = 0; j < (tile + 1) * DC_BLOCK; j += 16) {
                Tf32Parts a[2][1][4];
#pragma unroll
                for (int r = 0; r < 2; ++r) a_along(a[r][0], a_s + tile * 16 * DC_LM + j + 8 * r, DC_LM, lane);
                add_runs<4>(with_pairs, a, [&](Tf32Parts (&b)[2], int r, int n) { b_down(b, u_s + (j + 8 * r) * LV + v0 + 8 * n, LV, lane); });
            }
            // a token's output has the tokens up to it alone: where an infinity or a NaN of the block behind it came in with a weight of
            // zero, the output is added again
            if (!all_finite(with_pairs)) {
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (!is_finite(with_pairs[0][n][e])) {
                            const int t = tile * 16 + g8 + 8 * (e >> 1);
                            with_pairs[0][n][e] = acc[0][n][e] + sum_entry_by_entry(a_s + t * DC_LM, 1, u_s + v0 + 8 * n + 2 * t4 + (e & 1), LV, nullptr, t + 1);
                        }
            }
            __syncwarp();
            const int begin = p.chunk_begin[item], count = p.chunk_end[item] - begin;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = tile * 16 + 8 * half + g8;
                if (t >= count) continue;
                float* to = p.raw + ((seq_row0 + begin + t) * p.heads + h) * vdim + column0 + v0 + 2 * t4;
#pragma unroll
                for (int n = 0; n < 4; ++n) *(float2*)(to + 8 * n) = make_float2(with_pairs[0][n][2 * half], with_pairs[0][n][2 * half + 1]);
            }
        }
        float fresh[MT][2][4] = {};
#pragma unroll 1
        for (int j = 0; j < DC_TOKENS; j += 16) {
            Tf32Parts a[2][MT][4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float2 f = *(const float2*)&k_factor[item & 1][j + 8 * r + 2 * t4];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const float* x = k_s + (j + 8 * r + 2 * t4) * LK + c0 + 16 * m + g8;
                    a[r][m][0] = tf32_parts(x[0] * f.x);
                    a[r][m][1] = tf32_parts(x[8] * f.x);
                    a[r][m][2] = tf32_parts(x[LK] * f.y);
                    a[r][m][3] = tf32_parts(x[LK + 8] * f.y);
                }
            }
            add_runs<2>(fresh, a, [&](Tf32Parts (&b)[2], int r, int n) { b_down(b, u_s + (j + 8 * r) * LV + s0 + 8 * n, LV, lane); });
        }
        if (!all_finite(fresh)) {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (!is_finite(fresh[m][n][e]))
                            fresh[m][n][e] = sum_entry_by_entry(k_s + c0 + 16 * m + g8 + 8 * (e >> 1), LK, u_s + s0 + 8 * n + 2 * t4 + (e & 1), LV,
                                                                k_factor[item & 1], DC_TOKENS);
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n) {
#pragma unroll
                for (int e = 0; e < 4; ++e) S[m][n][e] = fmaf(decay, S[m][n][e], fresh[m][n][e]);
                float* to = s_s + (c0 + 16 * m + g8) * LV + s0 + 8 * n + 2 * t4;
                *(float2*)to = make_float2(S[m][n][0], S[m][n][1]);
                *(float2*)(to + 8 * LV) = make_float2(S[m][n][2], S[m][n][3]);
            }
        __syncthreads();                             // nobody reads u, the pairs' weights and the keys any more
        if (item + 1 < last) copy_second(item + 1);
    }
    float* to = kept + ((start + n_tok) & 1) * p.copy_floats;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            float* at = to + (size_t)(c0 + 16 * m + g8) * vdim + s0 + 8 * n + 2 * t4;
            *(float2*)at = make_float2(S[m][n][0], S[m][n][1]);
            *(float2*)(at + 8 * (size_t)vdim) = make_float2(S[m][n][2], S[m][n][3]);
        }
}

// Launch 3.  A warp a (token, head): bound by reading o and the gate once.
template <int VDIM, typename OutT>
__global__ void __launch_bounds__(256) delta_chunk_finish_kernel(DeltaChunks p, int items) {
    constexpr int EACH = VDIM / 32;
    const int lane = threadIdx.x & 31, item = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (item >= items) return;
    const size_t row = item / p.heads;
    const int h = item - (int)row * p.heads;
    const float* o = p.raw + (size_t)item * VDIM + lane;
    const float* gate = p.proj + row * p.proj_stride + p.g_off + h * VDIM + lane;
    float x[EACH], z[EACH], ss = 0.f;
#pragma unroll
    for (int i = 0; i < EACH; ++i) { x[i] = o[32 * i]; z[i] = gate[32 * i]; }
#pragma unroll
    for (int i = 0; i < EACH; ++i) ss = fmaf(x[i], x[i], ss);
    const float rinv = 1.0f / sqrtf(warp_sum(ss) / (float)VDIM + p.eps);
    OutT* out = (OutT*)p.out + (size_t)item * VDIM + lane;
#pragma unroll
    for (int i = 0; i < EACH; ++i) out[32 * i] = from_f32<OutT>(x[i] * rinv * p.norm[lane + 32 * i] * (z[i] / (1.0f + expf(-z[i]))));
}

// ----------------------------------------------------------------------------- host side

// Chunks of at most 64 tokens: chunk_seq/begin/end and, per sequence, its first chunk (one entry more at the end).  raw: num_rows *
// heads * vdim floats; scratch: num_chunks * heads * (64 (dim + vdim + 64 + 2) + 4) floats.
FRB_API int frb_delta_chunks(const float* conv, int conv_stride, int q_off, int k_off, int v_off, const float* proj, int proj_stride, int b_off,
                             int a_off, int g_off, const float* a_log, const float* dt_bias, const float* norm, const int* seq_slot,
                             const int* seq_start, const int* cu_q_len, float* state, long long copy_floats, long long state_offset, void* out,
                             int out_dtype, float* raw, int num_rows, int num_seqs, int heads, int kv_heads, int dim, int vdim, float eps,
                             const int* chunk_seq, const int* chunk_begin, const int* chunk_end, const int* seq_chunk0, int num_chunks,
                             float* scratch, cudaStream_t stream) {
    if (num_seqs == 0 || num_chunks == 0) return 0;
    FRB_CHECK_ARG((dim == 64 || dim == 128) && (vdim == 64 || vdim == 128) && kv_heads >= 1 && heads % kv_heads == 0 && heads <= 65535,
                  "delta chunks: %d heads of %d x %d over %d key heads", heads, dim, vdim, kv_heads);
    FRB_CHECK_ARG(((conv_stride | q_off | k_off) & 3) == 0 && ((copy_floats | state_offset) & 1) == 0 && ((uintptr_t)state & 7) == 0 &&
                      (((uintptr_t)conv | (uintptr_t)scratch | (uintptr_t)raw) & 15) == 0, "delta chunks: rows of %d entries are not in steps of 16 bytes",
                  conv_stride);
    FRB_CHECK_ARG((long long)num_rows * heads < (1ll << 31) - 8, "delta chunks: %d rows of %d heads", num_rows, heads);
    DeltaChunks p;
    p.conv = conv; p.proj = proj; p.a_log = a_log; p.dt_bias = dt_bias; p.norm = norm; p.seq_slot = seq_slot; p.seq_start = seq_start;
    p.cu_q_len = cu_q_len; p.chunk_seq = chunk_seq; p.chunk_begin = chunk_begin; p.chunk_end = chunk_end; p.seq_chunk0 = seq_chunk0;
    p.state = state; p.copy_floats = copy_floats; p.state_offset = state_offset; p.out = out; p.raw = raw;
    const size_t items = (size_t)num_chunks * heads;
    p.w = scratch;
    p.u = p.w + items * DC_TOKENS * dim;
    p.pairs = p.u + items * DC_TOKENS * vdim;
    p.q_factor = p.pairs + items * DC_TOKENS * DC_TOKENS;
    p.k_factor = p.q_factor + items * DC_TOKENS;
    p.decays = p.k_factor + items * DC_TOKENS;
    p.conv_stride = conv_stride; p.q_off = q_off; p.k_off = k_off; p.v_off = v_off; p.proj_stride = proj_stride; p.b_off = b_off; p.a_off = a_off;
    p.g_off = g_off; p.heads = heads; p.kv_heads = kv_heads; p.eps = eps;
    const size_t one = (size_t)(2 * DC_TOKENS * (dim + 8) + DC_TOKENS * (DC_TOKENS + 4)) * sizeof(float);
    const size_t two = (size_t)(2 * DC_TOKENS * (dim + 8) + DC_TOKENS * (dim + 4) + DC_TOKENS * DC_LM + (dim + DC_TOKENS) * (DC_SLICE + 4)) * sizeof(float);
    const dim3 chains(num_seqs, heads, vdim / DC_SLICE);
    const int rows_heads = num_rows * heads;
#define FRB_DELTA_CHUNKS(DIM, VDIM)                                                                                                  \
    do {                                                                                                                             \
        cudaFuncSetAttribute(delta_chunk_solve_kernel<DIM, VDIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)one);            \
        cudaFuncSetAttribute(delta_chunk_chain_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)two);                  \
        delta_chunk_solve_kernel<DIM, VDIM><<<dim3(num_chunks, heads), 256, one, stream>>>(p);                                       \
        delta_chunk_chain_kernel<DIM><<<chains, 512, two, stream>>>(p, vdim);                                                        \
        FRB_DISPATCH_DTYPE(out_dtype, OutT, {                                                                                        \
            delta_chunk_finish_kernel<VDIM, OutT><<<(rows_heads + 7) / 8, 256, 0, stream>>>(p, rows_heads);                          \
        });                                                                                                                          \
    } while (0)
    if (dim == 128 && vdim == 128) FRB_DELTA_CHUNKS(128, 128);
    else if (dim == 128) FRB_DELTA_CHUNKS(128, 64);
    else if (vdim == 128) FRB_DELTA_CHUNKS(64, 128);
    else FRB_DELTA_CHUNKS(64, 64);
#undef FRB_DELTA_CHUNKS
    FRB_RETURN_LAUNCH("delta_chunks");
}
