// The gated delta rule of delta_rule.cu for prompts, in chunks of 64 tokens.  Per head (q and k unit vectors, q also times
// dim^(-1/2); beta and one decay g a token):
//
//     u_i = beta_i (v_i - g_i S_(i-1)^T k_i),   S_i = g_i S_(i-1) + k_i u_i^T,   o_i = S_i^T q_i.
//
// With S the state at a chunk's start and w(j, i) the product of the decays of its tokens j + 1 .. i (w(i): from the chunk's start):
//     (I + M) u = beta v - beta w k^T S,   M_ij = beta_i w(j, i) (k_i . k_j) for j < i,
//     o_i = w(i) S^T q_i + sum_(j <= i) w(j, i) (q_i . k_j) u_j,   S <- w(end) S + sum_j w(j, end) k_j u_j^T.
//   1. every chunk and key head side by side: the products of the unit keys with one another and with the unit queries;
//   2. every chunk and head side by side: the weights, M and the pairs' weights for o; then (I + M) X = [beta w k | beta v] by
//      substitution, two threads for two columns, in float32: W and U' with u = U' - W S.  (The entries of (I + M)^(-1) are at most one: each is
//      what is left of a unit of v_j under steps that shorten, times beta k_i.)
//   3. along the chunks of a sequence, a block that keeps the state in registers: u = U' - W S, o, and the new state.  Heads of 128 value
//      columns: on tcgen05, a block a (sequence, head); of 64: on mma.sync.
//   4. the head's root mean square, weight and gate.
// A weight is the exponential of a sum of logarithms that has its tokens' alone, or a product of such factors: never a quotient, and no
// difference of two sums either, which behind one strong decay would have lost the digits of the mild ones.  The sums run over up to 16
// tokens inside a block and up to 48 between blocks: a rounding of their logarithms, which are large only where the weight is small.
//
// Everything is float32; the products run on tensor cores with each operand as two parts (tf32_parts.cuh: sums of 16 entries, added in
// float32 registers; f16_parts.cuh: of at most 128).  Four prompts of 2,048 tokens, 16 heads of 128 x 128 over 4 key heads: 320 us (34 +
// 128 + 129 + 34 for the launches in turn; the pairs' scales of single rows and the look at the outputs that they are for cost launch 2 two
// of its microseconds; delta_rule.cu token by token 1,367).  With launch 1's products made by launch 2 for every head, and
// launch 3 on mma.sync, 589 (189 + 368 + 34).  Launch 2 is bound by its substitution's reads of M from shared memory and by the
// latencies before it, two blocks an SM; launch 3 by the chain of its phases.
#include "f16_parts.cuh"
#include "tf32_parts.cuh"

#define DC_TOKENS 64
#define DC_BLOCK 16
#define DC_BLOCKS (DC_TOKENS / DC_BLOCK)
#define DC_SLICE 64           // value columns a block of launch 2 keeps
#define DC_LM (DC_TOKENS + 8)
#define DC_FACTORS (4 * DC_TOKENS + 4)
#define DC_W_SCALE 8          // exponents of the parts' scales
#define DC_Q_SCALE 17
#define DC_K_SCALE 14

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
    // for the chain on tcgen05, in place of w and pairs: their parts, and the unit keys' and queries'
    uint16_t* w_parts;       // [chunks][heads][part][dim / 64][DC_TOKENS][64], the row times 2^8 / (a power of two about w(i))
    uint16_t* pair_parts;    // [chunks][heads][part][DC_TOKENS][DC_TOKENS], rows with a scale each
    uint16_t *q_parts, *k_parts;     // [chunks][kv_heads][part][dim / 64][DC_TOKENS][64], times 2^17 and 2^14
    float* raw_pairs;        // [chunks][kv_heads][2][DC_TOKENS][DC_TOKENS]: the unit keys' products [j][i], the queries' with them [i][j], j <= i
    float* norms;            // [chunks][kv_heads][3][DC_TOKENS]: what makes the queries (with dim^(-1/2)) and keys unit vectors; the queries' scale off (0: zeros)
    float* factors;          // [chunks][heads][DC_FACTORS]: w's scale off; w(i), the query's scale off; w(j, end); the pairs' scales off; w(end)
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

// The exponent that brings entries of W's row i, at most 2^6 w(i), below 2^14.
__device__ __forceinline__ int dc_w_exponent(float start) { return DC_W_SCALE - max(ilogbf(fmaxf(start, 1e-30f)), -100); }

// Launch 1.  grid (chunk, key head): the products of the unit keys with one another and with the unit queries, once for all heads over
// them.  PARTS: also those rows as float16 parts, for the chain on tcgen05.
template <int DIM, bool PARTS>
__global__ void __launch_bounds__(256, 2) delta_chunk_pairs_kernel(DeltaChunks p) {
    constexpr int LQ = DIM + 8;
    extern __shared__ float4 dc_smem[];
    __shared__ float q_inv[DC_TOKENS], k_inv[DC_TOKENS];
    float* q_s = (float*)dc_smem;                   // [DC_TOKENS][LQ]
    float* k_s = q_s + DC_TOKENS * LQ;              // [DC_TOKENS][LQ]
    const int item = blockIdx.x, kvh = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    let_next_kernel_start();
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item];
    const size_t row0 = (size_t)p.cu_q_len[b] + p.chunk_begin[item], at = (size_t)item * p.kv_heads + kvh;
    const float* rows = p.conv + row0 * p.conv_stride;
    dc_copy_rows<DIM, 256>(q_s, LQ, rows + p.q_off + kvh * DIM, p.conv_stride, count);
    dc_copy_rows<DIM, 256>(k_s, LQ, rows + p.k_off + kvh * DIM, p.conv_stride, count);
    copies_commit();
    copies_wait<0>();
    __syncthreads();
    for (int t = warp; t < DC_TOKENS; t += 8) {
        float qq = 0.f, kk = 0.f;
        bool some = false;                           // an entry of the query that is not zero
#pragma unroll
        for (int d = 0; d < DIM; d += 32) {
            const float x = q_s[t * LQ + d + lane], y = k_s[t * LQ + d + lane];
            qq = fmaf(x, x, qq);
            kk = fmaf(y, y, kk);
            some = some || x != 0.f;
        }
        qq = warp_sum(qq);
        kk = warp_sum(kk);
        if (PARTS) some = __any_sync(0xffffffffu, some);
        if (lane == 0) {
            const float q = 1.0f / sqrtf((float)DIM) / sqrtf(qq + 1e-6f), k = 1.0f / sqrtf(kk + 1e-6f);
            q_inv[t] = q;
            k_inv[t] = k;
            p.norms[at * 3 * DC_TOKENS + t] = q;
            p.norms[at * 3 * DC_TOKENS + DC_TOKENS + t] = k;
            if (PARTS) p.norms[at * 3 * DC_TOKENS + 2 * DC_TOKENS + t] = some ? power_of_two(-DC_Q_SCALE) : 0.f;
        }
    }
    __syncthreads();
    if (PARTS) {
        constexpr int UNITS = DC_TOKENS * DIM / 8;
        const size_t to = at * 2 * DC_TOKENS * DIM;
        for (int u = tid; u < 2 * UNITS; u += 256) {
            const bool key = u >= UNITS;
            const int r = u % UNITS / (DIM / 8), c = u % (DIM / 8) * 8;
            const float* from = (key ? k_s : q_s) + r * LQ + c;
            const float scale = (key ? k_inv[r] : q_inv[r]) * power_of_two(key ? DC_K_SCALE : DC_Q_SCALE);
            uint4 hi, lo;
            split_four(*(const float4*)from, scale, hi.x, hi.y, lo.x, lo.y);
            split_four(*(const float4*)(from + 4), scale, hi.z, hi.w, lo.z, lo.w);
            uint16_t* parts = (key ? p.k_parts : p.q_parts) + to + piece_place(r, c);
            *(uint4*)parts = hi;
            *(uint4*)(parts + DC_TOKENS * DIM) = lo;
        }
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
    float* kk = p.raw_pairs + at * 2 * DC_TOKENS * DC_TOKENS;            // [j][i], then q k [i][j]
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < DC_BLOCKS; ++n)
            if (n <= tiles[m])
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = tiles[m] * DC_BLOCK + (lane >> 2) + 8 * (e >> 1), j = n * DC_BLOCK + 8 * odd + 2 * (lane & 3) + (e & 1);
                    if (j <= i && !is_finite(acc[m][n][e])) acc[m][n][e] = sum_entry_by_entry(left + i * LQ, 1, k_s + j * LQ, 1, nullptr, DIM);
                    const float value = acc[m][n][e] * k_inv[j] * (keys ? k_inv[i] : q_inv[i]);
                    if (keys) kk[j * DC_TOKENS + i] = value;
                    else kk[DC_TOKENS * DC_TOKENS + i * DC_TOKENS + j] = value;
                }
}

// Launch 2.  grid (chunk, head): the weights, M and the pairs' weights for o, and the substitution.  PARTS: what it leaves for launch 3 as
// float16 parts (the chain on tcgen05).
template <int DIM, int VDIM, bool PARTS>
__global__ void __launch_bounds__(256, 2) delta_chunk_solve_kernel(DeltaChunks p) {
    constexpr int LS = DC_TOKENS + 4;
    __shared__ float beta_s[DC_TOKENS], log_s[DC_TOKENS], to_s[DC_TOKENS], from_s[DC_TOKENS], start_s[DC_TOKENS], q_inv[DC_TOKENS], k_inv[DC_TOKENS], w_scale[DC_TOKENS];
    __shared__ float block_log[DC_BLOCKS], between[DC_BLOCKS][DC_BLOCKS];
    __shared__ __align__(16) float own[DC_TOKENS][DC_BLOCK + 4];         // w(j, i) of the tokens j of i's block; zero for later ones
    __shared__ __align__(16) float m_s[DC_TOKENS * LS];                  // M, column by column
    const int item = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int b = p.chunk_seq[item], count = p.chunk_end[item] - p.chunk_begin[item], kvh = h / (p.heads / p.kv_heads);
    const size_t row0 = (size_t)p.cu_q_len[b] + p.chunk_begin[item], at = (size_t)item * p.heads + h, kv_at = (size_t)item * p.kv_heads + kvh;
    const float* rows = p.conv + row0 * p.conv_stride;

    // the substitution's right-hand side, two columns of [k | v] for two neighbouring threads, on its way meanwhile: thread r of the two has
    // the rows 8 g + 4 r .. + 3
    float x[2][DC_TOKENS / 2];
    const int column = tid & ~1, r = tid & 1;
    const bool key = column < DIM;
    const auto row_of = [&](int i) { return 2 * (i & ~3) + 4 * r + (i & 3); };
    if (tid < DIM + VDIM) {
        const float* from = rows + (key ? p.k_off + kvh * DIM + column : p.v_off + h * VDIM + column - DIM);
        const bool pairs_of_columns = key || (p.v_off & 1) == 0;         // the keys' rows are in steps of 16 bytes
#pragma unroll
        for (int i = 0; i < DC_TOKENS / 2; ++i) {
            const float* at_row = from + (size_t)min(row_of(i), count - 1) * p.conv_stride;
            if (pairs_of_columns) {
                const float2 v = *(const float2*)at_row;
                x[0][i] = v.x;
                x[1][i] = v.y;
            } else {
                x[0][i] = at_row[0];
                x[1][i] = at_row[1];
            }
        }
    }
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
    __syncthreads();
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
    // the chunk's factors for launch 3: a token's decays to the chunk's end
    float rest = 0.f;
    if (tid < DC_TOKENS)
        for (int m = tid / DC_BLOCK + 1; m < DC_BLOCKS; ++m) rest += block_log[m];
    after_previous_kernel();                         // launch 1, whose products come from here on; it began when the rows were there
    // (with PARTS what takes the queries' scale off in the place of their norms, which are in their parts)
    if (tid < 2 * DC_TOKENS) (tid < DC_TOKENS ? q_inv : k_inv)[tid % DC_TOKENS] = p.norms[kv_at * 3 * DC_TOKENS + (PARTS && tid < DC_TOKENS ? 2 * DC_TOKENS : 0) + tid];
    __syncthreads();
    if (tid < DC_TOKENS) {
        const float to_end = from_s[tid] * expf(rest);
        if (PARTS) {
            float* factors = p.factors + at * DC_FACTORS;
            const int exponent = dc_w_exponent(start_s[tid]);
            w_scale[tid] = power_of_two(exponent);
            factors[tid] = power_of_two(-exponent);
            factors[DC_TOKENS + tid] = start_s[tid] * q_inv[tid];
            factors[2 * DC_TOKENS + tid] = to_end;
            if (tid == DC_TOKENS - 1) factors[4 * DC_TOKENS] = start_s[tid];
        } else {
            p.q_factor[at * DC_TOKENS + tid] = start_s[tid] * q_inv[tid];
            p.k_factor[at * DC_TOKENS + tid] = to_end * k_inv[tid];
            if (tid == DC_TOKENS - 1) p.decays[at] = start_s[tid];
        }
    }

    // four entries of M's columns at a time, then eight of the pairs' rows
    const float* kk = p.raw_pairs + kv_at * 2 * DC_TOKENS * DC_TOKENS;
    auto weight = [&](int i, int j) {
        const int ib = i / DC_BLOCK, jb = j / DC_BLOCK;
        return jb < ib ? to_s[i] * between[ib][jb] * from_s[j] : own[i][j % DC_BLOCK];
    };
#pragma unroll
    for (int u = tid; u < DC_TOKENS * DC_TOKENS / 4; u += 256) {
        const int j = u / (DC_TOKENS / 4), i0 = u % (DC_TOKENS / 4) * 4;
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i0 + 3 > j) {
            const float4 raw = *(const float4*)(kk + j * DC_TOKENS + i0);
            const float r[4] = {raw.x, raw.y, raw.z, raw.w};
            float* to = (float*)&m;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (i0 + e > j) to[e] = r[e] * weight(i0 + e, j) * beta_s[i0 + e];
        }
        *(float4*)(m_s + j * LS + i0) = m;
    }
    for (int u = tid; u < DC_TOKENS * DC_TOKENS / 8; u += 256) {
        const int i = u / (DC_TOKENS / 8), j0 = u % (DC_TOKENS / 8) * 8;
        float y[8] = {};
        if (j0 <= i) {
            const float* from = kk + DC_TOKENS * DC_TOKENS + i * DC_TOKENS + j0;
            const float4 a = *(const float4*)from, c = *(const float4*)(from + 4);
            const float r[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (j0 + e <= i) y[e] = r[e] * weight(i, j0 + e);
        }
        if (PARTS) {                                 // eight neighbouring threads have a row
            float top = 0.f;
#pragma unroll
            for (int e = 0; e < 8; e += 2) top = max3(top, fabsf(y[e]), fabsf(y[e + 1]));
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const int exponent = parts_exponent(top);
            if (j0 == 0) p.factors[at * DC_FACTORS + 3 * DC_TOKENS + i] = top > 0.f ? power_of_two(-exponent) : 0.f;
            uint4 hi, lo;
            split_four(make_float4(y[0], y[1], y[2], y[3]), power_of_two(exponent), hi.x, hi.y, lo.x, lo.y);
            split_four(make_float4(y[4], y[5], y[6], y[7]), power_of_two(exponent), hi.z, hi.w, lo.z, lo.w);
            uint16_t* to = p.pair_parts + at * 2 * DC_TOKENS * DC_TOKENS + piece_place(i, j0);
            *(uint4*)to = hi;
            *(uint4*)(to + DC_TOKENS * DC_TOKENS) = lo;
        } else {
            float4* to = (float4*)(p.pairs + at * DC_TOKENS * DC_TOKENS + i * DC_TOKENS + j0);
            to[0] = make_float4(y[0], y[1], y[2], y[3]);
            to[1] = make_float4(y[4], y[5], y[6], y[7]);
        }
    }
    __syncthreads();

    // substitution: two threads for two columns of [beta w k | beta v], each with half of the rows of both.  It is bound by the reads of M, one
    // entry a cycle for a whole warp: with two columns a thread they are half as many as with one (launch 2: 128 us instead of 153; with
    // four columns and four threads, whose exchanges are twice as many, 144; with two threads a column, 64 registers each, 178).
    if (tid >= DIM + VDIM) return;
#pragma unroll
    for (int i = 0; i < DC_TOKENS / 2; ++i) {
        const int row = row_of(i);
        const float factor = key ? beta_s[row] * start_s[row] * k_inv[row] : beta_s[row];
#pragma unroll
        for (int c = 0; c < 2; ++c) x[c][i] = row < count ? factor * x[c][i] : 0.f;
    }
    const int lane = tid & 31, width = key ? DIM : VDIM;
    float* to = key ? p.w + at * DC_TOKENS * DIM + column : p.u + at * DC_TOKENS * VDIM + column - DIM;
    uint16_t* w_parts = p.w_parts + at * 2 * DC_TOKENS * DIM;
    // four rows at a time, which one of the two threads has: it settles them among themselves, both learn them, and they leave every later row
#pragma unroll
    for (int g = 0; g < DC_TOKENS / 4; ++g) {
        const int own_group = g >> 1, owner = g & 1;
        const float* m = m_s + 4 * g * LS;
        const float4 m0 = *(const float4*)(m + 4 * g), m1 = *(const float4*)(m + LS + 4 * g), m2 = *(const float4*)(m + 2 * LS + 4 * g);
        float d[2][4];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float* from = x[c] + 4 * own_group;
            d[c][0] = from[0];
            d[c][1] = fmaf(m0.y, -d[c][0], from[1]);
            d[c][2] = fmaf(m1.z, -d[c][1], fmaf(m0.z, -d[c][0], from[2]));
            d[c][3] = fmaf(m2.w, -d[c][2], fmaf(m1.w, -d[c][1], fmaf(m0.w, -d[c][0], from[3])));
#pragma unroll
            for (int e = 0; e < 4; ++e) d[c][e] = __shfl_sync(0xffffffffu, d[c][e], (lane & ~1) | owner);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {                // a thread writes two of the four rows
            const int row = 4 * g + 2 * r + e;
            const float first = r ? d[0][2 + e] : d[0][e], second = r ? d[1][2 + e] : d[1][e];
            if (!PARTS || !key) {
                *(float2*)(to + (size_t)row * width) = make_float2(first, second);
            } else {
                const float scale = w_scale[row];
                uint32_t hi, lo;
                split_two(mul_pairs(pair_of(first, second), pair_of(scale, scale)), hi, lo);
                uint16_t* parts = w_parts + piece_place(row, column);
                *(uint32_t*)parts = hi;
                *(uint32_t*)(parts + DC_TOKENS * DIM) = lo;
            }
        }
        const float* later = m + 4 * r;
#pragma unroll
        for (int l = own_group + owner; l < DC_TOKENS / 8; ++l)
#pragma unroll
            for (int e = 0; e < 4; ++e) {                                // two rows at a time
                ulonglong2 w = *(const ulonglong2*)(later + e * LS + 8 * l);
                if (l == own_group && r == 0) w = make_ulonglong2(0, 0); // the rows themselves
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint64_t leaves = pair_of(-d[c][e], -d[c][e]);
                    float* y = x[c] + 4 * l;
                    halves_of(fma_pairs(w.x, leaves, pair_of(y[0], y[1])), y[0], y[1]);
                    halves_of(fma_pairs(w.y, leaves, pair_of(y[2], y[3])), y[2], y[3]);
                }
            }
    }
}

// Launch 3.  grid (sequence, head, slice of 64 value columns), 16 warps.  W and the queries are free once u is there, the pairs' weights
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
    after_previous_kernel();
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

// Launch 3 on tcgen05, for heads of 128 value columns.  grid (sequence, head): a block keeps the head's state, transposed: a lane of tensor
// memory is a value column, and two threads have half of its DIM entries each, in float32.  With every operand as two float16 parts (the
// small products first, 2^11 times too large, taken down by the first large one), for every chunk
//     D1 = S^T [W; Q]^T        128 x 64 x DIM, W first: the state's parts in tensor memory, W's and the queries' rows in shared memory;
//     u^T = U'^T - D1          two threads a column, 32 tokens each; its parts, and those of u w(j, end), go to tensor memory;
//     DS = (u w(j, end))^T K   128 x DIM x 64, the keys N-major;   DO = u^T pairs^T   128 x 64 x 64;
//     S <- w(end) S + DS^T, o = w(i) D1 + DO in float32 registers.
// The columns' parts have a power of two of their own each, from the largest entry of the state or of u.  What bounds it: the chain of a
// chunk's phases, 6,300 cycles (11.5 us on mma.sync): the first product 1,150, the third 1,250, the state's split 1,250, u and its two
// splits 2,000, the new state 560; the SMs that have a sequence's head, 64 of them for four prompts in sixteen heads, issue an
// instruction on nearly every cycle of the splits.  A number that is not finite, or a token whose outputs may have lost digits (PARTS_LEAST),
// makes the block take the sequence's head again, token by token.
#define DT_SHARES 2            // threads a column: each half of its entries and of a chunk's tokens (four: 127 us instead of 118)
#define DT_WARPS (4 * DT_SHARES)
#define DT_ROWS (32 * DT_WARPS)
#define DT_THREADS (DT_ROWS + 96)        // the columns' warps (w & 3: lanes; w >> 2: share), then one each for copies, products, outputs
#define DT_TOKENS (DC_TOKENS / DT_SHARES)

using namespace frb_tma;
using namespace frb_tc;

// A sequence's head token by token (delta_rule.cu's formula) by the columns' threads, DT_SHARES a column, each with its entries of the state.
// room: shared memory for the rows of 32 tokens and the threads' sums.  Bound by the reads of q and k from there: a token takes
// 1.4 us (one thread a column, its state spilled, the rows fetched token by token: 7.5 us).
template <int DIM>
static __device__ __noinline__ void dt_token_by_token(const DeltaChunks& p, int b, int h, float* room) {
    constexpr int VDIM = 128, SHARE = DIM / DT_SHARES, BATCH = 32;
    float *q_s = room, *k_s = q_s + BATCH * DIM, *v_s = k_s + BATCH * DIM;
    float4* scalars = (float4*)(v_s + BATCH * VDIM);                     // beta, decay, the query's product with the key
    float2* sums = (float2*)(scalars + BATCH);                           // [token & 1][share][column]
    const int tid = threadIdx.x, lane = tid & 31, share = tid / VDIM, column = tid % VDIM, kvh = h / (p.heads / p.kv_heads);
    auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(DT_ROWS) : "memory"); };
    const int start = p.seq_start[b], count = p.cu_q_len[b + 1] - p.cu_q_len[b];
    const size_t row0 = p.cu_q_len[b];
    float* state = p.state + (size_t)p.seq_slot[b] * 2 * p.copy_floats + p.state_offset + ((size_t)h * DIM + share * SHARE) * VDIM + column;
    const float* from = state + (start & 1) * p.copy_floats;
    float* to = state + ((start + count) & 1) * p.copy_floats;
    const float rate = expf(p.a_log[h]), bias = p.dt_bias[h];
    uint64_t S[SHARE / 2];
#pragma unroll
    for (int d = 0; d < SHARE / 2; ++d) S[d] = pair_of(from[(size_t)(2 * d) * VDIM], from[(size_t)(2 * d + 1) * VDIM]);
    for (int t0 = 0; t0 < count; t0 += BATCH) {
        const int here = min(BATCH, count - t0);
        meet();                                      // nobody reads the rows before any more
        for (int t = share; t < here; t += DT_SHARES) v_s[t * VDIM + column] = p.conv[(row0 + t0 + t) * p.conv_stride + p.v_off + h * VDIM + column];
        for (int t = tid >> 5; t < here; t += DT_WARPS) {
            const float* rows = p.conv + (row0 + t0 + t) * p.conv_stride;
            const float* logits = p.proj + (row0 + t0 + t) * p.proj_stride + h;
            float x[DIM / 32], y[DIM / 32], qq = 0.f, kk = 0.f, qk = 0.f;
#pragma unroll
            for (int d = 0; d < DIM / 32; ++d) {
                x[d] = rows[p.q_off + kvh * DIM + 32 * d + lane];
                y[d] = rows[p.k_off + kvh * DIM + 32 * d + lane];
                qq = fmaf(x[d], x[d], qq);
                kk = fmaf(y[d], y[d], kk);
                qk = fmaf(x[d], y[d], qk);
            }
            const float q = 1.0f / sqrtf((float)DIM) / sqrtf(warp_sum(qq) + 1e-6f), k = 1.0f / sqrtf(warp_sum(kk) + 1e-6f);
            qk = warp_sum(qk) * q * k;
#pragma unroll
            for (int d = 0; d < DIM / 32; ++d) {
                q_s[t * DIM + 32 * d + lane] = x[d] * q;
                k_s[t * DIM + 32 * d + lane] = y[d] * k;
            }
            if (lane == 0)
                scalars[t] = make_float4(1.0f / (1.0f + expf(-logits[p.b_off])), expf(-rate * dc_softplus(logits[p.a_off] + bias)), qk, 0.f);
        }
        meet();
        for (int t = 0; t < here; ++t) {
            const float4 f = scalars[t];
            const ulonglong2 *k2 = (const ulonglong2*)(k_s + t * DIM + share * SHARE), *q2 = (const ulonglong2*)(q_s + t * DIM + share * SHARE);
            const uint64_t decay = pair_of(f.y, f.y);
            uint64_t seen[2] = {0ull, 0ull}, from_state[2] = {0ull, 0ull};
#pragma unroll
            for (int d = 0; d < SHARE / 4; ++d) {
                const ulonglong2 k = k2[d], q = q2[d];
                S[2 * d] = mul_pairs(S[2 * d], decay);
                S[2 * d + 1] = mul_pairs(S[2 * d + 1], decay);
                seen[0] = fma_pairs(S[2 * d], k.x, seen[0]);
                seen[1] = fma_pairs(S[2 * d + 1], k.y, seen[1]);
                from_state[0] = fma_pairs(S[2 * d], q.x, from_state[0]);
                from_state[1] = fma_pairs(S[2 * d + 1], q.y, from_state[1]);
            }
            float a, b, c, e;
            halves_of(add_pairs(seen[0], seen[1]), a, b);
            halves_of(add_pairs(from_state[0], from_state[1]), c, e);
            float2* told = sums + (t & 1) * DT_SHARES * VDIM + column;
            told[share * VDIM] = make_float2(a + b, c + e);
            meet();
            float2 all = told[0];
#pragma unroll
            for (int i = 1; i < DT_SHARES; ++i) { all.x += told[i * VDIM].x; all.y += told[i * VDIM].y; }
            const float u = f.x * (v_s[t * VDIM + column] - all.x);
            const uint64_t us = pair_of(u, u);
#pragma unroll
            for (int d = 0; d < SHARE / 4; ++d) {
                const ulonglong2 k = k2[d];
                S[2 * d] = fma_pairs(k.x, us, S[2 * d]);
                S[2 * d + 1] = fma_pairs(k.y, us, S[2 * d + 1]);
            }
            if (share == 0) p.raw[((row0 + t0 + t) * p.heads + h) * VDIM + column] = fmaf(u, f.z, all.y);
        }
    }
#pragma unroll
    for (int d = 0; d < SHARE / 2; ++d) {
        float even, odd;
        halves_of(S[d], even, odd);
        to[(size_t)(2 * d) * VDIM] = even;
        to[(size_t)(2 * d + 1) * VDIM] = odd;
    }
}

template <int DIM>
__global__ void __launch_bounds__(DT_THREADS, 1) delta_chunk_chain_tc_kernel(const __grid_constant__ DeltaChunks p, int* __restrict__ status) {
    constexpr int VDIM = 128, SHARE = DIM / DT_SHARES;
    constexpr uint32_t ROWS_PART = DC_TOKENS * DIM * 2, PAIR_PART = DC_TOKENS * DC_TOKENS * 2;       // bytes of one part
    // tensor memory: the state's parts; D1 of W, later u's parts; D1 of Q; the parts of u w(j, end); DO; DS
    constexpr int S_HI = 0, S_LO = DIM / 2, D1_W = 128, D1_Q = 192, UK = 256, D_O = 320, D_S = 384;
    extern __shared__ uint8_t dt_smem[];
    __shared__ uint64_t w_full, q_full, k_full, pairs_full, u_full, s_ready, u_ready, d1w_done, d1q_done, ds_done, do_done, o_stored, o_free;
    __shared__ float tops[3][DT_SHARES][VDIM];
    __shared__ int first_rows[DT_SHARES][4];
    __shared__ __align__(16) float factors[3][DC_FACTORS];               // of chunk c at c % 3: a chunk's are read until the next one's state is split
    __shared__ uint32_t tmem_slot;
    __shared__ int failed_flag, odd_numbers;
    volatile int* failed = &failed_flag;
    uint8_t* w_s = (uint8_t*)(((uintptr_t)dt_smem + 1023) & ~(uintptr_t)1023);
    uint8_t* q_s = w_s + 2 * ROWS_PART;
    uint8_t* k_s = q_s + 2 * ROWS_PART;
    uint8_t* pairs_s = k_s + 2 * ROWS_PART;
    float* u_s = (float*)(pairs_s + 2 * PAIR_PART);                      // [DC_TOKENS][VDIM]: U'
    float* o_s = u_s + DC_TOKENS * VDIM;                                 // the same of the outputs
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int b = blockIdx.x, h = blockIdx.y, kvh = h / (p.heads / p.kv_heads);
    const int first = p.seq_chunk0[b], last = __shfl_sync(0xffffffffu, p.seq_chunk0[b + 1], 0), start = p.seq_start[b];
    const int n_tok = p.cu_q_len[b + 1] - p.cu_q_len[b], chunks = __shfl_sync(0xffffffffu, last - first, 0);
    const size_t seq_row0 = p.cu_q_len[b];

    if (threadIdx.x == 0) {
        bar_init(&w_full, 1); bar_init(&q_full, 1); bar_init(&k_full, 1); bar_init(&pairs_full, 1);
        bar_init(&u_full, 1); bar_init(&o_stored, DT_ROWS / 32); bar_init(&o_free, 1);
        bar_init(&s_ready, DT_ROWS / 32); bar_init(&u_ready, DT_ROWS / 32);
        bar_init(&d1w_done, 1); bar_init(&d1q_done, 1); bar_init(&ds_done, 1); bar_init(&do_done, 1);
        failed_flag = 0;
        odd_numbers = 0;
        bar_init_fence();
    }
    if (warp == DT_WARPS + 1) tmem_alloc(&tmem_slot, 512);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    after_previous_kernel();                         // barriers and tensor memory were set up while it still ran

    if (warp == DT_WARPS) {
        if (lane == 0) {
            for (int c = 0; c < chunks; ++c) {
                const size_t at = (size_t)(first + c) * p.heads + h, kv_at = (size_t)(first + c) * p.kv_heads + kvh;
                const uint32_t before = (c & 1) ^ 1;                     // of the phase that the chunk before has ended
                if (c && !bar_wait(&d1w_done, before, failed)) { atomicExch(status, 61); break; }
                bar_expect(&w_full, 2 * ROWS_PART + DC_FACTORS * 4);
                copy_bulk(w_s, p.w_parts + at * 2 * DC_TOKENS * DIM, 2 * ROWS_PART, &w_full);
                copy_bulk(factors[c % 3], p.factors + at * DC_FACTORS, DC_FACTORS * 4, &w_full);
                if (c && !bar_wait(&u_ready, before, failed)) { atomicExch(status, 73); break; }
                bar_expect(&u_full, DC_TOKENS * VDIM * 4);
                copy_bulk(u_s, p.u + at * DC_TOKENS * VDIM, DC_TOKENS * VDIM * 4, &u_full);
                if (c && !bar_wait(&d1q_done, before, failed)) { atomicExch(status, 62); break; }
                bar_expect(&q_full, 2 * ROWS_PART);
                copy_bulk(q_s, p.q_parts + kv_at * 2 * DC_TOKENS * DIM, 2 * ROWS_PART, &q_full);
                if (c && !bar_wait(&ds_done, before, failed)) { atomicExch(status, 63); break; }
                bar_expect(&k_full, 2 * ROWS_PART);
                copy_bulk(k_s, p.k_parts + kv_at * 2 * DC_TOKENS * DIM, 2 * ROWS_PART, &k_full);
                if (c && !bar_wait(&do_done, before, failed)) { atomicExch(status, 64); break; }
                bar_expect(&pairs_full, 2 * PAIR_PART);
                copy_bulk(pairs_s, p.pair_parts + at * 2 * DC_TOKENS * DC_TOKENS, 2 * PAIR_PART, &pairs_full);
            }
        }
    } else if (warp == DT_WARPS + 1) {
        // the whole warp goes through the loop (elect_one, tcgen05.cuh); its products run in the order of their issue
        constexpr uint32_t idesc64 = (1u << 4) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(VDIM >> 4) << 24);
        constexpr uint32_t idesc_k = (1u << 4) | (1u << 16) | ((uint32_t)(DIM >> 3) << 17) | ((uint32_t)(VDIM >> 4) << 24);
        const uint64_t w_at = tile_desc(smem_addr(w_s)), q_at = tile_desc(smem_addr(q_s)), pairs_at = tile_desc(smem_addr(pairs_s));
        const uint64_t k_at = desc_n_major(smem_addr(k_s));
        auto along = [](int k) { return (k / 4) * (DC_TOKENS * 128 >> 4) + (k % 4) * 2; };
        auto down = [](int k) { return k * (16 * 128 >> 4); };
        for (int c = 0; c < chunks; ++c) {
            const uint32_t phase = c & 1;
            if (!warp_wait_both(&w_full, phase, &s_ready, phase, failed)) { if (lane == 0) atomicExch(status, 65); break; }
            fence_after_sync();
            if (elect_one()) {
                products_of_parts<DIM / 16>(tmem + D1_W, tmem + S_HI, tmem + S_LO, w_at, w_at + (ROWS_PART >> 4), idesc64, along);
                mma_commit(&d1w_done);
            }
            __syncwarp();
            if (!warp_wait(&q_full, phase, failed)) { if (lane == 0) atomicExch(status, 66); break; }
            fence_after_sync();
            if (elect_one()) {
                products_of_parts<DIM / 16>(tmem + D1_Q, tmem + S_HI, tmem + S_LO, q_at, q_at + (ROWS_PART >> 4), idesc64, along);
                mma_commit(&d1q_done);
            }
            __syncwarp();
            if (!warp_wait_both(&k_full, phase, &u_ready, phase, failed)) { if (lane == 0) atomicExch(status, 67); break; }
            fence_after_sync();
            if (elect_one()) {
                products_of_parts<DC_TOKENS / 16>(tmem + D_S, tmem + UK, tmem + UK + 32, k_at, k_at + (ROWS_PART >> 4), idesc_k, down);
                mma_commit(&ds_done);
            }
            __syncwarp();
            if (!warp_wait(&pairs_full, phase, failed)) { if (lane == 0) atomicExch(status, 68); break; }
            fence_after_sync();
            if (elect_one()) {
                products_of_parts<DC_TOKENS / 16>(tmem + D_O, tmem + D1_W, tmem + D1_W + 32, pairs_at, pairs_at + (PAIR_PART >> 4), idesc64,
                                                  [](int k) { return k * 2; });
                mma_commit(&do_done);
            }
            __syncwarp();
        }
    } else if (warp == DT_WARPS + 2) {
        for (int c = 0; c < chunks; ++c) {           // a chunk's outputs, a token's 512 bytes a copy
            if (!warp_wait(&o_stored, c & 1, failed)) { if (lane == 0) atomicExch(status, 74); break; }
            const int begin = p.chunk_begin[first + c], count = p.chunk_end[first + c] - begin;
            for (int t = lane; t < count; t += 32)
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                             ::"l"(p.raw + ((seq_row0 + begin + t) * p.heads + h) * VDIM), "r"(smem_addr(o_s + t * VDIM)), "r"(VDIM * 4) : "memory");
            asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&o_free);
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        // A wait that gives up does not end the loop: the block's later waits then return at once, and every thread reaches the barriers.
        const int share = warp >> 2, quarter = warp & 3, column = quarter * 32 + lane, t0 = DT_TOKENS * share;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        float* kept = p.state + (size_t)p.seq_slot[b] * 2 * p.copy_floats + p.state_offset + (size_t)h * DIM * VDIM + (size_t)share * SHARE * VDIM + column;
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
            if (!bar_wait(bar, phase, failed)) { if (ok && lane == 0) atomicExch(status, code); ok = false; }
            __syncwarp();
            fence_after_sync();
        };
        auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(DT_ROWS) : "memory"); };
        auto largest = [&](int slot) {               // of what the column's threads have put there
            float top = tops[slot][0][column];
#pragma unroll
            for (int i = 1; i < DT_SHARES; ++i) top = fmaxf(top, tops[slot][i][column]);
            return top;
        };
        float S[SHARE], o[DT_TOKENS];
        uint64_t finite = 0ull;                      // becomes NaNs at the first number that is not finite
#pragma unroll
        for (int d = 0; d < SHARE; ++d) S[d] = (kept + (start & 1) * p.copy_floats)[(size_t)d * VDIM];
        float u_inv = 0.f, s_least = 0.f, u_least = 0.f;
        auto write_outputs = [&](int c) {            // what u gives the outputs of chunk c, behind what its state gave
            const float4* f4 = (const float4*)factors[c % 3];
            wait(&do_done, c & 1, 72);
            uint32_t v[DT_TOKENS / 16][16];
            load_columns<DT_TOKENS>(lanes + D_O + t0, v);
            tmem_wait_ld();
            if (c > 0) wait(&o_free, (c & 1) ^ 1, 75);           // the copies of the chunk before have read its outputs
            float smallest = INFINITY;               // of the column's outputs
#pragma unroll
            for (int t = 0; t < DT_TOKENS; t += 4) {
                const float4 fp = f4[(3 * DC_TOKENS + t0 + t) / 4];
                const uint64_t ps[2] = {pair_of(fp.x, fp.y), pair_of(fp.z, fp.w)};
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    const uint64_t sums = pair_of(__uint_as_float(v[(t + i) / 16][(t + i) % 16]), __uint_as_float(v[(t + i) / 16][(t + i) % 16 + 1]));
                    const uint64_t y = fma_pairs(sums, mul_pairs(pair_of(u_inv, u_inv), ps[i / 2]), pair_of(o[t + i], o[t + i + 1]));
                    float y0, y1;
                    halves_of(y, y0, y1);
                    smallest = min3(smallest, fabsf(y0), fabsf(y1));
                    finite = fma_pairs(y, 0ull, finite);
                    o_s[(t0 + t + i) * VDIM + column] = y0;
                    o_s[(t0 + t + i + 1) * VDIM + column] = y1;
                }
            }
            // Queries and pairs' weights are at most dim^(-1/2), so that what takes their scales off is at most 2^-17.  Where no column has
            // outputs that are all large enough by that: a token's row at a time; one before the first that is not zero may be of zeros.
            if (!__any_sync(0xffffffffu, smallest >= (s_least + u_least) * power_of_two(-17))) {
                const int first_token = first_rows[0][quarter] < DT_TOKENS ? first_rows[0][quarter] : DT_TOKENS + first_rows[1][quarter];
                for (int t = t0; t < t0 + DT_TOKENS; ++t) {
                    const float from_state = s_least * factors[c % 3][DC_TOKENS + t];
                    const float least = t < first_token ? from_state : fmaf(u_least, factors[c % 3][3 * DC_TOKENS + t], from_state);
                    if (!__any_sync(0xffffffffu, fabsf(o_s[t * VDIM + column]) >= least)) finite = pair_of(NAN, NAN);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&o_stored);
        };
        for (int c = 0; c < chunks; ++c) {
            const uint32_t phase = c & 1;
            const float4* f4 = (const float4*)factors[c % 3];            // W's, the queries' and the keys' factors, sixteen of four each
            float top[2] = {0.f, 0.f};
#pragma unroll
            for (int d = 0; d < SHARE; d += 2) top[d / 2 & 1] = max3(top[d / 2 & 1], fabsf(S[d]), fabsf(S[d + 1]));
            tops[0][share][column] = fmaxf(top[0], top[1]);
            meet();
            const float s_top = largest(0);
            const int s_exponent = parts_exponent(s_top);
            store_parts(S, power_of_two(s_exponent), lanes + S_HI + share * (SHARE / 2), lanes + S_LO + share * (SHARE / 2));
            tmem_wait_st();
            // the factors came with W: waited for before s_ready, behind which the next chunk's may come and end the barrier's next phase
            if (!bar_wait(&w_full, phase, failed)) ok = false;
            fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&s_ready);
            if (c > 0) write_outputs(c - 1);         // while W S is made

            // u of this thread's tokens
            wait(&d1w_done, phase, 69);
            const float s_inv = power_of_two(-s_exponent);
            uint32_t v[DT_TOKENS / 16][16];
            load_columns<DT_TOKENS>(lanes + D1_W + t0, v);
            float u[DT_TOKENS], uk[DT_TOKENS], u_top = 0.f, uk_top = 0.f;
            if (!bar_wait(&u_full, phase, failed)) ok = false;           // U'; the next chunk's comes behind u_ready
            __syncwarp();
#pragma unroll
            for (int t = 0; t < DT_TOKENS; ++t) u[t] = u_s[(t0 + t) * VDIM + column];
            tmem_wait_ld();
#pragma unroll
            for (int t = 0; t < DT_TOKENS; t += 4) {
                const float4 fw = f4[(t0 + t) / 4], fk = f4[(2 * DC_TOKENS + t0 + t) / 4];
                const float ws[4] = {fw.x, fw.y, fw.z, fw.w}, ks[4] = {fk.x, fk.y, fk.z, fk.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    u[t + i] = fmaf(-__uint_as_float(v[(t + i) / 16][(t + i) % 16]), s_inv * ws[i], u[t + i]);
                    uk[t + i] = u[t + i] * ks[i];
                }
                u_top = max3(u_top, fmaxf(fabsf(u[t]), fabsf(u[t + 1])), fmaxf(fabsf(u[t + 2]), fabsf(u[t + 3])));
                uk_top = max3(uk_top, fmaxf(fabsf(uk[t]), fabsf(uk[t + 1])), fmaxf(fabsf(uk[t + 2]), fabsf(uk[t + 3])));
            }
#pragma unroll
            for (int t = 0; t < DT_TOKENS; t += 2) finite = fma_pairs(pair_of(u[t], u[t + 1]), 0ull, finite);
            fence_before_sync();                                         // D1's columns are read before another share's parts go over them
            tops[1][share][column] = u_top;
            tops[2][share][column] = uk_top;
            meet();
            u_top = largest(1);
            const int u_exponent = parts_exponent(u_top), uk_exponent = parts_exponent(largest(2));
            fence_after_sync();
            store_parts(uk, power_of_two(uk_exponent), lanes + UK + t0 / 2, lanes + UK + 32 + t0 / 2);
            store_parts(u, power_of_two(u_exponent), lanes + D1_W + t0 / 2, lanes + D1_W + 32 + t0 / 2);
            tmem_wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&u_ready);
            u_inv = power_of_two(-u_exponent);
            s_least = PARTS_LEAST * warp_unit(s_top, s_exponent);
            u_least = PARTS_LEAST * warp_unit(u_top, u_exponent);
            const int first_here = first_row(u);
            if (lane == 0) first_rows[share][quarter] = first_here;              // read behind the next meeting, with the outputs

            // what the state gives the outputs, then the new state
            wait(&d1q_done, phase, 70);
            load_columns<DT_TOKENS>(lanes + D1_Q + t0, v);
            tmem_wait_ld();
#pragma unroll
            for (int t = 0; t < DT_TOKENS; t += 4) {
                const float4 fq = f4[(DC_TOKENS + t0 + t) / 4];
                const float qs[4] = {fq.x, fq.y, fq.z, fq.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) o[t + i] = __uint_as_float(v[(t + i) / 16][(t + i) % 16]) * (s_inv * qs[i]);
            }
            const float decay = factors[c % 3][4 * DC_TOKENS], uk_inv = power_of_two(-uk_exponent) * power_of_two(-DC_K_SCALE);
            wait(&ds_done, phase, 71);
            uint32_t fresh[SHARE / 16][16];
            load_columns<SHARE>(lanes + D_S + share * SHARE, fresh);
            tmem_wait_ld();
#pragma unroll
            for (int d = 0; d < SHARE; d += 2) {
                const uint64_t now = fma_pairs(pair_of(S[d], S[d + 1]), pair_of(decay, decay),
                                               mul_pairs(pair_of(__uint_as_float(fresh[d / 16][d % 16]), __uint_as_float(fresh[d / 16][d % 16 + 1])), pair_of(uk_inv, uk_inv)));
                halves_of(now, S[d], S[d + 1]);
            }
        }
        if (chunks > 0) {
            meet();
            write_outputs(chunks - 1);
        }
#pragma unroll
        for (int d = 0; d < SHARE; d += 2) finite = fma_pairs(pair_of(S[d], S[d + 1]), 0ull, finite);        // an earlier one reached the outputs
        float even, odd;
        halves_of(finite, even, odd);
        if (even != 0.f || odd != 0.f) odd_numbers = 1;
        meet();
        if (chunks > 0) {
            if (!odd_numbers && ok && !*failed) {
                float* to = kept + ((start + n_tok) & 1) * p.copy_floats;
#pragma unroll
                for (int d = 0; d < SHARE; ++d) to[(size_t)d * VDIM] = S[d];
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (failed_flag && warp == 0 && lane == 0) {
        // copies may still be on their way into this block's shared memory: give them a bounded time to land
        uint64_t* bars[5] = {&w_full, &q_full, &k_full, &pairs_full, &u_full};
        for (int i = 0; i < 5; ++i)
            for (uint32_t parity = 0; parity < 2; ++parity) { int zero = 0; bar_wait(bars[i], parity, &zero, 2000000); }
    }
    __syncthreads();
    if (warp == DT_WARPS + 1) tmem_free(tmem, 512);
    if (odd_numbers && !failed_flag && warp < DT_WARPS) dt_token_by_token<DIM>(p, b, h, (float*)w_s);       // over the outputs written, whose copies have ended
}

// The last launch.  A warp a (token, head): bound by reading o and the gate once.
template <int VDIM, typename OutT>
__global__ void __launch_bounds__(256) delta_chunk_finish_kernel(DeltaChunks p, int items) {
    constexpr int EACH = VDIM / 32;
    after_previous_kernel();
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
// heads * vdim floats; scratch: num_chunks * (heads * (64 (dim + vdim + 64 + 4) + 4) + 64 kv_heads (2 dim + 131)) floats.  status: one int on
// the device, zero before the call.
FRB_API int frb_delta_chunks(const float* conv, int conv_stride, int q_off, int k_off, int v_off, const float* proj, int proj_stride, int b_off,
                             int a_off, int g_off, const float* a_log, const float* dt_bias, const float* norm, const int* seq_slot,
                             const int* seq_start, const int* cu_q_len, float* state, long long copy_floats, long long state_offset, void* out,
                             int out_dtype, float* raw, int num_rows, int num_seqs, int heads, int kv_heads, int dim, int vdim, float eps,
                             const int* chunk_seq, const int* chunk_begin, const int* chunk_end, const int* seq_chunk0, int num_chunks,
                             float* scratch, int* status, cudaStream_t stream) {
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
    p.w_parts = (uint16_t*)p.w;
    p.pair_parts = (uint16_t*)p.pairs;
    p.factors = p.q_factor;
    p.q_parts = (uint16_t*)(p.factors + items * DC_FACTORS);
    p.k_parts = p.q_parts + (size_t)num_chunks * kv_heads * 2 * DC_TOKENS * dim;
    p.raw_pairs = (float*)(p.k_parts + (size_t)num_chunks * kv_heads * 2 * DC_TOKENS * dim);
    p.norms = p.raw_pairs + (size_t)num_chunks * kv_heads * 2 * DC_TOKENS * DC_TOKENS;
    p.conv_stride = conv_stride; p.q_off = q_off; p.k_off = k_off; p.v_off = v_off; p.proj_stride = proj_stride; p.b_off = b_off; p.a_off = a_off;
    p.g_off = g_off; p.heads = heads; p.kv_heads = kv_heads; p.eps = eps;
    const size_t one = (size_t)2 * DC_TOKENS * (dim + 8) * sizeof(float);
    const size_t two = (size_t)(2 * DC_TOKENS * (dim + 8) + DC_TOKENS * (dim + 4) + DC_TOKENS * DC_LM + (dim + DC_TOKENS) * (DC_SLICE + 4)) * sizeof(float);
    const dim3 chains(num_seqs, heads, vdim / DC_SLICE);
    const int rows_heads = num_rows * heads;
#define FRB_DELTA_CHUNKS(DIM, VDIM)                                                                                                  \
    do {                                                                                                                             \
        constexpr bool PARTS = VDIM == 128;                                                                                          \
        cudaFuncSetAttribute(delta_chunk_pairs_kernel<DIM, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)one);           \
        delta_chunk_pairs_kernel<DIM, PARTS><<<dim3(num_chunks, kv_heads), 256, one, stream>>>(p);                                   \
        launch_dependent_resident(2, delta_chunk_solve_kernel<DIM, VDIM, PARTS>, dim3(num_chunks, heads), dim3(256), 0, stream, p);  \
        if constexpr (PARTS) {                                                                                                       \
            const size_t tc = (size_t)(6 * DIM + 2 * DC_TOKENS + 4 * VDIM) * DC_TOKENS * 2 + 1024;                                   \
            cudaFuncSetAttribute(delta_chunk_chain_tc_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc);            \
            launch_dependent(delta_chunk_chain_tc_kernel<DIM>, dim3(num_seqs, heads), dim3(DT_THREADS), tc, stream, p, status);      \
        } else {                                                                                                                     \
            cudaFuncSetAttribute(delta_chunk_chain_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)two);              \
            launch_dependent(delta_chunk_chain_kernel<DIM>, chains, dim3(512), two, stream, p, vdim);                                \
        }                                                                                                                            \
        FRB_DISPATCH_DTYPE(out_dtype, OutT, {                                                                                        \
            launch_dependent_resident(8, delta_chunk_finish_kernel<VDIM, OutT>, dim3((rows_heads + 7) / 8), dim3(256), 0, stream, p, rows_heads); \
        });                                                                                                                          \
    } while (0)
    if (dim == 128 && vdim == 128) FRB_DELTA_CHUNKS(128, 128);
    else if (dim == 128) FRB_DELTA_CHUNKS(128, 64);
    else if (vdim == 128) FRB_DELTA_CHUNKS(64, 128);
    else FRB_DELTA_CHUNKS(64, 64);
#undef FRB_DELTA_CHUNKS
    FRB_RETURN_LAUNCH("delta_chunks");
}
