// The state-space scan of scans.cu for prompts, in chunks of 64 tokens.  Per head, with one decay a token and B, C shared by the heads of
// a group:
//
//     S <- a_t S + B_t (dt_t x_t)^T,   y_t = S^T C_t + D x_t,   a_t = exp(-exp(A_log) dt_t)          (S is [N, vdim])
//
// With w(j, i) the product of the decays of tokens j + 1 .. i of a chunk and u_j = dt_j x_j:
//   1. per chunk and group: the products C_i . B_j of its pairs j <= i, for all heads of the group, and the rows of B and C as parts;
//   2. per chunk and head: the decays, the pairs' weights P_ij = w(j, i) (C_i . B_j) as parts, the tokens' factors;
//   3. along the chunks, a block a (sequence, 128 columns of a group's values: two heads of 64 or one of 128): the state stays in
//      registers; y_i = w(start, i) (S^T C_i) + sum_(j <= i) P_ij u_j, S <- w(end) S + sum_j B_j (w(j, end) u_j)^T; then D x and the gate.
// A weight is the exponential of a sum of logarithms that has its tokens' alone, or a product of such factors: never a quotient, and no
// difference of two sums either, which behind one strong decay would have lost the digits of the mild ones.  The sums run over up to 16
// tokens inside a block and 48 between blocks: a rounding of their logarithms, which are large only where the weight is small.
//
// Everything is float32; launch 1's products run on mma.sync in TF32 parts (tf32_parts.cuh), sums of 16 entries, added in float32
// registers; launch 3's on tcgen05 in float16 parts (f16_parts.cuh), over at most 128 entries.
// Four prompts of 2,048 tokens, 64 heads of 128 x 64 in 8 groups: 45 + 44 + 180 us (45 + 45 + 178 without the look for outputs that may have lost
// digits), against 676 us of four launches on mma.sync with a state written and read for every chunk of 128 tokens (states 189, chain
// 65, outputs 382, pairs 40), and 1,210 token by token.
#include "f16_parts.cuh"
#include "silu.cuh"
#include "tf32_parts.cuh"

#define SC_CHUNK 128          // tokens of the callers' chunks: two of this file's
#define SC_TOKENS 64
#define SC_BLOCK 16
#define SC_BLOCKS (SC_TOKENS / SC_BLOCK)
#define SC_COLUMNS 128        // value columns of a block of launch 3
#define SC_FACTORS (4 * SC_TOKENS + 4)
#define SC_B_FAR 1048576.f    // 2^20: a new state is then off by less than 2^-24 of its columns' largest (64 products, 2^-50 each)

using namespace frb_tma;
using namespace frb_tc;

struct StateSpaceChunks {
    const float* proj;       // [T, proj_stride]: z of channel j at z_offset + j, dt of head h at dt_offset + h
    const float* xbc;        // [T, xbc_stride]: x of head h at h * vdim, B of group g at b_offset + g * N, C at c_offset + g * N
    const float *dt_bias, *a_log, *d;            // [heads]
    const int *seq_slot, *seq_start, *cu_q_len, *chunk_seq, *chunk_begin, *chunk_end, *seq_chunk0;
    float* state;            // [slots][2][copy_floats], this part's [heads][N][vdim] at state_offset
    long long copy_floats, state_offset;
    float* out;              // [T, heads * vdim]
    // of every half of a caller's chunk (a chunk here)
    uint16_t *c_parts, *b_parts;     // [chunk][group][part][N / 64][SC_TOKENS][64]: C's rows with a scale each, B's with one for the chunk
    uint16_t* pair_parts;    // [chunk][columns / 128][part][head of the columns][SC_TOKENS][SC_TOKENS]: P's rows with a scale each
    float* raw_pairs;        // [chunk][group][SC_TOKENS][SC_TOKENS]: C_i . B_j, j <= i
    float* scales;           // [chunk][group][SC_TOKENS + 4]: what takes the scales of C's rows off, and that of B (a NaN: no parts serve)
    float* factors;          // [chunk][head][SC_FACTORS]: w(start, i) and C's scale off; P's scales off; w(j, end); dt_j; w(end), B's scale off
    int proj_stride, z_offset, dt_offset, xbc_stride, b_offset, c_offset, heads, vdim, N, groups;

    __device__ __forceinline__ int tokens_of(int chunk) const {          // 0 or less: none
        const int item = chunk >> 1;
        return min(SC_TOKENS, chunk_end[item] - chunk_begin[item] - (chunk & 1) * SC_TOKENS);
    }
    __device__ __forceinline__ size_t row_of(int chunk) const {
        const int item = chunk >> 1;
        return (size_t)cu_q_len[chunk_seq[item]] + chunk_begin[item] + (chunk & 1) * SC_TOKENS;
    }
};

__device__ __forceinline__ float sc_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// Launch 1.  grid (chunk, group).  A warp takes a row tile of 16 and every other eight columns of the blocks up to it.
template <int N>
__global__ void __launch_bounds__(256, 2) state_space_pairs_kernel(StateSpaceChunks p) {
    constexpr int LC = N + 8, UNITS = SC_TOKENS * N / 8;
    extern __shared__ float4 sc_smem[];
    __shared__ float c_top[SC_TOKENS], b_top[SC_TOKENS];
    float* c_s = (float*)sc_smem;                   // [SC_TOKENS][LC]
    float* b_s = c_s + SC_TOKENS * LC;              // [SC_TOKENS][LC]
    const int chunk = blockIdx.x, g = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, count = p.tokens_of(chunk);
    const float* rows = p.xbc + p.row_of(chunk) * p.xbc_stride;
    const size_t at = (size_t)chunk * p.groups + g;
    for (int i = tid; i < 2 * SC_TOKENS * (N / 4); i += 256) {
        const int t = i / (N / 4) % SC_TOKENS, u = i % (N / 4);
        const bool is_b = i >= SC_TOKENS * (N / 4);
        float* to = (is_b ? b_s : c_s) + t * LC + 4 * u;
        if (t < count) copy16_async(to, rows + (size_t)t * p.xbc_stride + (is_b ? p.b_offset : p.c_offset) + g * N + 4 * u);
        else *(float4*)to = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    copies_commit();
    copies_wait<0>();
    __syncthreads();
    for (int t = warp; t < 2 * SC_TOKENS; t += 8) {
        const float* row = (t < SC_TOKENS ? c_s : b_s) + t % SC_TOKENS * LC;
        float top = 0.f;
#pragma unroll
        for (int n = 0; n < N; n += 32) top = fmaxf(top, fabsf(row[n + lane]));
        top = warp_max(top);
        if (lane == 0) (t < SC_TOKENS ? c_top : b_top)[t % SC_TOKENS] = top;
    }
    __syncthreads();
    // one scale for B: a row far larger than another would cost that one its digits
    const float b0 = b_top[lane], b1 = b_top[lane + 32], large = warp_max(fmaxf(b0, b1));
    const float least = -warp_max(-fminf(b0 > 0.f ? b0 : INFINITY, b1 > 0.f ? b1 : INFINITY));
    const int b_exponent = parts_exponent(large);
    if (tid < SC_TOKENS) p.scales[at * (SC_TOKENS + 4) + tid] = c_top[tid] > 0.f ? power_of_two(-parts_exponent(c_top[tid])) : 0.f;
    if (tid == 0) p.scales[at * (SC_TOKENS + 4) + SC_TOKENS] = least * SC_B_FAR < large ? NAN : power_of_two(-b_exponent);
    for (int u = tid; u < 2 * UNITS; u += 256) {
        const bool is_b = u >= UNITS;
        const int r = u % UNITS / (N / 8), c = u % (N / 8) * 8;
        const float* from = (is_b ? b_s : c_s) + r * LC + c;
        const float scale = power_of_two(is_b ? b_exponent : parts_exponent(c_top[r]));
        uint4 hi, lo;
        split_four(*(const float4*)from, scale, hi.x, hi.y, lo.x, lo.y);
        split_four(*(const float4*)(from + 4), scale, hi.z, hi.w, lo.z, lo.w);
        uint16_t* parts = (is_b ? p.b_parts : p.c_parts) + at * 2 * SC_TOKENS * N + piece_place(r, c);
        *(uint4*)parts = hi;
        *(uint4*)(parts + SC_TOKENS * N) = lo;
    }
    const int tile = warp & 3, odd = warp >> 2;
    float acc[SC_BLOCKS][4] = {};
#pragma unroll 2
    for (int k = 0; k < N; k += 16) {
        Tf32Parts a[2][1][4], bb[2][1][2];
#pragma unroll
        for (int r = 0; r < 2; ++r) a_along(a[r][0], c_s + tile * SC_BLOCK * LC + k + 8 * r, LC, lane);
#pragma unroll
        for (int n = 0; n < SC_BLOCKS; ++n) {
            if (n > tile) break;
#pragma unroll
            for (int r = 0; r < 2; ++r) b_along(bb[r][0], b_s + (n * SC_BLOCK + 8 * odd) * LC + k + 8 * r, LC, lane);
            float t[1][1][4];
            mma_runs(t, a, bb);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] += t[0][0][e];
        }
    }
    float* out = p.raw_pairs + at * SC_TOKENS * SC_TOKENS + (tile * SC_BLOCK + (lane >> 2)) * SC_TOKENS + 8 * odd + 2 * (lane & 3);
#pragma unroll
    for (int n = 0; n < SC_BLOCKS; ++n)
        if (n <= tile) {
            *(float2*)(out + n * SC_BLOCK) = make_float2(acc[n][0], acc[n][1]);
            *(float2*)(out + n * SC_BLOCK + 8 * SC_TOKENS) = make_float2(acc[n][2], acc[n][3]);
        }
}

// Launch 2.  grid (chunk, head), 128 threads: bound by reading the group's pairs and writing the head's parts once.
__global__ void __launch_bounds__(128) state_space_weights_kernel(StateSpaceChunks p) {
    __shared__ float log_s[SC_TOKENS], to_s[SC_TOKENS], from_s[SC_TOKENS], step_s[SC_TOKENS];
    __shared__ float block_log[SC_BLOCKS], between[SC_BLOCKS][SC_BLOCKS];
    __shared__ __align__(16) float own[SC_TOKENS][SC_BLOCK + 4];         // w(j, i) of the tokens j of i's block; zero for later ones
    const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, g = h / (p.heads / p.groups), count = p.tokens_of(chunk);
    const size_t row0 = p.row_of(chunk);
    float* factors = p.factors + ((size_t)chunk * p.heads + h) * SC_FACTORS;
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
        to_s[tid] = expf(before);
        from_s[tid] = expf(tail);
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
        for (int j = 0; j < SC_BLOCK; j += 4) *(float4*)&own[tid][j] = make_float4(row[j], row[j + 1], row[j + 2], row[j + 3]);
    } else {
        const int t = tid - SC_TOKENS;
        if (t < SC_BLOCKS * SC_BLOCKS) {             // the whole blocks between two
            const int i = t / SC_BLOCKS, j = t % SC_BLOCKS;
            float sum = 0.f;
            for (int m = j + 1; m < i; ++m) sum += block_log[m];
            between[i][j] = expf(sum);
        }
        float sum = 0.f, rest = 0.f;
        for (int m = 0; m < t / SC_BLOCK; ++m) sum += block_log[m];
        for (int m = t / SC_BLOCK + 1; m < SC_BLOCKS; ++m) rest += block_log[m];
        const float* scales = p.scales + ((size_t)chunk * p.groups + g) * (SC_TOKENS + 4);
        const float start = expf(sum) * to_s[t];
        factors[t] = start * scales[t];
        factors[2 * SC_TOKENS + t] = from_s[t] * expf(rest);
        factors[3 * SC_TOKENS + t] = step_s[t];
        if (t == SC_TOKENS - 1) {
            factors[4 * SC_TOKENS] = start;
            factors[4 * SC_TOKENS + 1] = scales[SC_TOKENS];
        }
    }
    __syncthreads();
    // eight entries of a row of P at a time; eight neighbouring threads have a row
    const int heads_here = SC_COLUMNS / p.vdim;
    const float* raw = p.raw_pairs + ((size_t)chunk * p.groups + g) * SC_TOKENS * SC_TOKENS;
    uint16_t* parts = p.pair_parts + ((size_t)chunk * (p.heads / heads_here) + h / heads_here) * 2 * heads_here * SC_TOKENS * SC_TOKENS
                      + (h % heads_here) * SC_TOKENS * SC_TOKENS;
#pragma unroll
    for (int u = tid; u < SC_TOKENS * SC_TOKENS / 8; u += 128) {
        const int i = u / (SC_TOKENS / 8), j0 = u % (SC_TOKENS / 8) * 8, ib = i / SC_BLOCK, jb = j0 / SC_BLOCK;
        float y[8] = {}, top = 0.f;
        if (j0 <= i) {
            const float4 a = *(const float4*)(raw + i * SC_TOKENS + j0), c = *(const float4*)(raw + i * SC_TOKENS + j0 + 4);
            const float r[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (j0 + e <= i) {
                    y[e] = r[e] * (jb < ib ? to_s[i] * (between[ib][jb] * from_s[j0 + e]) : own[i][(j0 + e) % SC_BLOCK]);
                    top = fmaxf(top, fabsf(y[e]));
                }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const int exponent = parts_exponent(top);
        if (j0 == 0) factors[SC_TOKENS + i] = top > 0.f ? power_of_two(-exponent) : 0.f;
        uint4 hi, lo;
        split_four(make_float4(y[0], y[1], y[2], y[3]), power_of_two(exponent), hi.x, hi.y, lo.x, lo.y);
        split_four(make_float4(y[4], y[5], y[6], y[7]), power_of_two(exponent), hi.z, hi.w, lo.z, lo.w);
        uint16_t* to = parts + piece_place(i, j0);
        *(uint4*)to = hi;
        *(uint4*)(to + heads_here * SC_TOKENS * SC_TOKENS) = lo;
    }
}

// Launch 3.  grid (sequence, columns / 128): a lane of tensor memory is a value column; two threads have half of its N state entries
// each, in float32, and half of a chunk's tokens.  The products of parts of a chunk:
//     DS = (u w(j, end))^T B   128 x N x 64, B's rows N-major;    D1 = S^T C^T   128 x 64 x N;    DO = u^T P^T   128 x 64 x 64, with two heads
//     128 x 64 x 128: a head's columns have u in their half of the inner size and zeros in the other's.
// The columns' parts have a power of two of their own each, from the largest entry of the state, of u or of u w(j, end).  Eight more warps take the
// outputs through D x and the gate while the next chunk is made: with these in the columns' warps a chunk took 4,000 cycles more.  A chunk is
// bound by the instructions of both, 9,000 to 10,000 cycles: the columns' splits 1,900, u 1,300, the waits for the products 1,900, the
// outputs' gates 4,000.  A number that is not finite, a token whose sums may have lost digits (PARTS_LEAST), or a chunk whose rows of B
// lie 2^20 apart makes the block take its columns of the sequence again, token by token.
#define ST_THREADS 640         // warps 0 copies, 1 products; 4-11 the columns' two halves (w & 3: lanes), 12-19 the outputs
#define ST_ROWS 256
#define ST_SHARE_TOKENS (SC_TOKENS / 2)
// registers a thread: at launch, and of each group of warps after it (their sum over the threads is below the launch's)
#define ST_REGS_LAUNCH 96
#define ST_REGS_ISSUE 40
#define ST_REGS_ROWS 152
#define ST_REGS_OUTPUTS 64
static_assert(128 * ST_REGS_ISSUE + ST_ROWS * (ST_REGS_ROWS + ST_REGS_OUTPUTS) <= ST_THREADS * ST_REGS_LAUNCH, "registers of the groups");

// A sequence's columns token by token, by the columns' threads, two a column, each with half of its state.  tid: among those threads;
// column0: the block's first; room: shared memory for the rows of 32 tokens and the threads' sums.  Bound by
// the reads of B and C from there: a token takes 1.3 us (one thread a column, its state spilled, the rows fetched token by token: 6.9 us).
template <int N>
static __device__ __forceinline__ void st_token_by_token(const StateSpaceChunks& p, int b, int column0, int tid, float* room, volatile int* failed) {
    constexpr int SHARE = N / 2, BATCH = 32;
    float *b_s = room, *c_s = b_s + BATCH * N, *x_s = c_s + BATCH * N, *z_s = x_s + BATCH * SC_COLUMNS;
    float2* steps = (float2*)(z_s + BATCH * SC_COLUMNS);                          // [token][head of the block]: the step, the decay less one
    float* sums = (float*)(steps + 2 * BATCH);                           // [token & 1][share][column]
    const int share = tid / SC_COLUMNS, column = column0 + tid % SC_COLUMNS, h0 = column0 / p.vdim, h = column / p.vdim;
    const int g = h / (p.heads / p.groups), heads_here = SC_COLUMNS / p.vdim;
    auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(ST_ROWS) : "memory"); };
    const int start = p.seq_start[b], count = p.cu_q_len[b + 1] - p.cu_q_len[b], at = tid % SC_COLUMNS;
    const size_t row0 = p.cu_q_len[b];
    float* state = p.state + (size_t)p.seq_slot[b] * 2 * p.copy_floats + p.state_offset + ((size_t)h * N + share * SHARE) * p.vdim + column % p.vdim;
    const float* from = state + (start & 1) * p.copy_floats;
    float* to = state + ((start + count) & 1) * p.copy_floats;
    const float dskip = p.d[h];
    uint64_t S[SHARE / 2];
#pragma unroll
    for (int n = 0; n < SHARE / 2; ++n) S[n] = pair_of(from[(size_t)(2 * n) * p.vdim], from[(size_t)(2 * n + 1) * p.vdim]);
    for (int t0 = 0; t0 < count; t0 += BATCH) {
        const int here = min(BATCH, count - t0);
        meet();                                      // nobody reads the rows before any more
        for (int t = share; t < here; t += 2) {
            x_s[t * SC_COLUMNS + at] = p.xbc[(row0 + t0 + t) * p.xbc_stride + column];
            z_s[t * SC_COLUMNS + at] = p.proj[(row0 + t0 + t) * p.proj_stride + p.z_offset + column];
        }
        for (int i = tid; i < here * (2 * N / 4); i += ST_ROWS) {
            const int t = i / (2 * N / 4), u = i % (2 * N / 4);
            const bool is_b = u < N / 4;
            const float* row = p.xbc + (row0 + t0 + t) * p.xbc_stride + (is_b ? p.b_offset : p.c_offset) + g * N + 4 * (u % (N / 4));
            *(float4*)((is_b ? b_s : c_s) + t * N + 4 * (u % (N / 4))) = *(const float4*)row;
        }
        if (tid < 2 * BATCH && tid / 2 < here && tid % 2 < heads_here) {
            const int hh = h0 + tid % 2;
            const float step = sc_softplus(p.proj[(row0 + t0 + tid / 2) * p.proj_stride + p.dt_offset + hh] + p.dt_bias[hh]);
            steps[tid] = make_float2(step, expm1f(-expf(p.a_log[hh]) * step));
        }
        meet();
        for (int t = 0; t < here; ++t) {
            const float2 f = steps[2 * t + h - h0];
            const ulonglong2 *b2 = (const ulonglong2*)(b_s + t * N + share * SHARE), *c2 = (const ulonglong2*)(c_s + t * N + share * SHARE);
            const float x = x_s[t * SC_COLUMNS + at];
            const uint64_t less_one = pair_of(f.y, f.y), u = pair_of(f.x * x, f.x * x);
            uint64_t y[2] = {0ull, 0ull};
#pragma unroll
            for (int n = 0; n < SHARE / 4; ++n) {
                const ulonglong2 b = b2[n], c = c2[n];
                S[2 * n] = fma_pairs(b.x, u, fma_pairs(less_one, S[2 * n], S[2 * n]));
                S[2 * n + 1] = fma_pairs(b.y, u, fma_pairs(less_one, S[2 * n + 1], S[2 * n + 1]));
                y[0] = fma_pairs(S[2 * n], c.x, y[0]);
                y[1] = fma_pairs(S[2 * n + 1], c.y, y[1]);
            }
            float even, odd;
            halves_of(add_pairs(y[0], y[1]), even, odd);
            float* told = sums + (t & 1) * 2 * SC_COLUMNS + at;
            told[share * SC_COLUMNS] = even + odd;
            meet();
            if (share == 0) {
                const float z = z_s[t * SC_COLUMNS + at];
                p.out[(row0 + t0 + t) * ((size_t)p.heads * p.vdim) + column] = fmaf(dskip, x, told[0] + told[SC_COLUMNS]) * (z / (1.0f + expf(-z)));
            }
        }
    }
    if (*failed) return;
#pragma unroll
    for (int n = 0; n < SHARE / 2; ++n) {
        float even, odd;
        halves_of(S[n], even, odd);
        to[(size_t)(2 * n) * p.vdim] = even;
        to[(size_t)(2 * n + 1) * p.vdim] = odd;
    }
}

template <int N, bool TWO>
__global__ void __launch_bounds__(ST_THREADS, 1) state_space_chain_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ StateSpaceChunks p, int* __restrict__ status) {
    constexpr int SHARE = N / 2, HEADS = TWO ? 2 : 1, UK = HEADS * SC_TOKENS;        // UK: columns of u's parts
    constexpr uint32_t ROWS_PART = SC_TOKENS * N * 2, PAIR_PART = HEADS * SC_TOKENS * SC_TOKENS * 2, X_BYTES = SC_TOKENS * SC_COLUMNS * 4;
    // tensor memory: the state's parts, later DO over their first columns; D1; u's parts; those of u w(j, end); DS
    constexpr int S_HI = 0, S_LO = N / 2, D_O = 0, D_1 = 128, U_HI = 192, U_LO = U_HI + UK / 2, UE_HI = 320, UE_LO = 352, D_S = 384;
    extern __shared__ uint8_t st_smem[];
    __shared__ uint64_t x_full, b_full, c_full, pairs_full, ready, d1_done, ds_done, do_done, o_stored, o_free[2];
    __shared__ float tops[3][2][SC_COLUMNS];
    __shared__ int first_rows[2][4];
    __shared__ __align__(16) float factors[2][HEADS][SC_FACTORS];
    __shared__ uint32_t tmem_slot;
    __shared__ int failed_flag, odd_numbers;
    volatile int* failed = &failed_flag;
    uint8_t* c_s = (uint8_t*)(((uintptr_t)st_smem + 1023) & ~(uintptr_t)1023);
    uint8_t* b_s = c_s + 2 * ROWS_PART;
    uint8_t* pairs_s = b_s + 2 * ROWS_PART;
    float* x_s = (float*)(pairs_s + 2 * PAIR_PART);                      // [chunk & 1][SC_TOKENS][SC_COLUMNS]
    float* o_s = x_s + 2 * SC_TOKENS * SC_COLUMNS;                       // of S^T C + sum P u
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int b = blockIdx.x, block = blockIdx.y, column0 = block * SC_COLUMNS, h0 = column0 / p.vdim, g = h0 / (p.heads / p.groups);
    const int first = 2 * p.seq_chunk0[b], last = p.seq_chunk0[b + 1], start = p.seq_start[b], n_tok = p.cu_q_len[b + 1] - p.cu_q_len[b];
    int chunks = 2 * last - first;
    if (chunks > 0 && p.tokens_of(first + chunks - 1) <= 0) --chunks;
    chunks = __shfl_sync(0xffffffffu, chunks, 0);

    if (threadIdx.x == 0) {
        bar_init(&x_full, 1); bar_init(&b_full, 1); bar_init(&c_full, 1); bar_init(&pairs_full, 1); bar_init(&ready, ST_ROWS / 32);
        bar_init(&d1_done, 1); bar_init(&ds_done, 1); bar_init(&do_done, 1); bar_init(&o_stored, ST_ROWS / 32); bar_init(&o_free[0], ST_ROWS / 32); bar_init(&o_free[1], ST_ROWS / 32);
        failed_flag = 0;
        odd_numbers = 0;
        bar_init_fence();
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 512);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    after_previous_kernel();                         // barriers and tensor memory were set up while it still ran

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ST_REGS_ISSUE));
        if (warp == 0) {
            for (int c = 0; c < chunks; ++c) {
                const int chunk = first + c;
                const uint32_t before = (c & 1) ^ 1;                     // of the phase that the chunk before has ended
                const size_t group_at = (size_t)chunk * p.groups + g, factor_bytes = HEADS * SC_FACTORS * 4;
                if (c && !warp_wait(&ready, before, failed)) { if (lane == 0) atomicExch(status, 81); break; }
                if (c > 1 && !warp_wait(&o_free[c & 1], (c >> 1 & 1) ^ 1, failed)) { if (lane == 0) atomicExch(status, 92); break; }
                if (lane == 0) {
                    bar_expect(&x_full, X_BYTES + factor_bytes);
                    load_2d(x_s + (c & 1) * SC_TOKENS * SC_COLUMNS, &map_x, column0, (int)p.row_of(chunk), &x_full);
                    copy_bulk(factors[c & 1], p.factors + ((size_t)chunk * p.heads + h0) * SC_FACTORS, factor_bytes, &x_full);
                }
                if (c && !warp_wait(&ds_done, before, failed)) { if (lane == 0) atomicExch(status, 82); break; }
                if (lane == 0) {
                    bar_expect(&b_full, 2 * ROWS_PART);
                    copy_bulk(b_s, p.b_parts + group_at * 2 * SC_TOKENS * N, 2 * ROWS_PART, &b_full);
                }
                if (c && !warp_wait(&d1_done, before, failed)) { if (lane == 0) atomicExch(status, 83); break; }
                if (lane == 0) {
                    bar_expect(&c_full, 2 * ROWS_PART);
                    copy_bulk(c_s, p.c_parts + group_at * 2 * SC_TOKENS * N, 2 * ROWS_PART, &c_full);
                }
                if (c && !warp_wait(&do_done, before, failed)) { if (lane == 0) atomicExch(status, 84); break; }
                if (lane == 0) {
                    bar_expect(&pairs_full, 2 * PAIR_PART);
                    copy_bulk(pairs_s, p.pair_parts + ((size_t)chunk * gridDim.y + block) * 2 * HEADS * SC_TOKENS * SC_TOKENS, 2 * PAIR_PART, &pairs_full);
                }
                __syncwarp();
            }
        } else if (warp == 1) {
            // the whole warp goes through the loop (elect_one, tcgen05.cuh); its products run in the order of their issue, so DO may be
            // asked for over the state's parts, which D1 has read
            constexpr uint32_t idesc64 = (1u << 4) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(SC_COLUMNS >> 4) << 24);
            constexpr uint32_t idesc_b = (1u << 4) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(SC_COLUMNS >> 4) << 24);
            const uint64_t c_at = tile_desc(smem_addr(c_s)), pairs_at = tile_desc(smem_addr(pairs_s)), b_at = desc_n_major(smem_addr(b_s));
            auto along = [](int k) { return (k / 4) * (SC_TOKENS * 128 >> 4) + (k % 4) * 2; };
            for (int c = 0; c < chunks; ++c) {
                const uint32_t phase = c & 1;
                if (!warp_wait_both(&ready, phase, &b_full, phase, failed)) { if (lane == 0) atomicExch(status, 85); break; }
                fence_after_sync();
                if (elect_one()) {
                    products_of_parts<SC_TOKENS / 16>(tmem + D_S, tmem + UE_HI, tmem + UE_LO, b_at, b_at + (ROWS_PART >> 4), idesc_b,
                                                      [](int k) { return k * (16 * 128 >> 4); });
                    mma_commit(&ds_done);
                }
                __syncwarp();
                if (!warp_wait(&c_full, phase, failed)) { if (lane == 0) atomicExch(status, 86); break; }
                fence_after_sync();
                if (elect_one()) {
                    products_of_parts<N / 16>(tmem + D_1, tmem + S_HI, tmem + S_LO, c_at, c_at + (ROWS_PART >> 4), idesc64, along);
                    mma_commit(&d1_done);
                }
                __syncwarp();
                if (!warp_wait(&pairs_full, phase, failed)) { if (lane == 0) atomicExch(status, 87); break; }
                fence_after_sync();
                if (elect_one()) {
                    products_of_parts<UK / 16>(tmem + D_O, tmem + U_HI, tmem + U_LO, pairs_at, pairs_at + (PAIR_PART >> 4), idesc64, along);
                    mma_commit(&do_done);
                }
                __syncwarp();
            }
        }
    } else if (warp < 12) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ST_REGS_ROWS));
        // A wait that gives up does not end the loop: the block's later waits then return at once, and every thread reaches the barriers.
        const int share = (warp - 4) >> 2, quarter = warp & 3, column = quarter * 32 + lane, t0 = ST_SHARE_TOKENS * share;
        const int hh = TWO ? quarter >> 1 : 0;       // the column's head among the block's
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        const size_t state_at = p.state_offset + ((size_t)(h0 + hh) * N + share * SHARE) * p.vdim + column % p.vdim;
        float* kept = p.state + (size_t)p.seq_slot[b] * 2 * p.copy_floats + state_at;
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
            if (!bar_wait(bar, phase, failed)) { if (ok && lane == 0) atomicExch(status, code); ok = false; }
            __syncwarp();
            fence_after_sync();
        };
        auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(ST_ROWS) : "memory"); };
        float S[SHARE];
        uint64_t finite = 0ull;                      // becomes NaNs at the first number that is not finite
#pragma unroll
        for (int n = 0; n < SHARE; ++n) S[n] = (kept + (start & 1) * p.copy_floats)[(size_t)n * p.vdim];
        if (TWO) {                                   // the other head's half of the inner size: zeros for good
            const uint32_t zeros[16] = {};
            tmem_st16(lanes + U_HI + (hh ^ 1) * 32 + 16 * share, zeros);
            tmem_st16(lanes + U_LO + (hh ^ 1) * 32 + 16 * share, zeros);
        }
        for (int c = 0; c < chunks; ++c) {
            const uint32_t phase = c & 1;
            const float4* f4 = (const float4*)factors[c & 1][hh];        // sixteen of four each: D1's, DO's, w(j, end), dt
            const int count = p.tokens_of(first + c);
            wait(&x_full, phase, 88);                // and the factors; what they overwrite was used before the chunk before was ready
            float u[ST_SHARE_TOKENS], u_top = 0.f, ue_top = 0.f, s_top = 0.f;
#pragma unroll
            for (int t = 0; t < ST_SHARE_TOKENS; ++t) u[t] = x_s[((c & 1) * SC_TOKENS + t0 + t) * SC_COLUMNS + column];
#pragma unroll
            for (int t = 0; t < ST_SHARE_TOKENS; t += 4) {
                const float4 f = f4[(3 * SC_TOKENS + t0 + t) / 4];
                halves_of(mul_pairs(pair_of(u[t], u[t + 1]), pair_of(f.x, f.y)), u[t], u[t + 1]);
                halves_of(mul_pairs(pair_of(u[t + 2], u[t + 3]), pair_of(f.z, f.w)), u[t + 2], u[t + 3]);
            }
            if (t0 + ST_SHARE_TOKENS > count) {      // behind the last token are other rows
#pragma unroll
                for (int t = 0; t < ST_SHARE_TOKENS; ++t)
                    if (t0 + t >= count) u[t] = 0.f;
            }
#pragma unroll
            for (int t = 0; t < ST_SHARE_TOKENS; t += 4) {
                const float4 fe = f4[(2 * SC_TOKENS + t0 + t) / 4];
                u_top = max3(max3(u_top, fabsf(u[t]), fabsf(u[t + 1])), fabsf(u[t + 2]), fabsf(u[t + 3]));
                float e[4];
                halves_of(mul_pairs(pair_of(u[t], u[t + 1]), pair_of(fe.x, fe.y)), e[0], e[1]);
                halves_of(mul_pairs(pair_of(u[t + 2], u[t + 3]), pair_of(fe.z, fe.w)), e[2], e[3]);
                ue_top = max3(max3(ue_top, fabsf(e[0]), fabsf(e[1])), fabsf(e[2]), fabsf(e[3]));
            }
#pragma unroll
            for (int n = 0; n < SHARE; n += 2) s_top = max3(s_top, fabsf(S[n]), fabsf(S[n + 1]));
            tops[0][share][column] = s_top;
            tops[1][share][column] = u_top;
            tops[2][share][column] = ue_top;
            const int first_here = first_row(u);
            if (lane == 0) first_rows[share][quarter] = first_here;
            fence_before_sync();                     // DO's columns are read before the state's parts go over them
            meet();
            fence_after_sync();
            s_top = fmaxf(tops[0][0][column], tops[0][1][column]);
            u_top = fmaxf(tops[1][0][column], tops[1][1][column]);
            const int s_exponent = parts_exponent(s_top), u_exponent = parts_exponent(u_top);
            const int ue_exponent = parts_exponent(fmaxf(tops[2][0][column], tops[2][1][column]));
            const float s_least = PARTS_LEAST * warp_unit(s_top, s_exponent), u_least = PARTS_LEAST * warp_unit(u_top, u_exponent);
            const int first_token = first_rows[0][quarter] < ST_SHARE_TOKENS ? first_rows[0][quarter] : ST_SHARE_TOKENS + first_rows[1][quarter];
            store_parts(S, power_of_two(s_exponent), lanes + S_HI + share * (SHARE / 2), lanes + S_LO + share * (SHARE / 2));
            store_parts(u, power_of_two(u_exponent), lanes + U_HI + hh * 32 + t0 / 2, lanes + U_LO + hh * 32 + t0 / 2);
#pragma unroll
            for (int t = 0; t < ST_SHARE_TOKENS; t += 4) {
                const float4 fe = f4[(2 * SC_TOKENS + t0 + t) / 4];
                halves_of(mul_pairs(pair_of(u[t], u[t + 1]), pair_of(fe.x, fe.y)), u[t], u[t + 1]);
                halves_of(mul_pairs(pair_of(u[t + 2], u[t + 3]), pair_of(fe.z, fe.w)), u[t + 2], u[t + 3]);
            }
            store_parts(u, power_of_two(ue_exponent), lanes + UE_HI + t0 / 2, lanes + UE_LO + t0 / 2);
            tmem_wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&ready);

            // the new state, then the outputs
            const float decay = factors[c & 1][hh][4 * SC_TOKENS], s_inv = power_of_two(-s_exponent), u_inv = power_of_two(-u_exponent);
            const float ue_inv = power_of_two(-ue_exponent) * factors[c & 1][hh][4 * SC_TOKENS + 1];
            wait(&ds_done, phase, 89);
#pragma unroll
            for (int n0 = 0; n0 < SHARE; n0 += 32) {
                uint32_t v[2][16];
                load_columns<32>(lanes + D_S + share * SHARE + n0, v);
                tmem_wait_ld();
#pragma unroll
                for (int n = 0; n < 32; n += 2) {
                    const uint64_t now = fma_pairs(pair_of(S[n0 + n], S[n0 + n + 1]), pair_of(decay, decay),
                                                   mul_pairs(pair_of(__uint_as_float(v[n / 16][n % 16]), __uint_as_float(v[n / 16][n % 16 + 1])), pair_of(ue_inv, ue_inv)));
                    halves_of(now, S[n0 + n], S[n0 + n + 1]);
                }
            }
            uint32_t v[2][16];
            uint64_t o[ST_SHARE_TOKENS / 2];
            auto sums_at = [&](int t) { return pair_of(__uint_as_float(v[t / 16][t % 16]), __uint_as_float(v[t / 16][t % 16 + 1])); };
            wait(&d1_done, phase, 90);
            load_columns<32>(lanes + D_1 + t0, v);
            tmem_wait_ld();
#pragma unroll
            for (int t = 0; t < ST_SHARE_TOKENS; t += 4) {
                const float4 f = f4[(t0 + t) / 4];
                const uint64_t fs[2] = {pair_of(f.x, f.y), pair_of(f.z, f.w)};
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    o[t / 2 + i] = mul_pairs(sums_at(t + 2 * i), mul_pairs(pair_of(s_inv, s_inv), fs[i]));
            }
            wait(&do_done, phase, 91);
            load_columns<32>(lanes + D_O + t0, v);
            tmem_wait_ld();
            if (c > 0) wait(&o_free[phase ^ 1], (c - 1) >> 1 & 1, 92);       // the chunk before has been read
            float spare = INFINITY;                  // by how much the column's sums exceed the least that holds its digits
#pragma unroll
            for (int t = 0; t < ST_SHARE_TOKENS; t += 4) {
                const float4 f = f4[(SC_TOKENS + t0 + t) / 4], g4 = f4[(t0 + t) / 4];
                const uint64_t fs[2] = {pair_of(f.x, f.y), pair_of(f.z, f.w)}, gs[2] = {pair_of(g4.x, g4.y), pair_of(g4.z, g4.w)};
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint64_t y = fma_pairs(sums_at(t + 2 * i), mul_pairs(pair_of(u_inv, u_inv), fs[i]), o[t / 2 + i]);
                    finite = fma_pairs(y, 0ull, finite);
                    float y0, y1, least0, least1;
                    halves_of(y, y0, y1);
                    halves_of(fma_pairs(pair_of(s_least, s_least), gs[i], mul_pairs(pair_of(u_least, u_least), fs[i])), least0, least1);
                    spare = min3(spare, fabsf(y0) - least0, fabsf(y1) - least1);
                    o_s[(t0 + t + 2 * i) * SC_COLUMNS + column] = y0;
                    o_s[(t0 + t + 2 * i + 1) * SC_COLUMNS + column] = y1;
                }
            }
            // no column whose sums all do: a token's row at a time; one before the first that is not zero may be of zeros
            if (!__any_sync(0xffffffffu, spare >= 0.f)) {
                for (int t = 0; t < ST_SHARE_TOKENS; ++t) {
                    const float y = fabsf(o_s[(t0 + t) * SC_COLUMNS + column]), from_state = s_least * factors[c & 1][hh][t0 + t];
                    const float least = t0 + t < first_token ? from_state : fmaf(u_least, factors[c & 1][hh][SC_TOKENS + t0 + t], from_state);
                    if (!__any_sync(0xffffffffu, y >= least)) finite = pair_of(NAN, NAN);
                }
            }
            __syncwarp();
            if (lane == 0) bar_arrive(&o_stored);
        }
#pragma unroll
        for (int n = 0; n < SHARE; n += 2) finite = fma_pairs(pair_of(S[n], S[n + 1]), 0ull, finite);        // an earlier one reached the outputs
        float even, odd;
        halves_of(finite, even, odd);
        if (even != 0.f || odd != 0.f) odd_numbers = 1;
        meet();
        if (chunks > 0 && odd_numbers) {
            // over the outputs written, of which the last have been by then; in the place of the last chunk's operands (inlined: these warps'
            // registers hold the state)
            wait(&o_free[(chunks - 1) & 1], (chunks - 1) >> 1 & 1, 92);
            st_token_by_token<N>(p, b, column0, threadIdx.x - 128, (float*)c_s, failed);
        } else if (chunks > 0 && ok && !*failed) {
            float* to = kept + ((start + n_tok) & 1) * p.copy_floats;
#pragma unroll
            for (int n = 0; n < SHARE; ++n) to[(size_t)n * p.vdim] = S[n];
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ST_REGS_OUTPUTS));
        // a thread two columns of every fourth token; z is asked for into L2 a chunk ahead
        const int tid = threadIdx.x - 384, column = column0 + 2 * (tid & 63), t0 = tid >> 6;
        const float dskip = p.d[column / p.vdim];
        auto z_of = [&](int chunk, int t) { return p.proj + (p.row_of(chunk) + t) * p.proj_stride + p.z_offset; };
        float gates[2][16];
        auto load = [&](int c, int half) {
            const int count = p.tokens_of(first + c);
            const float* z = z_of(first + c, t0) + column;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int t = half * (SC_TOKENS / 2) + 4 * k;
                float2 v = make_float2(0.f, 0.f);
                if (t0 + t < count) v = *(const float2*)(z + (size_t)t * p.proj_stride);
                gates[half][2 * k] = v.x;
                gates[half][2 * k + 1] = v.y;
            }
        };
        if (chunks > 0) load(0, 0);
        for (int c = 0; c < chunks; ++c) {
            const int count = p.tokens_of(first + c);
            float* out = p.out + (p.row_of(first + c) + t0) * ((size_t)p.heads * p.vdim) + column;
            const float* sums = o_s + t0 * SC_COLUMNS + 2 * (tid & 63);
            const float* x = x_s + ((c & 1) * SC_TOKENS + t0) * SC_COLUMNS + 2 * (tid & 63);
            if (c + 1 < chunks && (tid >> 2) < p.tokens_of(first + c + 1))
                asm volatile("prefetch.global.L2 [%0];" ::"l"(z_of(first + c + 1, tid >> 2) + column0 + 32 * (tid & 3)));
            auto write = [&](int half) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int t = half * (SC_TOKENS / 2) + 4 * k;
                    const float2 o = *(const float2*)(sums + t * SC_COLUMNS), xs = *(const float2*)(x + t * SC_COLUMNS);
                    const float2 y = make_float2(fmaf(dskip, xs.x, o.x) * gates[half][2 * k], fmaf(dskip, xs.y, o.y) * gates[half][2 * k + 1]);
                    if (t0 + t < count) *(float2*)(out + (size_t)t * p.heads * p.vdim) = y;
                }
            };
            silu_of(gates[0]);
            load(c, 1);
            if (!bar_wait(&o_stored, c & 1, failed)) { if (lane == 0) atomicExch(status, 93); }
            __syncwarp();
            write(0);
            if (c + 1 < chunks) load(c + 1, 0);
            silu_of(gates[1]);
            write(1);
            __syncwarp();
            if (lane == 0) bar_arrive(&o_free[c & 1]);
        }
    }
    fence_before_sync();
    __syncthreads();
    if (failed_flag && warp == 0 && lane == 0) {
        // copies may still be on their way into this block's shared memory: give them a bounded time to land
        uint64_t* bars[4] = {&x_full, &b_full, &c_full, &pairs_full};
        for (int i = 0; i < 4; ++i)
            for (uint32_t parity = 0; parity < 2; ++parity) { int zero = 0; bar_wait(bars[i], parity, &zero, 2000000); }
    }
    __syncthreads();
    if (warp == 1) tmem_free(tmem, 512);
}

// ----------------------------------------------------------------------------- host side

// Chunks of at most 128 tokens: chunk_seq/begin/end and, per sequence, its first chunk (one entry more at the end).  scratch:
// 2 * num_chunks * (groups * (64 (64 + 2 N + 1) + 4) + heads * (64 * 64 + 260)) floats.  status: one int on the device, zero before
// the call.  num_rows: the rows of xbc.
FRB_API int frb_state_space_chunks(const float* proj, int proj_stride, int z_offset, int dt_offset, const float* xbc, int xbc_stride,
                                   int b_offset, int c_offset, const float* dt_bias, const float* a_log, const float* d, const int* seq_slot,
                                   const int* seq_start, const int* cu_q_len, float* state, long long copy_floats, long long state_offset,
                                   float* out, int num_seqs, int heads, int vdim, int N, int groups, const int* chunk_seq,
                                   const int* chunk_begin, const int* chunk_end, const int* seq_chunk0, int num_chunks, int num_rows,
                                   float* scratch, int* status, cudaStream_t stream) {
    if (num_seqs == 0 || num_chunks == 0) return 0;
    FRB_CHECK_ARG((N == 64 || N == 128) && (vdim == 64 || vdim == 128) && groups >= 1 && heads % groups == 0 &&
                      heads / groups * vdim % SC_COLUMNS == 0 && heads <= 65535, "state-space chunks: %d heads of %d x %d in %d groups", heads, N,
                  vdim, groups);
    FRB_CHECK_ARG(((xbc_stride | b_offset | c_offset) & 3) == 0 && ((proj_stride | z_offset) & 1) == 0 &&
                      (((uintptr_t)xbc | (uintptr_t)scratch | (uintptr_t)out) & 15) == 0 && ((uintptr_t)proj & 7) == 0,
                  "state-space chunks: rows of %d entries are not in steps of 16 bytes", xbc_stride);
    StateSpaceChunks p;
    p.proj = proj; p.xbc = xbc; p.dt_bias = dt_bias; p.a_log = a_log; p.d = d; p.seq_slot = seq_slot; p.seq_start = seq_start;
    p.cu_q_len = cu_q_len; p.chunk_seq = chunk_seq; p.chunk_begin = chunk_begin; p.chunk_end = chunk_end; p.seq_chunk0 = seq_chunk0;
    p.state = state; p.copy_floats = copy_floats; p.state_offset = state_offset; p.out = out;
    const size_t chunks = 2 * (size_t)num_chunks, rows = chunks * groups * SC_TOKENS * N;
    p.c_parts = (uint16_t*)scratch;
    p.b_parts = (uint16_t*)(scratch + rows);
    p.pair_parts = (uint16_t*)(scratch + 2 * rows);
    p.raw_pairs = scratch + 2 * rows + chunks * heads * SC_TOKENS * SC_TOKENS;
    p.scales = p.raw_pairs + chunks * groups * SC_TOKENS * SC_TOKENS;
    p.factors = p.scales + chunks * groups * (SC_TOKENS + 4);
    p.proj_stride = proj_stride; p.z_offset = z_offset; p.dt_offset = dt_offset; p.xbc_stride = xbc_stride; p.b_offset = b_offset;
    p.c_offset = c_offset; p.heads = heads; p.vdim = vdim; p.N = N; p.groups = groups;
    const int two = vdim == 64 ? 2 : 1;
    const size_t pairs_smem = 2 * (size_t)SC_TOKENS * (N + 8) * sizeof(float);
    const size_t chain_smem = (size_t)SC_TOKENS * 2 * (4 * N + 2 * two * SC_TOKENS + 6 * SC_COLUMNS) + 1024;
    CUtensorMap map_x;
    EncodeFn encode = encoder();
    cuuint64_t dims[2] = {(cuuint64_t)xbc_stride, (cuuint64_t)num_rows}, strides[1] = {(cuuint64_t)xbc_stride * 4};
    cuuint32_t box[2] = {SC_COLUMNS, SC_TOKENS}, steps[2] = {1, 1};
    FRB_CHECK_ARG(encode && encode(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(xbc), dims, strides, box, steps,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
                  "state-space chunks: cuTensorMapEncodeTiled failed or is not available");
    const dim3 chains(num_seqs, heads * vdim / SC_COLUMNS);
#define FRB_STATE_SPACE(NN, TWO)                                                                                                      \
    do {                                                                                                                              \
        auto chain = state_space_chain_kernel<NN, TWO>;                                                                               \
        /* the groups of warps share out the registers that the block is launched with: fewer, and they would wait for ever */        \
        static const int registers = [&] {                                                                                            \
            cudaFuncAttributes attributes;                                                                                            \
            return cudaFuncGetAttributes(&attributes, chain) == cudaSuccess ? attributes.numRegs : 0;                                 \
        }();                                                                                                                          \
        FRB_CHECK_ARG(registers >= ST_REGS_LAUNCH, "state-space chunks: the kernel was compiled to %d registers", registers);         \
        cudaFuncSetAttribute(state_space_pairs_kernel<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pairs_smem);             \
        cudaFuncSetAttribute(chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chain_smem);                                    \
        state_space_pairs_kernel<NN><<<dim3((unsigned)chunks, groups), 256, pairs_smem, stream>>>(p);                                 \
        state_space_weights_kernel<<<dim3((unsigned)chunks, heads), 128, 0, stream>>>(p);                                             \
        launch_dependent(chain, chains, dim3(ST_THREADS), chain_smem, stream, map_x, p, status);                                             \
    } while (0)
    if (N == 128) { if (two == 2) FRB_STATE_SPACE(128, true); else FRB_STATE_SPACE(128, false); }
    else { if (two == 2) FRB_STATE_SPACE(64, true); else FRB_STATE_SPACE(64, false); }
#undef FRB_STATE_SPACE
    FRB_RETURN_LAUNCH("state_space_chunks");
}
