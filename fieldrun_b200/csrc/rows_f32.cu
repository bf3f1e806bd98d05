// Products of a few float32 rows with large float32 weights: the experts' and the dense products of float32 decode steps.
// Same formulas and lists as experts_generic.cu, tiles of at most eight rows; every product and sum is a float32
// multiply-add, a lane's over every 128th run of four entries, the lanes' added in a fixed order.
//
// What bounds it: the weights' bytes.  experts_generic gives a block 32 rows x 64 features and takes the inner size sixteen
// entries at a time with two barriers each: a single row costs as much as 32, and a block has 4 KB of weights on their way.
// Eight tokens of MiniMax-M2's experts (57 used, 3.2 GB of weights) took 4.59 ms there, 0.7 TB/s.  Here a warp reads eight
// weight rows side by side through a ring of its own in shared memory (asynchronous copies; a lane reads back only what it
// copied, so the ring needs no barrier), and every weight meets all rows of its tile in registers; the rows come through L1,
// which the weights bypass: 0.23 ms a product (7 TB/s).  Steps of up to eight rows an expert, and of sizes or so little work that the
// products on the tensor cores (products_f32.cu) do not take them, run here in tiles of eight rows that read an expert's weights
// again from L2.
#include "common.cuh"
#include "pairs.cuh"

#define RF_WARPS 4
#define RF_FEATS 8            // weight rows a warp takes
#define RF_ROWS 8             // most rows of a tile
#define RF_STAGES 4           // runs of 32 x 4 entries of every weight row on their way: 16 KB a warp

struct RowsParams {
    const float* W;           // [E][(paired ? 2 : 1) F][K]
    const float* X;           // rows of K
    const int* x_rows;        // sorted row -> row of X, or null
    const int *tile_expert, *tile_row0, *num_tiles, *offsets;
    float* out;               // [N, F]
    int F, K;
    float gate_limit;
};

__device__ __forceinline__ void rf_copy16(float4* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ float rf_dot4(float4 a, float4 b, float c) {
    c = fmaf(a.x, b.x, c);
    c = fmaf(a.y, b.y, c);
    c = fmaf(a.z, b.z, c);
    return fmaf(a.w, b.w, c);
}

// The sums of a warp's lanes, added by halves: value i of N ends in to[i].
template <int N>
__device__ __forceinline__ void rf_join(float (&acc)[N], int lane, float* to) {
    __syncwarp();
    int n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n /= 2;
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i >= n) break;
                const float keep = upper ? acc[i + n] : acc[i], send = upper ? acc[i] : acc[i + n];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        } else {
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
        }
    }
    constexpr int LEFT = N > 32 ? N / 32 : 1, SHARE = N < 32 ? 32 / N : 1;
#pragma unroll
    for (int j = 0; j < LEFT; ++j)
        if (lane % SHARE == 0) to[lane / SHARE * LEFT + j] = acc[j];
}

// One warp: eight weight rows (`w`, their addresses) with R rows of x over the 16-byte units [begin, end) of the inner size.
// Value f * R + r, weight row f with row r, ends in to[f * R + r]: the lanes' sums meet by halves.
template <int R>
__device__ __forceinline__ void rf_products(float4* ring, const float* const (&w)[RF_FEATS], const float* const (&x)[RF_ROWS], int begin,
                                            int end, int lane, float* to) {
    constexpr int N = RF_FEATS * R;
    float acc[N];
#pragma unroll
    for (int i = 0; i < N; ++i) acc[i] = 0.f;
    auto copy_run = [&](int stage, int u) {
        if (u < end)
#pragma unroll
            for (int f = 0; f < RF_FEATS; ++f) rf_copy16(ring + (stage * RF_FEATS + f) * 32 + lane, w[f] + 4 * (size_t)u);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < RF_STAGES - 1; ++s) copy_run(s, begin + 32 * s + lane);
    int stage = 0;
#pragma unroll 1
    for (int u = begin + lane; u - lane < end; u += 32) {
        copy_run((stage + RF_STAGES - 1) % RF_STAGES, u + 32 * (RF_STAGES - 1));
        if (u < end) {
            float4 xv[R];
#pragma unroll
            for (int r = 0; r < R; ++r) xv[r] = *(const float4*)(x[r] + 4 * (size_t)u);
            asm volatile("cp.async.wait_group %0;" ::"n"(RF_STAGES - 1) : "memory");
#pragma unroll
            for (int f = 0; f < RF_FEATS; ++f) {
                const float4 wv = ring[(stage * RF_FEATS + f) * 32 + lane];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[f * R + r] = rf_dot4(wv, xv[r], acc[f * R + r]);
            }
        }
        stage = (stage + 1) % RF_STAGES;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    rf_join<N>(acc, lane, to);
}

// PARTS: warps that share eight weight rows, each with its part of the inner size.
template <bool PAIRED, int PARTS>
__global__ void __launch_bounds__(32 * RF_WARPS, 3) rows_f32_kernel(RowsParams p) {
    extern __shared__ float4 rf_smem[];
    __shared__ float sums[RF_WARPS][RF_FEATS * RF_ROWS];
    after_previous_kernel();
    const int tile = blockIdx.y;
    if (tile >= p.num_tiles[0]) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int OUT = PAIRED ? RF_FEATS / 2 : RF_FEATS;                // output features of eight weight rows
    const int f0 = (blockIdx.x * (RF_WARPS / PARTS) + warp / PARTS) * OUT;
    const int e = p.tile_expert[tile], row0 = p.tile_row0[tile];
    const int rows = min(RF_ROWS, p.offsets[e + 1] - row0);
    const float* We = p.W + (size_t)e * (PAIRED ? 2 : 1) * p.F * p.K;
    const float* w[RF_FEATS];
#pragma unroll
    for (int i = 0; i < RF_FEATS; ++i)                                   // of a pair the gate rows, then the up rows; behind the last
        w[i] = We + ((size_t)(PAIRED && i >= OUT ? p.F : 0) + min(f0 + i % OUT, p.F - 1)) * p.K;      // feature that one again
    const float* x[RF_ROWS];
#pragma unroll
    for (int r = 0; r < RF_ROWS; ++r) {
        const int row = row0 + min(r, rows - 1);
        x[r] = p.X + (size_t)(p.x_rows ? p.x_rows[row] : row) * p.K;
    }
    const int units = p.K >> 2, part = (units + 32 * PARTS - 1) / (32 * PARTS) * 32;          // whole runs
    const int begin = min(warp % PARTS * part, units), end = min(begin + part, units);
    float4* ring = rf_smem + warp * RF_STAGES * RF_FEATS * 32;
    int bits;                                                            // log2 of the rows that a value's index counts
    if (rows <= 1) { rf_products<1>(ring, w, x, begin, end, lane, sums[warp]); bits = 0; }
    else if (rows <= 2) { rf_products<2>(ring, w, x, begin, end, lane, sums[warp]); bits = 1; }
    else if (rows <= 4) { rf_products<4>(ring, w, x, begin, end, lane, sums[warp]); bits = 2; }
    else { rf_products<8>(ring, w, x, begin, end, lane, sums[warp]); bits = 3; }
    if (PARTS > 1) __syncthreads(); else __syncwarp();
    const int first = warp / PARTS * PARTS;                              // the warps of these weight rows, added in their order
    for (int v = lane + 32 * (warp % PARTS); v < OUT << bits; v += 32 * PARTS) {
        const int r = v & ((1 << bits) - 1), f = f0 + (v >> bits);
        float sum = 0.f, up = 0.f;
#pragma unroll
        for (int k = 0; k < PARTS; ++k) {
            sum += sums[first + k][v];
            if (PAIRED) up += sums[first + k][(OUT << bits) + v];
        }
        if (f < p.F && r < rows) p.out[(size_t)(row0 + r) * p.F + f] = PAIRED ? paired_gate(sum, up, p.gate_limit) : sum;
    }
}

// Four entries of R rows of x; PAIRS: two rows at a time, for the same multiply-adds in half the instructions.
template <int R, bool PAIRS>
struct RowsOfX {
    float4 one[PAIRS ? 1 : R];
    uint64_t two[PAIRS ? R / 2 : 1][4];
};

template <int R, bool PAIRS>
__device__ __forceinline__ void rf_load_x(RowsOfX<R, PAIRS>& to, const float* const (&x)[R], int u, int end) {
#pragma unroll
    for (int r = 0; r < R; r += PAIRS ? 2 : 1) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), a = u < end ? *(const float4*)(x[r] + 4 * u) : zero;
        if (PAIRS) {
            const float4 b = u < end ? *(const float4*)(x[r + PAIRS] + 4 * u) : zero;
            to.two[r / 2][0] = pair_of(a.x, b.x);
            to.two[r / 2][1] = pair_of(a.y, b.y);
            to.two[r / 2][2] = pair_of(a.z, b.z);
            to.two[r / 2][3] = pair_of(a.w, b.w);
        } else {
            to.one[r] = a;
        }
    }
}

// A dense product of up to eight rows: one matrix, no lists.  As many blocks as are resident at once take a share of the weight rows each (their
// number over the blocks, to the row), eight at a time, for the whole launch; a block's warps have a part of the inner size each, always the same
// one, and add theirs in their order, so that a row's sums do not depend on the other rows.  A warp's ring runs on from eight rows to the next and,
// where the weights are complete, begins ahead of the wait for the kernel before.  A run's place in the ring is filled again as soon as its lane
// has read it, ahead of the join.  The rows of x stay in registers where a warp's part has at most HELD runs of them, else the next run's are asked
// for ahead.  `tiles`: two where seven or eight rows would not fit so; neighbouring blocks then have four rows each and the same weights.
//
// Bound by the weights' bytes up to four rows, beyond by the multiply-adds and the joins.  The kernel above, whose blocks begin and end
// once for 32 KB to 96 KB of weights, and this one in a stream of launches, microseconds for 1, 4, 6 and 8 rows: 8192 x 3072 weights 19.6 24.6
// 28.8 29.1 | 15.2 15.8 18.1 19.8 (15.4 at the memory's rate), 3072 x 6144 15.4 17.1 19.0 19.3 | 12.3 12.9 16.7 18.4, 8192 x 8192 49.6 55.9 60.9 62.3
// | 40.0 44.6 49.3 60.4, 1024 x 1024 2.9 3.4 4.0 4.1 | 1.9 2.1 2.4 2.5, 144 x 96 2.2 2.4 2.5 2.6 | 1.5 1.7 2.0 1.9.  Twelve warps an SM: with one block
// an SM whatever the inner size 65536 x 128 takes 28 us with one row and 51 with eight instead of 7 and 12 (28 and 38 by the kernel above).  Only with
// very many weight rows do a single row's joins cost more than that kernel's ends: 65536 x 3072 113 | 120, 200064 x 3072 338 | 362; with eight
// rows 163 | 126 and 469 | 419, but 131072 x 2048 194 | 232.  Rows two by two (fma.rn.f32x2) pay where the work is large enough for six or eight rows'
// multiply-adds to bound it: 200064 x 3072 414 -> 377 with eight, 8192 x 3072 21.8 -> 20.7, but 1024 x 1024 2.5 -> 3.2.  Six rows as eight: 8192 x 3072
// 20.6 instead of 18.9, 2048 x 8192 19.9 instead of 15.7.
#define RD_WARPS 12

template <int R, int HELD>
__global__ void __launch_bounds__(32 * RD_WARPS, 1) dense_rows_f32_kernel(const float* W, const float* X, float* __restrict__ out, int all_rows,
                                                                          int tiles, int F, int K, int weights_final) {
    extern __shared__ float4 rf_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    float* sums = (float*)(rf_smem + warps * RF_STAGES * RF_FEATS * 32);                       // [2][warps][RF_FEATS * R]
    const int share = blockIdx.x / tiles, shares = gridDim.x / tiles, tile = blockIdx.x - share * tiles;
    const int row0 = tile * R, rows = min(all_rows - row0, R);
    X += (size_t)row0 * K;
    out += (size_t)row0 * F;
    const int f_begin = (int)((long long)F * share / shares), f_end = (int)((long long)F * (share + 1) / shares);
    const int units = K >> 2, part = (units + 8 * warps - 1) / (8 * warps) * 8;               // whole lines of 128 bytes
    const int begin = min(warp * part, units), end = min(begin + part, units), with_work = (units + part - 1) / part;
    const int runs = (end - begin + 31) / 32, groups = (f_end - f_begin + RF_FEATS - 1) / RF_FEATS, all = groups * runs;
    float4* ring = rf_smem + warp * RF_STAGES * RF_FEATS * 32 + lane;
    // the place of the next run to be copied
    const float* from = W + (size_t)f_begin * K;
    int copy_run = 0, copy_left = f_end - f_begin, copied = 0;
    auto copy = [&](int stage) {
        if (copied < all) {
            const int u = begin + 32 * copy_run + lane;
            if (u < end)
#pragma unroll
                for (int f = 0; f < RF_FEATS; ++f)
                    if (f < copy_left) rf_copy16(ring + (stage * RF_FEATS + f) * 32, from + (size_t)f * K + 4 * u);
            ++copied;
            if (++copy_run == runs) { copy_run = 0; copy_left -= RF_FEATS; from += (size_t)RF_FEATS * K; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (!weights_final) wait_for_previous_kernel();
#pragma unroll
    for (int s = 0; s < RF_STAGES; ++s) copy(s);
    wait_for_previous_kernel();
    let_next_kernel_start();                          // not before: the next kernel may read, ahead of its wait, what is complete by now
    const float* x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = X + (size_t)min(r, rows - 1) * K;
    constexpr bool PAIRS = R >= 6 && HELD == 2;
    RowsOfX<R, PAIRS> held[HELD ? HELD : 1];
    auto load_x = [&](RowsOfX<R, PAIRS>& to, int run) { rf_load_x<R, PAIRS>(to, x, begin + 32 * run + lane, end); };
#pragma unroll
    for (int h = 0; h < (HELD ? HELD : 1); ++h) load_x(held[h], h);
    float acc[PAIRS ? 1 : RF_FEATS * R];
    uint64_t acc2[PAIRS ? RF_FEATS * R / 2 : 1];
    int stage = 0;
    auto multiply = [&](const RowsOfX<R, PAIRS>& xv, int run) {
        asm volatile("cp.async.wait_group %0;" ::"n"(RF_STAGES - 1) : "memory");
        if (begin + 32 * run + lane < end)
#pragma unroll
            for (int f = 0; f < RF_FEATS; ++f) {
                const float4 wv = ring[(stage * RF_FEATS + f) * 32];
                if (PAIRS) {
                    const uint64_t w2[4] = {pair_of(wv.x, wv.x), pair_of(wv.y, wv.y), pair_of(wv.z, wv.z), pair_of(wv.w, wv.w)};
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int r = 0; r < R / 2; ++r) {
                            uint64_t& sum = acc2[f * (R / 2) + r];
                            sum = fma_pairs(w2[k], xv.two[r][k], sum);
                        }
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[f * R + r] = rf_dot4(wv, xv.one[r], acc[f * R + r]);
                }
            }
        copy(stage);                                                     // what this lane copied there it has read
        stage = (stage + 1) % RF_STAGES;
    };
#pragma unroll 1
    for (int g = 0; g < groups; ++g) {
        if (PAIRS) {
#pragma unroll
            for (int i = 0; i < RF_FEATS * R / 2; ++i) acc2[i] = 0;
        } else {
#pragma unroll
            for (int i = 0; i < RF_FEATS * R; ++i) acc[i] = 0.f;
        }
        if (HELD) {
#pragma unroll
            for (int h = 0; h < HELD; ++h)
                if (h < runs) multiply(held[h], h);
        } else {
#pragma unroll 1
            for (int run = 0; run < runs; ++run) {
                RowsOfX<R, PAIRS> next;
                load_x(next, run + 1 < runs ? run + 1 : 0);
                multiply(held[0], run);
                held[0] = next;
            }
        }
        float each[RF_FEATS * R];
#pragma unroll
        for (int i = 0; i < RF_FEATS * R; ++i) {
            if (!PAIRS) each[i] = acc[i];
            else if (i % 2 == 0) halves_of(acc2[i / 2], each[i], each[i + 1]);
        }
        // (six rows as four and two: the lanes' sums meet by halves)
        constexpr int HALVES = R == 6 ? 4 : R;
        float first[RF_FEATS * HALVES], second[R == 6 ? RF_FEATS * 2 : 1];
#pragma unroll
        for (int f = 0; f < RF_FEATS; ++f)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (r < HALVES) first[f * HALVES + r] = each[f * R + r];
                else second[f * 2 + r - HALVES] = each[f * R + r];
            }
        float* group_sums = sums + (g & 1) * warps * (RF_FEATS * R);
        rf_join<RF_FEATS * HALVES>(first, lane, group_sums + warp * (RF_FEATS * R));
        if constexpr (R == 6) rf_join<RF_FEATS * 2>(second, lane, group_sums + warp * (RF_FEATS * R) + RF_FEATS * HALVES);
        __syncthreads();                                                 // the sums of two groups back are read by then
        for (int v = threadIdx.x; v < RF_FEATS * R; v += blockDim.x) {
            const bool last_two = v >= RF_FEATS * HALVES;
            const int at = last_two ? v - RF_FEATS * HALVES : v, each_row = last_two ? 2 : HALVES;
            const int r = at % each_row + (last_two ? HALVES : 0), f = f_begin + g * RF_FEATS + at / each_row;
            float sum = 0.f;
            for (int k = 0; k < with_work; ++k) sum += group_sums[k * (RF_FEATS * R) + v];
            if (f < f_end && r < rows) out[(size_t)r * F + f] = sum;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Warps of a block: twelve, or a run of the inner size each where that has fewer.  Beyond four runs a warp the rows of x do not stay in
// registers, and twelve warps that meet after every eight weight rows wait for one another: where there are more than eight weight rows for
// every SM six or four do, whichever leave fewer of their blocks' places empty (eight rows of 4096 x 8192 32 us instead of 38, of 8192 x 8192 60
// instead of 64, of 3072 x 12288 32 instead of 38; the kernel above 41, 62 and 35.  It stays ahead by up to a tenth where seven or eight
// rows meet some 640 groups of weight rows, 5120 x 8192, and neither count of blocks comes out even).
static int dense_rows_warps(int units, int groups, int sms) {
    if (units < 32 * RD_WARPS) return (units + 31) / 32;
    if (units <= 4 * 32 * RD_WARPS || groups <= sms) return RD_WARPS;
    return 2 * ((groups + 2 * sms - 1) / (2 * sms)) <= 3 * ((groups + 3 * sms - 1) / (3 * sms)) ? 6 : 4;
}

// out [rows, F] = X [rows, K] W^T, W [F][K], all float32; up to eight rows.  weights_final: W was complete before the kernel before this one
// began, and may be read while that one still runs.
FRB_API int frb_dense_rows_f32(const float* W, const float* X, float* out, int rows, int F, int K, int weights_final, cudaStream_t stream) {
    if (rows == 0 || F == 0) return 0;
    FRB_CHECK_ARG(rows > 0 && rows <= RF_ROWS, "dense float32 rows: %d rows are outside 1..%d", rows, RF_ROWS);
    FRB_CHECK_ARG(K > 0 && K % 4 == 0, "dense float32 rows: an inner size of %d is not a multiple of 4", K);
    FRB_CHECK_ARG((((uintptr_t)W | (uintptr_t)X) & 15) == 0, "dense float32 rows: operands must be 16-byte aligned");
    const int sms = frb_sm_count(), units = K / 4, groups = (F + RF_FEATS - 1) / RF_FEATS, warps = dense_rows_warps(units, groups, sms);
    const int part = (units + 8 * warps - 1) / (8 * warps) * 8, runs = (part + 31) / 32;
    // (with two tiles everywhere eight rows of 8192 x 3072 take 24.9 us instead of 20.7; with one, of 3072 x 6144 20.9 instead of 18.8, and six
    // rows 18.6 with two instead of 17.2, 20.0 with their four runs in registers)
    const int tiles = rows > 6 && runs > 2 && runs <= 4 ? 2 : 1;
    const int per_sm = RD_WARPS / warps, most = per_sm * sms / tiles, shares = groups < most ? groups : most, blocks = shares * tiles;
#define FRB_DENSE(R, HELD)                                                                                                        \
    do {                                                                                                                          \
        const size_t smem = (size_t)warps * (RF_STAGES * RF_FEATS * 32 * sizeof(float4) + 2 * RF_FEATS * R * sizeof(float));      \
        if (smem > 48 * 1024)                                                                                                     \
            cudaFuncSetAttribute(dense_rows_f32_kernel<R, HELD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);         \
        launch_dependent_resident(per_sm, dense_rows_f32_kernel<R, HELD>, dim3(blocks), dim3(32 * warps), smem, stream, W, X,     \
                                  out, rows, tiles, F, K, weights_final);                                                         \
    } while (0)
#define FRB_DENSE_ROWS(R)                                                                                                         \
    do {                                                                                                                          \
        if (runs == 1) FRB_DENSE(R, 1);                                                                                           \
        else if (runs == 2) FRB_DENSE(R, 2);                                                                                      \
        else if (runs <= 4) FRB_DENSE(R, 4);                                                                                      \
        else FRB_DENSE(R, 0);                                                                                                     \
    } while (0)
    if (rows == 1) FRB_DENSE_ROWS(1);
    else if (rows == 2) FRB_DENSE_ROWS(2);
    else if (rows <= 4 || tiles == 2) FRB_DENSE_ROWS(4);
    else if (rows <= 6 && runs == 1) FRB_DENSE(6, 1);
    else if (rows <= 6 && runs == 2) FRB_DENSE(6, 2);
    else if (rows <= 6) FRB_DENSE(6, 0);
    else if (runs == 1) FRB_DENSE(8, 1);
    else if (runs == 2) FRB_DENSE(8, 2);
    else FRB_DENSE(8, 0);
#undef FRB_DENSE_ROWS
#undef FRB_DENSE
    FRB_RETURN_LAUNCH("dense_rows_f32");
}

// W [E][(paired ? 2 : 1) * F][K]; X rows of K; out [N, F], all float32.  x_rows (nullable) maps a sorted row to its X row.
// max_tiles bounds the grid; the lists' tiles have at most eight rows.
FRB_API int frb_rows_f32(const float* W, const float* X, const int* x_rows, const int* tile_expert, const int* tile_row0,
                         const int* num_tiles, const int* offsets, int max_tiles, float* out, int F, int K, int paired, float gate_limit,
                         cudaStream_t stream) {
    if (max_tiles == 0 || F == 0) return 0;
    FRB_CHECK_ARG(K > 0 && K % 4 == 0, "float32 rows: an inner size of %d is not a multiple of 4", K);
    FRB_CHECK_ARG((((uintptr_t)W | (uintptr_t)X) & 15) == 0, "float32 rows: operands must be 16-byte aligned");
    FRB_CHECK_ARG(max_tiles <= 65535, "float32 rows: %d tiles exceed the grid", max_tiles);
    const RowsParams p = {W, X, x_rows, tile_expert, tile_row0, num_tiles, offsets, out, F, K, gate_limit};
    const int outs = paired ? RF_FEATS / 2 : RF_FEATS, groups = (F + outs - 1) / outs;      // runs of eight weight rows of a tile
    // A single tile's blocks of four runs are one or two a SM and end unevenly: there four warps share a run of weight rows.
    // (Six rows with 8192 x 3072 and 3072 x 6144 weights, which the kernel above has by now, an event pair around each launch, which
    // itself is about 6 us: 33 us on average, 52 and 57 with other splits of the same sizes into blocks of four and two runs.)  With many
    // tiles, or the weight rows of a vocabulary, a warp to a run has the fewer joins.
    const bool parts = (long long)groups * max_tiles < 16384;
    const dim3 grid(parts ? groups : (groups + RF_WARPS - 1) / RF_WARPS, max_tiles);
    const size_t smem = (size_t)RF_WARPS * RF_STAGES * RF_FEATS * 32 * sizeof(float4);
#define FRB_ROWS(PAIRED, PARTS)                                                                                                   \
    do {                                                                                                                          \
        cudaFuncSetAttribute(rows_f32_kernel<PAIRED, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);             \
        launch_dependent(rows_f32_kernel<PAIRED, PARTS>, grid, dim3(32 * RF_WARPS), smem, stream, p);                             \
    } while (0)
    if (paired) { if (parts) FRB_ROWS(true, 4); else FRB_ROWS(true, 1); }
    else { if (parts) FRB_ROWS(false, 4); else FRB_ROWS(false, 1); }
#undef FRB_ROWS
    FRB_RETURN_LAUNCH("rows_f32");
}
