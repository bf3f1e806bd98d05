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
    // (Six rows with 8192 x 3072 and 3072 x 6144 weights, an event pair around each launch, which itself is about 6 us: 33 us on
    // average, 52 and 57 with other splits of the same sizes into blocks of four and two runs.)  With many tiles a warp to a run has
    // the fewer joins.
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
