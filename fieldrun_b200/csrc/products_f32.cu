// Products of many float32 rows with float32 weights on the tensor cores (tcgen05), each operand as two float16 parts.
//
// y[row, f] = sum_k x[row, k] W_e[f, k].  Every row of x and every weight row is multiplied by a power of two that brings its
// largest entry to [2^14, 2^15), then split into hi = float16(v) and lo = float16(2^11 (v - hi)).  Entries down to 2^-29 of the row's
// largest keep 22 bits or more, smaller ones an absolute error of 2^-51 of that largest; the product is hi hi + 2^-11 (hi lo + lo hi),
// whose terms are exact in float32, and lo lo is below 2^-22 of it.  What would cost precision is the tensor cores' adder: it
// cuts the sum off instead of rounding it, so an error grows by about 1e-9 of the sum with every entry of the inner size
// (measured: 2.3e-7 of the result after 256 entries, 3.2e-6 after 3,072).  So the large products (hi hi) are summed in tensor
// memory over 256 entries at a time only and added in float32 registers, rounded, and the small ones, whose cut is 2^-11 of
// that, have accumulators of their own.  Against 64-bit sums the result is off by 3.6e-7 at any inner size from 2,048 to 6,144;
// the library's float32 product by 2e-7 to 1.4e-6, the kernel for any sizes (experts_generic.cu) by 1.7e-6.
//
// Some outputs are summed again entry by entry in float32: those of rows without a scale (rows with an infinity or a NaN or without an
// entry of 2^-112); those that came out as an infinity or a NaN; and those so small that entries below 2^-29 of their rows' largest may
// have had a part in them.  In units of the scaled rows each such entry is off by at most 2^-36 and meets entries below 2^15, so a sum
// of K is off by less than K 2^-20, both sides together: 2^-25 of any sum from 32 K on, where the largest product is 2^30.  Of rows
// of normally distributed numbers one output in 40,000 is below that.  The last two also hold where weights were written after
// the scales were made of them, and no longer suit them.
//
// What bounds it: 3,704 tokens on MiniMax-M2's 256 experts have to read 14.5 GB of weights (2.2 ms) and take 2.5 PFLOP of
// float16 products (1.6 ms at the tensor cores' peak).  The two products of those sizes take 4.9 ms (in tiles of eight rows on
// the ordinary pipes, rows_f32.cu: 28.8 ms); 3,704 rows with 8192 x 3072 weights 0.78 ms with their scales and parts, 720 TFLOP/s of
// float16 products (the library's float32 product 3.17 ms).  What holds it is the way from L2 to shared memory: a step of 6.3 MFLOP
// takes 64 KB a SM, and with the copies and barriers alone it takes 1,430 cycles of the 2,210 (without the products 1,800, without the
// split 1,990; 16 workers instead of eight: 2,400).
//
// A block (one per SM, for the whole launch) takes items of 128 features x 128 rows in turn.  Two producer threads fill a ring each
// by TMA: weights as float32 [128][64], rows as their two parts [2][128][64].  Eight warps read a weight tile, a row and half
// of the entries a lane, split it and store the parts to tensor memory, where they are the first operand of
// tcgen05.mma: shared memory, the busiest unit, then carries the weights twice and the rows of x three times a step instead of
// the split weights three times more.  The same warps take the finished sums out of tensor memory, between two tiles, so that
// the tensor cores have the next tile to work on meanwhile.
#include <cuda_fp16.h>

#include "tcgen05.cuh"

#define PF_FEATS 128
#define PF_ROWS 128
#define PF_K 64               // entries of the inner size a step
#define PF_CHUNK 4            // steps whose large products are summed in tensor memory
#define PF_WSTAGES 4
#define PF_XSTAGES 3
#define PF_WORKERS 8
#define PF_PART (PF_WORKERS / 4)                 // workers of the same 32 weight rows: each a part of the entries and of the columns
#define PF_COLS (PF_ROWS / PF_PART)              // columns of sums a worker has
#define PF_THREADS (96 + 32 * PF_WORKERS)       // warp 0: copies of weights, 1: MMAs, then the workers, the last: copies of rows
#define PF_WBYTES (PF_FEATS * PF_K * 4)
#define PF_XBYTES (2 * PF_ROWS * PF_K * 2)
// tensor memory: large sums twice (a chunk in the making, one being read), small sums, two stages of the weights' parts
#define PF_LARGE(buffer) ((buffer) * PF_ROWS)
#define PF_SMALL (2 * PF_ROWS)
#define PF_PARTS(stage) (3 * PF_ROWS + (stage) * 64)

using namespace frb_tma;
using namespace frb_tc;

// Tiles of at most 128 rows of one expert; without lists (a dense product) tile t is rows 128 t and on of the only weight matrix.
struct ProductsParams {
    const float* W;            // [E][F][K]
    const float* w_scale;      // [E * F]
    const float* x_scale;      // [rows_total]
    // what the parts were made from (split_rows), for the rows without a scale
    const float* x;
    const int* x_rows;
    int gated;
    float gate_limit;
    const int *tile_expert, *tile_row0, *num_tiles, *offsets;
    float* out;                // [rows, F]
    // outputs to be summed again: for every item and worker whether there are any, and, if so, a lane's columns
    uint8_t* again;            // [items * PF_WORKERS]
    unsigned long long* columns;               // [items * PF_WORKERS][32]
    int* status;
    int F, K, tiles;           // tiles: without lists
    long long rows_total;

    __device__ __forceinline__ int count() const { return num_tiles ? num_tiles[0] : tiles; }
    __device__ __forceinline__ int expert(int tile) const { return tile_expert ? tile_expert[tile] : 0; }
    __device__ __forceinline__ int first_row(int tile) const { return tile_row0 ? tile_row0[tile] : tile * PF_ROWS; }
    __device__ __forceinline__ int end_row(int e) const { return offsets ? offsets[e + 1] : (int)rows_total; }
};

__device__ __forceinline__ uint32_t half2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }

// The parts of four entries times their row's scale; lo is 2^11 times what hi leaves, so that it is no smaller than hi.
#define PF_LO 2048.f
__device__ __forceinline__ void split_four(float4 v, float scale, uint32_t& hi0, uint32_t& hi1, uint32_t& lo0, uint32_t& lo1) {
    const float a = v.x * scale, b = v.y * scale, c = v.z * scale, d = v.w * scale;
    const __half2 h0 = __floats2half2_rn(a, b), h1 = __floats2half2_rn(c, d);
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    hi0 = half2_bits(h0);
    hi1 = half2_bits(h1);
    lo0 = half2_bits(__floats2half2_rn((a - f0.x) * PF_LO, (b - f0.y) * PF_LO));
    lo1 = half2_bits(__floats2half2_rn((c - f1.x) * PF_LO, (d - f1.y) * PF_LO));
}

// A wait of a whole warp: either all of its lanes go on or none.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* failed) {
    return __all_sync(0xffffffffu, bar_wait(bar, parity, failed));
}

// The exponent of a scale, a power of two, whatever its sign: -1 marks a row of zeros.
__device__ __forceinline__ int scale_exponent(float scale) { return (int)(__float_as_uint(scale) >> 23 & 255) - 127; }

// Whether an output is zero for its row's or its weight row's zeros (the other being finite, and the sum zero still).
__device__ __forceinline__ bool is_of_zeros(float sum, float w_scale, float x_scale) {
    return sum == 0.f && (x_scale < 0.f ? w_scale != 0.f : w_scale < 0.f && x_scale != 0.f);
}

__global__ void __launch_bounds__(PF_THREADS, 1)
products_f32_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                    const __grid_constant__ ProductsParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t w_full[PF_WSTAGES], w_empty[PF_WSTAGES], x_full[PF_XSTAGES], x_empty[PF_XSTAGES];
    __shared__ uint64_t parts_full[2], parts_empty[2], large_done[2], large_read[2], item_read;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* w_ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* x_ring = w_ring + PF_WSTAGES * PF_WBYTES;
    const int feature_blocks = (p.F + PF_FEATS - 1) / PF_FEATS, steps = (p.K + PF_K - 1) / PF_K;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PF_WSTAGES; ++s) { bar_init(&w_full[s], 1); bar_init(&w_empty[s], PF_WORKERS); }
        for (int s = 0; s < PF_XSTAGES; ++s) { bar_init(&x_full[s], 1); bar_init(&x_empty[s], 1); }
        for (int s = 0; s < 2; ++s) {
            bar_init(&parts_full[s], PF_WORKERS);
            bar_init(&parts_empty[s], 1);
            bar_init(&large_done[s], 1);
            bar_init(&large_read[s], PF_WORKERS);
        }
        bar_init(&item_read, PF_WORKERS);
        failed = 0;
        bar_init_fence();
    }
    if (warp == 1) tmem_alloc(&tmem_base_slot, 512);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_base_slot;
    const int num_items = p.count() * feature_blocks;

    if (warp == 0) {
        if (lane == 0) {
            int ws = 0;
            uint32_t parity = 1;
            bool ok = true;
            for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
                const int tile = item / feature_blocks;
                const int w_row = p.expert(tile) * p.F + (item - tile * feature_blocks) * PF_FEATS;
                for (int step = 0; step < steps; ++step) {
                    if (!bar_wait(&w_empty[ws], parity, &failed)) { atomicExch(p.status, 41); ok = false; break; }
                    uint8_t* dst = w_ring + ws * PF_WBYTES;
                    bar_expect(&w_full[ws], PF_WBYTES);
                    load_2d(dst, &map_w, step * PF_K, w_row, &w_full[ws]);
                    load_2d(dst + PF_WBYTES / 2, &map_w, step * PF_K + 32, w_row, &w_full[ws]);
                    if (++ws == PF_WSTAGES) { ws = 0; parity ^= 1; }
                }
            }
        }
    } else if (warp == PF_THREADS / 32 - 1) {
        if (lane == 0) {
            int xs = 0;
            uint32_t parity = 1;
            bool ok = true;
            for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
                const int row0 = p.first_row(item / feature_blocks);
                for (int step = 0; step < steps; ++step) {
                    if (!bar_wait(&x_empty[xs], parity, &failed)) { atomicExch(p.status, 42); ok = false; break; }
                    uint8_t* dst = x_ring + xs * PF_XBYTES;
                    bar_expect(&x_full[xs], PF_XBYTES);
                    load_2d(dst, &map_x, step * PF_K, row0, &x_full[xs]);
                    load_2d(dst + PF_XBYTES / 2, &map_x, step * PF_K, (int)(row0 + p.rows_total), &x_full[xs]);
                    if (++xs == PF_XSTAGES) { xs = 0; parity ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int xs = 0, stage = 0, buffer = 0;
            uint32_t x_parity = 0, parts_parity = 0, read_parity = 1, item_parity = 1;
            bool ok = true;
            for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
                const int tile = item / feature_blocks;
                const int rows = min(PF_ROWS, p.end_row(p.expert(tile)) - p.first_row(tile));
                // float32 accumulators, float16 operands, both K-major, M = 128, N = the tile's rows in steps of 16
                const uint32_t idesc = (1u << 4) | ((uint32_t)(((rows + 15) & ~15) >> 3) << 17) | ((uint32_t)(PF_FEATS >> 4) << 24);
                if (!bar_wait(&item_read, item_parity, &failed)) { atomicExch(p.status, 43); break; }      // the small sums are free
                item_parity ^= 1;
                for (int step = 0; step < steps; ++step) {
                    const bool opens = step % PF_CHUNK == 0, closes = step % PF_CHUNK == PF_CHUNK - 1 || step == steps - 1;
                    if (opens && !bar_wait(&large_read[buffer], read_parity, &failed)) { atomicExch(p.status, 44); ok = false; break; }
                    if (!bar_wait(&parts_full[stage], parts_parity, &failed)) { atomicExch(p.status, 45); ok = false; break; }
                    if (!bar_wait(&x_full[xs], x_parity, &failed)) { atomicExch(p.status, 46); ok = false; break; }
                    fence_after_sync();
                    const uint32_t hi = tmem + PF_PARTS(stage), lo = hi + 32;
                    const uint32_t x_hi = smem_addr(x_ring + xs * PF_XBYTES), x_lo = x_hi + PF_XBYTES / 2;
#pragma unroll
                    for (int k = 0; k < PF_K / 16; ++k) {
                        const uint64_t desc_hi = tile_desc(x_hi + 32 * k);
                        mma_ts(tmem + PF_SMALL, lo + 8 * k, desc_hi, idesc, (step | k) != 0);
                        mma_ts(tmem + PF_SMALL, hi + 8 * k, tile_desc(x_lo + 32 * k), idesc, 1);
                        mma_ts(tmem + PF_LARGE(buffer), hi + 8 * k, desc_hi, idesc, !(opens && k == 0));
                    }
                    mma_commit(&x_empty[xs]);
                    mma_commit(&parts_empty[stage]);
                    if (++xs == PF_XSTAGES) { xs = 0; x_parity ^= 1; }
                    if (++stage == 2) { stage = 0; parts_parity ^= 1; }
                    if (closes) {
                        mma_commit(&large_done[buffer]);
                        if (++buffer == 2) { buffer = 0; read_parity ^= 1; }
                    }
                }
            }
        }
    } else {
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        const int r = quarter * 32 + lane;                               // the weight row of the tile that this lane splits
        int ws = 0, stage = 0, buffer = 0, step = 0;
        uint32_t w_parity = 0, parts_parity = 1, done_parity = 0;
        float sums[PF_COLS], scale = 0.f;
#pragma unroll
        for (int i = 0; i < PF_COLS; ++i) sums[i] = 0.f;
        // of the item in hand, and of the chunk that is finished but not taken yet (0: none, 1: one, 2: its item's last)
        int row0 = 0, rows = 0, f = 0, taken_row0 = 0, taken_rows = 0, taken_f = 0, taken_item = 0, pending = 0;
        float taken_scale = 0.f;

        // Each turn splits one step's weights, then takes the chunk that the turn before it finished: the tensor cores have this
        // turn's step to work on meanwhile.  A last turn without weights takes the last chunk.
        for (int item = blockIdx.x;;) {
            const bool more = item < num_items;
            if (more) {
                if (step == 0) {
                    const int tile = item / feature_blocks, e = p.expert(tile);
                    row0 = p.first_row(tile) + part * PF_COLS;
                    rows = min(PF_COLS, p.end_row(e) - row0);            // of this part's columns; 0 or less: none
                    f = (item - tile * feature_blocks) * PF_FEATS + r;
                    scale = p.w_scale[(long long)e * p.F + min(f, p.F - 1)];
                }
                if (!warp_wait(&w_full[ws], w_parity, &failed)) { if (lane == 0) atomicExch(p.status, 48); break; }
                // 32 entries of a row are 128 bytes of a box; 16-byte chunk c of row r lies at chunk c ^ (r & 7)
                const uint8_t* src = w_ring + ws * PF_WBYTES + part * (PF_WBYTES / 2) + r * 128;
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 w = *(const float4*)(src + ((c ^ (r & 7)) << 4));
                    split_four(w, scale, hi[2 * c], hi[2 * c + 1], lo[2 * c], lo[2 * c + 1]);
                }
                __syncwarp();
                if (lane == 0) bar_arrive(&w_empty[ws]);
                if (++ws == PF_WSTAGES) { ws = 0; w_parity ^= 1; }
                if (!warp_wait(&parts_empty[stage], parts_parity, &failed)) { if (lane == 0) atomicExch(p.status, 49); break; }
                fence_after_sync();
                tmem_st16(lanes + PF_PARTS(stage) + part * 16, hi);
                tmem_st16(lanes + PF_PARTS(stage) + 32 + part * 16, lo);
                tmem_wait_st();
                fence_before_sync();
                __syncwarp();
                if (lane == 0) bar_arrive(&parts_full[stage]);
                if (++stage == 2) { stage = 0; parts_parity ^= 1; }
            }
            if (pending) {
                if (!warp_wait(&large_done[buffer], done_parity, &failed)) { if (lane == 0) atomicExch(p.status, 47); break; }
                fence_after_sync();
                uint32_t v[2][16];
                const uint32_t large = lanes + PF_LARGE(buffer) + part * PF_COLS, small = lanes + PF_SMALL + part * PF_COLS;
                if (taken_rows > 0) tmem_ld16(large, v[0]);
#pragma unroll
                for (int c = 0; c < PF_COLS / 16; ++c) {
                    tmem_wait_ld();
                    if (c + 1 < PF_COLS / 16 && 16 * (c + 1) < taken_rows) tmem_ld16(large + 16 * (c + 1), v[(c + 1) & 1]);
                    if (16 * c < taken_rows)
#pragma unroll
                        for (int j = 0; j < 16; ++j) sums[16 * c + j] += __uint_as_float(v[c & 1][j]);
                }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) bar_arrive(&large_read[buffer]);
                if (++buffer == 2) { buffer = 0; done_parity ^= 1; }
                if (pending == 2) {                                      // the item's end: its small products, the scales, the result
                    if (taken_rows > 0) tmem_ld16(small, v[0]);
#pragma unroll
                    for (int c = 0; c < PF_COLS / 16; ++c) {
                        tmem_wait_ld();
                        if (c + 1 < PF_COLS / 16 && 16 * (c + 1) < taken_rows) tmem_ld16(small + 16 * (c + 1), v[(c + 1) & 1]);
                        if (16 * c < taken_rows)
#pragma unroll
                            for (int j = 0; j < 16; ++j) sums[16 * c + j] = fmaf(__uint_as_float(v[c & 1][j]), 1.0f / PF_LO, sums[16 * c + j]);
                    }
                    fence_before_sync();
                    __syncwarp();
                    if (lane == 0) bar_arrive(&item_read);
                    const int w_exponent = scale_exponent(taken_scale);
                    const float least = 32.f * (float)p.K;
                    uint32_t bad[2] = {0, 0};
                    const float own_x_scales[2] = {lane < taken_rows ? p.x_scale[taken_row0 + lane] : 0.f,
                                                   lane + 32 < taken_rows ? p.x_scale[taken_row0 + lane + 32] : 0.f};
#pragma unroll
                    for (int n = 0; n < PF_COLS; ++n) {
                        const float x_scale = __shfl_sync(0xffffffffu, own_x_scales[n / 32], n % 32);
                        if (n < taken_rows && taken_f < p.F) {
                            const long long row = (long long)taken_row0 + n;
                            const float size = fabsf(sums[n]);
                            if (!(size >= least && size <= 3.402823466e38f && taken_scale > 0.f && x_scale > 0.f) &&
                                !is_of_zeros(sums[n], taken_scale, x_scale)) bad[n / 32] |= 1u << n % 32;
                            p.out[row * p.F + taken_f] = ldexpf(sums[n], -(w_exponent + scale_exponent(x_scale)));
                        }
                        sums[n] = 0.f;
                    }
                    const bool any = __any_sync(0xffffffffu, (bad[0] | bad[1]) != 0);
                    const long long unit = (long long)taken_item * PF_WORKERS + warp - 2;
                    if (any) p.columns[unit * 32 + lane] = (unsigned long long)bad[1] << 32 | bad[0];
                    if (lane == 0) p.again[unit] = any;
                }
            }
            if (!more) break;
            pending = step == steps - 1 ? 2 : step % PF_CHUNK == PF_CHUNK - 1 ? 1 : 0;
            if (pending) { taken_row0 = row0; taken_rows = rows; taken_f = f; taken_item = item; taken_scale = scale; }
            if (++step == steps) { step = 0; item += gridDim.x; }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (failed && warp == 0 && lane == 0) {
        // copies may still be on their way into this block's shared memory: give them a bounded time to land
        for (int s = 0; s < PF_WSTAGES; ++s) { int again = 0; bar_wait(&w_full[s], 0, &again); }
        for (int s = 0; s < PF_XSTAGES; ++s) { int again = 0; bar_wait(&x_full[s], 0, &again); }
    }
    __syncthreads();
    if (warp == 1) tmem_free(tmem, 512);
}

// The outputs to be summed again, a warp each: a warp takes the workers' outputs of an item that have some, and their columns in turn.  A
// kernel of its own: called from the workers' loop the same cost that a quarter of its speed.  3,704 rows with 8192 x 3072 and 3072 x 6144
// weights, on average: 626 us with this kernel, 28 of them its own; 800 the other way; 606 with no output summed again but those of rows
// without a scale.
__global__ void __launch_bounds__(256, 4) products_f32_again_kernel(const __grid_constant__ ProductsParams p) {
    const int lane = threadIdx.x & 31, feature_blocks = (p.F + PF_FEATS - 1) / PF_FEATS;
    const long long units = (long long)p.count() * feature_blocks * PF_WORKERS, warps = (long long)gridDim.x * 8;
    for (long long first = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); first < units; first += 32 * warps) {
        const long long mine = first + lane * warps;
        for (uint32_t left = __ballot_sync(0xffffffffu, mine < units && p.again[mine]); left; left &= left - 1) {
            const long long unit = first + (__ffs(left) - 1) * warps;
            const int item = (int)(unit / PF_WORKERS), worker = (int)(unit % PF_WORKERS), tile = item / feature_blocks, e = p.expert(tile);
            // the worker of warp w: weight rows 32 (w & 3) on, columns of part (w - 2) / 4
            const int f = (item - tile * feature_blocks) * PF_FEATS + ((worker + 2) & 3) * 32 + lane;
            const long long row0 = p.first_row(tile) + (worker >> 2) * PF_COLS, w_row = (long long)e * p.F + min(f, p.F - 1);
            const long long rows_here = p.end_row(e) - row0;             // whatever a launch that gave up has left in `again`: no row beyond
            const unsigned long long there = rows_here >= 64 ? ~0ull : rows_here > 0 ? (1ull << rows_here) - 1 : 0;
            const unsigned long long columns = f < p.F ? p.columns[unit * 32 + lane] & there : 0;
            unsigned long long all = (unsigned long long)__reduce_or_sync(0xffffffffu, (uint32_t)(columns >> 32)) << 32 |
                                     __reduce_or_sync(0xffffffffu, (uint32_t)columns);
            for (; all; all &= all - 1) {
                const int n = __ffsll((long long)all) - 1;
                const long long row = row0 + n;
                const float* x = p.x + (p.x_rows ? p.x_rows[row] : row) * (p.gated ? 2ll * p.K : (long long)p.K);
                for (uint32_t mask = __ballot_sync(0xffffffffu, (columns >> n & 1) != 0); mask; mask &= mask - 1) {
                    const int of = __ffs(mask) - 1;
                    const float* w = p.W + __shfl_sync(0xffffffffu, w_row, of) * p.K;
                    float sum = 0.f;
#pragma unroll 8
                    for (int k = 4 * lane; k < p.K; k += 128) {
                        const float4 a = *(const float4*)(w + k);
                        float4 b = *(const float4*)(x + k);
                        if (p.gated) {
                            const float4 up = *(const float4*)(x + p.K + k);
                            b = make_float4(paired_gate(b.x, up.x, p.gate_limit), paired_gate(b.y, up.y, p.gate_limit),
                                            paired_gate(b.z, up.z, p.gate_limit), paired_gate(b.w, up.w, p.gate_limit));
                        }
                        sum = fmaf(a.x, b.x, sum);
                        sum = fmaf(a.y, b.y, sum);
                        sum = fmaf(a.z, b.z, sum);
                        sum = fmaf(a.w, b.w, sum);
                    }
                    sum = warp_sum(sum);
                    if (lane == of) p.out[row * p.F + f] = sum;
                }
            }
        }
    }
}

// ----------------------------------------------------------------------------- scales and parts

// The power of two that brings `top` to [2^14, 2^15); -1 for a row of zeros, 0 for one with an infinity or a NaN or whose scale
// would leave float32.
__device__ __forceinline__ float row_scale(float top) {
    if (!(top <= 3.402823466e38f)) return 0.f;
    if (top == 0.f) return -1.f;
    const int exponent = 14 - ilogbf(top);
    return exponent <= 126 ? __uint_as_float((uint32_t)(exponent + 127) << 23) : 0.f;
}

// fmaxf drops a NaN: a row's largest entry, or a NaN if it holds one.
__device__ __forceinline__ float larger_or_nan(float a, float b) { return a != a || b != b ? __int_as_float(0x7fffffff) : fmaxf(a, b); }

__device__ __forceinline__ float largest_of_four(float4 v, float top) {
    return larger_or_nan(larger_or_nan(larger_or_nan(fabsf(v.x), fabsf(v.y)), larger_or_nan(fabsf(v.z), fabsf(v.w))), top);
}

__device__ __forceinline__ float warp_top(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = larger_or_nan(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// A warp a weight row: bound by reading the weights once (100 MB in 15 us).
__global__ void __launch_bounds__(256) weight_scales_kernel(const float* __restrict__ w, float* __restrict__ scale, long long rows, int K) {
    const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const float4* src = (const float4*)(w + row * K);
    float top = 0.f;
#pragma unroll 4
    for (int u = threadIdx.x & 31; u < K / 4; u += 32) top = largest_of_four(src[u], top);
    top = warp_top(top);
    if ((threadIdx.x & 31) == 0) scale[row] = row_scale(top);
}

// A block a row: parts[0][i] and parts[1][i] of the row x[rows[i]] (of row i without `rows`), or, GATED, of the unit
// paired_gate(x[i][k], x[i][K + k]) of a row of 2 K entries.  The row stays in shared memory between its maximum and its parts.
template <bool GATED>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, const int* __restrict__ rows, __half* __restrict__ parts,
                                                         float* __restrict__ scale, long long count, int K, float gate_limit) {
    extern __shared__ float4 split_row[];
    __shared__ float tops[8];
    const int units = K / 4;
    for (long long i = blockIdx.x; i < count; i += gridDim.x) {
        const float4* src = (const float4*)(x + (size_t)(rows ? rows[i] : i) * (GATED ? 2 * (size_t)K : (size_t)K));
        float top = 0.f;
        for (int u = threadIdx.x; u < units; u += 256) {
            float4 v = src[u];
            if (GATED) {
                const float4 up = src[units + u];
                v = make_float4(paired_gate(v.x, up.x, gate_limit), paired_gate(v.y, up.y, gate_limit), paired_gate(v.z, up.z, gate_limit),
                                paired_gate(v.w, up.w, gate_limit));
            }
            split_row[u] = v;
            top = largest_of_four(v, top);
        }
        top = warp_top(top);
        if ((threadIdx.x & 31) == 0) tops[threadIdx.x >> 5] = top;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 8; ++w) top = larger_or_nan(top, tops[w]);
        const float s = row_scale(top);
        uint2* hi = (uint2*)(parts + (size_t)i * K);
        uint2* lo = (uint2*)(parts + (size_t)(count + i) * K);
        for (int u = threadIdx.x; u < units; u += 256) {
            uint32_t h0 = 0, h1 = 0, l0 = 0, l1 = 0;
            if (s != 0.f) split_four(split_row[u], s, h0, h1, l0, l1);
            hi[u] = make_uint2(h0, h1);
            lo[u] = make_uint2(l0, l1);
        }
        if (threadIdx.x == 0) scale[i] = s;
        __syncthreads();                                                 // the row and the warps' maxima are read by then
    }
}

// ----------------------------------------------------------------------------- host side

// A map over row-major [rows, cols] with boxes of [box_rows][128 bytes] under the 128-byte swizzle; zeros outside.
static bool map_rows_of_128_bytes(CUtensorMap* map, const void* base, CUtensorMapDataType type, uint32_t size, uint64_t rows, uint64_t cols,
                                  uint32_t box_rows) {
    EncodeFn fn = encoder();
    if (!fn) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * size};
    cuuint32_t box[2] = {128 / size, box_rows};
    cuuint32_t elem[2] = {1, 1};
    return fn(map, type, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

FRB_API int frb_weight_scales(const float* w, float* scale, long long rows, int K, cudaStream_t stream) {
    if (rows == 0) return 0;
    FRB_CHECK_ARG(K > 0 && K % 8 == 0 && ((uintptr_t)w & 15) == 0, "weight scales: rows of %d entries", K);
    weight_scales_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, stream>>>(w, scale, rows, K);
    FRB_RETURN_LAUNCH("weight_scales");
}

// parts float16 [2][count][K], scale [count]; gated: x has rows of 2 K entries, gate then up.
FRB_API int frb_split_rows(const float* x, const int* rows, void* parts, float* scale, long long count, int K, int gated, float gate_limit,
                           cudaStream_t stream) {
    if (count == 0) return 0;
    FRB_CHECK_ARG(K > 0 && K % 8 == 0 && K <= 32768 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)parts & 15) == 0, "split rows: rows of %d entries", K);
    const size_t smem = (size_t)K * sizeof(float);
    const unsigned grid = (unsigned)(count < (1 << 20) ? count : (1 << 20));
    if (smem > 40 * 1024) {
        cudaFuncSetAttribute(split_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(split_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    if (gated) split_rows_kernel<true><<<grid, 256, smem, stream>>>(x, rows, (__half*)parts, scale, count, K, gate_limit);
    else split_rows_kernel<false><<<grid, 256, smem, stream>>>(x, rows, (__half*)parts, scale, count, K, gate_limit);
    FRB_RETURN_LAUNCH("split_rows");
}

// W float32 [E][F][K] with w_scale [E * F]; parts float16 [2][rows_total][K] with x_scale [rows_total], made from x (with x_rows,
// gated, gate_limit as for frb_split_rows), the rows of each expert together; tiles of at most 128 rows (null lists: the tiles of
// one weight matrix); out float32 [rows_total, F].  again: scratch, FRB_PRODUCTS_AGAIN bytes for every tile and 128 features.  status:
// one int on the device, zero before the call.
#define FRB_PRODUCTS_AGAIN (PF_WORKERS * (32 * 8 + 1))
FRB_API int frb_products_f32(const float* W, const float* w_scale, int num_experts, const void* parts, const float* x_scale, long long rows_total,
                             const float* x, const int* x_rows, int gated, float gate_limit, const int* tile_expert, const int* tile_row0,
                             const int* num_tiles, const int* offsets, int max_tiles, float* out, int F, int K, void* again, int* status,
                             cudaStream_t stream) {
    if (max_tiles == 0 || F == 0) return 0;
    FRB_CHECK_ARG(K > 0 && K % 8 == 0, "float32 products: an inner size of %d is not a multiple of 8", K);
    FRB_CHECK_ARG((((uintptr_t)W | (uintptr_t)parts | (uintptr_t)x) & 15) == 0 && ((uintptr_t)again & 7) == 0,
                  "float32 products: operands must be 16-byte aligned");
    FRB_CHECK_ARG(2 * rows_total + PF_ROWS < (1ll << 31) && (long long)num_experts * F < (1ll << 31) - PF_FEATS,
                  "float32 products: %lld rows or %d experts of %d features exceed a coordinate", rows_total, num_experts, F);
    const long long items = (long long)max_tiles * ((F + PF_FEATS - 1) / PF_FEATS);
    FRB_CHECK_ARG(items < (1ll << 31) - (1 << 16), "float32 products: %d tiles of %d features exceed the count of items", max_tiles, F);
    CUtensorMap map_w, map_x;
    FRB_CHECK_ARG(map_rows_of_128_bytes(&map_w, W, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)num_experts * F, K, PF_FEATS) &&
                      map_rows_of_128_bytes(&map_x, parts, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, 2 * rows_total, K, PF_ROWS),
                  "float32 products: cuTensorMapEncodeTiled failed or is not available");
    const ProductsParams p = {W, w_scale, x_scale, x, x_rows, gated, gate_limit, tile_expert, tile_row0, num_tiles, offsets, out,
                              (uint8_t*)again + items * PF_WORKERS * 32 * 8, (unsigned long long*)again, status, F, K, max_tiles, rows_total};
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const size_t smem = PF_WSTAGES * PF_WBYTES + PF_XSTAGES * PF_XBYTES + 1024;
    cudaFuncSetAttribute(products_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    products_f32_kernel<<<(unsigned)(items < sms ? items : sms), PF_THREADS, smem, stream>>>(map_w, map_x, p);
    products_f32_again_kernel<<<4 * sms, 256, 0, stream>>>(p);
    FRB_RETURN_LAUNCH("products_f32");
}
