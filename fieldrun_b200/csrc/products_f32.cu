// Products of many float32 rows with float32 weights on the tensor cores (tcgen05), each operand as two float16 parts.
//
// y[row, f] = sum_k x[row, k] W_e[f, k].  Every row of x and every weight row is multiplied by a power of two that brings its
// largest entry to [2^14, 2^15), then split into hi = float16(v) and lo = float16(2^11 (v - hi)).  Entries down to 2^-29 of the row's
// largest keep 22 bits or more, smaller ones an absolute error of 2^-51 of that largest; the product is hi hi + 2^-11 (hi lo + lo hi),
// whose terms are exact in float32, and lo lo is below 2^-22 of it.  What would cost precision is the tensor cores' adder: it
// cuts the sum off instead of rounding it, so an error grows by about 1e-9 of the sum with every entry of the inner size
// (measured: 2.3e-7 of the result after 256 entries, 3.2e-6 after 3,072).  So the products of 64 entries at a time are summed in tensor
// memory, the small ones (hi lo, lo hi) first, 2^11 times too large; the first of the large ones takes their sum down by 2^11 as it
// is added.  The sums of 64 entries are added in float32 registers, rounded.  Against 64-bit sums the result is off by 1.5e-7 to 2.2e-7
// at inner sizes from 1,024 to 6,144 (sums of 256 entries in tensor memory: 3.6e-7); the library's float32 product by 2e-7 to 1.4e-6,
// the kernel for any sizes (experts_generic.cu) by 1.7e-6.
//
// Some outputs are summed again entry by entry in float32: those of rows without a scale (rows with an infinity or a NaN or without an
// entry of 2^-112); those that came out as an infinity or a NaN; and those so small that entries below 2^-29 of their rows' largest may
// have had a part in them.  In units of the scaled rows each such entry is off by at most 2^-36 and meets entries below 2^15, so a sum
// of K is off by less than K 2^-20, both sides together: 2^-25 of any sum from 32 K on, where the largest product is 2^30.  Of rows
// of normally distributed numbers one output in 40,000 is below that.  The last two also hold where weights were written after
// the scales were made of them, and no longer suit them.
//
// What bounds it: 3,704 tokens on MiniMax-M2's 256 experts have to read 14.5 GB of weights (2.2 ms) and take 2.5 PFLOP of
// float16 products (1.6 ms at the tensor cores' peak).  The two products of those sizes take 3.25 ms (in tiles of eight rows on
// the ordinary pipes, rows_f32.cu: 28.8 ms): their steps run at the memory's rate, and at an item's end, where all SMs write at
// once, the next item's steps wait for some 8,000 of its 70,000 cycles.  3,704 rows with 8192 x 3072 and 3072 x 6144 weights take
// 770 us, 1.27 PFLOP/s of float16 products; there the way from L2 to shared memory holds it, 45 bytes a cycle and SM (72 KB a step of
// 1,640 cycles, 960 of them products).  How it came there, those two sums in microseconds: one lane issuing the products, whose
// operands then have to be moved to uniform registers one by one, and splitting, adding and writing in the same warps 4770 and
// 1190; a whole warp issuing, and sums and results in warps of their own 3430 and 830; 160 rows instead of 128, with one accumulator
// instead of two 3360 and 776; the difference v - hi by the multiply-add that takes float16 as it is 3210 and 773.  As slow or slower:
// copies of 32 rows, as many as the tile has (3400 and 875); another order of the inner size in each block of features (3290 and 781).
//
// A block (one per SM, for the whole launch) takes items of 128 features x 160 rows in turn.  Two producer threads fill a ring each
// by TMA: weights as float32 [128][64], rows as their two parts [2][160][64].  Eight warps read a weight tile, a row and half
// of the entries a lane, split it and store the parts to tensor memory, where they are the first operand of
// tcgen05.mma: shared memory then carries the weights twice and the rows of x three times a step instead of the split weights
// three times more.  Eight more warps take the sums of one step out of tensor memory while the tensor cores make the next one's.
#include "f16_parts.cuh"

#define PF_FEATS 128
#define PF_ROWS 160
#define PF_K 64               // entries of the inner size a step
#define PF_STAGES 3           // steps whose weights, rows and parts are held
#define PF_WORKERS 8                             // splitters, and as many collectors
#define PF_PART (PF_WORKERS / 4)                 // workers of the same 32 weight rows: each a part of the entries, or of the columns
#define PF_COLS (PF_ROWS / PF_PART)              // columns of sums a collector has
#define PF_MASKS ((PF_COLS + 31) / 32)
#define PF_SPLITTERS 4                           // the first splitter's warp, and the first collector's
#define PF_COLLECTORS (PF_SPLITTERS + PF_WORKERS)
#define PF_THREADS (32 * (PF_COLLECTORS + PF_WORKERS))
#define PF_TABLE 128                             // items of a block whose place is looked up at its start
#define PF_GROUP 12                              // tiles of a dense product whose items are taken together
// registers a thread: at launch, and of each group of warps after it (their sum over the threads is below the launch's)
#define PF_REGS_LAUNCH 96
#define PF_REGS_ISSUE 56
#define PF_REGS_SPLIT 88
#define PF_REGS_COLLECT 120
static_assert(128 * PF_REGS_ISSUE + 32 * PF_WORKERS * (PF_REGS_SPLIT + PF_REGS_COLLECT) <= PF_THREADS * PF_REGS_LAUNCH, "registers of the groups");
#define PF_WBYTES (PF_FEATS * PF_K * 4)
#define PF_XBYTES (2 * PF_ROWS * PF_K * 2)
// tensor memory: the sums of two steps (one in the making, one being read), three stages of the weights' parts
#define PF_SUMS(buffer) ((buffer) * PF_ROWS)
#define PF_PARTS(stage) (2 * PF_ROWS + (stage) * 64)
static_assert(PF_PARTS(PF_STAGES) <= 512, "columns of tensor memory");

using namespace frb_tma;
using namespace frb_tc;

// An item: a tile's rows, and 128 features from f0 on.
struct Item {
    int row0, rows, f0, expert;
};

// Tiles of at most PF_ROWS rows of one expert; without lists (a dense product) tile t is rows PF_ROWS t and on of the only weight matrix.
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
    // outputs to be summed again: for every item and collector whether there are any, and, if so, a lane's columns
    uint8_t* again;            // [items * PF_WORKERS]
    uint32_t* columns;         // [items * PF_WORKERS][PF_MASKS][32]
    int* status;
    int F, K, tiles;           // tiles: without lists
    uint32_t zero;             // 0, which the compiler does not know
    long long rows_total;

    __device__ __forceinline__ int count() const { return num_tiles ? num_tiles[0] : tiles; }
    __device__ __forceinline__ int feature_blocks() const { return (F + PF_FEATS - 1) / PF_FEATS; }

    // The items in the order they are taken.  An expert's: its tiles' features in turn, so that its weights are read in one piece.  A dense
    // product's: PF_GROUP tiles side by side, so that the blocks at work read the same few rows and weights (147 SMs: 12 tiles, 12 blocks
    // of features).
    __device__ __forceinline__ Item item(int i, int tiles_in_all) const {
        const int blocks = feature_blocks(), group = tile_expert ? 1 : PF_GROUP;
        const int first = i / (group * blocks) * group, within = i - first * blocks, width = min(group, tiles_in_all - first);
        const int tile = first + within % width;
        Item it;
        it.f0 = within / width * PF_FEATS;
        it.expert = tile_expert ? tile_expert[tile] : 0;
        it.row0 = tile_row0 ? tile_row0[tile] : tile * PF_ROWS;
        it.rows = min(PF_ROWS, (offsets ? offsets[it.expert + 1] : (int)rows_total) - it.row0);
        return it;
    }
};

// The exponent of a scale, a power of two, whatever its sign: -1 marks a row of zeros.
__device__ __forceinline__ int scale_exponent(float scale) { return (int)(__float_as_uint(scale) >> 23 & 255) - 127; }

// Whether an output is zero for its row's or its weight row's zeros (the other being finite, and the sum zero still).
__device__ __forceinline__ bool is_of_zeros(float sum, float w_scale, float x_scale) {
    return sum == 0.f && (x_scale < 0.f ? w_scale != 0.f : w_scale < 0.f && x_scale != 0.f);
}

// A collector's columns of an item: the sums in units of the scales, to out [rows, features]; which of them are to be summed again.
__device__ __forceinline__ void write_item(const ProductsParams& p, int row0, int rows, int f, float w_scale, const float (&x_scales)[PF_MASKS],
                                           float (&sums)[PF_COLS], long long unit, int lane) {
    const float least = 32.f * (float)p.K;
    uint32_t bad[PF_MASKS] = {};
    const int w_exponent = scale_exponent(w_scale);
    // scales in the middle of float32's range, as a rule: one factor takes both off
    bool middle = w_scale > 0.f && abs(w_exponent) < 64;
#pragma unroll
    for (int i = 0; i < PF_MASKS; ++i) middle = middle && x_scales[i] > 0.f && abs(scale_exponent(x_scales[i])) < 64;
    float* out = p.out + (long long)row0 * p.F + f;
    const bool here = f < p.F;
    if (__all_sync(0xffffffffu, middle)) {
        const float w_factor = __uint_as_float((uint32_t)(127 - w_exponent) << 23);
        float factors[PF_MASKS];
#pragma unroll
        for (int i = 0; i < PF_MASKS; ++i) factors[i] = __uint_as_float((uint32_t)(127 - scale_exponent(x_scales[i])) << 23);
#pragma unroll
        for (int n = 0; n < PF_COLS; ++n) {
            const float factor = w_factor * __shfl_sync(0xffffffffu, factors[n / 32], n % 32), size = fabsf(sums[n]);
            if (n < rows && here) {
                if (!(size >= least && size <= 3.402823466e38f)) bad[n / 32] |= 1u << n % 32;
                *out = sums[n] * factor;
            }
            out += p.F;
            sums[n] = 0.f;
        }
    } else {
#pragma unroll
        for (int n = 0; n < PF_COLS; ++n) {
            const float x_scale = __shfl_sync(0xffffffffu, x_scales[n / 32], n % 32), size = fabsf(sums[n]);
            if (n < rows && here) {
                if (!(size >= least && size <= 3.402823466e38f && w_scale > 0.f && x_scale > 0.f) && !is_of_zeros(sums[n], w_scale, x_scale))
                    bad[n / 32] |= 1u << n % 32;
                // by halves of the exponent, which are factors of float32: a product that the first half cuts off is zero in the end
                const int exponent = w_exponent + scale_exponent(x_scale), half = exponent >> 1;
                *out = sums[n] * __uint_as_float((uint32_t)(127 - half) << 23) * __uint_as_float((uint32_t)(127 - (exponent - half)) << 23);
            }
            out += p.F;
            sums[n] = 0.f;
        }
    }
    uint32_t some = 0;
#pragma unroll
    for (int i = 0; i < PF_MASKS; ++i) some |= bad[i];
    const bool any = __any_sync(0xffffffffu, some != 0);
    if (any)
#pragma unroll
        for (int i = 0; i < PF_MASKS; ++i) p.columns[(unit * PF_MASKS + i) * 32 + lane] = bad[i];
    if (lane == 0) p.again[unit] = any;
}

__global__ void __launch_bounds__(PF_THREADS, 1)
products_f32_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                    const __grid_constant__ ProductsParams p) {
    extern __shared__ uint8_t smem_raw[];
    // weights as float32: copied, split; a step's rows copied and its weights' parts stored; its products done; its sums read
    __shared__ uint64_t w_full[PF_STAGES], w_empty[PF_STAGES], ready[PF_STAGES], done[PF_STAGES], sums_read[2];
    __shared__ Item table[PF_TABLE];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int failed;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    uint8_t* w_ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* x_ring = w_ring + PF_STAGES * PF_WBYTES;
    const int steps = (p.K + PF_K - 1) / PF_K;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PF_STAGES; ++s) {
            bar_init(&w_full[s], 1);
            bar_init(&w_empty[s], PF_WORKERS);
            bar_init(&ready[s], PF_WORKERS + 1);
            bar_init(&done[s], 1);
        }
        for (int s = 0; s < 2; ++s) bar_init(&sums_read[s], PF_WORKERS);
        failed = 0;
        bar_init_fence();
    }
    if (warp == 1) tmem_alloc(&tmem_base_slot, 512);
    const int tiles = p.count(), all_items = tiles * p.feature_blocks();
    const int items = all_items > (int)blockIdx.x ? (all_items - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (threadIdx.x < PF_TABLE && threadIdx.x < items) table[threadIdx.x] = p.item(blockIdx.x + threadIdx.x * gridDim.x, tiles);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    auto item_at = [&](int i) { return i < PF_TABLE ? table[i] : p.item(blockIdx.x + i * gridDim.x, tiles); };

    if (warp < PF_SPLITTERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PF_REGS_ISSUE));
        if (warp == 0) {
            if (lane == 0) {
                int stage = 0;
                uint32_t parity = 1;
                bool ok = true;
                for (int i = 0; i < items && ok; ++i) {
                    const Item it = item_at(i);
                    for (int step = 0; step < steps; ++step) {
                        if (!bar_wait(&w_empty[stage], parity, &failed)) { atomicExch(p.status, 41); ok = false; break; }
                        uint8_t* dst = w_ring + stage * PF_WBYTES;
                        bar_expect(&w_full[stage], PF_WBYTES);
                        load_2d(dst, &map_w, step * PF_K, it.expert * p.F + it.f0, &w_full[stage]);
                        load_2d(dst + PF_WBYTES / 2, &map_w, step * PF_K + 32, it.expert * p.F + it.f0, &w_full[stage]);
                        if (++stage == PF_STAGES) { stage = 0; parity ^= 1; }
                    }
                }
            }
        } else if (warp == 2) {
            if (lane == 0) {
                int stage = 0;
                uint32_t parity = 1;
                bool ok = true;
                for (int i = 0; i < items && ok; ++i) {
                    const int row0 = item_at(i).row0;
                    for (int step = 0; step < steps; ++step) {
                        if (!bar_wait(&done[stage], parity, &failed)) { atomicExch(p.status, 42); ok = false; break; }
                        uint8_t* dst = x_ring + stage * PF_XBYTES;
                        bar_expect(&ready[stage], PF_XBYTES);
                        load_2d(dst, &map_x, step * PF_K, row0, &ready[stage]);
                        load_2d(dst + PF_XBYTES / 2, &map_x, step * PF_K, (int)(row0 + p.rows_total), &ready[stage]);
                        if (++stage == PF_STAGES) { stage = 0; parity ^= 1; }
                    }
                }
            }
        } else if (warp == 1) {
            // the whole warp goes through the loop, so that an MMA's operands are the same in all of its lanes: uniform registers
            const uint32_t x_base = smem_addr(x_ring);
            int stage = 0, buffer = 0;
            uint32_t ready_parity = 0, read_parity = 1;
            bool ok = true;
            for (int i = 0; i < items && ok; ++i) {
                // float32 accumulators, float16 operands, both K-major, M = 128, N = the tile's rows in steps of 16
                const int columns = (item_at(i).rows + 15) & ~15;
                const uint32_t idesc = __shfl_sync(0xffffffffu, (1u << 4) | ((uint32_t)(columns >> 3) << 17) | ((uint32_t)(PF_FEATS >> 4) << 24), 0);
                for (int step = 0; step < steps; ++step) {
                    if (!warp_wait_both(&ready[stage], ready_parity, &sums_read[buffer], read_parity, &failed)) {
                        if (lane == 0) atomicExch(p.status, 43);
                        ok = false;
                        break;
                    }
                    fence_after_sync();
                    const uint32_t hi = tmem + PF_PARTS(stage), lo = hi + 32, sums = tmem + PF_SUMS(buffer);
                    const uint64_t x_hi = tile_desc(x_base + stage * PF_XBYTES), x_lo = x_hi + (PF_XBYTES / 2 >> 4);
                    if (elect_one()) {
                        // the small products first, 2^11 times too large; the first large one takes their sum down
#pragma unroll
                        for (int k = 0; k < PF_K / 16; ++k) mma_ts(sums, lo + 8 * k, x_hi + 2 * k, idesc, k != 0);
#pragma unroll
                        for (int k = 0; k < PF_K / 16; ++k) mma_ts(sums, hi + 8 * k, x_lo + 2 * k, idesc, 1);
                        mma_ts_scaled<11>(sums, hi, x_hi, idesc);
#pragma unroll
                        for (int k = 1; k < PF_K / 16; ++k) mma_ts(sums, hi + 8 * k, x_hi + 2 * k, idesc, 1);
                        mma_commit(&done[stage]);
                    }
                    __syncwarp();
                    if (++stage == PF_STAGES) { stage = 0; ready_parity ^= 1; }
                    if (++buffer == 2) { buffer = 0; read_parity ^= 1; }
                }
            }
        }
    } else if (warp < PF_COLLECTORS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PF_REGS_SPLIT));
        const int quarter = warp & 3, part = (warp - PF_SPLITTERS) >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + part * 16;
        const int r = quarter * 32 + lane;                               // the weight row of the tile that this lane splits
        int stage = 0;
        uint32_t w_parity = 0, done_parity = 1;
        auto scale_of = [&](int i) {
            const Item it = item_at(i);
            return p.w_scale[(long long)it.expert * p.F + min(it.f0 + r, p.F - 1)];
        };
        float scale, next_scale = items > 0 ? scale_of(0) : 0.f;
        bool ok = true;
        for (int i = 0; i < items && ok; ++i) {
            scale = next_scale;
            if (i + 1 < items) next_scale = scale_of(i + 1);
            for (int step = 0; step < steps; ++step) {
                if (!warp_wait(&w_full[stage], w_parity, &failed)) { if (lane == 0) atomicExch(p.status, 44); ok = false; break; }
                // 32 entries of a row are 128 bytes of a box; 16-byte chunk c of row r lies at chunk c ^ (r & 7)
                const uint8_t* src = w_ring + stage * PF_WBYTES + part * (PF_WBYTES / 2) + r * 128;
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 w = *(const float4*)(src + ((c ^ (r & 7)) << 4));
                    split_four(w, scale, hi[2 * c], hi[2 * c + 1], lo[2 * c], lo[2 * c + 1]);
                }
                // The stage is given back once every read of it has ended.  Reads alone may still be on their way: the compiler moves them
                // behind an arrive and a wait, down to the conversions that need them, and by then the next copy may have come.  So the
                // arrive's address is made of what they brought.
                uint32_t brought = 0;
#pragma unroll
                for (int c = 0; c < 8; ++c) brought ^= hi[2 * c];
                __syncwarp();
                if (lane == 0) bar_arrive((uint64_t*)((uint8_t*)&w_empty[stage] + (brought & p.zero)));
                if (!warp_wait(&done[stage], done_parity, &failed)) { if (lane == 0) atomicExch(p.status, 45); ok = false; break; }
                fence_after_sync();
                tmem_st16(lanes + PF_PARTS(stage), hi);
                tmem_st16(lanes + PF_PARTS(stage) + 32, lo);
                tmem_wait_st();
                fence_before_sync();
                __syncwarp();
                if (lane == 0) bar_arrive(&ready[stage]);
                if (++stage == PF_STAGES) { stage = 0; w_parity ^= 1; done_parity ^= 1; }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PF_REGS_COLLECT));
        const int quarter = warp & 3, part = (warp - PF_COLLECTORS) >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + part * PF_COLS;
        int stage = 0, buffer = 0;
        uint32_t done_parity = 0;
        float sums[PF_COLS];
#pragma unroll
        for (int c = 0; c < PF_COLS; ++c) sums[c] = 0.f;
        bool ok = true;
        for (int i = 0; i < items && ok; ++i) {
            const Item it = item_at(i);
            const int row0 = it.row0 + part * PF_COLS, rows = it.rows - part * PF_COLS, f = it.f0 + quarter * 32 + lane;   // rows <= 0: none
            const float w_scale = p.w_scale[(long long)it.expert * p.F + min(f, p.F - 1)];
            float x_scales[PF_MASKS];
#pragma unroll
            for (int m = 0; m < PF_MASKS; ++m) x_scales[m] = 32 * m + lane < min(rows, PF_COLS) ? p.x_scale[row0 + 32 * m + lane] : 1.f;
            for (int step = 0; step < steps; ++step) {
                if (!warp_wait(&done[stage], done_parity, &failed)) { if (lane == 0) atomicExch(p.status, 46); ok = false; break; }
                fence_after_sync();
#pragma unroll
                for (int c = 0; c < PF_COLS / 16; ++c)
                    if (16 * c < rows) {
                        uint32_t v[16];
                        tmem_ld16(lanes + PF_SUMS(buffer) + 16 * c, v);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; ++j) sums[16 * c + j] += __uint_as_float(v[j]);
                    }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) bar_arrive(&sums_read[buffer]);
                if (++stage == PF_STAGES) { stage = 0; done_parity ^= 1; }
                buffer ^= 1;
            }
            if (ok) write_item(p, row0, rows, f, w_scale, x_scales, sums, ((long long)i * gridDim.x + blockIdx.x) * PF_WORKERS + warp - PF_COLLECTORS, lane);
        }
    }
    fence_before_sync();
    __syncthreads();
    if (failed && warp == 0 && lane == 0) {
        // copies may still be on their way into this block's shared memory: give them a bounded time to land
        for (int s = 0; s < PF_STAGES; ++s) { int again = 0; bar_wait(&w_full[s], 0, &again); }
        for (int s = 0; s < PF_STAGES; ++s) { int again = 0; bar_wait(&ready[s], 0, &again); }
    }
    __syncthreads();
    if (warp == 1) tmem_free(tmem, 512);
}

// The outputs to be summed again, a warp each: a warp takes a collector's outputs of an item that have some, and their columns in turn.  A
// kernel of its own: called from the workers' loop the same cost that a quarter of its speed (with tiles of 128 rows, 3,704 rows with 8192 x
// 3072 and 3072 x 6144 weights, on average: 626 us with a kernel of its own, 800 without).  With those weights it takes 25 and 35 us beside
// 450 and 314 of the products.
__global__ void __launch_bounds__(256, 4) products_f32_again_kernel(const __grid_constant__ ProductsParams p) {
    const int lane = threadIdx.x & 31, tiles = p.count();
    const long long units = (long long)tiles * p.feature_blocks() * PF_WORKERS, warps = (long long)gridDim.x * 8;
    for (long long first = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); first < units; first += 32 * warps) {
        const long long mine = first + lane * warps;
        for (uint32_t left = __ballot_sync(0xffffffffu, mine < units && p.again[mine]); left; left &= left - 1) {
            const long long unit = first + (__ffs(left) - 1) * warps;
            const int worker = (int)(unit % PF_WORKERS);
            const Item it = p.item((int)(unit / PF_WORKERS), tiles);
            // the collector of that number: weight rows 32 (number & 3) on, columns of part number / 4
            const int f = it.f0 + (worker & 3) * 32 + lane;
            const int first_row = it.row0 + (worker >> 2) * PF_COLS, rows_here = min(it.rows - (worker >> 2) * PF_COLS, PF_COLS);
            const long long w_row = (long long)it.expert * p.F + min(f, p.F - 1);
#pragma unroll 1
            for (int m = 0; m < PF_MASKS; ++m) {
                const int there = rows_here - 32 * m;                    // whatever a launch that gave up has left in `again`: no row beyond
                const uint32_t within = there >= 32 ? ~0u : there > 0 ? (1u << there) - 1 : 0;
                const uint32_t columns = f < p.F ? p.columns[(unit * PF_MASKS + m) * 32 + lane] & within : 0;
                for (uint32_t all = __reduce_or_sync(0xffffffffu, columns); all; all &= all - 1) {
                    const int n = __ffs(all) - 1;
                    const long long row = (long long)first_row + 32 * m + n;
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
// gated, gate_limit as for frb_split_rows), the rows of each expert together; tiles of at most PF_ROWS rows (null lists: the tiles of
// one weight matrix); out float32 [rows_total, F].  again: scratch, FRB_PRODUCTS_AGAIN bytes for every tile and 128 features.  status:
// one int on the device, zero before the call.
#define FRB_PRODUCTS_AGAIN (PF_WORKERS * (32 * 4 * PF_MASKS + 1))
FRB_API int frb_products_f32(const float* W, const float* w_scale, int num_experts, const void* parts, const float* x_scale, long long rows_total,
                             const float* x, const int* x_rows, int gated, float gate_limit, const int* tile_expert, const int* tile_row0,
                             const int* num_tiles, const int* offsets, int max_tiles, float* out, int F, int K, void* again, int* status,
                             cudaStream_t stream) {
    if (max_tiles == 0 || F == 0) return 0;
    FRB_CHECK_ARG(K > 0 && K % 8 == 0, "float32 products: an inner size of %d is not a multiple of 8", K);
    FRB_CHECK_ARG((((uintptr_t)W | (uintptr_t)parts | (uintptr_t)x) & 15) == 0 && ((uintptr_t)again & 3) == 0,
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
                              (uint8_t*)again + items * PF_WORKERS * 32 * 4 * PF_MASKS, (uint32_t*)again, status, F, K, max_tiles, 0u, rows_total};
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // the groups of warps share out the registers that the block is launched with: fewer, and they would wait for each other's for ever
    static const int registers = [] {
        cudaFuncAttributes attributes;
        return cudaFuncGetAttributes(&attributes, products_f32_kernel) == cudaSuccess ? attributes.numRegs : 0;
    }();
    FRB_CHECK_ARG(registers >= PF_REGS_LAUNCH, "float32 products: the kernel was compiled to %d registers", registers);
    const size_t smem = PF_STAGES * (PF_WBYTES + PF_XBYTES) + 1024;
    cudaFuncSetAttribute(products_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    products_f32_kernel<<<(unsigned)(items < sms ? items : sms), PF_THREADS, smem, stream>>>(map_w, map_x, p);
    products_f32_again_kernel<<<4 * sms, 256, 0, stream>>>(p);
    FRB_RETURN_LAUNCH("products_f32");
}
