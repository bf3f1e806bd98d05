// Float32 attention of prompts on the fifth-generation tensor cores (tcgen05), every operand as two float16 parts (f16_parts.cuh).
//
// Same formulas and options as attention_f32.cu, whose tiles keep the other head sizes and steps of few queries.  A first kernel splits
// the keys and values that the step's queries may see, page by page, each page times a power of two, into scratch that lies as the
// products want it in shared memory (K-major rows of 128 bytes, 128-byte swizzle); keys behind a sequence's end become zeros.
// Then a block takes 128 queries of one head, split once into tensor memory, and walks the pages:
//   S = Q K^T      128 x 64 x HD, three products of parts: the small ones (lo hi, hi lo) first, 2^11 times too large, taken down by
//                  the first of the large ones.  Two buffers, for even and odd pages;
//   softmax        eight warps, a thread a query: four take the even pages, four the odd ones, each with a maximum and a sum of its
//                  own.  Weights of at most 2^14 go back over the scores' columns as two parts;
//   P V            128 x VD x 64 in the same order of parts, from zero for every page: the tensor cores' adder cuts off instead of rounding, so
//                  a page's sum is added to the query's in float32 registers, rounded, when the next page's weights are on their way;
//   the end        the two threads of a query join their sums.
// A query is taken again key by key where a result is not finite (an infinity or a NaN makes its page's, or its query's, parts NaNs, and
// with them all results that the page has a part in), and where parts of one scale may not hold its digits: entries 2^29 times smaller
// than the largest of their query or page, which may be a token's that the query does not see, are off by 2^-51 of that largest.  So a
// query keeps the largest scales of the pages that it sees, and looks at the end whether its scores could be off by what they say
// (FT_SCORE_UNIT) and whether its result is small beside it (FT_VALUE_UNITS): a result that passes is as exact as one without such an entry.
//
// What bounds it: six prompts of 17 to 1,500 tokens (48 heads over 8 of 128) are 48 GFLOP, 144 of parts: 90 us at the tensor cores' rate.
// They take 220 us and 13 for the pages' parts (tiles on mma.sync 1,115).  A page of a tile is 36 products, 1,600 cycles, and takes 1,900: a
// group's weights, their product, the next scores, and its next weights follow one another.  A block's beginning and end, 10,000 and 7,500
// cycles beside the 20,000 of ten pages, are the rest: the tensor memory that it needs leaves no room for a second block.  On the way, in
// microseconds: 268 with the queries read and the results written a row a thread, and a page's sums added after the next page's
// weights; 231 by way of shared memory; 224 with stages given back by the rows instead of by commits.
#include "attention_f32.cuh"
#include "f16_parts.cuh"

#define FT_QUERIES 128
#define FT_STAGES 3
#define FT_THREADS 384         // warps 0-2: copies, products, the sequence's place in the scratch; 4-7 even pages, 8-11 odd ones
#define FT_ROW_THREADS 256
// registers a thread: at launch, and of the first four warps and the others after it (their sum is the launch's)
#define FT_REGS_LAUNCH 168
#define FT_REGS_ISSUE 56
#define FT_REGS_ROWS 224
static_assert(128 * FT_REGS_ISSUE + FT_ROW_THREADS * FT_REGS_ROWS <= FT_THREADS * FT_REGS_LAUNCH, "registers of the groups");
#define FT_LARGEST 1099511627776.f         // 2^40: queries and keys beyond it have no parts; those of a query or page below
#define FT_SMALLEST 8.6736173798840355e-19f      // 2^-60 are split with that one's scale (their products are below 2^-20 of any score)
#define FT_NO_SHIFT 1e30f      // a query's shift before its first visible key
// An entry that its scale leaves below 2^-13 is off by at most 2^-36.  Scores: HD products with parts of the other operand below 2^15, times
// this unit at most: off by less than 2^-21 (2^-29 for errors of random signs), far less than the rounding of scores that large.
#define FT_SCORE_UNIT 0.00390625f          // 2^-8
// Results: a key's weight off by 2^-36 meets values below 2^15, beside a result of at least 2^11 of the same units: 2^-32 of it a key.  The
// largest weight being 2^14, only values 2^18 times larger than the result make it smaller than that.
#define FT_VALUE_UNITS 2048.f

using namespace frb_tma;
using namespace frb_tc;

// The pages that a sequence's new queries may see, in the order of the scratch: the pages of the first tokens that stay visible, then
// those from its first query's window on.
struct PageRun {
    int first, kept, count;
    __device__ __forceinline__ int place(int page) const { return page < kept ? page : kept + page - first; }
};

__device__ __forceinline__ PageRun pages_of(const F32Attention& p, int start, int q_len) {
    PageRun r;
    r.first = first_visible_key(start, p.window, p.chunk) / FRB_PAGE;
    r.kept = kept_runs(p.keep_first, FRB_PAGE, r.first);
    r.count = q_len > 0 ? r.kept + (start + q_len - 1) / FRB_PAGE - r.first + 1 : 0;
    return r;
}

// ----------------------------------------------------------------------------- the pages' parts

// A block a page of one key head (blockIdx.z 0) or value head (1).  Scratch: keys [page][key head][part][HD / 64][64 keys][64 entries],
// values [page][value head][part][VD][64 keys]; inv: what takes a page's scale off, [page][key head], then [page][value head].
template <int HD, int VD>
__global__ void __launch_bounds__(256)
attention_f32_split_kernel(F32Attention p, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, const int* __restrict__ seq_q_len,
                           int num_seqs, int total_pages, uint4* __restrict__ key_parts, uint4* __restrict__ value_parts, float* __restrict__ inv) {
    __shared__ int found[3];                               // sequence, page of it, keys of the page that the sequence holds
    __shared__ float tops[8];
    const bool values = blockIdx.z != 0;
    const int head = blockIdx.y, heads = values ? p.v_heads : p.num_kv_heads, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (head >= heads) return;
    if (warp == 0) {
        if (lane == 0) found[0] = -1;
        __syncwarp();
        for (int b0 = 0, before = 0; b0 < num_seqs; b0 += 32) {
            const int b = b0 + lane;
            PageRun r = {0, 0, 0};
            if (b < num_seqs) r = pages_of(p, seq_start[b], seq_q_len[b]);
            int end = r.count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int lower = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= o) end += lower;
            }
            const int begin = before + end - r.count, i = blockIdx.x - begin;
            if (i >= 0 && i < r.count) {
                const int page = run_at(i, r.kept, r.first);
                found[0] = b;
                found[1] = page;
                found[2] = min(FRB_PAGE, seq_start[b] + seq_q_len[b] - page * FRB_PAGE);
            }
            before += __shfl_sync(0xffffffffu, end, 31);
            if (before > (int)blockIdx.x) break;
        }
    }
    __syncthreads();
    if (found[0] < 0) return;
    const int there = found[2];
    const size_t page = p.page_table[(size_t)seq_slot[found[0]] * p.max_pages + found[1]];
    constexpr int K_UNITS = FRB_PAGE * HD / 8, V_UNITS = VD * FRB_PAGE / 8, MOST = (K_UNITS > V_UNITS ? K_UNITS : V_UNITS) / 256;
    const int units = values ? V_UNITS : K_UNITS;
    const float4* src = (const float4*)(values ? p.v_pages + (page * heads + head) * VD * FRB_PAGE : p.k_pages + (page * heads + head) * FRB_PAGE * HD);
    float4 v[MOST][2];
    float top = 0.f;
    bool whole = true;                                     // no infinity, no NaN
#pragma unroll
    for (int i = 0; i < MOST; ++i) {
        const int u = threadIdx.x + 256 * i;
        if (u < units) {
            v[i][0] = src[2 * u];
            v[i][1] = src[2 * u + 1];
            float* e = (float*)v[i];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int key = values ? (u & 7) * 8 + j : u / (HD / 8);
                if (key >= there) e[j] = 0.f;
                whole = whole && fabsf(e[j]) <= 3.402823466e38f;
                top = fmaxf(top, fabsf(e[j]));
            }
        }
    }
    top = warp_max(whole ? top : INFINITY);
    if (lane == 0) tops[warp] = top;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) top = fmaxf(top, tops[w]);
    whole = top <= (values ? 3.402823466e38f : FT_LARGEST);
    const int exponent = whole ? min(14 - ilogbf(fmaxf(top, values ? 1.1754943508222875e-38f : FT_SMALLEST)), 126) : 0;
    const float scale = power_of_two(exponent);
    if (threadIdx.x == 0) inv[(values ? (size_t)total_pages * p.num_kv_heads : 0) + (size_t)blockIdx.x * heads + head] = top > 0.f ? power_of_two(-exponent) : 0.f;
    uint4* dst = (values ? value_parts : key_parts) + ((size_t)blockIdx.x * heads + head) * 2 * units;
#pragma unroll
    for (int i = 0; i < MOST; ++i) {
        const int u = threadIdx.x + 256 * i;
        if (u < units) {
            uint4 hi, lo;
            split_four(v[i][0], scale, hi.x, hi.y, lo.x, lo.y);
            split_four(v[i][1], scale, hi.z, hi.w, lo.z, lo.w);
            if (!whole) hi = lo = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
            // unit (row, chunk of eight entries); keys: 64 entries of all 64 rows, then the next 64
            const int row = values ? u >> 3 : u / (HD / 8), chunk = values ? u & 7 : u % (HD / 8);
            const int at = (chunk >> 3) * (FRB_PAGE * 8) + row * 8 + ((chunk & 7) ^ (row & 7));
            dst[at] = hi;
            dst[units + at] = lo;
        }
    }
}

// ----------------------------------------------------------------------------- the tiles

// grid (head, tile of 128 queries).  MODIFIED: capped scores or slopes.
template <int HD, int VD, bool MODIFIED>
__global__ void __launch_bounds__(FT_THREADS, 1)
attention_f32_tc_kernel(F32Attention p, const int* __restrict__ tile_seq, const int* __restrict__ tile_q0, const int* __restrict__ seq_slot,
                        const int* __restrict__ seq_start, const int* __restrict__ seq_q_len, const int* __restrict__ cu_q_len, int total_pages,
                        const uint8_t* __restrict__ key_parts, const uint8_t* __restrict__ value_parts, const float* __restrict__ inv,
                        int* __restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t q_full, k_full[FT_STAGES], k_empty[FT_STAGES], v_full[FT_STAGES], v_empty[FT_STAGES];
    __shared__ uint64_t s_full[2], p_full[2], o_full[2];          // of even and odd pages
    __shared__ float q_top[2][FT_QUERIES], told[2][4][FT_QUERIES];
    __shared__ int again[FT_QUERIES], held[FT_QUERIES], base_slot, failed_flag;
    __shared__ uint32_t tmem_slot;
    volatile int* failed = &failed_flag;
    constexpr uint32_t K_PART = FRB_PAGE * HD * 2, V_PART = VD * FRB_PAGE * 2;     // bytes of one part of a page
    constexpr int Q_HI = 0, Q_LO = HD / 2;
    auto sp_cols = [](int e) { return HD + FRB_PAGE * e; };
    auto o_cols = [](int e) { return HD + 2 * FRB_PAGE + VD * e; };
    static_assert(HD + 2 * FRB_PAGE + 2 * VD <= 512, "columns of tensor memory");

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int head = blockIdx.x, tile = gridDim.y - 1 - blockIdx.y;          // the last tiles of a sequence see the most keys
    const int seq = tile_seq[tile], q0 = tile_q0[tile], q_len = seq_q_len[seq], start = seq_start[seq];
    const int rows = min(FT_QUERIES, q_len - q0), pos0 = start + q0;
    const size_t token0 = (size_t)cu_q_len[seq] + q0;
    const int group = p.num_heads / p.num_kv_heads, g = head / group, vg = g / (p.num_kv_heads / p.v_heads);
    const PageRun run = pages_of(p, start, q_len);
    const int first_page = first_visible_key(pos0, p.window, p.chunk) / FRB_PAGE, kept = kept_runs(p.keep_first, FRB_PAGE, first_page);
    const int pages = __shfl_sync(0xffffffffu, kept + (pos0 + rows - 1) / FRB_PAGE - first_page + 1, 0);

    uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* k_ring = base;
    uint8_t* v_ring = base + FT_STAGES * 2 * K_PART;

    // The queries are on their way while barriers and tensor memory are set up: a warp of the rows fetches its 32 queries' half of the
    // entries, eight neighbouring lanes 128 bytes of a query at a time.
    float4 fetched[HD / 64][8];
    if (warp >= 4)
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = (warp & 3) * 32 + 4 * i + (lane >> 3);
                fetched[c][i] = r < rows ? *(const float4*)(p.q + ((token0 + r) * p.num_heads + head) * HD + ((warp - 4) >> 2) * (HD / 2) + 32 * c + 4 * (lane & 7))
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
            }

    if (threadIdx.x == 0) {
        bar_init(&q_full, 8);
        for (int s = 0; s < FT_STAGES; ++s) { bar_init(&k_full[s], 1); bar_init(&k_empty[s], 1); bar_init(&v_full[s], 1); bar_init(&v_empty[s], 1); }
        for (int e = 0; e < 2; ++e) { bar_init(&s_full[e], 1); bar_init(&p_full[e], 4); bar_init(&o_full[e], 1); }
        failed_flag = 0;
        bar_init_fence();
    }
    if (threadIdx.x < FT_QUERIES) again[threadIdx.x] = held[threadIdx.x] = 0;
    if (warp == 1) tmem_alloc(&tmem_slot, 512);
    if (warp == 2) {                                       // the scratch's pages before this sequence's
        int before = 0;
        for (int b = lane; b < seq; b += 32) before += pages_of(p, seq_start[b], seq_q_len[b]).count;
        before = __reduce_add_sync(0xffffffffu, before);
        if (lane == 0) base_slot = before;
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    // the scratch's place of the tile's n-th page
    auto place = [&](int n) { return (size_t)base_slot + run.place(run_at(n, kept, first_page)); };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FT_REGS_ISSUE));
        if (warp == 0) {
            if (lane == 0) {
                for (int n = 0; n < pages; ++n) {
                    const int s = n % FT_STAGES;
                    const uint32_t parity = ((n / FT_STAGES) & 1) ^ 1;
                    if (n == FT_STAGES - 1 && !bar_wait(&q_full, 0, failed)) { atomicExch(status, 54); break; }     // the queries pass through there
                    if (!bar_wait(&k_empty[s], parity, failed)) { atomicExch(status, 51); break; }
                    bar_expect(&k_full[s], 2 * K_PART);
                    copy_bulk(k_ring + s * 2 * K_PART, key_parts + (place(n) * p.num_kv_heads + g) * 2 * K_PART, 2 * K_PART, &k_full[s]);
                    if (!bar_wait(&v_empty[s], parity, failed)) { atomicExch(status, 52); break; }
                    bar_expect(&v_full[s], 2 * V_PART);
                    copy_bulk(v_ring + s * 2 * V_PART, value_parts + (place(n) * p.v_heads + vg) * 2 * V_PART, 2 * V_PART, &v_full[s]);
                }
            }
        } else if (warp == 1) {
            // The whole warp goes through the loop (elect_one, tcgen05.cuh).  Its products run in the order of their issue, so the scores
            // of page n + 2 may be asked for over the weights of page n, whose product has been.
            constexpr uint32_t idesc_s = (1u << 4) | ((uint32_t)(FRB_PAGE >> 3) << 17) | ((uint32_t)(FT_QUERIES >> 4) << 24);
            constexpr uint32_t idesc_o = (1u << 4) | ((uint32_t)(VD >> 3) << 17) | ((uint32_t)(FT_QUERIES >> 4) << 24);
            const uint32_t k_at = smem_addr(k_ring), v_at = smem_addr(v_ring);
            auto scores = [&](int n) -> bool {
                const int s = n % FT_STAGES, e = n & 1;
                if (!warp_wait(&k_full[s], (n / FT_STAGES) & 1, failed)) { if (lane == 0) atomicExch(status, 53); return false; }
                fence_after_sync();
                const uint64_t hi = tile_desc(k_at + s * 2 * K_PART), lo = hi + (K_PART >> 4);
                if (elect_one()) {
                    products_of_parts<HD / 16>(tmem + sp_cols(e), tmem + Q_HI, tmem + Q_LO, hi, lo, idesc_s,
                                               [](int k) { return (k / 4) * (FRB_PAGE * 128 >> 4) + (k % 4) * 2; });
                    mma_commit(&s_full[e]);
                }
                __syncwarp();
                return true;
            };
            bool ok = warp_wait(&q_full, 0, failed);
            if (!ok && lane == 0) atomicExch(status, 54);
            if (ok) ok = scores(0) && (pages < 2 || scores(1));
            for (int n = 0; n < pages && ok; ++n) {
                const int s = n % FT_STAGES, e = n & 1;
                if (!warp_wait_both(&v_full[s], (n / FT_STAGES) & 1, &p_full[e], (n >> 1) & 1, failed)) { if (lane == 0) atomicExch(status, 55); break; }
                fence_after_sync();
                const uint64_t hi = tile_desc(v_at + s * 2 * V_PART), lo = hi + (V_PART >> 4);
                if (elect_one()) {
                    products_of_parts<FRB_PAGE / 16>(tmem + o_cols(e), tmem + sp_cols(e), tmem + sp_cols(e) + FRB_PAGE / 2, hi, lo, idesc_o,
                                                     [](int k) { return k * 2; });
                    mma_commit(&o_full[e]);
                }
                __syncwarp();
                if (n + 2 < pages) ok = scores(n + 2);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FT_REGS_ROWS));
        // A wait that gives up does not end the loop: the block's later waits then return at once, and every thread reaches the barriers
        // of the end.
        const int e = (warp - 4) >> 2, quarter = warp & 3, row = quarter * 32 + lane;        // the query = the lane of tensor memory
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        const bool valid = row < rows;
        const int pos = valid ? pos0 + row : -1, low = valid ? first_visible_key(pos, p.window, p.chunk) : 0;
        const float slope = MODIFIED && p.slopes ? p.slopes[head] : 0.f;
        float q_factor;                                    // the scale of the softmax, and what takes the query's off
        bool ok = true;
        {
            // This thread's half of its query, by way of shared memory (the rings' last stage, whose first copies wait for q_full): chunk c of
            // row r lies at chunk c ^ (r & 7).
            float4 q[HD / 8];
            float4* staged = (float4*)((e == 0 ? k_ring + (FT_STAGES - 1) * 2 * K_PART : v_ring + (FT_STAGES - 1) * 2 * V_PART) + quarter * 4096);
            float top = 0.f;
            bool whole = true;
#pragma unroll
            for (int c = 0; c < HD / 64; ++c) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = 4 * i + (lane >> 3);
                    staged[r * 8 + ((lane & 7) ^ (r & 7))] = fetched[c][i];
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) q[8 * c + i] = staged[lane * 8 + (i ^ (lane & 7))];
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll
            for (int i = 0; i < HD / 8; ++i) {
                const float m = fmaxf(fmaxf(fabsf(q[i].x), fabsf(q[i].y)), fmaxf(fabsf(q[i].z), fabsf(q[i].w)));
                whole = whole && fabsf(q[i].x) <= FT_LARGEST && fabsf(q[i].y) <= FT_LARGEST && fabsf(q[i].z) <= FT_LARGEST && fabsf(q[i].w) <= FT_LARGEST;
                top = fmaxf(top, m);
            }
            q_top[e][row] = whole ? top : INFINITY;
            asm volatile("bar.sync 1, %0;" ::"n"(FT_ROW_THREADS) : "memory");
            top = fmaxf(q_top[0][row], q_top[1][row]);
            whole = top <= FT_LARGEST;
            const int exponent = whole ? 14 - ilogbf(fmaxf(top, FT_SMALLEST)) : 0;
            const float scale = power_of_two(exponent);
            q_factor = p.scale * power_of_two(-exponent);
#pragma unroll
            for (int c = 0; c < HD / 64; ++c) {            // 16 columns: 32 entries
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 8; ++i) split_four(q[8 * c + i], scale, hi[2 * i], hi[2 * i + 1], lo[2 * i], lo[2 * i + 1]);
                if (!whole)
#pragma unroll
                    for (int i = 0; i < 16; ++i) hi[i] = lo[i] = 0x7fff7fffu;
                tmem_st16(lanes + Q_HI + e * (HD / 4) + 16 * c, hi);
                tmem_st16(lanes + Q_LO + e * (HD / 4) + 16 * c, lo);
            }
            tmem_wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&q_full);
        }
        float o[VD], sum = 0.f, shift = FT_NO_SHIFT;       // weights are 2^(score log2(e) + shift)
#pragma unroll
        for (int i = 0; i < VD; ++i) o[i] = 0.f;
        float corr_before = 1.f, value_before = 0.f;       // of the page whose sums are still to be added
        float key_largest = 0.f, value_largest = 0.f;      // of the pages that the query sees: what takes their scales off
        auto add_page = [&](int n) {
            if (!bar_wait(&o_full[e], (n >> 1) & 1, failed)) { if (ok && lane == 0) atomicExch(status, 58); ok = false; }
            __syncwarp();
            fence_after_sync();
            if (quarter == 0 && lane == 0) bar_arrive(&v_empty[n % FT_STAGES]);      // the product has ended: its values' stage is free
            const uint64_t corr = pair_of(corr_before, corr_before), factor = pair_of(value_before, value_before);
#pragma unroll
            for (int c0 = 0; c0 < VD / 16; c0 += 4) {
                uint32_t v[4][16];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld16(lanes + o_cols(e) + 16 * (c0 + c), v[c]);
                tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        float& even = o[16 * (c0 + c) + i];
                        float& odd = o[16 * (c0 + c) + i + 1];
                        halves_of(fma_pairs(pair_of(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])), factor,
                                            mul_pairs(pair_of(even, odd), corr)), even, odd);
                    }
            }
        };
        const float* key_inv = inv + g;
        const float* value_inv = inv + (size_t)total_pages * p.num_kv_heads + vg;
        for (int n = e; n < pages; n += 2) {
            const size_t at = place(n);
            const float key_factor = key_inv[at * p.num_kv_heads], value_factor = value_inv[at * p.v_heads];
            const int key0 = run_at(n, kept, first_page) * FRB_PAGE;
            if (n >= 2) add_page(n - 2);
            if (!bar_wait(&s_full[e], (n >> 1) & 1, failed)) { if (ok && lane == 0) atomicExch(status, 59); ok = false; }
            __syncwarp();
            fence_after_sync();
            if (quarter == 0 && lane == 0) bar_arrive(&k_empty[n % FT_STAGES]);      // and so is the keys' one here
            uint32_t raw[4][16];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld16(lanes + sp_cols(e) + 16 * c, raw[c]);
            tmem_wait_ld();
            float scale = fmaxf(q_factor * key_factor, 1e-30f);      // products are below 2^38: what is smaller makes no score either
            if (MODIFIED) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float s = __uint_as_float(raw[c][i]) * scale;
                        if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
                        raw[c][i] = __float_as_uint(s - slope * (float)(pos - (key0 + 16 * c + i)));
                    }
                scale = 1.f;
            }
            if (!__all_sync(0xffffffffu, valid && key0 + FRB_PAGE - 1 <= pos && (key0 >= low || key0 + FRB_PAGE <= p.keep_first))) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (!key_visible(key0 + 16 * c + i, low, pos, p.keep_first)) raw[c][i] = 0xff800000u;
            }
            float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 16; i += 2)
                    top[(i >> 1) & 3] = max3(top[(i >> 1) & 3], __uint_as_float(raw[c][i]), __uint_as_float(raw[c][i + 1]));
            // the scale times log2(e) in two float32 numbers: a score's power of two is off by the rounding of what is left of it beside the
            // maximum, not of the score itself.  The first is rounded down, so that the second is positive: a hidden key stays at -infinity
            constexpr float LOG2E = 1.4426950408889634f, LOG2E_LO = (float)(1.4426950408889634 - (double)LOG2E);
            static_assert(LOG2E_LO > 0.f, "the second number is positive");
            const float c_hi = __fmul_rd(scale, LOG2E), c_lo = fmaf(scale, LOG2E_LO, fmaf(scale, LOG2E, -c_hi));
            const float page_top = max3(fmaxf(top[0], top[1]), top[2], top[3]);
            const float shift_now = page_top == -INFINITY ? shift : fminf(shift, 14.f - page_top * c_hi);
            if (page_top != -INFINITY) {
                key_largest = fmaxf(key_largest, key_factor);
                value_largest = fmaxf(value_largest, value_factor);
            }
            const float corr = exp2_fast(shift_now - shift);
            shift = shift_now;
            const uint64_t hi_pair = pair_of(c_hi, c_hi), lo_pair = pair_of(c_lo, c_lo), shift_pair = pair_of(shift, shift);
            uint64_t sums[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
            for (int half = 0; half < 2; ++half) {         // 32 keys: 16 columns of either part
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const uint32_t* at2 = &raw[2 * half + i / 8][2 * (i % 8)];
                    const uint64_t x = pair_of(__uint_as_float(at2[0]), __uint_as_float(at2[1]));
                    float y0, y1;
                    halves_of(fma_pairs(x, lo_pair, fma_pairs(x, hi_pair, shift_pair)), y0, y1);
                    const uint64_t w = pair_of(exp2_fast(y0), exp2_fast(y1));
                    sums[i & 3] = add_pairs(sums[i & 3], w);
                    split_two(w, hi[i], lo[i]);
                }
                // over the scores, which are all in registers: the large parts in their first half's columns
                tmem_st16(lanes + sp_cols(e) + 16 * half, hi);
                tmem_st16(lanes + sp_cols(e) + FRB_PAGE / 2 + 16 * half, lo);
            }
            float even, odd;
            halves_of(add_pairs(add_pairs(sums[0], sums[1]), add_pairs(sums[2], sums[3])), even, odd);
            sum = fmaf(sum, corr, even + odd);
            tmem_wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&p_full[e]);                   // its weights are there, and the sums of its page before are read
            corr_before = corr;
            value_before = value_factor;
        }
        const int last = pages - 1 - ((pages - 1 - e) & 1);          // this group's last page, if it has one
        if (last >= 0) add_page(last);
        // The two threads of a query tell each other their shift and sum, and leave their values' sums in shared memory (the rings are free
        // when both groups have come here: every product has ended), chunk c of row r at chunk c ^ (r & 7).
        told[e][0][row] = shift;
        told[e][1][row] = sum;
        told[e][2][row] = q_factor * key_largest;
        told[e][3][row] = value_largest;
        asm volatile("bar.sync 1, %0;" ::"n"(FT_ROW_THREADS) : "memory");
        float4* mine4 = (float4*)(base + e * (FT_QUERIES * VD * 4)) + row * (VD / 4);
#pragma unroll
        for (int i = 0; i < VD / 4; ++i) mine4[i ^ (row & 7)] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
        if (e == 0) {                                      // a query's factors for the two sums
            const float shift0 = told[0][0][row], shift1 = told[1][0][row];
            float least = fminf(shift0, shift1), total = 0.f;
            if (p.sinks) {
                const float sink = p.sinks[head] * 1.4426950408889634f;
                least = fminf(least, 14.f - sink);
                total = exp2_fast(sink + least);
            }
            const float w0 = exp2_fast(least - shift0), w1 = exp2_fast(least - shift1);
            total += fmaf(told[0][1][row], w0, told[1][1][row] * w1);
            float factor = 1.0f / total;
            if (p.gate && valid) factor *= 1.0f / (1.0f + expf(-p.gate[(token0 + row) * p.gate_stride + head]));
            q_top[0][row] = w0 * factor;
            q_top[1][row] = w1 * factor;
            if (fmaxf(told[0][2][row], told[1][2][row]) > FT_SCORE_UNIT) again[row] = 1;
            told[0][0][row] = FT_VALUE_UNITS * fmaxf(told[0][3][row], told[1][3][row]) * (fmaxf(w0, w1) * factor);      // the least that holds its digits
        }
        asm volatile("bar.sync 1, %0;" ::"n"(FT_ROW_THREADS) : "memory");
        for (int u = threadIdx.x - 128; u < rows * (VD / 4); u += FT_ROW_THREADS) {
            const int r = u / (VD / 4), chunk = u % (VD / 4), at = r * (VD / 4) + (chunk ^ (r & 7));
            const float4 a = ((const float4*)base)[at], b = ((const float4*)(base + FT_QUERIES * VD * 4))[at];
            const float wa = q_top[0][r], wb = q_top[1][r];
            const float4 y = make_float4(fmaf(a.x, wa, b.x * wb), fmaf(a.y, wa, b.y * wb), fmaf(a.z, wa, b.z * wb), fmaf(a.w, wa, b.w * wb));
            ((float4*)(p.out + ((token0 + r) * p.num_heads + head) * VD))[chunk] = y;
            const float largest = fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w)));
            if (!(fabsf(y.x) <= 3.402823466e38f && fabsf(y.y) <= 3.402823466e38f && fabsf(y.z) <= 3.402823466e38f && fabsf(y.w) <= 3.402823466e38f)) again[r] = 1;
            if (largest >= told[0][0][r]) held[r] = 1;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(FT_ROW_THREADS) : "memory");
        const int* table = p.page_table + (size_t)seq_slot[seq] * p.max_pages;
        const bool whole = ok && !*failed;
        for (uint32_t left = __ballot_sync(0xffffffffu, valid && (again[row] != 0 || held[row] == 0) && whole && (lane & 1) == e); left; left &= left - 1) {
            const int r = quarter * 32 + __ffs(left) - 1;
            f32_query_key_by_key(p, table, head, g, vg, pos0 + r, token0 + r);
        }
    }
    fence_before_sync();
    __syncthreads();
    if (failed_flag && warp == 0 && lane == 0) {
        // copies may still be on their way into this block's shared memory: give them a bounded time to land
        for (int s = 0; s < FT_STAGES; ++s) { int zero = 0; bar_wait(&k_full[s], 0, &zero); zero = 0; bar_wait(&v_full[s], 0, &zero); }
    }
    __syncthreads();
    if (warp == 1) tmem_free(tmem, 512);
}

// ----------------------------------------------------------------------------- host side

// tile_seq/tile_q0: the step's tiles of 128 queries; total_pages: pages that the sequences' new queries may see, in all.  Scratch: the
// keys' parts, total_pages * kv heads * 64 * head_dim * 4 bytes, the values', total_pages * value heads * 64 * v_dim * 4 bytes, and
// total_pages * (kv heads + value heads) floats.  status: one int on the device, zero before the call.
FRB_API int frb_attention_f32_tc(const float* q, const float* k_pages, const float* v_pages, const int* page_table, int max_pages,
                                 const int* tile_seq, const int* tile_q0, int num_tiles, const int* seq_slot, const int* seq_start,
                                 const int* seq_q_len, const int* cu_q_len, int num_seqs, int total_pages, float* scratch, int* status,
                                 float* out, int num_heads, int num_kv_heads, int head_dim, int v_dim, float scale, int window,
                                 const float* slopes, int chunk, const float* sinks, const float* gate, int gate_stride, float softcap,
                                 int keep_first, int num_v_heads, cudaStream_t stream) {
    if (num_tiles == 0) return 0;
    FRB_CHECK_ARG((head_dim == 64 && (v_dim == 64 || v_dim == 128)) || (head_dim == 128 && v_dim == 128),
                  "float32 attention on tcgen05: heads of %d over values of %d", head_dim, v_dim);
    FRB_CHECK_ARG(scale > 0.f, "float32 attention on tcgen05: a softmax scale of %g is not positive", (double)scale);
    FRB_CHECK_ARG(num_tiles <= 65535 && num_kv_heads <= 65535 && total_pages > 0, "float32 attention on tcgen05: %d tiles of %d pages exceed the grid",
                  num_tiles, total_pages);
    FRB_CHECK_ARG((((uintptr_t)scratch | (uintptr_t)out) & 15) == 0, "float32 attention on tcgen05: scratch must be 16-byte aligned");
    F32Attention p;
    const int bad = f32_attention_params(&p, q, k_pages, v_pages, page_table, max_pages, out, num_heads, num_kv_heads, head_dim, v_dim, scale,
                                         window, slopes, chunk, sinks, gate, gate_stride, softcap, keep_first, num_v_heads);
    if (bad) return bad;
    float* key_parts = scratch;
    float* value_parts = key_parts + (size_t)total_pages * num_kv_heads * FRB_PAGE * head_dim;
    float* inv = value_parts + (size_t)total_pages * num_v_heads * FRB_PAGE * v_dim;
    const dim3 pages(total_pages, num_kv_heads, 2), grid(num_heads, num_tiles);
    const size_t smem = (size_t)FT_STAGES * FRB_PAGE * (head_dim + v_dim) * 4 + 1024;
#define FRB_TC_TILES(HD, VD, MODIFIED)                                                                                                    \
    do {                                                                                                                                  \
        auto kernel = attention_f32_tc_kernel<HD, VD, MODIFIED>;                                                                          \
        cudaFuncAttributes attributes;                                                                                                    \
        /* the groups of warps share out the registers that the block is launched with: fewer, and they would wait for ever */            \
        static const int registers = cudaFuncGetAttributes(&attributes, kernel) == cudaSuccess ? attributes.numRegs : 0;                  \
        FRB_CHECK_ARG(registers >= FT_REGS_LAUNCH, "float32 attention on tcgen05: the kernel was compiled to %d registers", registers);   \
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                                             \
        attention_f32_split_kernel<HD, VD><<<pages, 256, 0, stream>>>(p, seq_slot, seq_start, seq_q_len, num_seqs, total_pages,           \
                                                                      (uint4*)key_parts, (uint4*)value_parts, inv);                       \
        kernel<<<grid, FT_THREADS, smem, stream>>>(p, tile_seq, tile_q0, seq_slot, seq_start, seq_q_len, cu_q_len, total_pages,           \
                                                   (const uint8_t*)key_parts, (const uint8_t*)value_parts, inv, status);                  \
    } while (0)
    const bool modified = slopes || softcap > 0.f;
    if (head_dim == 128) { if (modified) FRB_TC_TILES(128, 128, true); else FRB_TC_TILES(128, 128, false); }
    else if (v_dim == 128) { if (modified) FRB_TC_TILES(64, 128, true); else FRB_TC_TILES(64, 128, false); }
    else { if (modified) FRB_TC_TILES(64, 64, true); else FRB_TC_TILES(64, 64, false); }
#undef FRB_TC_TILES
    FRB_RETURN_LAUNCH("attention_f32_tc");
}
