// Attention over the paged cache in float32 for the head sizes that models have: the float32 path's prompts in tiles of 64
// queries, and its single tokens in chunks of 256 keys that run side by side.  Same formulas and options as
// attention_generic.cu (window, chunk, first tokens, slopes, sinks, cap, gates, a value head of another size, key heads that
// share a value head), which keeps the sizes these kernels do not take; attention_f32_tc.cu takes all but the smallest steps of prompts with
// heads of 64 and 128.  Everything is float32; the tiles' products run on tensor
// cores with each operand as two TF32 parts (tf32_parts.cuh).
//
// What bounds them.  Prompts: the instructions that split the operands and the tensor cores; attention_generic runs a block per
// token, which reads the token's keys and values for itself through scalar loads, and a warp's 32 keys through one chain of
// multiply-adds: 15.2 ms for six prompts of 17 to 1,500 tokens (48 heads over 8 of 128, 3.1 TFLOP/s).  Tiles of 64 queries with 8 x 4
// scores and 8 x 8 sums a thread on the ordinary pipes took 1.59 ms (30 TFLOP/s), on the tensor cores 1.12 ms (43).  Single tokens: the
// keys' and values' bytes; there a block per token and key head left 48 blocks on 148 SMs, each walking its whole sequence: 1.20 ms
// for six sequences of 17 to 1,500 keys; the whole layer went from 1.33 to 0.08 ms, most of it the dense products.
#include "attention_f32.cuh"
#include "tf32_parts.cuh"

__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
    c = fmaf(a.x, b.x, c);
    c = fmaf(a.y, b.y, c);
    c = fmaf(a.z, b.z, c);
    return fmaf(a.w, b.w, c);
}

// ----------------------------------------------------------------------------- prompts

#define TILE_Q 64             // queries of one head a block takes
#define TILE_THREADS 128

// A block takes 64 neighbouring queries of one head and walks the pages of 64 keys that any of them sees; a warp has 16 of the
// queries.  Both products run on tensor cores with each operand as two TF32 parts; the weights stay in the registers that the
// scores are in, which are those that the second product wants them in.  A page's sums are added to the queries' in float32,
// rounded (over thousands of keys the tensor cores' adder, which cuts off, would cost more than a rounding).  The next page's keys
// are on their way while this page's values are summed, its values while the next scores are computed.  NT: column tiles of eight
// value entries.
//
// A query whose results are not all finite is taken again by its warp, key by key and with the hidden ones left out: an infinity has no
// parts, and a hidden value counts here with a weight of zero, which an infinity or a NaN does not bear.
template <int NT>
__global__ void __launch_bounds__(TILE_THREADS, 2)
attention_f32_tiles_kernel(F32Attention p, const int* __restrict__ tile_seq, const int* __restrict__ tile_q0,
                           const int* __restrict__ seq_slot, const int* __restrict__ seq_start, const int* __restrict__ seq_q_len,
                           const int* __restrict__ cu_q_len) {
    constexpr int LV = FRB_PAGE + 8;
    extern __shared__ float4 f32_smem[];
    const int hd = p.head_dim, vd = p.v_dim;
    const int hd8 = (hd + 7) & ~7, ld = ((hd + 31) & ~31) + 8;           // entries of the inner size; a row's place
    float* q_s = (float*)f32_smem;                         // [TILE_Q][ld]
    float* k_s = q_s + TILE_Q * ld;                        // [FRB_PAGE][ld]
    float* v_s = k_s + FRB_PAGE * ld;                      // [8 NT][LV]
    // the last tiles of the sequences see the most keys: they begin first.  A tile of the step's lists is 128 queries: two blocks
    const int unit = gridDim.y - 1 - blockIdx.y;
    const int head = blockIdx.x, seq = tile_seq[unit >> 1];
    const int q0 = tile_q0[unit >> 1] + TILE_Q * (unit & 1), q_len = seq_q_len[seq];
    if (q0 >= q_len) return;
    const int rows = min(TILE_Q, q_len - q0);
    const int pos0 = seq_start[seq] + q0, last = pos0 + rows - 1;
    const size_t token0 = (size_t)cu_q_len[seq] + q0;
    const int group = p.num_heads / p.num_kv_heads, g = head / group, vg = g / (p.num_kv_heads / p.v_heads);
    const int first_page = first_visible_key(pos0, p.window, p.chunk) / FRB_PAGE;
    const int kept = kept_runs(p.keep_first, FRB_PAGE, first_page);
    const int pages = kept + last / FRB_PAGE - first_page + 1;
    const int* table = p.page_table + (size_t)seq_slot[seq] * p.max_pages;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g8 = lane >> 2, t4 = lane & 3;
    const int units = hd >> 2;

    // entries that no copy fills: the queries' and keys' padding, queries beyond the tile, value rows beyond v_dim
    for (int i = tid; i < TILE_Q * (ld / 4); i += TILE_THREADS) {
        const int r = i / (ld / 4), u = i - r * (ld / 4);
        if (u >= units || r >= rows) *(float4*)(q_s + r * ld + 4 * u) = make_float4(0.f, 0.f, 0.f, 0.f);
        if (u >= units) *(float4*)(k_s + r * ld + 4 * u) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int i = vd * LV + tid; i < 8 * NT * LV; i += TILE_THREADS) v_s[i] = 0.f;

    auto copy_keys = [&](int n) {
        const float* src = p.k_pages + ((size_t)table[run_at(n, kept, first_page)] * p.num_kv_heads + g) * FRB_PAGE * hd;
        for (int r = warp; r < FRB_PAGE; r += TILE_THREADS / 32)
            for (int u = lane; u < units; u += 32) copy16_async(k_s + r * ld + 4 * u, src + r * hd + 4 * u);
    };
    auto copy_values = [&](int n) {
        const float* src = p.v_pages + ((size_t)table[run_at(n, kept, first_page)] * p.v_heads + vg) * FRB_PAGE * vd;
        for (int d = tid >> 4; d < vd; d += TILE_THREADS / 16) copy16_async(v_s + d * LV + 4 * (tid & 15), src + d * FRB_PAGE + 4 * (tid & 15));
    };
    for (int r = warp; r < rows; r += TILE_THREADS / 32)
        for (int u = lane; u < units; u += 32) copy16_async(q_s + r * ld + 4 * u, p.q + ((token0 + r) * p.num_heads + head) * hd + 4 * u);
    copy_keys(0);
    copies_commit();
    copy_values(0);
    copies_commit();

    const float slope = p.slopes ? p.slopes[head] : 0.f;
    const int pos[2] = {pos0 + warp * 16 + g8, pos0 + warp * 16 + g8 + 8};
    const int lo[2] = {first_visible_key(pos[0], p.window, p.chunk), first_visible_key(pos[1], p.window, p.chunk)};
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, acc[NT][4] = {};
    const float* q_rows = q_s + warp * 16 * ld;

    for (int n = 0; n < pages; ++n) {
        const int j0 = run_at(n, kept, first_page) * FRB_PAGE;
        copies_wait<1>();                                  // this page's keys; its values may still be on their way
        __syncthreads();
        float s[1][8][4] = {}, small[1][8][4] = {};
#pragma unroll 2
        for (int c = 0; c < hd8; c += 8) {
            Tf32Parts a[1][4], b[8][2];
            a_along(a[0], q_rows + c, ld, lane);
#pragma unroll
            for (int j = 0; j < 8; ++j) b_along(b[j], k_s + 8 * j * ld + c, ld, lane);
            mma_tiles_apart(s, small, a, b);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[0][j][e] += small[0][j][e];
        const bool edge = j0 + FRB_PAGE - 1 > pos0 || p.window > 0 || p.chunk > 0;      // some query may not see some key
        float corr[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float top = m[half];
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int key = j0 + 8 * j + 2 * t4 + e;
                    float& x = s[0][j][2 * half + e];
                    x = f32_score(p, x, slope, pos[half], key, !edge || key_visible(key, lo[half], pos[half], p.keep_first));
                    top = fmaxf(top, x);
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float use = top == -INFINITY ? 0.f : top;           // a query that has seen no key yet
            corr[half] = expf(m[half] - use);
            m[half] = top;
            l[half] *= corr[half];
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float& x = s[0][j][2 * half + e];
                    x = expf(x - use);
                    l[half] += x;                                     // this lane's keys; the four lanes' sums meet at the end
                }
        }
        __syncthreads();                                   // nobody reads the keys any more
        if (n + 1 < pages) copy_keys(n + 1);
        copies_commit();
        copies_wait<1>();                                  // this page's values
        if (j0 + FRB_PAGE - 1 > last) {                    // keys behind the last one seen: whatever a page holds there counts for nothing
            __syncthreads();
            for (int i = tid; i < vd * FRB_PAGE; i += TILE_THREADS)
                if (j0 + i % FRB_PAGE > last) v_s[i / FRB_PAGE * LV + i % FRB_PAGE] = 0.f;
        }
        __syncthreads();
        constexpr int RUN = NT < 8 ? NT : 8;               // column tiles whose page's sums are in registers together
#pragma unroll
        for (int n0 = 0; n0 < NT; n0 += RUN) {
            float page[1][RUN][4] = {};
#pragma unroll
            for (int j = 0; j < 8; ++j) {                  // the scores' registers, keys 2 t and 2 t + 1 of a run of eight
                const Tf32Parts a[1][4] = {{tf32_parts(s[0][j][0]), tf32_parts(s[0][j][2]), tf32_parts(s[0][j][1]), tf32_parts(s[0][j][3])}};
                Tf32Parts b[RUN][2];
#pragma unroll
                for (int i = 0; i < RUN; ++i) b_along(b[i], v_s + 8 * (n0 + i) * LV + 8 * j, LV, lane);
                mma_tiles(page, a, b);
            }
#pragma unroll
            for (int i = 0; i < RUN; ++i) {
                float (&o)[4] = acc[n0 + i];
                o[0] = fmaf(o[0], corr[0], page[0][i][0]);
                o[1] = fmaf(o[1], corr[0], page[0][i][1]);
                o[2] = fmaf(o[2], corr[1], page[0][i][2]);
                o[3] = fmaf(o[3], corr[1], page[0][i][3]);
            }
        }
        __syncthreads();
        if (n + 1 < pages) copy_values(n + 1);
        copies_commit();
    }
    copies_wait<0>();
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int r = warp * 16 + 8 * half + g8;
        float total = l[half];
        total += __shfl_xor_sync(0xffffffffu, total, 1);
        total += __shfl_xor_sync(0xffffffffu, total, 2);
        float factor = 1.f;
        if (p.sinks) {
            const float sink = p.sinks[head], top = fmaxf(m[half], sink);
            factor = expf(m[half] - top);
            total = total * factor + expf(sink - top);
        }
        float inv = factor / total, sum = 0.f;                           // sum: becomes a NaN at the first result that is not finite
        if (r < rows) {
            if (p.gate) inv *= 1.0f / (1.0f + expf(-p.gate[(token0 + r) * p.gate_stride + head]));
            float* out = p.out + ((token0 + r) * p.num_heads + head) * vd;
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int d = 8 * i + 2 * t4 + e;
                    if (d < vd) {
                        const float x = acc[i][2 * half + e] * inv;
                        out[d] = x;
                        sum = fmaf(x, 0.f, sum);
                    }
                }
        }
        uint32_t again = __ballot_sync(0xffffffffu, sum != 0.f);         // four lanes a query
        __syncwarp();                                                    // the results above are written before they are written again
        for (int i = 0; again; ++i, again >>= 4)
            if (again & 15) f32_query_key_by_key(p, table, head, g, vg, pos0 + warp * 16 + 8 * half + i, token0 + warp * 16 + 8 * half + i);
    }
}

// ----------------------------------------------------------------------------- single tokens

#define TOKEN_PAGES 4         // pages a block takes: chunks of 256 keys
#define TOKEN_HEADS 8         // query heads of a key head that a block takes at a time

// A block takes four pages of one key head of one sequence for all its query heads (eight at a time).  Keys and values go from
// global memory to registers, sixteen 16-byte loads a lane on their way at once: a warp takes one page of keys (eight lanes a
// key, each with its part of every head's query in registers), then a quarter of the value entries over all four pages (sixteen
// lanes an entry, four keys a lane, the sums of every head in registers until the end).  KJ: head_dim / 32, VR: v_dim / 8, GB:
// query heads of a key head.
template <int KJ, int VR, int GB>
__global__ void __launch_bounds__(128)
attention_f32_token_kernel(F32Attention p, const int* __restrict__ tok_pos, const int* __restrict__ tok_slot, float* __restrict__ part_o,
                           float* __restrict__ part_ml, int max_chunks) {
    __shared__ float4 weights[GB][TOKEN_PAGES * FRB_PAGE / 4];
    after_previous_kernel();
    constexpr int HD = 32 * KJ, VD = 8 * VR;
    const int c = blockIdx.x, g = blockIdx.y, t = blockIdx.z;
    const int pos = tok_pos[t], lo = first_visible_key(pos, p.window, p.chunk);
    const int first_page = lo / FRB_PAGE, kept = kept_runs(p.keep_first, FRB_PAGE, first_page);
    const int pages = kept + pos / FRB_PAGE - first_page + 1, begin = c * TOKEN_PAGES;
    if (begin >= pages) return;
    const int count = min(TOKEN_PAGES, pages - begin);
    const int* table = p.page_table + (size_t)tok_slot[t] * p.max_pages;
    const int group = p.num_heads / p.num_kv_heads, vg = g / (p.num_kv_heads / p.v_heads);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* scores = (float*)weights;

    for (int h0 = 0; h0 < group; h0 += GB) {
        const int heads = min(GB, group - h0), head0 = g * group + h0;
        if (warp < count) {
            const int l8 = lane & 7, sub = lane >> 3;
            float4 q[GB][KJ];
#pragma unroll
            for (int h = 0; h < GB; ++h)
#pragma unroll
                for (int j = 0; j < KJ; ++j)
                    q[h][j] = h < heads ? *(const float4*)(p.q + ((size_t)t * p.num_heads + head0 + h) * HD + 32 * j + 4 * l8)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
            const int run = run_at(begin + warp, kept, first_page);
            const float* keys = p.k_pages + ((size_t)table[run] * p.num_kv_heads + g) * FRB_PAGE * HD;
            const float slope = p.slopes && l8 < heads ? p.slopes[head0 + l8] : 0.f;
#pragma unroll 1
            for (int k0 = 0; k0 < FRB_PAGE; k0 += 16) {
                float4 k[4][KJ];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < KJ; ++j) k[i][j] = *(const float4*)(keys + (size_t)(k0 + 4 * i + sub) * HD + 32 * j + 4 * l8);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float mine = 0.f;
#pragma unroll
                    for (int h = 0; h < GB; ++h) {
                        float s = 0.f;
#pragma unroll
                        for (int j = 0; j < KJ; ++j) s = dot4(q[h][j], k[i][j], s);
                        s += __shfl_xor_sync(0xffffffffu, s, 4);
                        s += __shfl_xor_sync(0xffffffffu, s, 2);
                        s += __shfl_xor_sync(0xffffffffu, s, 1);
                        if (l8 == h) mine = s;
                    }
                    const int at = k0 + 4 * i + sub, key = run * FRB_PAGE + at;
                    if (l8 < GB)
                        scores[l8 * TOKEN_PAGES * FRB_PAGE + warp * FRB_PAGE + at] =
                            f32_score(p, mine, slope, pos, key, key_visible(key, lo, pos, p.keep_first));
                }
            }
        }
        __syncthreads();
        for (int h = warp; h < heads; h += 4) {            // the chunk's softmax, a warp a head
            float* row = scores + h * TOKEN_PAGES * FRB_PAGE;
            float s[2 * TOKEN_PAGES], top = -INFINITY, sum = 0.f;
#pragma unroll
            for (int i = 0; i < 2 * TOKEN_PAGES; ++i) {
                s[i] = i < 2 * count ? row[32 * i + lane] : -INFINITY;
                top = fmaxf(top, s[i]);
            }
            top = warp_max(top);
            const float use = top == -INFINITY ? 0.f : top;
#pragma unroll
            for (int i = 0; i < 2 * TOKEN_PAGES; ++i) {
                const float w = expf(s[i] - use);
                row[32 * i + lane] = w;
                sum += w;
            }
            sum = warp_sum(sum);
            if (lane == 0) {
                float* ml = part_ml + (((size_t)t * p.num_heads + head0 + h) * max_chunks + c) * 2;
                ml[0] = top;
                ml[1] = sum;
            }
        }
        __syncthreads();
        {
            const int side = lane >> 4, l16 = lane & 15, d0 = warp * (VD / 4) + side;      // entries d0, d0 + 2, ...
            float acc[GB][VR];
#pragma unroll
            for (int h = 0; h < GB; ++h)
#pragma unroll
                for (int j = 0; j < VR; ++j) acc[h][j] = 0.f;
#pragma unroll 1
            for (int n = 0; n < count; ++n) {
                const int page = table[run_at(begin + n, kept, first_page)];
                const float* values = p.v_pages + ((size_t)page * p.v_heads + vg) * FRB_PAGE * VD + 4 * l16;
                float4 v[VR];
#pragma unroll
                for (int j = 0; j < VR; ++j) v[j] = *(const float4*)(values + (size_t)(d0 + 2 * j) * FRB_PAGE);
                const int key = run_at(begin + n, kept, first_page) * FRB_PAGE;
                if (key < lo || key + FRB_PAGE - 1 > pos) {          // values that the token does not see are left out, whatever they are
                    const int k0 = key + 4 * l16;
                    const bool seen[4] = {key_visible(k0, lo, pos, p.keep_first), key_visible(k0 + 1, lo, pos, p.keep_first),
                                          key_visible(k0 + 2, lo, pos, p.keep_first), key_visible(k0 + 3, lo, pos, p.keep_first)};
#pragma unroll
                    for (int j = 0; j < VR; ++j)
                        v[j] = make_float4(seen[0] ? v[j].x : 0.f, seen[1] ? v[j].y : 0.f, seen[2] ? v[j].z : 0.f, seen[3] ? v[j].w : 0.f);
                }
#pragma unroll
                for (int h = 0; h < GB; ++h) {
                    const float4 w = weights[h][n * (FRB_PAGE / 4) + l16];
                    if (h < heads)
#pragma unroll
                        for (int j = 0; j < VR; ++j) acc[h][j] = dot4(w, v[j], acc[h][j]);
                }
            }
            // the sixteen lanes' sums: VR is halved as long as it is even, a lane keeping the half that its bit names
#pragma unroll
            for (int h = 0; h < GB; ++h) {
                if (h >= heads) break;
                int n = VR, base = 0;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) {
                    if (n % 2 == 0) {
                        n /= 2;
                        const bool upper = (lane & o) != 0;
#pragma unroll
                        for (int j = 0; j < VR / 2; ++j) {
                            if (j >= n) break;
                            const float keep = upper ? acc[h][j + n] : acc[h][j], send = upper ? acc[h][j] : acc[h][j + n];
                            acc[h][j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                        }
                        base += upper ? n : 0;
                    } else {
#pragma unroll
                        for (int j = 0; j < VR; ++j) {
                            if (j >= n) break;
                            acc[h][j] += __shfl_xor_sync(0xffffffffu, acc[h][j], o);
                        }
                    }
                }
                float* to = part_o + (((size_t)t * p.num_heads + head0 + h) * max_chunks + c) * VD;
#pragma unroll
                for (int j = 0; j < VR; ++j) {
                    if (j >= n) break;
                    to[d0 + 2 * (base + j)] = acc[h][j];             // lanes that share an entry write the same sum
                }
            }
        }
        __syncthreads();
    }
}

// The chunks of a (token, head) joined in their order, with the sink and the head's gate.
__global__ void __launch_bounds__(128)
attention_f32_merge_kernel(F32Attention p, const int* __restrict__ tok_pos, const float* __restrict__ part_o,
                           const float* __restrict__ part_ml, int max_chunks) {
    after_previous_kernel();
    const int t = blockIdx.x, head = blockIdx.y, vd = p.v_dim;
    const int pos = tok_pos[t], first_page = first_visible_key(pos, p.window, p.chunk) / FRB_PAGE;
    const int pages = kept_runs(p.keep_first, FRB_PAGE, first_page) + pos / FRB_PAGE - first_page + 1;
    const int chunks = (pages + TOKEN_PAGES - 1) / TOKEN_PAGES;
    const size_t row = ((size_t)t * p.num_heads + head) * max_chunks;
    float top = -INFINITY, total = 0.f, acc = 0.f;
    for (int c = 0; c < chunks; ++c) top = fmaxf(top, part_ml[2 * (row + c)]);
    if (p.sinks) top = fmaxf(top, p.sinks[head]);
    const float use = top == -INFINITY ? 0.f : top;
    const int d = threadIdx.x;
#pragma unroll 4
    for (int c = 0; c < chunks; ++c) {
        const float w = expf(part_ml[2 * (row + c)] - use);
        total += w * part_ml[2 * (row + c) + 1];
        if (d < vd) acc = fmaf(w, part_o[(row + c) * vd + d], acc);
    }
    if (p.sinks) total += expf(p.sinks[head] - use);
    float inv = 1.0f / total;
    if (p.gate) inv *= 1.0f / (1.0f + expf(-p.gate[(size_t)t * p.gate_stride + head]));
    if (d < vd) p.out[((size_t)t * p.num_heads + head) * vd + d] = acc * inv;
}

// ----------------------------------------------------------------------------- host side

// Prompts.  tile_seq/tile_q0: the step's tiles of 128 queries (sequence, first query among its new tokens).
FRB_API int frb_attention_f32_tiles(const float* q, const float* k_pages, const float* v_pages, const int* page_table, int max_pages,
                                    const int* tile_seq, const int* tile_q0, int num_tiles, const int* seq_slot, const int* seq_start,
                                    const int* seq_q_len, const int* cu_q_len, float* out, int num_heads, int num_kv_heads, int head_dim,
                                    int v_dim, float scale, int window, const float* slopes, int chunk, const float* sinks, const float* gate,
                                    int gate_stride, float softcap, int keep_first, int num_v_heads, cudaStream_t stream) {
    if (num_tiles == 0) return 0;
    FRB_CHECK_ARG(head_dim >= 4 && head_dim <= 128 && head_dim % 4 == 0 && v_dim >= 1 && v_dim <= 128,
                  "float32 attention tiles: heads of %d over values of %d", head_dim, v_dim);
    FRB_CHECK_ARG(2ll * num_tiles <= 65535, "float32 attention tiles: %d tiles exceed the grid", num_tiles);
    F32Attention p;
    const int bad = f32_attention_params(&p, q, k_pages, v_pages, page_table, max_pages, out, num_heads, num_kv_heads, head_dim, v_dim, scale,
                                         window, slopes, chunk, sinks, gate, gate_stride, softcap, keep_first, num_v_heads);
    if (bad) return bad;
    const int ld = ((head_dim + 31) & ~31) + 8;
#define FRB_TILES(NT)                                                                                                               \
    do {                                                                                                                            \
        const size_t smem = ((size_t)(TILE_Q + FRB_PAGE) * ld + (size_t)8 * NT * (FRB_PAGE + 8)) * sizeof(float);                   \
        cudaFuncSetAttribute(attention_f32_tiles_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);              \
        attention_f32_tiles_kernel<NT><<<dim3(num_heads, 2 * num_tiles), TILE_THREADS, smem, stream>>>(p, tile_seq, tile_q0,        \
                                                                                    seq_slot, seq_start, seq_q_len, cu_q_len);       \
    } while (0)
    if (v_dim <= 32) FRB_TILES(4);
    else if (v_dim <= 64) FRB_TILES(8);
    else FRB_TILES(16);
#undef FRB_TILES
    FRB_RETURN_LAUNCH("attention_f32_tiles");
}

// One token a sequence.  part_o [T, heads, max_chunks, v_dim] and part_ml [T, heads, max_chunks, 2]: scratch.
FRB_API int frb_attention_f32_token(const float* q, const float* k_pages, const float* v_pages, const int* page_table, int max_pages,
                                    const int* tok_pos, const int* tok_slot, int num_tokens, float* part_o, float* part_ml, int max_chunks,
                                    float* out, int num_heads, int num_kv_heads, int head_dim, int v_dim, float scale, int window,
                                    const float* slopes, int chunk, const float* sinks, const float* gate, int gate_stride, float softcap,
                                    int keep_first, int num_v_heads, cudaStream_t stream) {
    if (num_tokens == 0) return 0;
    FRB_CHECK_ARG(head_dim % 32 == 0 && head_dim >= 32 && head_dim <= 128 && (v_dim == head_dim || (head_dim == 64 && v_dim == 128)),
                  "float32 attention of single tokens: heads of %d over values of %d", head_dim, v_dim);
    FRB_CHECK_ARG(num_kv_heads <= 65535 && num_tokens <= 65535 && num_heads <= 65535, "float32 attention of %d tokens and %d heads exceeds the grid",
                  num_tokens, num_heads);
    F32Attention p;
    const int bad = f32_attention_params(&p, q, k_pages, v_pages, page_table, max_pages, out, num_heads, num_kv_heads, head_dim, v_dim, scale,
                                         window, slopes, chunk, sinks, gate, gate_stride, softcap, keep_first, num_v_heads);
    if (bad) return bad;
    const int group = num_heads / num_kv_heads;
    const dim3 grid(max_chunks, num_kv_heads, num_tokens);
#define FRB_TOKEN(KJ, VR, GB) launch_dependent_resident(2, attention_f32_token_kernel<KJ, VR, GB>, grid, dim3(128), 0, stream, p, tok_pos, \
                                                        tok_slot, part_o, part_ml, max_chunks)
#define FRB_TOKEN_GROUP(KJ, VR)                                                                                       \
    do {                                                                                                              \
        if (group == 1) FRB_TOKEN(KJ, VR, 1);                                                                         \
        else if (group == 2) FRB_TOKEN(KJ, VR, 2);                                                                    \
        else if (group <= 4) FRB_TOKEN(KJ, VR, 4);                                                                    \
        else if (group <= 6) FRB_TOKEN(KJ, VR, 6);                                                                    \
        else FRB_TOKEN(KJ, VR, 8);                                                                                    \
    } while (0)
    if (head_dim == 32) FRB_TOKEN_GROUP(1, 4);
    else if (head_dim == 64 && v_dim == 64) FRB_TOKEN_GROUP(2, 8);
    else if (head_dim == 64) FRB_TOKEN_GROUP(2, 16);
    else if (head_dim == 96) FRB_TOKEN_GROUP(3, 12);
    else FRB_TOKEN_GROUP(4, 16);
#undef FRB_TOKEN_GROUP
#undef FRB_TOKEN
    launch_dependent_resident(8, attention_f32_merge_kernel, dim3(num_tokens, num_heads), dim3(128), 0, stream, p, tok_pos, (const float*)part_o,
                              (const float*)part_ml, max_chunks);
    FRB_RETURN_LAUNCH("attention_f32_token");
}
