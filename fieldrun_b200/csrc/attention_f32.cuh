// What the float32 attention kernels share: the call's parameters, a score, and a query taken key by key.
#pragma once

#include "common.cuh"

struct F32Attention {
    const float* q;           // [T, nh, hd]
    const float* k_pages;     // [pages, nkv, PAGE, hd]
    const float* v_pages;     // [pages, v_heads, vd, PAGE]
    const float* slopes;      // [nh] or null
    const float* sinks;       // [nh] or null
    const float* gate;        // [T, gate_stride] or null
    const int* page_table;    // [slots, max_pages]
    float* out;               // [T, nh * vd]
    float scale, softcap;
    int gate_stride, chunk, keep_first, window, max_pages, num_heads, num_kv_heads, v_heads, head_dim, v_dim;
};

// The score of key j for the query at `pos` from the raw product, or -infinity where the key is hidden.
__device__ __forceinline__ float f32_score(const F32Attention& p, float raw, float slope, int pos, int j, bool visible) {
    float s = raw * p.scale;
    if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
    return visible ? s - slope * (float)(pos - j) : -INFINITY;
}

// One query of one head key by key in float32, a warp a query: the sums of attention_generic.
static __device__ __forceinline__ void f32_query_key_by_key(const F32Attention& p, const int* table, int head, int g, int vg, int pos, size_t token) {
    const int lane = threadIdx.x & 31, hd = p.head_dim, vd = p.v_dim, lo = first_visible_key(pos, p.window, p.chunk);
    const int first = lo / 32, kept = kept_runs(p.keep_first, 32, first), blocks = kept + pos / 32 - first + 1;
    const float* q = p.q + (token * p.num_heads + head) * hd;
    const float slope = p.slopes ? p.slopes[head] : 0.f;
    float m = -INFINITY, l = 0.f, acc[4] = {};
    for (int n = 0; n < blocks; ++n) {
        const int j0 = run_at(n, kept, first) * 32, j = j0 + lane, page = table[j0 / FRB_PAGE], in_page = j0 % FRB_PAGE;
        const bool visible = key_visible(j, lo, pos, p.keep_first);
        const float* k = p.k_pages + (((size_t)page * p.num_kv_heads + g) * FRB_PAGE + in_page + lane) * hd;
        const float* v = p.v_pages + ((size_t)page * p.v_heads + vg) * FRB_PAGE * vd + in_page;
        float s = 0.f;
        if (visible)
            for (int d = 0; d < hd; ++d) s = fmaf(q[d], k[d], s);
        s = f32_score(p, s, slope, pos, j, visible);
        const float top = fmaxf(m, warp_max(s)), corr = expf(m - top), w = visible ? expf(s - top) : 0.f;
        l = l * corr + warp_sum(w);
        m = top;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] *= corr;
        for (int kk = 0; kk < 32; ++kk) {
            const float wk = __shfl_sync(0xffffffffu, w, kk);
            if (key_visible(j0 + kk, lo, pos, p.keep_first))
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (lane + 32 * i < vd) acc[i] = fmaf(wk, v[(size_t)(lane + 32 * i) * FRB_PAGE + kk], acc[i]);
        }
    }
    if (p.sinks) {
        const float sink = p.sinks[head], top = fmaxf(m, sink), corr = expf(m - top);
        l = l * corr + expf(sink - top);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] *= corr;
    }
    float inv = 1.0f / l;
    if (p.gate) inv *= 1.0f / (1.0f + expf(-p.gate[token * p.gate_stride + head]));
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (lane + 32 * i < vd) p.out[(token * p.num_heads + head) * vd + lane + 32 * i] = acc[i] * inv;
}

static int f32_attention_params(F32Attention* p, const float* q, const float* k_pages, const float* v_pages, const int* page_table,
                                int max_pages, float* out, int num_heads, int num_kv_heads, int head_dim, int v_dim, float scale, int window,
                                const float* slopes, int chunk, const float* sinks, const float* gate, int gate_stride, float softcap,
                                int keep_first, int num_v_heads) {
    FRB_CHECK_ARG(num_kv_heads >= 1 && num_heads % num_kv_heads == 0, "attention: %d heads are not a multiple of %d kv heads", num_heads,
                  num_kv_heads);
    FRB_CHECK_ARG(num_v_heads >= 1 && num_kv_heads % num_v_heads == 0, "attention: %d key heads over %d value heads", num_kv_heads, num_v_heads);
    FRB_CHECK_ARG(keep_first >= 0 && !(keep_first > 0 && chunk > 0), "attention: %d first tokens together with chunks", keep_first);
    FRB_CHECK_ARG((((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0, "attention: queries and pages must be 16-byte aligned");
    p->q = q; p->k_pages = k_pages; p->v_pages = v_pages; p->slopes = slopes; p->sinks = sinks; p->gate = gate; p->page_table = page_table;
    p->out = out; p->scale = scale; p->softcap = softcap; p->gate_stride = gate_stride; p->chunk = chunk;
    p->keep_first = window > 0 ? keep_first : 0; p->window = window; p->max_pages = max_pages; p->num_heads = num_heads;
    p->num_kv_heads = num_kv_heads; p->v_heads = num_v_heads; p->head_dim = head_dim; p->v_dim = v_dim;
    return 0;
}
