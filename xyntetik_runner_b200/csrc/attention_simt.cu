// Causal attention over the paged cache on CUDA cores, float32 arithmetic:
// the attention of the true 32-bit path (and the checking twin of the
// tensor-core kernel).  One warp per (token, query head).  For the query at
// position p, head h, kv head h / (H/K):
//   s_t = (q . k_t) * scale   for t0 <= t <= p,  t0 = max(0, p - window + 1) (0 without a window)
//   a = softmax(s),  o = sum_t a_t v_t
// with kept first keys and a bias by distance as options (attention_mask.cuh)
// (src/model.c:3548-3589; softmax src/model.c:3409-3415).  Keys are taken in
// chunks of 32 in ascending order with a running maximum, so a query's result
// depends on its position and the keys only -- not on how the step was cut or
// what else is in the batch.  The reference's kernels are `k_attn`
// (src/kernels.cu:2043-2141) and the split `k_attn_dec` + `k_attn_merge`
// (src/kernels.cu:2171-2270).
//
// Every token's keys and values, its own included, are read from the cache:
// the store kernel runs before this one.
#include "common.cuh"
#include "attention_mask.cuh"
#include <math.h>

struct AttnArgs {
    const void* q;               // [n, q_row_stride] ; head h at offset h * hd
    void* out;                   // [n, H * hd]
    const void* cache_k;         // this layer's K block of page 0
    const int* positions;        // [n]
    const int* tok_seg;          // [n]
    const int* block_tables;     // [n_seg][max_pages]
    long long page_stride, v_offset, q_row_stride;
    int n, H, K, hd, max_pages, page_size, window;
    float scale;
    const float* sink;           // [H] or null: exp(sink[h]) joins the softmax's denominator once (no key, no value)
    float softcap;               // c > 0: every score becomes c tanh(score / c); 0: scores as they are
    int keep_first;              // with a window: the first keys that stay visible behind it
    XrBias bias;
};

#define AS_MAX_HD 256

template <typename T>
__global__ void __launch_bounds__(128)
k_attention_simt(AttnArgs a) {
    __shared__ float qs[4][AS_MAX_HD];
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long long idx = (long long)blockIdx.x * 4 + warp;
    if (idx >= (long long)a.n * a.H) return;
    int t = (int)(idx / a.H), h = (int)(idx % a.H);
    int kvh = h / (a.H / a.K);
    int pos = a.positions[t];
    const int* bt = a.block_tables + (size_t)a.tok_seg[t] * a.max_pages;
    const T* qrow = (const T*)a.q + (size_t)t * a.q_row_stride + (size_t)h * a.hd;
    for (int i = lane; i < a.hd; i += 32) qs[warp][i] = xr_to_f32<T>(qrow[i]);
    __syncwarp();

    int t0 = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    const int ND = AS_MAX_HD / 32;
    float acc[ND];
#pragma unroll
    for (int i = 0; i < ND; i++) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;
    const T* kbase = (const T*)a.cache_k;

    // the kept keys ahead of the window first, then the window: 32 keys at a time
    const int kept = min(a.keep_first, t0), kept_chunks = (kept + 31) / 32;
    const float* bias = a.bias.table != nullptr ? a.bias.table + (size_t)h * a.bias.len : nullptr;
    for (int c = 0; c < kept_chunks || t0 + 32 * (c - kept_chunks) <= pos; c++) {
        const int k0 = c < kept_chunks ? 32 * c : t0 + 32 * (c - kept_chunks), end = c < kept_chunks ? kept - 1 : pos;
        int kp = k0 + lane;
        bool valid = kp <= end;
        long long off = 0;
        float s = -INFINITY;
        if (valid) {
            int page = bt[kp / a.page_size];
            off = (long long)page * a.page_stride + ((long long)kvh * a.page_size + (kp % a.page_size)) * a.hd;
            const T* kr = kbase + off;
            float dot = 0.f;
            for (int i = 0; i < a.hd; i++) dot = fmaf(qs[warp][i], xr_to_f32<T>(kr[i]), dot);
            if (bias != nullptr) dot += xr_bias_at(bias, a.bias.len, pos - kp);
            s = dot * a.scale;
            if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
        }
        float cm = xr_warp_max(s);
        float m_new = fmaxf(m, cm);
        float corr = expf(m - m_new);            // 0 on the first chunk (m = -inf)
        float p = valid ? expf(s - m_new) : 0.f;
        l = l * corr + xr_warp_sum(p);
#pragma unroll
        for (int i = 0; i < ND; i++) acc[i] *= corr;
        int cnt = min(32, end - k0 + 1);
        for (int j = 0; j < cnt; j++) {
            float pj = __shfl_sync(0xffffffffu, p, j);
            long long oj = __shfl_sync(0xffffffffu, off, j);
            const T* vr = kbase + oj + a.v_offset;
#pragma unroll
            for (int i = 0; i < ND; i++) {
                int dd = lane + 32 * i;
                if (dd < a.hd) acc[i] = fmaf(pj, xr_to_f32<T>(vr[dd]), acc[i]);
            }
        }
        m = m_new;
    }
    T* orow = (T*)a.out + (size_t)t * a.H * a.hd + (size_t)h * a.hd;
    if (a.sink != nullptr) l += expf(a.sink[h] - m);
    float inv = 1.0f / l;
#pragma unroll
    for (int i = 0; i < ND; i++) {
        int dd = lane + 32 * i;
        if (dd < a.hd) orow[dd] = xr_from_f32<T>(acc[i] * inv);
    }
}

// ---------------------------------------------------------------------------------------------
// The same for portions of many tokens, float32, head sizes 64, 128 and 256, without a window: a block takes 16 packed rows (16 / G
// tokens of one request, the G query heads of one kv head) and brings every chunk of 32 keys and values to shared memory once
// for all of them, two chunks deep by asynchronous copies; a warp has two rows, a lane a key for the scores and HD / 32 columns
// for the sums.  A row's arithmetic is the other kernel's, operation for operation (scores in ascending columns, chunks of 32 from
// key 0 on, values in ascending keys), so the two give the same bits.
// What bounds it: shared memory (a lane's key row is read once for two rows) and, for short prompts, the chain of chunks.  300 tokens of one
// request, 8 heads on 2 of keys, 128 columns: 36 us, where a warp a row, which reads every key again for each row, takes 258.
// ---------------------------------------------------------------------------------------------
#define AT_RPW 2
#define AT_WARPS 8
#define AT_ROWS (AT_RPW * AT_WARPS)

template <int HD>
__global__ void __launch_bounds__(32 * AT_WARPS)
k_attention_simt_rows(AttnArgs a) {
    constexpr int LD = HD + 4, ND = HD / 32;               // floats between key rows: a lane a row, 16 bytes at a time, without conflicts
    extern __shared__ __align__(16) float at_sm[];
    float* ks = at_sm;                                     // [2][32][LD]
    float* vs = ks + 2 * 32 * LD;                          // [2][32][HD]
    float* qs = vs + 2 * 32 * HD;                          // [AT_ROWS][HD]
    float* ps = qs + AT_ROWS * HD;                         // [AT_ROWS][32]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = a.H / a.K, kvh = blockIdx.y, tokens = AT_ROWS / G;
    const int tile0 = blockIdx.x * tokens, tile1 = min(a.n, tile0 + tokens);
    const float* kbase = (const float*)a.cache_k;
    for (int e = threadIdx.x; e < AT_ROWS * HD; e += 32 * AT_WARPS) {
        const int r = e / HD, t = min(tile0 + r / G, a.n - 1);
        qs[e] = ((const float*)a.q)[(size_t)t * a.q_row_stride + (size_t)(kvh * G + r % G) * HD + e % HD];
    }
    // the tokens of one request at a time (nearly always all of the tile's)
    for (int first = tile0; first < tile1;) {
        const int seg = a.tok_seg[first];
        int last = first;
        while (last + 1 < tile1 && a.tok_seg[last + 1] == seg) last++;
        const int* bt = a.block_tables + (size_t)seg * a.max_pages;
        int most = 0;                                      // the largest position: the keys that are fetched
        for (int t = first; t <= last; t++) most = max(most, a.positions[t]);
        const int chunks = most / 32 + 1;
        int pos[AT_RPW], head[AT_RPW];
#pragma unroll
        for (int i = 0; i < AT_RPW; i++) {
            const int r = warp * AT_RPW + i, t = tile0 + r / G;
            head[i] = kvh * G + r % G;
            pos[i] = t >= first && t <= last ? a.positions[t] : -1;              // -1: not a row of this request
        }
        auto fetch = [&](int c) {
            float* kd = ks + (c & 1) * 32 * LD;
            float* vd = vs + (c & 1) * 32 * HD;
            for (int e = threadIdx.x; e < 32 * (HD / 4); e += 32 * AT_WARPS) {
                const int j = e / (HD / 4), d = e % (HD / 4) * 4, kp = c * 32 + j;
                if (kp > most) continue;
                const float* row = kbase + (long long)bt[kp / a.page_size] * a.page_stride + ((long long)kvh * a.page_size + kp % a.page_size) * HD + d;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(kd + j * LD + d)), "l"(row) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(vd + j * HD + d)), "l"(row + a.v_offset) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float m[AT_RPW], l[AT_RPW], acc[AT_RPW][ND];
#pragma unroll
        for (int i = 0; i < AT_RPW; i++) {
            m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
            for (int d = 0; d < ND; d++) acc[i][d] = 0.f;
        }
        __syncthreads();                                   // the queries are there; the request before is done with the buffers
        fetch(0);
        for (int c = 0; c < chunks; c++) {
            if (c + 1 < chunks) {
                fetch(c + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            const int kp = c * 32 + lane;
            const float* kr = ks + ((c & 1) * 32 + lane) * LD;
            const float* qw = qs + warp * AT_RPW * HD;
            float dot[AT_RPW];
#pragma unroll
            for (int i = 0; i < AT_RPW; i++) dot[i] = 0.f;
#pragma unroll 8
            for (int d = 0; d < HD; d += 4) {
                const float4 k = *reinterpret_cast<const float4*>(kr + d);
                float4 q[AT_RPW];
#pragma unroll
                for (int i = 0; i < AT_RPW; i++) q[i] = *reinterpret_cast<const float4*>(qw + i * HD + d);
#pragma unroll
                for (int i = 0; i < AT_RPW; i++) dot[i] = fmaf(q[i].x, k.x, dot[i]);
#pragma unroll
                for (int i = 0; i < AT_RPW; i++) dot[i] = fmaf(q[i].y, k.y, dot[i]);
#pragma unroll
                for (int i = 0; i < AT_RPW; i++) dot[i] = fmaf(q[i].z, k.z, dot[i]);
#pragma unroll
                for (int i = 0; i < AT_RPW; i++) dot[i] = fmaf(q[i].w, k.w, dot[i]);
            }
            bool whole = true;                             // every row of the warp sees all 32 keys
#pragma unroll
            for (int i = 0; i < AT_RPW; i++) {
                float s = -INFINITY;
                const bool valid = kp <= pos[i];
                if (valid) {
                    float x = dot[i];
                    if (a.bias.table != nullptr) x += xr_bias_at(a.bias.table + (size_t)head[i] * a.bias.len, a.bias.len, pos[i] - kp);
                    s = x * a.scale;
                    if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
                }
                const bool any = c * 32 <= pos[i];         // (a row that is done keeps what it has)
                const float m_new = fmaxf(m[i], xr_warp_max(s));
                const float corr = any ? expf(m[i] - m_new) : 1.f;
                const float p = valid ? expf(s - m_new) : 0.f;
                if (any) {
                    l[i] = l[i] * corr + xr_warp_sum(p);
                    m[i] = m_new;
                }
#pragma unroll
                for (int d = 0; d < ND; d++) acc[i][d] *= corr;
                ps[(warp * AT_RPW + i) * 32 + lane] = p;
                whole = whole && c * 32 + 31 <= pos[i];
            }
            __syncwarp();
            const float* pw = ps + warp * AT_RPW * 32;
            const float* vr = vs + (c & 1) * 32 * HD + lane * (ND < 4 ? ND : 4);
            auto value = [&](int j, bool masked) {
                float v[ND];
                if constexpr (ND == 2) { const float2 x = *reinterpret_cast<const float2*>(vr + j * HD); v[0] = x.x; v[1] = x.y; }
                else {
#pragma unroll
                    for (int d = 0; d < ND; d += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(vr + j * HD + d * 32);
                        v[d] = x.x; v[d + 1] = x.y; v[d + 2] = x.z; v[d + 3] = x.w;
                    }
                }
#pragma unroll
                for (int i = 0; i < AT_RPW; i++) {
                    if (masked && c * 32 + j > pos[i]) continue;        // (a key the row does not see may hold anything)
                    const float p = pw[i * 32 + j];
#pragma unroll
                    for (int d = 0; d < ND; d++) acc[i][d] = fmaf(p, v[d], acc[i][d]);
                }
            };
            if (whole) {
#pragma unroll 8
                for (int j = 0; j < 32; j++) value(j, false);
            } else {
                const int cnt = min(32, most - c * 32 + 1);
                for (int j = 0; j < cnt; j++) value(j, true);
            }
            __syncthreads();                               // this buffer is free for the chunk after next
        }
#pragma unroll
        for (int i = 0; i < AT_RPW; i++) {
            if (pos[i] < 0) continue;
            const int r = warp * AT_RPW + i, t = tile0 + r / G;
            if (a.sink != nullptr) l[i] += expf(a.sink[head[i]] - m[i]);
            const float inv = 1.0f / l[i];
            float* orow = (float*)a.out + (size_t)t * a.H * HD + (size_t)head[i] * HD + lane * (ND < 4 ? ND : 4);
            if constexpr (ND == 2) *reinterpret_cast<float2*>(orow) = make_float2(acc[i][0] * inv, acc[i][1] * inv);
            else {
#pragma unroll
                for (int d = 0; d < ND; d += 4)
                    *reinterpret_cast<float4*>(orow + d * 32) = make_float4(acc[i][d] * inv, acc[i][d + 1] * inv, acc[i][d + 2] * inv, acc[i][d + 3] * inv);
            }
        }
        first = last + 1;
    }
}

template <int HD>
static int launch_simt_rows(const AttnArgs& a, cudaStream_t stream) {
    constexpr size_t SMEM = (2 * 32 * (HD + 4) + 2 * 32 * HD + AT_ROWS * HD + AT_ROWS * 32) * sizeof(float);
    static bool ready[XR_DEVICES];
    if (!xr_once_per_device(ready, [] { return xr_allow_smem(k_attention_simt_rows<HD>, SMEM); })) return XR_ERR_LAUNCH;
    const int tokens = AT_ROWS / (a.H / a.K);
    k_attention_simt_rows<HD><<<dim3((a.n + tokens - 1) / tokens, a.K), 32 * AT_WARPS, SMEM, stream>>>(a);
    return xr_launch_status();
}

// portions: how many requests the tokens belong to (0: not known).
XR_EXPORT int xr_attention_simt(const void* q, void* out, int dtype, const void* cache_k, const int* positions,
                                const int* tok_seg, const int* block_tables, long long page_stride,
                                long long v_offset, long long q_row_stride, int n, int H, int K, int hd,
                                int max_pages, int page_size, int window, float scale, const float* sink, float softcap,
                                int keep_first, const float* bias, int bias_len, int portions, cudaStream_t stream) {
    if (n < 1 || H < 1 || K < 1 || H % K != 0 || hd < 1 || hd > AS_MAX_HD || page_size < 1 || window < 0 || softcap < 0.f ||
        keep_first < 0 || (bias != nullptr && bias_len < 1))
        return XR_ERR_ARG;
    AttnArgs a{q, out, cache_k, positions, tok_seg, block_tables, page_stride, v_offset, q_row_stride,
               n, H, K, hd, max_pages, page_size, window, scale, sink, softcap, window > 0 ? keep_first : 0, {bias, bias_len}};
    // Many tokens a request: the rows of 16 / G tokens share their keys.  A step of single tokens has nothing to share, and a window
    // starts every row's chunks elsewhere.  (The copies and stores are 16 bytes wide.)  8 tokens of one request, 8 heads on 2, 128
    // columns, a warp a row against this: 11 / 9 us, behind 1,000 keys 590 / 111, behind 4,000 2,340 / 418.
    const int G = H / K;
    const bool even = !(((uintptr_t)out | (uintptr_t)cache_k) & 15) && !((page_stride | v_offset) & 3);
    if (dtype == XR_F32 && portions > 0 && n >= 8 * portions && window == 0 && G <= AT_ROWS && AT_ROWS % G == 0 && even && K <= 65535) {
        if (hd == 64) return launch_simt_rows<64>(a, stream);
        if (hd == 128) return launch_simt_rows<128>(a, stream);
        if (hd == 256) return launch_simt_rows<256>(a, stream);
    }
    long long warps = (long long)n * H;
    long long blocks = (warps + 3) / 4;
    if (blocks > 0x7fffffffLL) return XR_ERR_ARG;
    if (dtype == XR_F32) k_attention_simt<float><<<(unsigned)blocks, 128, 0, stream>>>(a);
    else if (dtype == XR_BF16) k_attention_simt<__nv_bfloat16><<<(unsigned)blocks, 128, 0, stream>>>(a);
    else return XR_ERR_ARG;
    return xr_launch_status();
}
