// Matrix-memory recurrence (the mLSTM cell of xLSTM) with a stabilising running maximum, per request and head.
//
// State per (request slot, head): S [D][V], n [D], m (float32, zero when the slot is assigned).  For a token with
// query q (times D^-1/2), key k, value v, pre-activations a_i, a_f of the gates and cap c:
//   li = c tanh(a_i / c)                      (log of the input gate)
//   lf = logsigmoid(c tanh(a_f / c))          (log of the forget gate)
//   m' = max(lf + m, li);  f = exp(lf + m - m');  i = exp(li - m')
//   S' = f S + i k v^T;    n' = f n + i k
//   o  = S'^T q / (max(|n' . q|, exp(-m')) + 1e-6)
// Everything above is float32; q, k, v come from the projections in the activation dtype.
//
// Three kernels.  k_mlstm_gates walks a request's tokens once per head: m, f, i, n and the denominator of every token
// (scalars per token and head), and leaves n and m in the state.  k_mlstm_scan walks them once per (head, slice of
// 32 value columns) with S in shared memory, each thread updating its own cells, and writes o.  k_mlstm_out divides
// each head's o by its root mean square, multiplies by the norm weight and the sigmoid of the output gate.
// The walk is token by token in both, so the state after a token does not depend on how the tokens were cut into
// steps, bit for bit.
#include "chunked.cuh"
#include <math.h>

#define ML_VS 32          // value columns per block of the scan
#define ML_RG 8           // row groups (warps) per block of the scan
#define ML_CHUNK 8        // tokens whose q, k, v are staged together (the register scan stages one token per warp: = ML_RG)

__device__ __forceinline__ float ml_logsigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// a decay's logarithm is at most zero; one that is no number stays so (fminf would make it zero, a decay of one)
__device__ __forceinline__ float ml_log_decay(float x) { return x > 0.f ? 0.f : x; }

// state layout per slot: [H][D * V + D + 1]
__host__ __device__ __forceinline__ size_t ml_state_head(int D, int V) { return (size_t)D * V + D + 1; }

// Tokens are taken `stage` at a time, in four steps a chunk, so that nothing but a few scalar operations per token is
// serial: (1) the logarithms of the gates of the chunk's tokens, a thread a token; (2) one thread walks the chunk's
// scalars: m, f, i and exp(-m) of every token; (3) every thread owns elements of n and walks the chunk with them,
// n <- f n + i k, leaving n[d] q[d] of every token in shared memory; (4) the warps sum those products token by token
// (always in the same order) and write (f, i, denominator).
template <typename T>
__global__ void __launch_bounds__(256)
k_mlstm_gates(const T* __restrict__ proj, long long ldp, int q_col, int k_col, const float* __restrict__ gates,
              float* __restrict__ state, float* __restrict__ coef, const int* __restrict__ seg_start,
              const int* __restrict__ seg_len, const int* __restrict__ seg_slot, int H, int D, int V, float cap, int stage) {
    xr_pdl_launch();
    extern __shared__ float gsm[];
    float* prod = gsm;                          // [stage][D]: n[d] q[d] of the chunk's tokens
    float* lg = prod + (size_t)stage * D;       // [stage][2]: log input gate, log forget gate
    float* fi = lg + 2 * stage;                 // [stage][3]: f, i, exp(-m)
    __shared__ float m_run;
    const int h = blockIdx.x, seg = blockIdx.y;
    const int start = seg_start[seg], len = seg_len[seg], slot = seg_slot[seg];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    xr_pdl_wait();
    float* st = state + ((size_t)slot * H + h) * ml_state_head(D, V);
    float* n_g = st + (size_t)D * V;
    constexpr int OWN = 4;                      // elements of n per thread: D <= 4 * 256
    float nreg[OWN];
#pragma unroll
    for (int i = 0; i < OWN; i++) { const int d = threadIdx.x + i * blockDim.x; nreg[i] = d < D ? n_g[d] : 0.f; }
    if (threadIdx.x == 0) m_run = n_g[D];
    const float qs = 1.0f / sqrtf((float)D);
    for (int j0 = 0; j0 < len; j0 += stage) {
        const int cnt = min(stage, len - j0);
        for (int j = threadIdx.x; j < cnt; j += blockDim.x) {
            const int t = start + j0 + j;
            const float ai = gates[(size_t)t * 2 * H + h], af = gates[(size_t)t * 2 * H + H + h];
            lg[2 * j] = cap * tanhf(ai / cap);
            lg[2 * j + 1] = ml_logsigmoid(cap * tanhf(af / cap));
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            float m = m_run;
            for (int j = 0; j < cnt; j++) {
                const float li = lg[2 * j], lf = lg[2 * j + 1];
                const float m_new = fmaxf(lf + m, li);
                fi[3 * j] = expf(lf + m - m_new); fi[3 * j + 1] = expf(li - m_new); fi[3 * j + 2] = expf(-m_new);
                m = m_new;
            }
            m_run = m;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < OWN; i++) {
            const int d = threadIdx.x + i * blockDim.x;
            if (d < D) {
                float nn = nreg[i];
#pragma unroll 8
                for (int j = 0; j < cnt; j++) {
                    const T* row = proj + (size_t)(start + j0 + j) * ldp + (size_t)h * D + d;
                    nn = fmaf(fi[3 * j], nn, fi[3 * j + 1] * xr_to_f32<T>(row[k_col]));
                    prod[j * D + d] = nn * (xr_to_f32<T>(row[q_col]) * qs);
                }
                nreg[i] = nn;
            }
        }
        __syncthreads();
        for (int j = warp; j < cnt; j += nw) {
            float part = 0.f;
            for (int d = lane; d < D; d += 32) part += prod[j * D + d];
            const float qn = xr_warp_sum(part);
            if (lane == 0) {
                float* c = coef + ((size_t)(start + j0 + j) * H + h) * 3;
                c[0] = fi[3 * j]; c[1] = fi[3 * j + 1]; c[2] = fmaxf(fabsf(qn), fi[3 * j + 2]) + 1e-6f;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < OWN; i++) { const int d = threadIdx.x + i * blockDim.x; if (d < D) n_g[d] = nreg[i]; }
    if (threadIdx.x == 0) n_g[D] = m_run;
}

template <typename T>
__global__ void __launch_bounds__(ML_VS * ML_RG)
k_mlstm_scan_wide(const T* __restrict__ proj, long long ldp, int q_col, int k_col, int v_col, const float* __restrict__ coef,
             float* __restrict__ state, float* __restrict__ out, const int* __restrict__ seg_start,
             const int* __restrict__ seg_len, const int* __restrict__ seg_slot, int H, int D, int V) {
    xr_pdl_launch();
    extern __shared__ float sm[];
    float* S = sm;                                   // [D][ML_VS]
    float* ks = S + (size_t)D * ML_VS;               // [ML_CHUNK][D]
    float* qsm = ks + (size_t)ML_CHUNK * D;          // [ML_CHUNK][D]
    float* vs = qsm + (size_t)ML_CHUNK * D;          // [ML_CHUNK][ML_VS]
    float* red = vs + ML_CHUNK * ML_VS;              // [ML_CHUNK][ML_RG][ML_VS]
    float* cf = red + ML_CHUNK * ML_RG * ML_VS;      // [ML_CHUNK][3]
    const int col = threadIdx.x & (ML_VS - 1), rg = threadIdx.x / ML_VS;
    const int v0 = blockIdx.x * ML_VS, h = blockIdx.y, seg = blockIdx.z;
    const int start = seg_start[seg], len = seg_len[seg], slot = seg_slot[seg];
    const bool col_ok = v0 + col < V;
    xr_pdl_wait();
    float* Sg = state + ((size_t)slot * H + h) * ml_state_head(D, V);
    for (int d = rg; d < D; d += ML_RG) S[d * ML_VS + col] = col_ok ? Sg[(size_t)d * V + v0 + col] : 0.f;
    const float qscale = 1.0f / sqrtf((float)D);
    for (int j0 = 0; j0 < len; j0 += ML_CHUNK) {
        const int cnt = min(ML_CHUNK, len - j0);
        __syncthreads();
        for (int e = threadIdx.x; e < cnt * D; e += blockDim.x) {
            const int j = e / D, d = e % D;
            const T* row = proj + (size_t)(start + j0 + j) * ldp;
            ks[j * D + d] = xr_to_f32<T>(row[k_col + h * D + d]);
            qsm[j * D + d] = xr_to_f32<T>(row[q_col + h * D + d]) * qscale;
        }
        for (int e = threadIdx.x; e < cnt * ML_VS; e += blockDim.x) {
            const int j = e / ML_VS, c = e % ML_VS;
            vs[e] = v0 + c < V ? xr_to_f32<T>(proj[(size_t)(start + j0 + j) * ldp + v_col + h * V + v0 + c]) : 0.f;
        }
        for (int e = threadIdx.x; e < cnt * 3; e += blockDim.x) cf[e] = coef[((size_t)(start + j0 + e / 3) * H + h) * 3 + e % 3];
        __syncthreads();
        for (int j = 0; j < cnt; j++) {
            const float f = cf[j * 3], iv = cf[j * 3 + 1] * vs[j * ML_VS + col];
            float num = 0.f;
            for (int d = rg; d < D; d += ML_RG) {
                const float s = fmaf(f, S[d * ML_VS + col], iv * ks[j * D + d]);
                S[d * ML_VS + col] = s;
                num = fmaf(s, qsm[j * D + d], num);
            }
            red[(j * ML_RG + rg) * ML_VS + col] = num;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < cnt * ML_VS; e += blockDim.x) {
            const int j = e / ML_VS, c = e % ML_VS;
            if (v0 + c >= V) continue;
            float num = 0.f;
#pragma unroll
            for (int r = 0; r < ML_RG; r++) num += red[(j * ML_RG + r) * ML_VS + c];
            out[(size_t)(start + j0 + j) * H * V + (size_t)h * V + v0 + c] = num / cf[j * 3 + 2];
        }
    }
    __syncthreads();
    if (col_ok)
        for (int d = rg; d < D; d += ML_RG) Sg[(size_t)d * V + v0 + col] = S[d * ML_VS + col];
}

// The same walk with S in registers, for key sizes up to 256: thread (row group rg, column) keeps rows
// rg * RPT .. rg * RPT + RPT - 1 of its column (RPT = rows per thread, 8 * RPT >= D; rows beyond D stay zero), and reads
// the staged k and q of a token as float4 that the whole warp shares.
template <typename T, int RPT>
__global__ void __launch_bounds__(ML_VS * ML_RG)
k_mlstm_scan(const T* __restrict__ proj, long long ldp, int q_col, int k_col, int v_col, const float* __restrict__ coef,
             float* __restrict__ state, float* __restrict__ out, const int* __restrict__ seg_start,
             const int* __restrict__ seg_len, const int* __restrict__ seg_slot, int H, int D, int V) {
    xr_pdl_launch();
    constexpr int DP = ML_RG * RPT;
    __shared__ __align__(16) float ks[ML_CHUNK][DP];
    __shared__ __align__(16) float qsm[ML_CHUNK][DP];
    __shared__ float vs[ML_CHUNK][ML_VS];
    __shared__ float red[ML_CHUNK][ML_RG][ML_VS];
    __shared__ float cf[ML_CHUNK][3];
    const int col = threadIdx.x & (ML_VS - 1), rg = threadIdx.x / ML_VS;
    const int v0 = blockIdx.x * ML_VS, h = blockIdx.y, seg = blockIdx.z;
    const int start = seg_start[seg], len = seg_len[seg], slot = seg_slot[seg];
    const bool col_ok = v0 + col < V;
    xr_pdl_wait();
    float* Sg = state + ((size_t)slot * H + h) * ml_state_head(D, V);
    float S[RPT];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
        const int d = rg * RPT + i;
        S[i] = (col_ok && d < D) ? Sg[(size_t)d * V + v0 + col] : 0.f;
    }
    const float qscale = 1.0f / sqrtf((float)D);
    // the next chunk's k, q, v and scalars are on their way to registers while this chunk is computed
    constexpr int NL = ML_CHUNK * DP / (ML_VS * ML_RG);           // elements of k (and of q) per thread and chunk
    T kreg[NL], qreg[NL], vreg = xr_from_f32<T>(0.f);
    float creg = 0.f;
    auto prefetch = [&](int j0) {
        const int cnt = min(ML_CHUNK, len - j0);
#pragma unroll
        for (int i = 0; i < NL; i++) {
            const int e = threadIdx.x + i * (ML_VS * ML_RG), j = e / DP, d = e % DP;
            const bool ok = j < cnt && d < D;
            const T* row = proj + (size_t)(start + j0 + (ok ? j : 0)) * ldp + (size_t)h * D + (ok ? d : 0);
            kreg[i] = ok ? row[k_col] : xr_from_f32<T>(0.f);
            qreg[i] = ok ? row[q_col] : xr_from_f32<T>(0.f);
        }
        const int j = threadIdx.x / ML_VS;
        vreg = (j < cnt && col_ok) ? proj[(size_t)(start + j0 + j) * ldp + v_col + h * V + v0 + col] : xr_from_f32<T>(0.f);
        if ((int)threadIdx.x < cnt * 3) creg = coef[((size_t)(start + j0 + threadIdx.x / 3) * H + h) * 3 + threadIdx.x % 3];
    };
    prefetch(0);
    for (int j0 = 0; j0 < len; j0 += ML_CHUNK) {
        const int cnt = min(ML_CHUNK, len - j0);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NL; i++) {
            const int e = threadIdx.x + i * (ML_VS * ML_RG), j = e / DP, d = e % DP;
            ks[j][d] = xr_to_f32<T>(kreg[i]);
            qsm[j][d] = xr_to_f32<T>(qreg[i]) * qscale;
        }
        vs[threadIdx.x / ML_VS][col] = xr_to_f32<T>(vreg);
        if (threadIdx.x < ML_CHUNK * 3) cf[threadIdx.x / 3][threadIdx.x % 3] = creg;
        __syncthreads();
        if (j0 + ML_CHUNK < len) prefetch(j0 + ML_CHUNK);
        for (int j = 0; j < cnt; j++) {
            const float f = cf[j][0], iv = cf[j][1] * vs[j][col];
            const float4* k4 = reinterpret_cast<const float4*>(&ks[j][rg * RPT]);
            const float4* q4 = reinterpret_cast<const float4*>(&qsm[j][rg * RPT]);
            float num = 0.f;
#pragma unroll
            for (int i = 0; i < RPT / 4; i++) {
                const float4 kk = k4[i], qq = q4[i];
                S[4 * i] = fmaf(f, S[4 * i], iv * kk.x);         num = fmaf(S[4 * i], qq.x, num);
                S[4 * i + 1] = fmaf(f, S[4 * i + 1], iv * kk.y); num = fmaf(S[4 * i + 1], qq.y, num);
                S[4 * i + 2] = fmaf(f, S[4 * i + 2], iv * kk.z); num = fmaf(S[4 * i + 2], qq.z, num);
                S[4 * i + 3] = fmaf(f, S[4 * i + 3], iv * kk.w); num = fmaf(S[4 * i + 3], qq.w, num);
            }
            red[j][rg][col] = num;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < cnt * ML_VS; e += blockDim.x) {
            const int j = e / ML_VS, c = e % ML_VS;
            if (v0 + c >= V) continue;
            float num = 0.f;
#pragma unroll
            for (int r = 0; r < ML_RG; r++) num += red[j][r][c];
            out[(size_t)(start + j0 + j) * H * V + (size_t)h * V + v0 + c] = num / cf[j][2];
        }
    }
    if (col_ok) {
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            const int d = rg * RPT + i;
            if (d < D) Sg[(size_t)d * V + v0 + col] = S[i];
        }
    }
}

// o [n][H][V] float32 -> y [n][H * V] (activation dtype): o / rms(o over the head) * w * act(g); one warp per (token, head).
// The weight of head h starts at w + h * w_head (0: one weight of V values for all heads); act is the sigmoid, or SiLU
// with `gate_silu`.
// (TG: the gate's dtype, the activation dtype or float32)
template <typename T, typename TG = T>
__global__ void __launch_bounds__(128)
k_mlstm_out(const float* __restrict__ o, const TG* __restrict__ proj, long long ldp, int g_col, const float* __restrict__ w,
            T* __restrict__ y, int n, int H, int V, float eps, int w_head, int gate_silu) {
    xr_pdl_launch();
    xr_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long idx = (long long)blockIdx.x * 4 + warp;
    if (idx >= (long long)n * H) return;
    const int t = (int)(idx / H), h = (int)(idx % H);
    const float* src = o + ((size_t)t * H + h) * V;
    float ss = 0.f;
    for (int i = lane; i < V; i += 32) ss = fmaf(src[i], src[i], ss);
    ss = xr_warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)V + eps);
    const TG* g = proj + (size_t)t * ldp + g_col + (size_t)h * V;
    T* dst = y + (size_t)t * H * V + (size_t)h * V;
    for (int i = lane; i < V; i += 32) {
        const float z = xr_to_f32<TG>(g[i]);
        float gate = 1.0f / (1.0f + expf(-z));
        if (gate_silu) gate *= z;
        dst[i] = xr_from_f32<T>(src[i] * inv * (w != nullptr ? w[(size_t)h * w_head + i] : 1.0f) * gate);
    }
}
// The same with a head's values, gates and weights in a warp's registers, four columns an access (PER accesses a lane), all on their way at once:
// heads of up to 512 values, a multiple of four, on borders of an access.  2,048 tokens, 8 heads of 256, inside a step: 17.4 -> 9.8 us (gates in bfloat16), 20.3
// -> 10.5 (in float32).
__device__ __forceinline__ float4 ml_read4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ml_read4(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ void ml_write4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void ml_write4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
template <typename T, typename TG, int PER>
__global__ void __launch_bounds__(128)
k_mlstm_out_vec(const float* __restrict__ o, const TG* __restrict__ proj, long long ldp, int g_col, const float* __restrict__ w,
                T* __restrict__ y, int n, int H, int V, float eps, int w_head, int gate_silu) {
    xr_pdl_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long idx = (long long)blockIdx.x * 4 + warp;
    xr_pdl_wait();
    if (idx >= (long long)n * H) return;
    const int t = (int)(idx / H), h = (int)(idx % H);
    const float* src = o + ((size_t)t * H + h) * V;
    const TG* g = proj + (size_t)t * ldp + g_col + (size_t)h * V;
    T* dst = y + (size_t)t * H * V + (size_t)h * V;
    float4 x[PER], z[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int i = 4 * (lane + 32 * k);
        x[k] = z[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < V) { x[k] = ml_read4(src + i); z[k] = ml_read4(g + i); }
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < PER; k++) { ss = fmaf(x[k].x, x[k].x, ss); ss = fmaf(x[k].y, x[k].y, ss); ss = fmaf(x[k].z, x[k].z, ss); ss = fmaf(x[k].w, x[k].w, ss); }
    ss = xr_warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)V + eps);
    auto one = [&](float v, float z, float wt) {
        float gate = 1.0f / (1.0f + expf(-z));
        if (gate_silu) gate *= z;
        return v * inv * wt * gate;
    };
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int i = 4 * (lane + 32 * k);
        if (i >= V) continue;
        const float4 wt = w != nullptr ? ml_read4(w + (size_t)h * w_head + i) : make_float4(1.f, 1.f, 1.f, 1.f);
        ml_write4(dst + i, make_float4(one(x[k].x, z[k].x, wt.x), one(x[k].y, z[k].y, wt.y), one(x[k].z, z[k].z, wt.z), one(x[k].w, z[k].w, wt.w)));
    }
}
template <typename T, typename TG>
static void launch_mlstm_out(const float* o, const TG* proj, long long ldp, int g_col, const float* w, T* y, int n, int H, int V, float eps, int w_head, int gate_silu,
                             cudaStream_t stream) {
    const dim3 grid((unsigned)(((long long)n * H + 3) / 4)), block(128);
    const bool vec = V <= 512 && !((V | g_col | w_head) & 3) && ldp % 4 == 0 && !(((uintptr_t)o | (uintptr_t)w) & 15) && !((uintptr_t)proj & (4 * sizeof(TG) - 1)) &&
                     !((uintptr_t)y & (4 * sizeof(T) - 1));
#define MO(PER) xr_launch((k_mlstm_out_vec<T, TG, PER>), grid, block, 0, stream, o, proj, ldp, g_col, w, y, n, H, V, eps, w_head, gate_silu)
    if (vec && V <= 128) MO(1);
    else if (vec && V <= 256) MO(2);
    else if (vec) MO(4);
    else xr_launch((k_mlstm_out<T, TG>), grid, block, 0, stream, o, proj, ldp, g_col, w, y, n, H, V, eps, w_head, gate_silu);
#undef MO
}

// ---------------------------------------------------------------------------------------------
// Portions of many tokens go through the recurrence in chunks (chunked.cuh), with  a_t = f  and  s_t = i  in logarithms:
//   log f_t = lf_t + m_(t-1) - m_t <= 0,   s_t = exp(li_t - m_t),   floor_t = exp(-m_t).
// m is a running maximum of sums, m_t = max(m_(t-1) + lf_t, li_t): a block per (head, portion), a thread a run of tokens; a run is
// the map m -> max(m + A, B), the runs' maps are joined over the block, then every thread walks its run from its own start.
// ---------------------------------------------------------------------------------------------
#define ML_RUN 8
__global__ void __launch_bounds__(256)
k_mlstm_scalars(const float* __restrict__ gates, float* __restrict__ state, float* __restrict__ log_f, float* __restrict__ in_scale,
                float* __restrict__ floor_n, const int* __restrict__ seg_start, const int* __restrict__ seg_len, const int* __restrict__ seg_slot,
                int H, int D, int V, float cap) {
    xr_pdl_launch();
    __shared__ float sa[256], sb[256];
    const int h = blockIdx.x, seg = blockIdx.y, tid = threadIdx.x;
    const int start = seg_start[seg], len = seg_len[seg];
    const int per = (len + 255) / 256, i0 = min(len, tid * per), i1 = min(len, i0 + per);
    float* m_at = state + ((size_t)seg_slot[seg] * H + h) * ml_state_head(D, V) + (size_t)D * V + D;
    xr_pdl_wait();
    if (len <= 0) return;
    const float m0 = *m_at;
    auto logs = [&](int i, float& li, float& lf) {
        const float* row = gates + (size_t)(start + i) * 2 * H + h;
        li = cap * tanhf(row[0] / cap);
        lf = ml_logsigmoid(cap * tanhf(row[H] / cap));
    };
    // a run of up to ML_RUN tokens (portions of up to 2,048): both logarithms of all of them in registers, their loads on their way at once and the
    // functions taken once.  8 heads, 2,048 tokens inside a step, 18 to 24 -> 11.8 us.
    float lis[ML_RUN], lfs[ML_RUN];
    const bool held = per <= ML_RUN;
    if (held) {
#pragma unroll
        for (int k = 0; k < ML_RUN; k++) {
            const float* row = gates + (size_t)(start + min(i0 + k, len - 1)) * 2 * H + h;
            lis[k] = xr_ld_now(row); lfs[k] = xr_ld_now(row + H);
        }
#pragma unroll
        for (int k = 0; k < ML_RUN; k++) { xr_ld_fence(lis[k]); xr_ld_fence(lfs[k]); }
#pragma unroll
        for (int k = 0; k < ML_RUN; k++)
            if (i0 + k < i1) { lis[k] = cap * tanhf(lis[k] / cap); lfs[k] = ml_logsigmoid(cap * tanhf(lfs[k] / cap)); }
    }
    float A = 0.f, B = -INFINITY;
    auto join = [&](float li, float lf) { B = fmaxf(B + lf, li); A += lf; };
    if (held) {
#pragma unroll
        for (int k = 0; k < ML_RUN; k++)
            if (i0 + k < i1) join(lis[k], lfs[k]);
    } else {
        for (int i = i0; i < i1; i++) {
            float li, lf;
            logs(i, li, lf);
            join(li, lf);
        }
    }
    sa[tid] = A; sb[tid] = B;
    __syncthreads();
    for (int o = 1; o < 256; o <<= 1) {                  // the maps of all runs up to this one, joined
        float pa = 0.f, pb = -INFINITY;
        if (tid >= o) { pa = sa[tid - o]; pb = sb[tid - o]; }
        __syncthreads();
        if (tid >= o) { sb[tid] = fmaxf(pb + sa[tid], sb[tid]); sa[tid] += pa; }
        __syncthreads();
    }
    float m = tid == 0 ? m0 : fmaxf(m0 + sa[tid - 1], sb[tid - 1]), first_m = 0.f, first_lf = 0.f;
    auto token = [&](int i, float li, float lf) {
        const float m_new = fmaxf(lf + m, li);
        const size_t at = (size_t)(start + i) * H + h;
        if (i == i0) { first_m = m_new; first_lf = lf; }
        else log_f[at] = ml_log_decay(lf + m - m_new);
        in_scale[at] = expf(li - m_new); floor_n[at] = expf(-m_new);
        m = m_new;
    };
    if (held) {
#pragma unroll
        for (int k = 0; k < ML_RUN; k++)
            if (i0 + k < i1) token(i0 + k, lis[k], lfs[k]);
    } else {
        for (int i = i0; i < i1; i++) {
            float li, lf;
            logs(i, li, lf);
            token(i, li, lf);
        }
    }
    // a run's first decay leads over from the very m that the run before ended with (joined in another order, the sums differ in
    // their last bits, and S is kept relative to m)
    __syncthreads();
    sa[tid] = m;
    __syncthreads();
    if (i0 < i1) log_f[(size_t)(start + i0) * H + h] = ml_log_decay(first_lf + (tid == 0 ? m0 : sa[tid - 1]) - first_m);
    if (len > 0 && i0 < len && i1 == len) *m_at = m;     // (every thread has read it, barriers ago)
}

// q / sqrt(D), k and v as float32 rows [n][2 H D + H V]
template <typename T>
__global__ void __launch_bounds__(256)
k_mlstm_rows(const T* __restrict__ proj, long long ldp, int q_col, int k_col, int v_col, float* __restrict__ out, int n, int HD, int HV, float qs) {
    xr_pdl_launch();
    xr_pdl_wait();
    const int cols = 2 * HD + HV;
    for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < (size_t)n * cols; e += (size_t)gridDim.x * 256) {
        const size_t t = e / cols;
        const int c = (int)(e % cols);
        const T* row = proj + t * ldp;
        out[e] = c < HD ? xr_to_f32<T>(row[q_col + c]) * qs : (c < 2 * HD ? xr_to_f32<T>(row[k_col + c - HD]) : xr_to_f32<T>(row[v_col + c - 2 * HD]));
    }
}
// Eight columns a thread (grid: columns, tokens) of bfloat16 rows on 16-byte borders: without a division an element.  2,048 tokens of 4,096
// columns inside a step, 23.9 -> 10.2 us.
static __global__ void __launch_bounds__(256)
k_mlstm_rows_vec(const __nv_bfloat16* __restrict__ proj, long long ldp, int q_col, int k_col, int v_col, float* __restrict__ out, int n, int HD, int HV, float qs) {
    xr_pdl_launch();
    const int cols = 2 * HD + HV, c = (blockIdx.x * 256 + threadIdx.x) * 8;
    xr_pdl_wait();
    if (c >= cols) return;
    const int from = c < HD ? q_col + c : (c < 2 * HD ? k_col + c - HD : v_col + c - 2 * HD);
    const float f = c < HD ? qs : 1.0f;
    for (int t = blockIdx.y; t < n; t += gridDim.y) {
        const uint4 u = *reinterpret_cast<const uint4*>(proj + (size_t)t * ldp + from);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
        float4* dst = reinterpret_cast<float4*>(out + (size_t)t * cols + c);
#pragma unroll
        for (int i = 0; i < 2; i++)
            dst[i] = make_float4(__uint_as_float(w[2 * i] << 16) * f, __uint_as_float(w[2 * i] & 0xffff0000u) * f, __uint_as_float(w[2 * i + 1] << 16) * f,
                                 __uint_as_float(w[2 * i + 1] & 0xffff0000u) * f);
    }
}

template <typename T>
static int mlstm_chunked(const T* proj, long long ldp, int q_col, int k_col, int v_col, const float* gates, float* state, float* o, const int* seg_start,
                         const int* seg_len, const int* seg_slot, int n, int n_seg, int H, int D, int V, float cap, float* scratch,
                         long long scratch_floats, cudaStream_t stream) {
    const int HD = H * D, HV = H * V;
    const long long cols = 2LL * HD + HV;
    if (scratch_floats < ck_floats(n, n_seg, H, D, V, H, true) + n * (cols + 3LL * H) + 16) return XR_ERR_ARG;
    float* rows = reinterpret_cast<float*>(((uintptr_t)scratch + 15) & ~(uintptr_t)15);
    float* log_f = rows + n * cols;
    float* in_scale = log_f + (size_t)n * H;
    float* floor_n = in_scale + (size_t)n * H;
    float* rest = reinterpret_cast<float*>(((uintptr_t)(floor_n + (size_t)n * H) + 15) & ~(uintptr_t)15);
    const long long head = (long long)ml_state_head(D, V);
    ChunkArgs a{rows, rows + HD, rows + 2 * HD, cols, cols, cols, H, V, nullptr, nullptr, in_scale, nullptr, nullptr, nullptr, nullptr, state, (long long)H * head,
                head, 1, seg_start, seg_len, seg_slot, n_seg, o, 1.0f, floor_n};
    double* cum = ck_lay_out(a, rest, n, D, true);
    a.cum = cum;
    const size_t total = (size_t)n * cols;
    const int most = xr_sm_count() * 8, blocks = (int)((total + 255) / 256 < (size_t)most ? (total + 255) / 256 : most);
    if (sizeof(T) == 2 && !((ldp | q_col | k_col | v_col | HD | HV) & 7) && !(((uintptr_t)proj | (uintptr_t)rows) & 15))
        xr_launch(k_mlstm_rows_vec, dim3(((2 * HD + HV) / 8 + 255) / 256, n < 65535 ? n : 65535), dim3(256), 0, stream, (const __nv_bfloat16*)proj, ldp, q_col, k_col,
                  v_col, rows, n, HD, HV, 1.0f / sqrtf((float)D));
    else xr_launch((k_mlstm_rows<T>), dim3(blocks), dim3(256), 0, stream, proj, ldp, q_col, k_col, v_col, rows, n, HD, HV, 1.0f / sqrtf((float)D));
    xr_launch(k_mlstm_scalars, dim3(H, n_seg), dim3(256), 0, stream, gates, state, log_f, in_scale, floor_n, seg_start, seg_len, seg_slot, H, D, V, cap);
    xr_launch(ck_cumulate, dim3((H + 127) / 128, (unsigned)ck_chunks(n, n_seg)), dim3(128), 0, stream, (const float*)log_f, (long long)H, cum, H, a);
    return ck_run<CK_TOKEN, true>(a, n, D, stream);
}

// proj [n][ldp] (activation dtype): q at q_col [H][D], k at k_col [H][D], v at v_col [H][V], output gate at g_col [H][V];
// gates [n][2H] float32 (input-gate pre-activations, then forget-gate ones, biases included);
// state [slots][H][D*V + D + 1] float32;  coef [n][H][3], o [n][H][V]: float32 scratch;  y [n][H*V] activation dtype.
// scratch (null: the walk): the recurrence in chunks, where it takes the sizes; xr_chunked_floats says how much it needs.
XR_EXPORT int xr_mlstm(const void* proj, int dtype, long long ldp, int q_col, int k_col, int v_col, int g_col, const float* gates,
                       float* state, float* coef, float* o, const float* norm_w, void* y, const int* seg_start,
                       const int* seg_len, const int* seg_slot, int n, int n_seg, int H, int D, int V, float cap, float eps,
                       float* scratch, long long scratch_floats, cudaStream_t stream) {
    if (n < 1 || n_seg < 1 || H < 1 || D < 1 || V < 1 || !(cap > 0.f) || n_seg > 65535 || H > 65535) return XR_ERR_ARG;
    // tokens a chunk of the gates kernel: what fits 44 KB of shared memory, at most 32; its threads own up to 4 elements of n each
    if (D > 1024) return XR_ERR_ARG;
    int stage = (int)((44 * 1024 / sizeof(float)) / ((size_t)D + 5));
    stage = stage > 32 ? 32 : stage;
    const size_t smem_g = (size_t)stage * (D + 5) * sizeof(float);
    const size_t smem_s = ((size_t)D * ML_VS + 2 * (size_t)ML_CHUNK * D + ML_CHUNK * ML_VS + ML_CHUNK * ML_RG * ML_VS + ML_CHUNK * 3) * sizeof(float);
    if (smem_g > 48 * 1024 || smem_s > 220 * 1024) return XR_ERR_ARG;
    dim3 gg(H, n_seg), gs((V + ML_VS - 1) / ML_VS, H, n_seg);
#define SCAN_ARGS(T) gs, dim3(ML_VS * ML_RG), 0, stream, (const T*)proj, ldp, q_col, k_col, v_col, (const float*)coef, state, o, seg_start, seg_len, seg_slot, H, D, V
#define SCAN(T)                                                                                                                       \
    do {                                                                                                                              \
        if (D <= 32) xr_launch((k_mlstm_scan<T, 4>), SCAN_ARGS(T));                                                                   \
        else if (D <= 64) xr_launch((k_mlstm_scan<T, 8>), SCAN_ARGS(T));                                                              \
        else if (D <= 128) xr_launch((k_mlstm_scan<T, 16>), SCAN_ARGS(T));                                                            \
        else if (D <= 256) xr_launch((k_mlstm_scan<T, 32>), SCAN_ARGS(T));                                                            \
        else xr_launch((k_mlstm_scan_wide<T>), gs, dim3(ML_VS * ML_RG), smem_s, stream, (const T*)proj, ldp, q_col, k_col, v_col,      \
                       (const float*)coef, state, o, seg_start, seg_len, seg_slot, H, D, V);                                          \
    } while (0)
#define ML(T)                                                                                                                         \
    do {                                                                                                                              \
        if (D > 256 && smem_s > 48 * 1024 &&                                                                                                     \
            cudaFuncSetAttribute(k_mlstm_scan_wide<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_s) != cudaSuccess)      \
            return XR_ERR_LAUNCH;                                                                                                     \
        if (scratch != nullptr && ck_takes(D, V) && ck_chunks(n, n_seg) <= 65535) {                                                   \
            const int rc = mlstm_chunked<T>((const T*)proj, ldp, q_col, k_col, v_col, gates, state, o, seg_start, seg_len, seg_slot, n, n_seg, H, D, V, \
                                            cap, scratch, scratch_floats, stream);                                                    \
            if (rc != XR_OK) return rc;                                                                                               \
        } else {                                                                                                                      \
        xr_launch((k_mlstm_gates<T>), gg, dim3(D <= 128 ? 128 : 256), smem_g, stream, (const T*)proj, ldp, q_col, k_col, gates, state, coef, seg_start, \
                  seg_len, seg_slot, H, D, V, cap, stage);                                                                            \
        SCAN(T);                                                                                                                      \
        }                                                                                                                             \
        launch_mlstm_out<T, T>((const float*)o, (const T*)proj, ldp, g_col, norm_w, (T*)y, n, H, V, eps, V, 0, stream);               \
    } while (0)
    if (dtype == XR_F32) ML(float);
    else if (dtype == XR_BF16) ML(__nv_bfloat16);
    else return XR_ERR_ARG;
#undef ML
#undef SCAN
#undef SCAN_ARGS
    return xr_launch_status();
}

// The last step alone, for other recurrences: y [n][H * V] (dtype `dtype`) = o / rms(o per head) * w * act(gate), gate [n][ld_gate]
// (dtype `gate_dtype`: that of y, or float32) from column 0, head h at h * V; w null: no weight; w_head: elements between the heads'
// weights (0: one weight for all heads).
XR_EXPORT int xr_head_norm_gate(const float* o, const void* gate, int gate_dtype, long long ld_gate, const float* w, int w_head, int gate_silu,
                                void* y, int dtype, int n, int H, int V, float eps, cudaStream_t stream) {
    if (n < 1 || H < 1 || V < 1 || w_head < 0) return XR_ERR_ARG;
    typedef __nv_bfloat16 bf;
    if (dtype == XR_F32 && gate_dtype == XR_F32)
        launch_mlstm_out(o, (const float*)gate, ld_gate, 0, w, (float*)y, n, H, V, eps, w_head, gate_silu, stream);
    else if (dtype == XR_BF16 && gate_dtype == XR_BF16)
        launch_mlstm_out(o, (const bf*)gate, ld_gate, 0, w, (bf*)y, n, H, V, eps, w_head, gate_silu, stream);
    else if (dtype == XR_BF16 && gate_dtype == XR_F32)
        launch_mlstm_out(o, (const float*)gate, ld_gate, 0, w, (bf*)y, n, H, V, eps, w_head, gate_silu, stream);
    else return XR_ERR_ARG;
    return xr_launch_status();
}
