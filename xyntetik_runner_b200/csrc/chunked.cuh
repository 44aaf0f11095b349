// Linear recurrences over a matrix memory, cut into chunks of 64 tokens and computed as products, in float32 throughout.
//
//   S_t = diag(a_t) S_(t-1) + s_t k_t v_t^T,    o_t = S_t^T q_t        (S [D][V] per head)
//
// with a_t one decay for all of a head (constant, or per token) or one per key channel.  With c_t the sum of log a from the chunk's
// first token to t, S the memory before the chunk:
//   o_i = (q_i exp(c_i))^T S + sum_(j <= i) P_ij v_j,      P_ij = s_j sum_d q_i[d] k_j[d] exp(c_i[d] - c_j[d])
//   S'  = diag(exp(c_last)) S + sum_j (k_j s_j exp(c_last - c_j)) v_j^T
// Four kernels: ck_scores (per chunk and head: the row [q_i exp(c_i) | P_i] of every token and its key k~_j = k_j s_j exp(c_last - c_j)),
// ck_states (the sum of S'), ck_scan (the memories before every chunk, one after another, in the place of the sums, and the slot's new
// state) and ck_out (one product of [64 x (D + 64)] with [S; v]).  c is summed and subtracted in float64, so that a difference of two sums keeps float32's relative
// precision however far both have gone; every exponential's argument is at or below zero, except in the short cut of decays per
// channel (ck_scores).
//
// Why: the token-by-token walk (recurrent.cu, mlstm.cu) is a chain of as many steps as the portion has tokens and reads q, k and v
// from shared memory for every few state elements; as products the same work is bound by the float32 FMA pipes and spread over all
// chunks at once.  It costs about half as many operations again and the memories' way through L2, so it is for portions of many
// tokens: parts/chunks.py compares the two by a step's portions (every one, a single token too, is a chunk of its own with a memory of its
// own).  The sums come in another order than the walk's, so a state depends in its last bits on where portions were cut and on what stood
// beside them; callers that promise the same bits take the walk.
// 2,048 tokens of one request, 8 heads, us, walk / chunks: constant decay, 128 x 128 values: 166 / 75; decay per channel, 128 x 256:
// 223 / 138; mLSTM, 128 x 256: 906 / 193.  Root mean square error of the read-outs against float64, 2,040 tokens, walk / chunks: 2.3e-7 /
// 1.7e-7; 2.1e-6 / 1.8e-7; 6.9e-7 / 6.5e-7.
#pragma once
#include "common.cuh"
#include <math.h>

#define CK_L 64                     // tokens a chunk
#define CK_VT 64                    // value columns a block
#define CK_KB 32                    // ck_out: terms a block of its sums
#define CK_ST 3                     // ck_out: blocks in flight
enum { CK_HEAD = 0, CK_TOKEN = 1, CK_KEY = 2 };

struct ChunkArgs {
    const float* q; const float* k; const float* v;      // token t's rows at + t * ld; head h's q and k at h D, its v at h V
    long long ld_q, ld_k, ld_v;
    int H, V;
    const float* decay;              // CK_HEAD: [H], in (0, 1]
    const double* cum;               // c: CK_TOKEN [n][H], CK_KEY [n][H D]
    const float* in_scale;           // s: [n][H], or null (one)
    float* rows;                     // [chunks][H][64][D + 64]
    float* keys;                     // k~: [chunks][H][64][D]
    float* mem;                      // [chunks][H][D][V]
    float* mem_n;                    // NORM: [chunks][H][D]
    float* state; long long state_stride, head_stride;   // a slot's head h at + h * head_stride: [V][D], or with `rows_first` [D][V]
    int rows_first;
    const int* seg_start; const int* seg_len; const int* seg_slot;
    int n_seg;
    float* o;                        // [n][H V]
    float read_scale;
    const float* floor_n;            // NORM: [n][H]: the least denominator
};

// exp(x) of a float64 argument in float32: the argument's rounding to float32 is put back to first order, so that the result is
// good to float32's last bits however large |x| is.
__device__ __forceinline__ float ck_exp(double x) {
    const float hi = (float)x;
    const float e = expf(hi);
    return hi < -87.f ? e : fmaf(e, (float)(x - (double)hi), e);
}

// chunk -> its portion's tokens: (portion, first token of the step, tokens); portion -1: there is none
struct ChunkPlace { int seg, t0, count, first; };
__device__ __forceinline__ ChunkPlace ck_place(const ChunkArgs& a, int chunk) {
    int before = 0;
    for (int s = 0; s < a.n_seg; s++) {
        const int len = a.seg_len[s], c = (len + CK_L - 1) / CK_L;
        if (chunk < before + c) {
            const int i = (chunk - before) * CK_L;
            return {s, a.seg_start[s] + i, min(CK_L, len - i), before};
        }
        before += c;
    }
    return {-1, 0, 0, 0};
}

// ---- the sums c: a thread a (chunk, column), tokens in ascending order.  (A logarithm below -200 counts as -200: its decay is zero in
// float32 all the same, and differences of sums behind it keep their digits.) -------------------------------------------------
static __global__ void __launch_bounds__(128)
ck_cumulate(const float* __restrict__ log_a, long long ld, double* __restrict__ cum, int cols, ChunkArgs a) {
    xr_pdl_launch();
    const int c = blockIdx.x * 128 + threadIdx.x;
    const ChunkPlace p = ck_place(a, blockIdx.y);
    xr_pdl_wait();
    if (p.seg < 0 || c >= cols) return;
    double sum = 0.0;
    for (int i0 = 0; i0 < p.count; i0 += 16) {
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; i++) x[i] = xr_ld_now(log_a + (size_t)(p.t0 + min(i0 + i, p.count - 1)) * ld + c);
#pragma unroll
        for (int i = 0; i < 16; i++) xr_ld_fence(x[i]);
#pragma unroll
        for (int i = 0; i < 16; i++)
            if (i0 + i < p.count) { sum += (double)(x[i] < -200.f ? -200.f : x[i]); cum[(size_t)(p.t0 + i0 + i) * cols + c] = sum; }
    }
}

// ---- [q exp(c) | P] ----------------------------------------------------------------------------------------------------
// 256 threads, 4 x 4 scores each.  CK_KEY: where no channel's decay over the chunk goes below exp(-CK_DEEP), P is the product of
// q exp(c) and k exp(-c), which stay within float32's range (a score whose keys are too large for that is summed pair by pair).  Else, by sixteens of tokens with r the sum at the end of the sixteen
// before: a later sixteen's queries times exp(c_i - r) with the earlier keys times exp(r - c_j), both factors at most one, and inside a
// sixteen every pair's exponentials channel by channel.
#define CK_DEEP 60.0
// CK_KEY: one score, every channel's exponential on its own.  q, k: the two tokens' rows of the head, ci, cj their sums c.
template <int D>
static __device__ __noinline__ float ck_pair(const float* q, const float* k, const double* ci, const double* cj) {
    float sum = 0.f;
    for (int d = 0; d < D; d++) sum = fmaf(q[d] * k[d], ck_exp(ci[d] - cj[d]), sum);
    return sum;
}

template <int D, int KIND>
__global__ void __launch_bounds__(256)
ck_scores(ChunkArgs a) {
    xr_pdl_launch();
    constexpr int LD = D + 4, LR = D + CK_L;
    extern __shared__ __align__(16) float ck_sm[];
    float* qs = ck_sm;                       // [64][LD]
    float* ks = qs + CK_L * LD;              // [64][LD]; CK_KEY: 48 rows more behind it
    __shared__ double cs[CK_L];
    __shared__ float ends[CK_L];
    __shared__ int deep;
    const int h = blockIdx.x, tid = threadIdx.x;
    const ChunkPlace p = ck_place(a, blockIdx.y);
    xr_pdl_wait();
    if (p.seg < 0) return;
    if (tid == 0) deep = 0;
    const int last = p.t0 + p.count - 1;
    if (KIND != CK_KEY && tid < CK_L) {
        // c, and what a key's outer product is worth at the chunk's end
        const int t = min(tid, p.count - 1);
        const double lad = KIND == CK_HEAD ? log((double)a.decay[h]) : 0.0;
        cs[tid] = KIND == CK_HEAD ? (tid + 1) * lad : a.cum[(size_t)(p.t0 + t) * a.H + h];
        float f = KIND == CK_HEAD ? (t == p.count - 1 ? 1.f : ck_exp((p.count - 1 - t) * lad)) : ck_exp(a.cum[(size_t)last * a.H + h] - a.cum[(size_t)(p.t0 + t) * a.H + h]);
        if (a.in_scale != nullptr) f *= a.in_scale[(size_t)(p.t0 + t) * a.H + h];
        ends[tid] = f;
    }
    __syncthreads();
    // (a sum that is no number says nothing about the tokens before it)
    if (KIND == CK_KEY && tid < D && !(a.cum[((size_t)(p.t0 + p.count - 1) * a.H + h) * D + tid] >= -CK_DEEP)) deep = 1;
    if (KIND == CK_KEY) __syncthreads();
    float* out = a.rows + ((size_t)blockIdx.y * a.H + h) * CK_L * LR;
    float* keys = a.keys + ((size_t)blockIdx.y * a.H + h) * CK_L * D;
    for (int e = tid * 4; e < CK_L * D; e += 1024) {
        const int t = e / D, d = e % D;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q, r = q, kt = q;
        if (t < p.count) {
            q = *reinterpret_cast<const float4*>(a.q + (size_t)(p.t0 + t) * a.ld_q + h * D + d);
            k = *reinterpret_cast<const float4*>(a.k + (size_t)(p.t0 + t) * a.ld_k + h * D + d);
            if (KIND == CK_KEY) {
                const double* c = a.cum + ((size_t)(p.t0 + t) * a.H + h) * D + d;
                const double c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
                const double* cl = a.cum + ((size_t)last * a.H + h) * D + d;
                kt = make_float4(k.x * ck_exp(cl[0] - c0), k.y * ck_exp(cl[1] - c1), k.z * ck_exp(cl[2] - c2), k.w * ck_exp(cl[3] - c3));
                r = make_float4(q.x * ck_exp(c0), q.y * ck_exp(c1), q.z * ck_exp(c2), q.w * ck_exp(c3));
                if (!deep) {
                    q = r;
                    k = make_float4(k.x * ck_exp(-c0), k.y * ck_exp(-c1), k.z * ck_exp(-c2), k.w * ck_exp(-c3));
                } else if (t >= 16) {
                    const double* b = a.cum + ((size_t)(p.t0 + t / 16 * 16 - 1) * a.H + h) * D + d;
                    q = make_float4(q.x * ck_exp(c0 - b[0]), q.y * ck_exp(c1 - b[1]), q.z * ck_exp(c2 - b[2]), q.w * ck_exp(c3 - b[3]));
                }
            } else {
                const float f = ck_exp(cs[t]);
                r = make_float4(q.x * f, q.y * f, q.z * f, q.w * f);
                float g = ends[t];
                kt = make_float4(k.x * g, k.y * g, k.z * g, k.w * g);
            }
        }
        *reinterpret_cast<float4*>(qs + t * LD + d) = q;
        *reinterpret_cast<float4*>(ks + t * LD + d) = k;
        *reinterpret_cast<float4*>(out + t * LR + d) = r;
        *reinterpret_cast<float4*>(keys + t * D + d) = kt;
    }
    __syncthreads();
    // thread: tokens i = ti + 16 r, keys j = tj + 16 r (r = 0..3): rows 16 apart, so that a warp's sixteen tj read neighbouring rows
    const int ti = tid >> 4, tj = tid & 15;
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int s = 0; s < 4; s++) acc[r][s] = 0.f;
    if (KIND == CK_KEY && deep) {
        float* kb = ks + CK_L * LD;          // [48][LD]
#pragma unroll
        for (int r = 1; r < 4; r++) {        // the sixteen's queries with all earlier keys
            __syncthreads();
            if (16 * r < p.count) {
                const double* b = a.cum + ((size_t)(p.t0 + 16 * r - 1) * a.H + h) * D;
                for (int e = tid; e < 16 * r * D; e += 256) {
                    const int j = e / D, d = e % D;
                    kb[j * LD + d] = ks[j * LD + d] * ck_exp(b[d] - a.cum[((size_t)(p.t0 + j) * a.H + h) * D + d]);
                }
            }
            __syncthreads();
            if (16 * r < p.count)
                for (int d = 0; d < D; d += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(qs + (ti + 16 * r) * LD + d);
#pragma unroll
                    for (int s = 0; s < r; s++) {
                        const float4 y = *reinterpret_cast<const float4*>(kb + (tj + 16 * s) * LD + d);
                        acc[r][s] = fmaf(x.x, y.x, acc[r][s]); acc[r][s] = fmaf(x.y, y.y, acc[r][s]);
                        acc[r][s] = fmaf(x.z, y.z, acc[r][s]); acc[r][s] = fmaf(x.w, y.w, acc[r][s]);
                    }
                }
        }
        if (tj <= ti)
#pragma unroll
            for (int r = 0; r < 4; r++) {    // inside a sixteen
                const int i = ti + 16 * r, j = tj + 16 * r;
                if (i >= p.count) continue;
                const float* qi = a.q + (size_t)(p.t0 + i) * a.ld_q + h * D;
                const double* ci = a.cum + ((size_t)(p.t0 + i) * a.H + h) * D;
                const double* cj = a.cum + ((size_t)(p.t0 + j) * a.H + h) * D;
                float sum = 0.f;
                for (int d = 0; d < D; d++) sum = fmaf(qi[d] * ks[j * LD + d], ck_exp(ci[d] - cj[d]), sum);
                acc[r][r] = sum;
            }
    } else {
        // (16 channels at a time on their own, then added: see ck_out)
        for (int d0 = 0; d0 < D; d0 += 16) {
            float part[4][4];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int s = 0; s < 4; s++) part[r][s] = 0.f;
#pragma unroll 2
            for (int d = d0; d < d0 + 16; d += 4) {
                float4 x[4], y[4];
#pragma unroll
                for (int r = 0; r < 4; r++) x[r] = *reinterpret_cast<const float4*>(qs + (ti + 16 * r) * LD + d);
#pragma unroll
                for (int s = 0; s < 4; s++) y[s] = *reinterpret_cast<const float4*>(ks + (tj + 16 * s) * LD + d);
#pragma unroll
                for (int r = 0; r < 4; r++)
#pragma unroll
                    for (int s = 0; s <= r; s++) {       // (later keys' sixteens are masked whole)
                        part[r][s] = fmaf(x[r].x, y[s].x, part[r][s]); part[r][s] = fmaf(x[r].y, y[s].y, part[r][s]);
                        part[r][s] = fmaf(x[r].z, y[s].z, part[r][s]); part[r][s] = fmaf(x[r].w, y[s].w, part[r][s]);
                    }
            }
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int s = 0; s <= r; s++) acc[r][s] += part[r][s];
        }
    }
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const int j = tj + 16 * s;
        const float in = a.in_scale != nullptr && j < p.count ? a.in_scale[(size_t)(p.t0 + j) * a.H + h] : 1.f;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int i = ti + 16 * r;
            float x = 0.f;
            if (j <= i && i < p.count) {
                x = acc[r][s];
                if (KIND == CK_KEY && !(fabsf(x) < INFINITY)) {
                    const size_t ti64 = (size_t)(p.t0 + i), tj64 = (size_t)(p.t0 + j);
                    x = ck_pair<D>(a.q + ti64 * a.ld_q + h * D, a.k + tj64 * a.ld_k + h * D, a.cum + (ti64 * a.H + h) * D, a.cum + (tj64 * a.H + h) * D);
                }
                x *= in;
                if (KIND != CK_KEY && i != j) x *= ck_exp(cs[i] - cs[j]);
            }
            out[i * LR + D + j] = x;
        }
    }
}

// ---- sum_j k~_j v_j^T -----------------------------------------------------------------------------------------------
// 256 threads over D x 64: (D / 16) x 4 each, four channels and four columns at a time; all of the chunk's keys (as ck_scores left them)
// and values on their way at once.  (With the keys' exponentials taken here, once for every 64 value columns, the recurrence with decays
// per channel took 164 us at 2,048 tokens, 8 heads of 128 x 256; 138 so.)
template <int D, bool NORM>
__global__ void __launch_bounds__(256)
ck_states(ChunkArgs a) {
    xr_pdl_launch();
    constexpr int RD = D / 16;               // channels a thread: 4 (tid / 16) + 64 m + (0..3)
    __shared__ __align__(16) float ks[CK_L][D], vs[CK_L][CK_VT];
    const int v0 = blockIdx.x * CK_VT, h = blockIdx.y, tid = threadIdx.x;
    const ChunkPlace p = ck_place(a, blockIdx.z);
    xr_pdl_wait();
    if (p.seg < 0) return;
    const size_t at = (size_t)blockIdx.z * a.H + h;
    for (int e = tid * 4; e < CK_L * D; e += 1024)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(&ks[0][0] + e)), "l"(a.keys + at * CK_L * D + e) : "memory");
    for (int e = tid * 4; e < CK_L * CK_VT; e += 1024) {
        const int j = e / CK_VT, c = e % CK_VT, live = j < p.count ? 16 : 0;          // (no token: zeros)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(&vs[0][0] + e)),
                     "l"(a.v + (size_t)(p.t0 + (live ? j : 0)) * a.ld_v + (size_t)h * a.V + v0 + c), "r"(live) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int td = tid >> 4, tv = tid & 15;
    float acc[RD][4];
#pragma unroll
    for (int r = 0; r < RD; r++)
#pragma unroll
        for (int s = 0; s < 4; s++) acc[r][s] = 0.f;
#pragma unroll 4
    for (int j = 0; j < CK_L; j++) {
        const float4 v = *reinterpret_cast<const float4*>(&vs[j][4 * tv]);
#pragma unroll
        for (int m = 0; m < RD / 4; m++) {
            const float4 k = *reinterpret_cast<const float4*>(&ks[j][64 * m + 4 * td]);
            const float kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
            for (int r = 0; r < 4; r++) {
                acc[4 * m + r][0] = fmaf(kk[r], v.x, acc[4 * m + r][0]); acc[4 * m + r][1] = fmaf(kk[r], v.y, acc[4 * m + r][1]);
                acc[4 * m + r][2] = fmaf(kk[r], v.z, acc[4 * m + r][2]); acc[4 * m + r][3] = fmaf(kk[r], v.w, acc[4 * m + r][3]);
            }
        }
    }
    float* out = a.mem + at * D * a.V + v0 + 4 * tv;
#pragma unroll
    for (int m = 0; m < RD / 4; m++)
#pragma unroll
        for (int r = 0; r < 4; r++)
            *reinterpret_cast<float4*>(out + (size_t)(64 * m + 4 * td + r) * a.V) = make_float4(acc[4 * m + r][0], acc[4 * m + r][1], acc[4 * m + r][2], acc[4 * m + r][3]);
    if (NORM && blockIdx.x == 0 && tid < D) {
        float sum = 0.f;
        for (int j = 0; j < CK_L; j++) sum += ks[j][tid];
        a.mem_n[at * D + tid] = sum;
    }
}

// ---- the memories before the chunks ------------------------------------------------------------------------------------
// A thread an element of S (NORM: and, behind them, of the sum of keys), chunk after chunk; eight chunks' sums in flight.
template <int D, int KIND, bool NORM>
__global__ void __launch_bounds__(256)
ck_scan(ChunkArgs a) {
    xr_pdl_launch();
    const int seg = blockIdx.z, h = blockIdx.y, V = a.V, total = D * V;
    int e = blockIdx.x * 256 + threadIdx.x;
    const bool norm = NORM && e >= total;
    if (e >= total + (NORM ? D : 0)) return;
    const int len = a.seg_len[seg], chunks = (len + CK_L - 1) / CK_L;
    int first = 0;
    for (int s = 0; s < seg; s++) first += (a.seg_len[s] + CK_L - 1) / CK_L;
    xr_pdl_wait();
    if (chunks == 0) return;
    const int d = norm ? e - total : e / V, v = norm ? 0 : e % V;
    float* st = a.state + (size_t)a.seg_slot[seg] * a.state_stride + (size_t)h * a.head_stride +
                (norm ? (size_t)total + d : (a.rows_first ? (size_t)d * V + v : (size_t)v * D + d));
    float* m = norm ? a.mem_n + ((size_t)first * a.H + h) * D + d : a.mem + ((size_t)first * a.H + h) * total + e;
    const size_t step = (size_t)a.H * (norm ? D : total);
    const double lad = KIND == CK_HEAD ? log((double)a.decay[h]) : 0.0;
    float S = *st;
    for (int c0 = 0; c0 < chunks; c0 += 8) {
        float u[8];
        double cl[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int c = min(c0 + i, chunks - 1), last = min(len, (c + 1) * CK_L) - 1;
            u[i] = xr_ld_now(m + c * step);
            const int t = a.seg_start[seg] + last;
            cl[i] = KIND == CK_HEAD ? (last - c * CK_L + 1) * lad : (KIND == CK_TOKEN ? a.cum[(size_t)t * a.H + h] : a.cum[((size_t)t * a.H + h) * D + d]);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) xr_ld_fence(u[i]);
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (c0 + i < chunks) {
                m[(size_t)(c0 + i) * step] = S;
                S = fmaf(ck_exp(cl[i]), S, u[i]);
            }
    }
    *st = S;
}

// Token i's read-out in columns v0 .. v0 + 3 once more, with the values up to its own only: the product above also takes the chunk's later
// values, times zero, which is no zero where one of them is infinite or no number.  The same sums in the same order.
template <int D>
static __device__ __noinline__ float4 ck_out_causal(const float* row, const float* mem, const float* vals, long long ld_v, int V, int i) {
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 <= D + i; k0 += CK_KB) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = k0; k < k0 + CK_KB && k <= D + i; k++) {
            const float4 y = *reinterpret_cast<const float4*>(k < D ? mem + (size_t)k * V : vals + (size_t)(k - D) * ld_v);
            acc = make_float4(fmaf(row[k], y.x, acc.x), fmaf(row[k], y.y, acc.y), fmaf(row[k], y.z, acc.z), fmaf(row[k], y.w, acc.w));
        }
        sum = make_float4(sum.x + acc.x, sum.y + acc.y, sum.z + acc.z, sum.w + acc.w);
    }
    return sum;
}

// ---- [q exp(c) | P] [S; v] ----------------------------------------------------------------------------------------------
// 64 tokens x 64 columns a block of four warps; a thread 8 tokens (8 apart) x 4 columns; both operands in blocks of 32 through a ring
// of three stages.  A block's 32 terms are summed on their own and then added: the sums' rounding grows with their length.
template <int D, bool NORM>
__global__ void __launch_bounds__(128)
ck_out(ChunkArgs a) {
    xr_pdl_launch();
    constexpr int LR = D + CK_L, LA = CK_KB + 4, BLOCKS = LR / CK_KB;
    extern __shared__ __align__(16) float ck_sm[];
    float* as = ck_sm;                               // [CK_ST][64][LA]
    float* bs = as + CK_ST * CK_L * LA;              // [CK_ST][32][CK_VT]
    __shared__ float den[CK_L];
    const int v0 = blockIdx.x * CK_VT, h = blockIdx.y, tid = threadIdx.x;
    const ChunkPlace p = ck_place(a, blockIdx.z);
    xr_pdl_wait();
    if (p.seg < 0) return;
    const size_t at = (size_t)blockIdx.z * a.H + h;
    const float* rows = a.rows + at * CK_L * LR;
    const float* mem = a.mem + at * D * a.V + v0;
    const float* vals = a.v + (size_t)p.t0 * a.ld_v + (size_t)h * a.V + v0;
    auto fill = [&](int b) {
        float* ad = as + (b % CK_ST) * CK_L * LA;
        float* bd = bs + (b % CK_ST) * CK_KB * CK_VT;
        for (int e = tid; e < CK_L * (CK_KB / 4); e += 128) {
            const int t = e / (CK_KB / 4), k = e % (CK_KB / 4) * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(ad + t * LA + k)), "l"(rows + t * LR + b * CK_KB + k) : "memory");
        }
        for (int e = tid; e < CK_KB * (CK_VT / 4); e += 128) {
            const int r = e / (CK_VT / 4), c = e % (CK_VT / 4) * 4, k = b * CK_KB + r, j = k - D;
            const float* src = k < D ? mem + (size_t)k * a.V + c : vals + (size_t)(j < p.count ? j : 0) * a.ld_v + c;
            const int bytes = k < D || j < p.count ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(bd + r * CK_VT + c)), "l"(src), "r"(bytes) : "memory");
        }
    };
    const int tt = tid >> 4, tc = tid & 15;          // tokens tt + 8 r, columns 4 tc + (0..3)
    float sum[8][4];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
        for (int s = 0; s < 4; s++) sum[r][s] = 0.f;
#pragma unroll
    for (int b = 0; b < CK_ST - 1; b++) { fill(b); asm volatile("cp.async.commit_group;" ::: "memory"); }
    if (NORM) {
        // the denominators: the same rows times [sum of keys; ones], two threads a token; in float64, because they may cancel
        const float* nm = a.mem_n + at * D;
        const float* r = rows + (tid >> 1) * LR;
        double part[4] = {0.0, 0.0, 0.0, 0.0};
        for (int k = (tid & 1) * 4; k < LR; k += 8) {
            const float4 x = *reinterpret_cast<const float4*>(r + k);
            const float4 y = k < D ? *reinterpret_cast<const float4*>(nm + k) : make_float4(1.f, 1.f, 1.f, 1.f);
            part[0] = fma((double)x.x, (double)y.x, part[0]); part[1] = fma((double)x.y, (double)y.y, part[1]);
            part[2] = fma((double)x.z, (double)y.z, part[2]); part[3] = fma((double)x.w, (double)y.w, part[3]);
        }
        double sum64 = (part[0] + part[1]) + (part[2] + part[3]);
        sum64 += __shfl_xor_sync(0xffffffffu, sum64, 1);
        const float total = (float)sum64;
        if (!(tid & 1)) den[tid >> 1] = (tid >> 1) < p.count ? fmaxf(fabsf(total), a.floor_n[(size_t)(p.t0 + (tid >> 1)) * a.H + h]) + 1e-6f : 1.f;
    }
    for (int b = 0; b < BLOCKS; b++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(CK_ST - 2) : "memory");
        __syncthreads();
        if (b + CK_ST - 1 < BLOCKS) fill(b + CK_ST - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* ab = as + (b % CK_ST) * CK_L * LA + tt * LA;
        const float* bb = bs + (b % CK_ST) * CK_KB * CK_VT + 4 * tc;
        float acc[8][4];
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
            for (int s = 0; s < 4; s++) acc[r][s] = 0.f;
#pragma unroll
        for (int k = 0; k < CK_KB; k += 4) {
            float4 x[8], y[4];
#pragma unroll
            for (int r = 0; r < 8; r++) x[r] = *reinterpret_cast<const float4*>(ab + 8 * r * LA + k);
#pragma unroll
            for (int i = 0; i < 4; i++) y[i] = *reinterpret_cast<const float4*>(bb + (k + i) * CK_VT);
#pragma unroll
            for (int r = 0; r < 8; r++) {
                acc[r][0] = fmaf(x[r].x, y[0].x, acc[r][0]); acc[r][1] = fmaf(x[r].x, y[0].y, acc[r][1]); acc[r][2] = fmaf(x[r].x, y[0].z, acc[r][2]); acc[r][3] = fmaf(x[r].x, y[0].w, acc[r][3]);
            }
#pragma unroll
            for (int r = 0; r < 8; r++) {
                acc[r][0] = fmaf(x[r].y, y[1].x, acc[r][0]); acc[r][1] = fmaf(x[r].y, y[1].y, acc[r][1]); acc[r][2] = fmaf(x[r].y, y[1].z, acc[r][2]); acc[r][3] = fmaf(x[r].y, y[1].w, acc[r][3]);
            }
#pragma unroll
            for (int r = 0; r < 8; r++) {
                acc[r][0] = fmaf(x[r].z, y[2].x, acc[r][0]); acc[r][1] = fmaf(x[r].z, y[2].y, acc[r][1]); acc[r][2] = fmaf(x[r].z, y[2].z, acc[r][2]); acc[r][3] = fmaf(x[r].z, y[2].w, acc[r][3]);
            }
#pragma unroll
            for (int r = 0; r < 8; r++) {
                acc[r][0] = fmaf(x[r].w, y[3].x, acc[r][0]); acc[r][1] = fmaf(x[r].w, y[3].y, acc[r][1]); acc[r][2] = fmaf(x[r].w, y[3].z, acc[r][2]); acc[r][3] = fmaf(x[r].w, y[3].w, acc[r][3]);
            }
        }
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
            for (int s = 0; s < 4; s++) sum[r][s] += acc[r][s];
    }
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int i = tt + 8 * r;
        if (i >= p.count) continue;
        float4 y = make_float4(sum[r][0], sum[r][1], sum[r][2], sum[r][3]);
        if (!(fabsf(y.x) < INFINITY && fabsf(y.y) < INFINITY && fabsf(y.z) < INFINITY && fabsf(y.w) < INFINITY))
            y = ck_out_causal<D>(rows + (size_t)i * LR, mem + 4 * tc, vals + 4 * tc, a.ld_v, a.V, i);
        if (NORM) {
            const float f = den[i];
            y = make_float4(y.x / f, y.y / f, y.z / f, y.w / f);
        } else {
            y = make_float4(y.x * a.read_scale, y.y * a.read_scale, y.z * a.read_scale, y.w * a.read_scale);
        }
        *reinterpret_cast<float4*>(a.o + (size_t)(p.t0 + i) * a.H * a.V + (size_t)h * a.V + v0 + 4 * tc) = y;
    }
}

// ---- host ---------------------------------------------------------------------------------------------------------------
static inline bool ck_takes(int D, int V) { return (D == 64 || D == 128) && V >= CK_VT && V % CK_VT == 0; }
// chunks of a step of n tokens in n_seg portions, at most
static inline long long ck_chunks(int n, int n_seg) { return n / CK_L + n_seg; }
// float32 of scratch: rows, keys, memories (and sums of keys), then float64 sums c of `cum_cols` columns a token
static inline long long ck_floats(int n, int n_seg, int H, int D, int V, int cum_cols, bool norm) {
    const long long per = (long long)CK_L * (2 * D + CK_L) + (long long)D * V + (norm ? D : 0);
    return ck_chunks(n, n_seg) * H * per + 2LL * n * cum_cols + 8;
}
// lays the scratch out; returns where the sums c begin
static inline double* ck_lay_out(ChunkArgs& a, float* scratch, int n, int D, bool norm) {
    const long long heads = ck_chunks(n, a.n_seg) * a.H;
    a.rows = scratch;
    a.keys = a.rows + heads * CK_L * (D + CK_L);
    a.mem = a.keys + heads * CK_L * D;
    a.mem_n = norm ? a.mem + heads * D * a.V : nullptr;
    float* end = a.mem + heads * D * a.V + (norm ? heads * D : 0);
    return reinterpret_cast<double*>(((uintptr_t)end + 15) & ~(uintptr_t)15);
}

template <int D, int KIND, bool NORM>
static int ck_launch(const ChunkArgs& a, int n, cudaStream_t stream) {
    const unsigned chunks = (unsigned)ck_chunks(n, a.n_seg), vt = (unsigned)(a.V / CK_VT);
    if (chunks > 65535 || a.H > 65535 || a.n_seg > 65535) return XR_ERR_ARG;
    constexpr size_t S1 = (2 * CK_L + (KIND == CK_KEY ? 48 : 0)) * (size_t)(D + 4) * sizeof(float);
    constexpr size_t S4 = (size_t)CK_ST * (CK_L * (CK_KB + 4) + CK_KB * CK_VT) * sizeof(float);
    static bool ready[XR_DEVICES];
    if (!xr_once_per_device(ready, [] { return xr_allow_smem(ck_scores<D, KIND>, S1) && xr_allow_smem(ck_out<D, NORM>, S4); })) return XR_ERR_LAUNCH;
    xr_launch((ck_scores<D, KIND>), dim3(a.H, chunks), dim3(256), S1, stream, a);
    xr_launch((ck_states<D, NORM>), dim3(vt, a.H, chunks), dim3(256), 0, stream, a);
    xr_launch((ck_scan<D, KIND, NORM>), dim3((D * a.V + (NORM ? D : 0) + 255) / 256, a.H, a.n_seg), dim3(256), 0, stream, a);
    xr_launch((ck_out<D, NORM>), dim3(vt, a.H, chunks), dim3(128), S4, stream, a);
    return xr_launch_status();
}
template <int KIND, bool NORM>
static int ck_run(const ChunkArgs& a, int n, int D, cudaStream_t stream) {
    return D == 64 ? ck_launch<64, KIND, NORM>(a, n, stream) : ck_launch<128, KIND, NORM>(a, n, stream);
}
// 16 bytes a load: rows and columns on a 16-byte border
static inline bool ck_aligned(const ChunkArgs& a) {
    return !(((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.o) & 15) && !((a.ld_q | a.ld_k | a.ld_v) & 3);
}
