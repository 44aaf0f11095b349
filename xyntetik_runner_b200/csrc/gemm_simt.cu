// out[t][r] = sum_k X[t][k] * W[r][k] (+ bias[r]) on CUDA cores with float32
// FMA: the matrix product of the true 32-bit path, and of any weight the
// tensor-core kernel does not take.  X and W are read in their stored type
// (float32 or bfloat16, widened exactly); products and sums are float32, never
// TF32.  Each output element is one thread's sum over k in ascending order, so
// a token's result does not depend on how many other tokens are in the call
// (the property the reference demands of its batched kernels,
// src/kernels.cu:2415-2454).  The reference's counterparts are the warp-per-row
// kernels `k_mv_*` / `k_mv_*_b` (src/kernels.cu:116-144, 534-549).
#include "simt_tile.cuh"

// What bounds it: the FMA pipes (70 TFLOP/s measured) where there are enough tiles, else the chain of copies and of K dependent
// multiply-adds, which is why a product with few tiles takes small ones: see launch_simt.  Earlier form (one 64 x 64 tile, blocks of
// 16, no ring) against this, bfloat16 W, us: 256 tokens x 1,024 rows of 1,024: 70 / 29; 256 x 5,632 x 1,024: 156 / 91; 256 x 1,024 x 2,816:
// 185 / 71; 2,048 x 5,632 x 1,024: 970 / 577 (41 TFLOP/s); 1 x 1,024 x 2,816: 160 / 35.
template <typename TX, typename TW, typename TO, bool ACCUM, int WM, int WN, int TM, int TN>
__global__ void __launch_bounds__(32 * WM * WN)
k_gemm_simt(const TX* __restrict__ X, const TW* __restrict__ W, const float* __restrict__ bias,
            TO* __restrict__ out, int n, int n_out, int K, long long ldx, long long ldo, float alpha, int vec) {
    constexpr int BM = 4 * TM * WM, BN = 8 * TN * WN;
    extern __shared__ __align__(16) unsigned char gs_sm[];
    const int t0 = blockIdx.y * BM, r0 = blockIdx.x * BN;
    float acc[TM][TN];
    gs_tile<TX, TW, WM, WN, TM, TN>(
        gs_sm, K, vec, [&](int i) { return t0 + i < n ? X + (size_t)(t0 + i) * ldx : (const TX*)nullptr; },
        [&](int i) { return r0 + i < n_out ? W + (size_t)(r0 + i) * K : (const TW*)nullptr; }, acc);
    const int tm = gs_token<WN, TM>(), rn = gs_row<WN, TN>();
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int t = t0 + tm + 4 * i;
        if (t >= n) continue;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int r = r0 + rn + 8 * j;
            if (r >= n_out) continue;
            float v = alpha * acc[i][j];
            if (bias) v += bias[r];
            const size_t o = (size_t)t * ldo + r;
            if (ACCUM) out[o] = xr_from_f32<TO>(xr_to_f32<TO>(out[o]) + v);
            else out[o] = xr_from_f32<TO>(v);
        }
    }
}

// The same sums without the ring, for operands that 16-byte copies do not fit and for K of a few values: 64 x 64 outputs of 256 threads,
// 16 values of k at a time through registers into shared memory, k-major.  Element by element the ring's copies are stores that every
// later load waits for; here a thread has eight loads in flight and four blocks share an SM.  What bounds it: shared memory, 8 words
// for 16 multiply-adds.
#define GP_BM 64
#define GP_BN 64
#define GP_BK 16
template <typename TX, typename TW, typename TO, bool ACCUM>
__global__ void __launch_bounds__(256)
k_gemm_simt_plain(const TX* __restrict__ X, const TW* __restrict__ W, const float* __restrict__ bias,
                  TO* __restrict__ out, int n, int n_out, int K, long long ldx, long long ldo, float alpha) {
    __shared__ float Xs[GP_BK][GP_BM + 4];
    __shared__ float Ws[GP_BK][GP_BN + 4];
    const int tid = threadIdx.x, t0 = blockIdx.y * GP_BM, r0 = blockIdx.x * GP_BN;
    const int ty = tid / 16, tx = tid % 16, lrow = tid / 4, lk = (tid % 4) * 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += GP_BK) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = k0 + lk + q, t = t0 + lrow, r = r0 + lrow;
            Xs[lk + q][lrow] = t < n && k < K ? xr_to_f32<TX>(X[(size_t)t * ldx + k]) : 0.f;
            Ws[lk + q][lrow] = r < n_out && k < K ? xr_to_f32<TW>(W[(size_t)r * K + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GP_BK; kk++) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = Xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + ty * 4 + i;
        if (t >= n) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = r0 + tx * 4 + j;
            if (r >= n_out) continue;
            float v = alpha * acc[i][j];
            if (bias) v += bias[r];
            const size_t o = (size_t)t * ldo + r;
            if (ACCUM) out[o] = xr_from_f32<TO>(xr_to_f32<TO>(out[o]) + v);
            else out[o] = xr_from_f32<TO>(v);
        }
    }
}

template <typename TX, typename TW, typename TO, bool ACCUM, int WM, int WN, int TM, int TN>
static int launch_simt_tile(const void* X, const void* W, const float* bias, void* out, int n, int n_out, int K, long long ldx, long long ldo,
                            float alpha, int vec, cudaStream_t stream) {
    constexpr int BM = 4 * TM * WM, BN = 8 * TN * WN;
    constexpr size_t SMEM = gs_smem<TX, TW, BM, BN>();
    const dim3 grid((n_out + BN - 1) / BN, (n + BM - 1) / BM);
    if (grid.y > 65535) return XR_ERR_ARG;
    static bool ready[XR_DEVICES];
    if (SMEM > 48 * 1024 && !xr_once_per_device(ready, [] { return xr_allow_smem(k_gemm_simt<TX, TW, TO, ACCUM, WM, WN, TM, TN>, SMEM); }))
        return XR_ERR_LAUNCH;
    k_gemm_simt<TX, TW, TO, ACCUM, WM, WN, TM, TN><<<grid, 32 * WM * WN, SMEM, stream>>>((const TX*)X, (const TW*)W, bias, (TO*)out, n, n_out, K, ldx, ldo, alpha, vec);
    return xr_launch_status();
}

// Which tile: every element's arithmetic is the same in all of them.  The widest of which there are enough to keep the machine busy:
// wide ones read fewer words a multiply-add from shared memory, narrow ones spread a small product over more SMs.  Measured, us, tiles
// 8x32 / 32x32 / 32x64 / 64x64 / 128x128: 44 x 1,024 x 1,024: 17 21 29 43 114; 256 x 1,024 x 1,024: 35 29 29 45 115; 256 x 5,632 x 1,024:
// 163 103 91 98 117; 256 x 32,000 x 1,024: 881 535 464 433 451; 2,048 x 5,632 x 1,024: 1,235 745 642 613 577.
// Operands off the 16-byte borders, and K of at most 16, take the kernel without the ring where its tiles fill a third of the SMs:
// 760 x 1,525 x 5,123 625 / 477 (with the ring / without), 1,765 x 949 x 553 114 / 78, 1,097 x 152 x 3,633 238 / 215, 1,587 x 5,939 x 58 68 / 51, 1,487 x 3,097 x 4 17 / 12;
// with fewer tiles the ring is ahead: 117 x 172 x 255 14 / 19, 756 x 258 x 179 37 / 51, 46 x 5 x 2,553 105 / 134.
template <typename TX, typename TW, typename TO, bool ACCUM>
static int launch_simt_out(const void* X, const void* W, const float* bias, void* out, int n, int n_out, int K, long long ldx, long long ldo,
                           float alpha, cudaStream_t stream) {
#define GS(WM, WN, TM, TN) return launch_simt_tile<TX, TW, TO, ACCUM, WM, WN, TM, TN>(X, W, bias, out, n, n_out, K, ldx, ldo, alpha, vec, stream)
    const long long sms = xr_sm_count();
    constexpr int PX = 16 / (int)sizeof(TX), PW = 16 / (int)sizeof(TW);
    const int vec = !(((uintptr_t)X | (uintptr_t)W) & 15) && ldx % PX == 0 && K % PX == 0 && K % PW == 0;
    auto tiles = [&](int bm, int bn) { return (long long)((n + bm - 1) / bm) * ((n_out + bn - 1) / bn); };
    if ((!vec || K <= GP_BK) && n > 64 && 3 * tiles(GP_BM, GP_BN) > sms && (n + GP_BM - 1) / GP_BM <= 65535) {
        k_gemm_simt_plain<TX, TW, TO, ACCUM><<<dim3((n_out + GP_BN - 1) / GP_BN, (n + GP_BM - 1) / GP_BM), 256, 0, stream>>>(
            (const TX*)X, (const TW*)W, bias, (TO*)out, n, n_out, K, ldx, ldo, alpha);
        return xr_launch_status();
    }
    int pick;
    if (n <= 8 || tiles(32, 32) < sms) pick = 0;
    else if (tiles(128, 128) >= 4 * sms) pick = 4;
    else if (tiles(64, 64) >= 4 * sms) pick = 3;
    else pick = tiles(32, 64) >= 2 * sms ? 2 : 1;
    switch (pick) {
        case 0: GS(1, 4, 2, 1);            // 8 tokens x 32 rows
        case 1: GS(2, 2, 4, 2);            // 32 x 32
        case 2: GS(2, 2, 4, 4);            // 32 x 64
        case 3: GS(2, 2, 8, 4);            // 64 x 64
        default: GS(4, 2, 8, 8);           // 128 x 128
    }
#undef GS
}

template <typename TX, typename TW>
static int launch_simt(const void* X, const void* W, const float* bias, void* out, int out_dtype, int accumulate,
                       int n, int n_out, int K, long long ldx, long long ldo, float alpha, cudaStream_t stream) {
    if (accumulate) {
        if (out_dtype != XR_F32) return XR_ERR_ARG;
        return launch_simt_out<TX, TW, float, true>(X, W, bias, out, n, n_out, K, ldx, ldo, alpha, stream);
    }
    if (out_dtype == XR_F32) return launch_simt_out<TX, TW, float, false>(X, W, bias, out, n, n_out, K, ldx, ldo, alpha, stream);
    if (out_dtype == XR_BF16) return launch_simt_out<TX, TW, __nv_bfloat16, false>(X, W, bias, out, n, n_out, K, ldx, ldo, alpha, stream);
    return XR_ERR_ARG;
}

// X: [n, K] with row stride ldx; W: [n_out, K] dense; out: [n, n_out] with row stride ldo.
// accumulate != 0 adds into a float32 `out` (the residual stream).  alpha multiplies every sum, ahead of the bias.
XR_EXPORT int xr_gemm_simt(const void* X, int x_dtype, const void* W, int w_dtype, const float* bias, void* out,
                           int out_dtype, int accumulate, int n, int n_out, int K, long long ldx, long long ldo,
                           float alpha, cudaStream_t stream) {
    if (n < 1 || n_out < 1 || K < 1 || ldx < K || ldo < n_out) return XR_ERR_ARG;
    if (x_dtype == XR_F32 && w_dtype == XR_F32) return launch_simt<float, float>(X, W, bias, out, out_dtype, accumulate, n, n_out, K, ldx, ldo, alpha, stream);
    if (x_dtype == XR_F32 && w_dtype == XR_BF16) return launch_simt<float, __nv_bfloat16>(X, W, bias, out, out_dtype, accumulate, n, n_out, K, ldx, ldo, alpha, stream);
    if (x_dtype == XR_BF16 && w_dtype == XR_F32) return launch_simt<__nv_bfloat16, float>(X, W, bias, out, out_dtype, accumulate, n, n_out, K, ldx, ldo, alpha, stream);
    if (x_dtype == XR_BF16 && w_dtype == XR_BF16) return launch_simt<__nv_bfloat16, __nv_bfloat16>(X, W, bias, out, out_dtype, accumulate, n, n_out, K, ldx, ldo, alpha, stream);
    return XR_ERR_ARG;
}
