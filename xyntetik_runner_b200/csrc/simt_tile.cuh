// The inner part of the float32 products on CUDA cores: a tile of sums  acc(token, row) = sum_k x(token)[k] w(row)[k].
//
// A block: WM x WN warps, a warp 4 TM tokens x 8 TN rows, a thread TM x TN sums in registers (rows 8 apart, tokens 4 apart, so that
// the eight rows and four tokens that a warp reads at a time lie in different banks).  Both operands come in blocks of GS_BK values
// of k through a ring of GS_STAGES shared-memory stages, as stored (bfloat16 is widened in registers), by 16-byte asynchronous
// copies where the caller says that addresses, strides and K allow it (`vec`), else element by element.  Every sum is one thread's,
// over k in ascending order, whatever the tile: the tiles differ in speed only.
#pragma once
#include "common.cuh"

#define GS_BK 32
#define GS_STAGES 4

__device__ __forceinline__ void gs_copy_async(void* dst, const void* src, bool live) {
    const unsigned at = (unsigned)__cvta_generic_to_shared(dst);
    const int n = live ? 16 : 0;                          // (bytes that are not copied are filled with zeros)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(src), "r"(n) : "memory");
}
// four consecutive values of k
__device__ __forceinline__ float4 gs_read4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 gs_read4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
// elements between rows of a stage: 16 bytes more than the block, see above
template <typename T> __host__ __device__ constexpr int gs_stride() { return GS_BK + 16 / (int)sizeof(T); }
template <typename TX, typename TW, int BM, int BN> constexpr size_t gs_smem() {
    return (size_t)GS_STAGES * (BM * gs_stride<TX>() * sizeof(TX) + BN * gs_stride<TW>() * sizeof(TW));
}


// xrow(i), wrow(i): the address of the tile's i-th token's or row's first value, null where there is none (it counts as zeros).
template <typename TX, typename TW, int WM, int WN, int TM, int TN, typename XRow, typename WRow>
__device__ __forceinline__ void gs_tile(unsigned char* sm, int K, bool vec, XRow xrow, WRow wrow, float (&acc)[TM][TN]) {
    constexpr int BM = 4 * TM * WM, BN = 8 * TN * WN, THREADS = 32 * WM * WN;
    constexpr int SX = gs_stride<TX>(), SW = gs_stride<TW>();
    TX* xs = reinterpret_cast<TX*>(sm);                             // [GS_STAGES][BM][SX]
    TW* ws = reinterpret_cast<TW*>(xs + GS_STAGES * BM * SX);       // [GS_STAGES][BN][SW]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tm = (warp / WN) * 4 * TM + (lane >> 3), rn = (warp % WN) * 8 * TN + (lane & 7);
    const int blocks = (K + GS_BK - 1) / GS_BK;
    const TX* any_x = xrow(0);                                      // (a tile's first token and row exist)
    const TW* any_w = wrow(0);

    auto fill = [&](int b) {
        TX* xd = xs + (b % GS_STAGES) * BM * SX;
        TW* wd = ws + (b % GS_STAGES) * BN * SW;
        const int k0 = b * GS_BK;
        if (vec) {
            constexpr int PX = 16 / (int)sizeof(TX), PW = 16 / (int)sizeof(TW);      // values a copy moves
#pragma unroll
            for (int e = tid; e < BM * (GS_BK / PX); e += THREADS) {
                const int row = e / (GS_BK / PX), k = e % (GS_BK / PX) * PX;
                const TX* p = xrow(row);
                const bool ok = p != nullptr && k0 + k < K;
                gs_copy_async(xd + row * SX + k, ok ? p + k0 + k : any_x, ok);
            }
#pragma unroll
            for (int e = tid; e < BN * (GS_BK / PW); e += THREADS) {
                const int row = e / (GS_BK / PW), k = e % (GS_BK / PW) * PW;
                const TW* p = wrow(row);
                const bool ok = p != nullptr && k0 + k < K;
                gs_copy_async(wd + row * SW + k, ok ? p + k0 + k : any_w, ok);
            }
        } else {
            for (int e = tid; e < BM * GS_BK; e += THREADS) {
                const int row = e / GS_BK, k = e % GS_BK;
                const TX* p = xrow(row);
                xd[row * SX + k] = p != nullptr && k0 + k < K ? p[k0 + k] : xr_from_f32<TX>(0.f);
            }
            for (int e = tid; e < BN * GS_BK; e += THREADS) {
                const int row = e / GS_BK, k = e % GS_BK;
                const TW* p = wrow(row);
                wd[row * SW + k] = p != nullptr && k0 + k < K ? p[k0 + k] : xr_from_f32<TW>(0.f);
            }
        }
    };

#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.f;
#pragma unroll
    for (int b = 0; b < GS_STAGES - 1; b++) {
        if (b < blocks) fill(b);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int b = 0; b < blocks; b++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GS_STAGES - 2) : "memory");
        __syncthreads();                                   // block b has arrived for everyone, and block b - 1 is read by everyone
        if (b + GS_STAGES - 1 < blocks) fill(b + GS_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const TX* xb = xs + (b % GS_STAGES) * BM * SX + tm * SX;
        const TW* wb = ws + (b % GS_STAGES) * BN * SW + rn * SW;
        // (the next four k's values are on their way from shared memory while these are multiplied)
        float4 x[2][TM], w[2][TN];
        auto read = [&](int kk, int at) {
#pragma unroll
            for (int i = 0; i < TM; i++) x[at][i] = gs_read4(xb + 4 * i * SX + kk);
#pragma unroll
            for (int j = 0; j < TN; j++) w[at][j] = gs_read4(wb + 8 * j * SW + kk);
        };
        read(0, 0);
#pragma unroll
        for (int kk = 0; kk < GS_BK; kk += 4) {
            constexpr bool AHEAD = TM * TN <= 32;          // (a thread with more sums has the registers for one set)
            const int at = AHEAD ? (kk / 4) & 1 : 0;
            if (AHEAD && kk + 4 < GS_BK) read(kk + 4, at ^ 1);
            if (!AHEAD && kk > 0) read(kk, 0);
            // (one sum's four terms in ascending k, TM x TN sums between them)
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(x[at][i].x, w[at][j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(x[at][i].y, w[at][j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(x[at][i].z, w[at][j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(x[at][i].w, w[at][j].w, acc[i][j]);
        }
    }
}
// where this thread's sums lie in the tile: token gs_token + 4 i, row gs_row + 8 j
template <int WN, int TM> __device__ __forceinline__ int gs_token() { return (int)(threadIdx.x >> 5) / WN * 4 * TM + (int)(threadIdx.x & 31) / 8; }
template <int WN, int TN> __device__ __forceinline__ int gs_row() { return (int)(threadIdx.x >> 5) % WN * 8 * TN + (int)(threadIdx.x & 7); }
