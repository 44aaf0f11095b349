// The bfloat16 product for one token or two on CUDA cores: out[t][r] = sum_k X[t][k] W[r][k], W packed tile by tile (gemm_tc.cu), float32
// sums of exact products.  Included by gemm_tc.cu, whose epilogues and parameters it shares.
//
// What bounds a product of so few tokens inside a step is not its weights' bytes but the chain from the kernel ahead's end to its own: on
// tensor cores copy, multiply, read back, store partial sums, and a kernel to add them.  Here a lane holds its weights in registers before
// the kernel ahead is known to be complete (W is constant); behind the wait there are one read of the tokens into shared memory,
// multiply-adds, three shuffles and the store, with no cut along K outside the CTA.
//
// A unit: 8 rows of the product (gated: the gate and up rows of 4 features); a warp reads it with two 512-byte loads a K block of 64 (a
// lane 16 bytes of two rows, 8 lanes a row).  WK warps share a unit's K blocks, 8 / WK units a CTA of eight warps; their sums meet in
// shared memory, added in ascending order.
// Alone, weights from memory, us, tensor cores (with the finish of a cut) / here: 1 token, 1,024 x 1,024 4.8 / 2.5, 1,024 x 4,096 5.5 / 3.2,
// 2,048 x 3,072 6.4 / 3.4, 4,096 x 6,144 11.2 / 9.4, gated 4,096 x 14,336 37.7 / 35.5 (6.6 TB/s); 2 tokens, 1,024 x 4,096 5.6 / 3.8.
// Eight K blocks ahead in two CTAs an SM: 4,096 x 6,144 9.4, gated 4,096 x 14,336 38.4; a CTA an SM: Lilalorn w1024 283 -> 317.
#pragma once

#define GV_AHEAD 4                  // K blocks of weights that a lane holds
// "splits used" of a product that ran here: its one slice of sums is left to the caller's next kernel, or it is complete
#define GV_DEFERRED (1 << 16)
#define GV_COMPLETE (1 << 17)

__device__ __forceinline__ uint4 gv_load(const __nv_bfloat16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float gv_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float gv_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// two sums at a time: a += x * y
__device__ __forceinline__ void gv_fma2(float2& a, float2 x, float2 y) {
    asm("{\n\t.reg .b64 a, x, y;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tfma.rn.f32x2 a, x, y, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+f"(a.x), "+f"(a.y) : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
}

// grid (CTAs that walk the units, token tiles of p.bn rows with a matrix each (grouped) or 1)
template <int NT, bool GATED>
__global__ void __launch_bounds__(256, 3)
k_gemv(const __nv_bfloat16* __restrict__ W, const __nv_bfloat16* X, long long ldx, int wk_log, TcParams p) {
    extern __shared__ __align__(16) unsigned char gv_sm[];
    constexpr int OUT = GATED ? 4 : 8;                                       // outputs of a unit
    const int kb = p.w_kblocks, kp = kb * TC_BK;
    // [NT][K blocks][2][8 lanes][4]: the halves of a lane's eight values apart, so that eight lanes read 128 bytes side by side
    float* xs = reinterpret_cast<float*>(gv_sm);
    __shared__ float red[2][8 * NT * 8];                                     // [turn][warp][token][row]
    xr_pdl_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, WK = 1 << wk_log, per = 8 >> wk_log, wk = warp & (WK - 1);
    const int units = (p.n_out + OUT - 1) / OUT;
    size_t tok0 = 0;
    if (p.tile_group != nullptr) {
        // which matrix a tile meets was decided by a kernel of this step
        xr_pdl_wait();
        const int group = p.tile_group[blockIdx.y];
        if (group < 0) return;
        W += (size_t)group * p.group_row_tiles * kb * (TC_BM * TC_BK);
        tok0 = (size_t)blockIdx.y * p.bn;
    }
    const int nb = (kb - wk + WK - 1) >> wk_log;                             // this warp's K blocks: wk, wk + WK, ...
    const size_t step = (size_t)WK * (TC_BM * TC_BK);
    const __nv_bfloat16* wl = W + (size_t)wk * (TC_BM * TC_BK) + lane / 8 * TC_BK + lane % 8 * 8;
    constexpr int SECOND = (GATED ? 16 : 4) * TC_BK;                         // from a lane's first row to its second
    auto unit_at = [&](int unit) {
        const int in_tile = unit % 16, first = GATED ? in_tile / 4 * 32 + in_tile % 4 * 4 : in_tile * 8;
        return wl + (size_t)(unit / 16) * kb * (TC_BM * TC_BK) + first * TC_BK;
    };
    uint4 w[GV_AHEAD][2];
    int unit = blockIdx.x * per + (warp >> wk_log);
    const __nv_bfloat16* at = unit_at(unit);
#pragma unroll
    for (int i = 0; i < GV_AHEAD; i++)
        if (i < nb && unit < units) { w[i][0] = gv_load(at + i * step); w[i][1] = gv_load(at + i * step + SECOND); }
    if (p.tile_group == nullptr) xr_pdl_wait();
    for (int e = tid * 8; e < NT * kp; e += 256 * 8) {
        const int t = e / kp, k = e % kp;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (t < p.n && k < p.K) v = *reinterpret_cast<const uint4*>(X + (tok0 + t) * ldx + k);
        float* to = xs + e / TC_BK * TC_BK + e % TC_BK / 2;
        *reinterpret_cast<float4*>(to) = make_float4(gv_lo(v.x), gv_hi(v.x), gv_lo(v.y), gv_hi(v.y));
        *reinterpret_cast<float4*>(to + 32) = make_float4(gv_lo(v.z), gv_hi(v.z), gv_lo(v.w), gv_hi(v.w));
    }
    __syncthreads();
    const float* xl = xs + wk * TC_BK + lane % 8 * 4;
    const int stride = gridDim.x * per;
    for (int turn = 0, base = blockIdx.x * per; base < units; base += stride, turn ^= 1) {
        const int next = unit + stride;
        const __nv_bfloat16* next_at = unit_at(next);
        float2 acc[NT][2];
#pragma unroll
        for (int t = 0; t < NT; t++) acc[t][0] = acc[t][1] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int c = 0; c < nb; c += GV_AHEAD) {
            // what a lane holds next: the same unit's blocks GV_AHEAD on, or the next unit's from its first on
            const bool last = c + GV_AHEAD >= nb;
            const __nv_bfloat16* from = last ? next_at : at + (c + GV_AHEAD) * step;
            const int more = last ? (next < units ? nb : 0) : nb - c - GV_AHEAD, here = nb - c;
#pragma unroll
            for (int i = 0; i < GV_AHEAD; i++) {
                const uint4 a = w[i][0], b = w[i][1];
                if (i < more) { w[i][0] = gv_load(from); w[i][1] = gv_load(from + SECOND); }
                from += step;
                if (i >= here) continue;
                const float2 aw[4] = {{gv_lo(a.x), gv_hi(a.x)}, {gv_lo(a.y), gv_hi(a.y)}, {gv_lo(a.z), gv_hi(a.z)}, {gv_lo(a.w), gv_hi(a.w)}};
                const float2 bw[4] = {{gv_lo(b.x), gv_hi(b.x)}, {gv_lo(b.y), gv_hi(b.y)}, {gv_lo(b.z), gv_hi(b.z)}, {gv_lo(b.w), gv_hi(b.w)}};
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    const float4* x = reinterpret_cast<const float4*>(xl + t * kp + ((c + i) << wk_log) * TC_BK);
                    const float4 x0 = x[0], x1 = x[8];
                    const float2 xw[4] = {{x0.x, x0.y}, {x0.z, x0.w}, {x1.x, x1.y}, {x1.z, x1.w}};
#pragma unroll
                    for (int q = 0; q < 4; q++) { gv_fma2(acc[t][0], aw[q], xw[q]); gv_fma2(acc[t][1], bw[q], xw[q]); }
                }
            }
        }
#pragma unroll
        for (int t = 0; t < NT; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float v = acc[t][h].x + acc[t][h].y;
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                if (lane % 8 == 0) red[turn][(warp * NT + t) * 8 + h * 4 + lane / 8] = v;
            }
        __syncthreads();                                                     // (two turns' sums: the next turn's barrier guards these)
        const int i = tid % OUT, t = tid / OUT % NT, u = tid / (OUT * NT), r = (base + u) * OUT + i;
        if (u < per && t < p.n && r < p.n_out) {
            float s = 0.f, up = 0.f;
            for (int k = 0; k < WK; k++) {
                const float* from = red[turn] + ((u * WK + k) * NT + t) * 8 + i;
                s += from[0];
                if (GATED) up += from[4];
            }
            const size_t o = (tok0 + t) * p.ldo + r;
            if (p.epilogue == TC_EPI_PARTIAL) p.partial[(size_t)t * p.n_out + r] = p.alpha * s;
            else if (!GATED && p.epilogue == TC_EPI_ADD) ((float*)p.out)[o] += fmaf(p.alpha, s, p.bias != nullptr ? p.bias[r] : 0.f);
            else {
                const float v = GATED ? tc_gate(p.act, p.act_limit, s, up) : tc_act(p.act, fmaf(p.alpha, s, p.bias != nullptr ? p.bias[r] : 0.f));
                if (p.out_dtype == XR_BF16) ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(v);
                else ((float*)p.out)[o] = v;
            }
        }
        unit = next;
        at = next_at;
    }
}

// Whether a product of n tokens goes here, by K and the bytes of all matrices that it may read.  Where the lines lie is what whole decode
// steps took (us; runs of one rule differ by 0.2 %); the product alone says less, because behind it others wait with their weights fetched, and a
// product here keeps registers where one on tensor cores keeps shared memory.
//   one token, tensor cores alone / this rule: Lilalorn w1024 428 / 271, w2048 552 / 387, Turudra w2048 734 / 587, Besolix w2048 376 / 350, Llama-3.2-1B 739 /
//   731, Llama-3-8B 3,015 / 2,974.  K: up to 3,072 alone 8B 3,024; 5,632 too Besolix w2048 341, Pitolix w2048 281 (280), 8,192 too Llama-3.2-1B 793, Semesun w2048
//   333 (343): up to 4,096 no model is slower than without.  Bytes: up to 32 MB alone Turudra w2048 691, Pitolix w2048 301 (280); 100 MB, which
//   takes in gate and up of Llama-3.2-1B (67 MB) and heads of 66, 738 there, Lilalorn w2048 394, Semesun w1024 213 (217).  Experts' up to 64 MB alone
//   Turudra w2048 (69 MB) 657; nothing measured lies above.
//   two tokens: Lilalorn w1024 434 / 319, Turudra w1024 508 / 404, Semesun w1024 309 / 271; models 2,048 wide, of which few products are so short, stay within
//   1 % (Lilalorn 566 / 571, Turudra 775 / 774).  K up to 1,024 alone Lilalorn w1024 369; 2,048 too Llama-3.2-1B 759 -> 786, Turudra w2048 788, Lilalorn w2048
//   540.  Up to 8 MB alone Lilalorn w1024 374, up to 16 Buzarax w1024 336 (328), up to 40 the same as 24.  Three tokens and more need as many multiply-adds
//   again for bytes that are the same: four tokens 243 / 260 at Pitolix w1024.
static inline bool gemv_takes(int n, int K, long long bytes, bool grouped) {
    if (n == 1) return K <= 4096 && bytes <= (grouped ? 128000000 : 64000000);
    return n == 2 && K <= 1536 && bytes <= 24000000;
}

// `tiles` token tiles of p.bn rows each (grouped), or 1; p.n: tokens (of a tile)
static int launch_gemv(const void* X, const void* W, long long ldx, const TcParams& p, int tiles, cudaStream_t stream) {
    const int kb = p.w_kblocks, units = p.gated ? (p.n_out + 3) / 4 : (p.n_out + 7) / 8;
    if (tiles > 65535) return XR_ERR_ARG;
    int wk = 0;
    while (wk < 3 && (kb + (1 << wk) - 1) >> wk > GV_AHEAD) wk++;
    // (few units: more warps on each, down to two K blocks a warp)
    while (wk < 3 && (long long)(units + (8 >> wk) - 1) / (8 >> wk) * tiles < xr_sm_count() && kb >> wk > 2) wk++;
    // as many CTAs as are resident at once walk the units, so that a lane's loads run on from one unit into the next
    const int blocks = (units + (8 >> wk) - 1) / (8 >> wk), most = (3 * xr_sm_count() + tiles - 1) / tiles;
    const dim3 grid(blocks < most ? blocks : most, tiles);
    const size_t smem = (size_t)p.n * kb * TC_BK * sizeof(float);           // (32 KB at most)
#define GV(NT, G) xr_launch((k_gemv<NT, G>), grid, dim3(256), smem, stream, (const __nv_bfloat16*)W, (const __nv_bfloat16*)X, ldx, wk, p)
    if (p.gated) {
        if (p.n == 1) GV(1, true); else GV(2, true);
    } else {
        if (p.n == 1) GV(1, false); else GV(2, false);
    }
#undef GV
    return xr_launch_status();
}
