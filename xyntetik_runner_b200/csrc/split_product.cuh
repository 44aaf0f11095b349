// Products of float32 rows X with a bfloat16 matrix W, in float32's precision, on the 5th-generation tensor cores (tcgen05).
//
// A float32 value is the exact sum of three bfloat16 values: its first eight significant bits, the next eight of what is left, and
// the last eight.  (Cut off, not rounded: every difference is exact, and no piece overflows.)  W is bfloat16 as stored, so all products
// are exact and what rounds is the sums.  The tensor core's own accumulation cuts bits off at every step, so no long sum is left to it:
// a block of 64 values of k gets an accumulator of its own, four instructions long, which is then added in registers, rounded to
// nearest; the two lower pieces' sums, 2^-8 and 2^-16 of the size, accumulate over all of k.  Root mean square error against float64, normal
// values, in units of 2^-24 of the result's size, beside the FMA kernel's (gemm_simt.cu, one thread's sum over ascending k): K 256 1.4 / 4.8,
// 1,024 1.5 / 9.6, 2,816 1.7 / 16, 8,192 2.0 / 27.
//
// A CTA: 128 rows of W (the M of the instruction) x BN tokens x one slice of K.  Roles:
//   warp 0  : TMA of W, 64-row boxes                          warp 1 : the MMAs and tensor memory
//   workers : read X from L2 two blocks ahead, cut a block up and write its pieces to shared memory in the layout that the 128-byte
//             swizzle means, then add the accumulator of the block before in registers
// What bounds it: shared memory (a block of k and 64 tokens: W 16 KB written once and read twice, the pieces 24 KB written and read once),
// so the two lower pieces lie one behind the other and are ONE instruction's N; the workers' instructions; and waits, some 200 cycles
// each even where they are over, so that the issuing thread has one a block: the workers' arrival says that the stage was free, that W is
// there and that the accumulator before last is read.  us, FMA kernel / here: 1 x 1,024 x 2,816 35 / 8, 16 x 5,632 x 1,024 29 / 10, 256 x
// 1,024 x 1,024 29 / 11, 256 x 5,632 x 1,024 90 / 26, 256 x 32,000 x 1,024 433 / 93, 2,048 x 5,632 x 1,024 577 / 126 (187 TFLOP/s; three
// waits a block for the issuing thread 152; an unrolled end of 7,000 cycles, not in the instruction cache, 145).
//
// Slices of K are CTAs of a cluster: at the end they exchange their sums through distributed shared memory, added slice by slice in
// ascending order, each CTA finishing its share of the tokens.  How many slices there are depends on W's shape only, and the sums do not
// depend on BN: a token's row is the same bits whatever stands beside it in the call.
#pragma once
#include "tc_product.cuh"

struct SplitParams {
    const float* x; long long ldx;    // X [n][...], rows ldx values apart
    int n, K;
    int rows;            // rows of W that a block of X's columns meets (TWO: features, each with two rows)
    int second;          // TWO: rows of W between a feature's two
    int tiles;           // row tiles of such a block; block b reads X's columns from b K on
    int* status;         // device word: non-zero when a wait gave up
};

template <int BN> struct SplitShape {
    static constexpr int WORK = BN >= 32 ? 8 : 4;                  // warps that cut and add
    static constexpr int COLS = BN * 4 / WORK;                     // accumulator columns a thread
    static constexpr int XI = BN * 16 / (32 * WORK);               // times four values of a block of X a thread
    static constexpr int THREADS = 32 * (2 + WORK);
    static constexpr int STAGES = BN >= 64 ? 2 : (BN >= 32 ? 3 : 4);
    static constexpr int W_BYTES = TC_BM * TC_BK * 2, P_BYTES = BN * TC_BK * 2, STAGE = W_BYTES + 3 * P_BYTES;
    static constexpr int SMEM = STAGES * STAGE + 1024 + (3 * STAGES + 2) * 8 + 16;
    static_assert(BN * TC_BM * 4 <= STAGES * STAGE, "the sums fit where the stages were");
    static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs an SM");
};
// x = h + m + l, each a bfloat16 in its upper 16 bits.  What is no finite number stays whole in h.
__device__ __forceinline__ void sp_cut(float x, uint32_t& h, uint32_t& m, uint32_t& l) {
    const uint32_t b = __float_as_uint(x);
    const bool finite = (b & 0x7f800000u) != 0x7f800000u;
    h = finite ? b & 0xffff0000u : ((b & 0x007fffffu) ? 0x7fc00000u : b);
    const float r = finite ? x - __uint_as_float(h) : 0.f;
    m = __float_as_uint(r) & 0xffff0000u;
    l = __float_as_uint(r - __uint_as_float(m));
}
// two values at a time without the question; `odd` becomes no number if one of them is not finite
__device__ __forceinline__ float2 sp_sub2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 sp_add2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float sp_upper(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ uint32_t sp_pair(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }      // upper halves, a below b

// COLS consecutive accumulator columns of this thread's lane
template <int COLS> __device__ __forceinline__ void sp_ld(uint32_t taddr, float (&v)[COLS]) {
    static_assert(COLS % 16 == 0, "sixteen at a time");
#pragma unroll
    for (int c = 0; c < COLS; c += 16)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=f"(v[c]), "=f"(v[c + 1]), "=f"(v[c + 2]), "=f"(v[c + 3]), "=f"(v[c + 4]), "=f"(v[c + 5]), "=f"(v[c + 6]), "=f"(v[c + 7]),
              "=f"(v[c + 8]), "=f"(v[c + 9]), "=f"(v[c + 10]), "=f"(v[c + 11]), "=f"(v[c + 12]), "=f"(v[c + 13]), "=f"(v[c + 14]), "=f"(v[c + 15])
            : "r"(taddr + c) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int c = 0; c < COLS; c++) asm volatile("" : "+f"(v[c]));            // (no use of a value moves ahead of the wait)
}
__device__ __forceinline__ void sp_cut2(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l, float2& odd) {
    const float2 v = make_float2(x, y), hf = make_float2(sp_upper(x), sp_upper(y)), r = sp_sub2(v, hf), mf = make_float2(sp_upper(r.x), sp_upper(r.y)), lf = sp_sub2(r, mf);
    odd = sp_add2(odd, r);
    h = sp_pair(__float_as_uint(x), __float_as_uint(y));
    m = sp_pair(__float_as_uint(r.x), __float_as_uint(r.y));
    l = sp_pair(__float_as_uint(lf.x), __float_as_uint(lf.y));
}
__device__ __forceinline__ void sp_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ float sp_ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// Epi: `Row row(r)` what a row needs of constants (asked for once a thread if TWO), `Pre pre(t, r)` what an output needs beside its sums
// (loads only), `put(t, r, sum, second sum, row, pre)` the output.  r: the row of W (TWO: the feature), counted over all blocks.
// grid (slices, token tiles, row tiles of all blocks), cluster (slices, 1, 1).
template <int BN, bool TWO, class Epi>
__global__ void __launch_bounds__(SplitShape<BN>::THREADS, 2)
k_split_product(const __grid_constant__ CUtensorMap map_w, SplitParams p, Epi epi) {
    using Sh = SplitShape<BN>;
    constexpr int STAGES = Sh::STAGES, COLS = Sh::COLS, WORK = Sh::WORK, XI = Sh::XI, TMEM_COLS = 4 * BN, BOX = TC_BM / 2;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_w = (uint64_t*)(smem + STAGES * Sh::STAGE);
    uint64_t* full_x = full_w + STAGES;           // the workers are through with the block, see above
    uint64_t* empty = full_x + STAGES;
    uint64_t* acc_full = empty + STAGES;          // [2]
    uint32_t* tmem_slot = (uint32_t*)(acc_full + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    xr_pdl_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slices = gridDim.x, slice = blockIdx.x, tok0 = blockIdx.y * BN;
    const int block = blockIdx.z / p.tiles, row0 = (int)(blockIdx.z % p.tiles) * (TWO ? BOX : TC_BM), w_row0 = block * p.rows + row0;
    const int total_kb = (p.K + TC_BK - 1) / TC_BK;
    const int kb0 = slice * total_kb / slices, nkb = (slice + 1) * total_kb / slices - kb0;        // at least one: slices <= total_kb

    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(&full_w[s], 1); mbar_init(&full_x[s], WORK); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; b++) mbar_init(&acc_full[b], 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA of W: constants, so the ring fills before the kernel ahead is known to be complete ----------------
        if (tc_elect()) {
            int issued = 0;
            uint32_t s = 0, phase = 1;
            for (int i = 0; i < nkb; i++) {
                if (i >= STAGES && !mbar_wait(&empty[s], phase, abort_flag)) break;
                uint8_t* st = smem + s * Sh::STAGE;
                mbar_expect_tx(&full_w[s], Sh::W_BYTES);
                tma_load_2d(st, &map_w, (kb0 + i) * TC_BK, w_row0, &full_w[s]);
                tma_load_2d(st + Sh::W_BYTES / 2, &map_w, (kb0 + i) * TC_BK, w_row0 + (TWO ? p.second : BOX), &full_w[s]);
                issued = i + 1;
                if (++s == STAGES) { s = 0; phase ^= 1; }
            }
            if (*abort_flag)      // copies already issued still write shared memory: wait for them (bounded)
                for (int i = max(0, issued - STAGES); i < issued; i++)
                    for (uint32_t w = 0; w < XR_SPIN_LIMIT && !mbar_try_wait(&full_w[i % STAGES], (i / STAGES) & 1); w++) {}
        }
    } else if (warp == 1) {
        // ---------------- MMAs ----------------
        if (tc_elect()) {
            const uint64_t first = smem_desc_sw128(smem_u32(smem));
            bool ok = true;
            uint32_t s = 0, phase = 0;
            for (int i = 0; i < nkb && ok; i++) {
                ok = mbar_wait(&full_x[s], phase, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint64_t w_desc = first + s * (Sh::STAGE >> 4), h_desc = w_desc + (Sh::W_BYTES >> 4), ml_desc = h_desc + (Sh::P_BYTES >> 4);
#pragma unroll
                for (int k = 0; k < TC_BK / 16; k++) tc_mma(tmem_base + 2 * BN, w_desc + 2 * k, ml_desc + 2 * k, instr_desc(2 * BN), (i > 0 || k > 0) ? 1u : 0u);
#pragma unroll
                for (int k = 0; k < TC_BK / 16; k++) tc_mma(tmem_base + (i & 1) * BN, w_desc + 2 * k, h_desc + 2 * k, instr_desc(BN), k > 0 ? 1u : 0u);
                tc_commit(&empty[s]);
                tc_commit(&acc_full[i & 1]);
                if (++s == STAGES) { s = 0; phase ^= 1; }
            }
        }
    } else {
        // ---------------- X cut up, sums ----------------
        const int ct = tid - 64, k4 = ct & 15, r0 = ct >> 4;
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp - 2) >> 2) * COLS;
        float acc[COLS];
#pragma unroll
        for (int c = 0; c < COLS; c++) acc[c] = 0.f;
        auto add = [&](int i) {            // block i's accumulator
            // (a lane may see the barrier's end ahead of others, and tcgen05.ld is for a warp that has come together)
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[i & 1], (i >> 1) & 1, abort_flag))) return false;
            tc_fence_after();
            float v[COLS];
            sp_ld<COLS>(taddr + (i & 1) * BN, v);
#pragma unroll
            for (int c = 0; c < COLS; c++) acc[c] += v[c];
            tc_fence_before();             // (ahead of the next arrival, which says that it is read)
            return true;
        };
        // (a token that is not there is read as the last one: its sums are nobody's)
        const float* xb = p.x + (size_t)block * p.K + 4 * k4;
        uint32_t row_at[XI];                  // (in 16 bytes)
#pragma unroll
        for (int j = 0; j < XI; j++) row_at[j] = (uint32_t)((size_t)min(tok0 + r0 + 2 * WORK * j, p.n - 1) * (size_t)p.ldx >> 2);
        float4 even[XI], odd[XI];
        auto load = [&](int i, float4 (&v)[XI]) {
            if (i >= nkb) return;
            const int k = (kb0 + i) * TC_BK;
            const float4* from = reinterpret_cast<const float4*>(xb + k);
            if (k + TC_BK <= p.K || k + 4 * k4 < p.K) {
#pragma unroll
                for (int j = 0; j < XI; j++) v[j] = xr_ld_now4(from + row_at[j]);
            } else {
#pragma unroll
                for (int j = 0; j < XI; j++) v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        uint32_t s = 0, phase = 0;
        const uint32_t at = (uint32_t)(r0 * 128 + (((k4 >> 1) ^ (r0 & 7)) << 4) + (k4 & 1) * 8);       // (rows 8 apart: the same place in the swizzle)
        auto turn = [&](int i, float4 (&v)[XI]) {
            // (W's copy was made when the stage was free; a wait that gave up has set the flag, and all waits behind it are short)
            mbar_wait(&full_w[s], phase, abort_flag);
            uint8_t* dst = smem + s * Sh::STAGE + Sh::W_BYTES + at;
            float2 none = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < XI; j++) {
                uint2 h, m, l;
                sp_cut2(v[j].x, v[j].y, h.x, m.x, l.x, none);
                sp_cut2(v[j].z, v[j].w, h.y, m.y, l.y, none);
                uint8_t* d = dst + j * (2 * WORK * 128);
                *reinterpret_cast<uint2*>(d) = h;
                *reinterpret_cast<uint2*>(d + Sh::P_BYTES) = m;
                *reinterpret_cast<uint2*>(d + 2 * Sh::P_BYTES) = l;
            }
            none.x += none.y;
            if (none.x != none.x)          // something here is no finite number: once more, value by value
#pragma unroll 1
                for (int j = 0; j < XI; j++) {
                    const float4 x = j == 0 ? v[0] : (j == 1 ? v[1 % XI] : (j == 2 ? v[2 % XI] : v[3 % XI]));
                    uint32_t h[4], m[4], l[4];
                    sp_cut(x.x, h[0], m[0], l[0]); sp_cut(x.y, h[1], m[1], l[1]);
                    sp_cut(x.z, h[2], m[2], l[2]); sp_cut(x.w, h[3], m[3], l[3]);
                    uint8_t* d = dst + j * (2 * WORK * 128);
                    *reinterpret_cast<uint2*>(d) = make_uint2(sp_pair(h[0], h[1]), sp_pair(h[2], h[3]));
                    *reinterpret_cast<uint2*>(d + Sh::P_BYTES) = make_uint2(sp_pair(m[0], m[1]), sp_pair(m[2], m[3]));
                    *reinterpret_cast<uint2*>(d + 2 * Sh::P_BYTES) = make_uint2(sp_pair(l[0], l[1]), sp_pair(l[2], l[3]));
                }
            load(i + 2, v);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) sp_arrive(&full_x[s]);
            if (++s == STAGES) { s = 0; phase ^= 1; }
            return i == 0 || add(i - 1);
        };
        static_assert(XI <= 4, "the slow way's choice");
        xr_pdl_wait();
        load(0, even);
        load(1, odd);
        bool ok = true;
        for (int i = 0; i < nkb && ok; i += 2) {
            ok = turn(i, even);
            if (ok && i + 1 < nkb) ok = turn(i + 1, odd);
        }
        if (ok && add(nkb - 1)) {
            // (every MMA is complete, so the stages are free: the sums go there, [token][row])
            float* red = (float*)smem + ((warp - 2) >> 2) * COLS * TC_BM + (warp & 3) * 32 + lane;
#pragma unroll
            for (int c = 0; c < COLS; c += 16) {
                float mid[16], low[16];
                tc_ld16(taddr + 2 * BN + c, mid);
                tc_ld16(taddr + 3 * BN + c, low);
#pragma unroll
                for (int q = 0; q < 16; q++) red[(c + q) * TC_BM] = acc[c + q] + (mid[q] + low[q]);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    if (slices > 1) tc_cluster_sync(); else __syncthreads();
    // (the other warps' writes below are to what this step produces: the kernel ahead may still read it)
    xr_pdl_wait();
    {
        // (short code: it runs once a CTA, and what is not in the instruction cache costs more than the loop's turns)
        constexpr int per = TWO ? BOX : TC_BM, U = 4;
        const int share = BN / slices, c0 = slice * share, live = min(share, p.n - tok0 - c0);       // tokens that this CTA finishes
        const uint32_t mine = smem_u32(smem);
        static_assert(!TWO || Sh::THREADS % BOX == 0, "TWO: a thread's outputs are one feature's");
        typename Epi::Row row{};
        if (TWO && row0 + tid % BOX < p.rows) row = epi.row(w_row0 + tid % BOX);
        for (int e0 = tid; e0 < per * live; e0 += U * Sh::THREADS) {
            float a[U], b[U];
            typename Epi::Pre pre[U];
            int r[U], c[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                // (an output that is not there is read as the first one)
                const int e = e0 + u * Sh::THREADS, at = e < per * live && row0 + e % per < p.rows ? e : 0;
                r[u] = at % per; c[u] = c0 + at / per;
                pre[u] = epi.pre(tok0 + c[u], w_row0 + r[u]);
                a[u] = b[u] = 0.f;
            }
            if (slices == 1) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const float* from = (const float*)smem + c[u] * TC_BM + r[u];
                    a[u] = from[0];
                    if (TWO) b[u] = from[BOX];
                }
            } else {
#pragma unroll 1
                for (int s = 0; s < slices; s++) {
                    const uint32_t from = tc_map_to_rank(mine, s);
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        a[u] += sp_ld_cluster(from + (uint32_t)(c[u] * TC_BM + r[u]) * 4);
                        if (TWO) b[u] += sp_ld_cluster(from + (uint32_t)(c[u] * TC_BM + r[u] + BOX) * 4);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int e = e0 + u * Sh::THREADS;
                if (e < per * live && row0 + e % per < p.rows) epi.put(tok0 + c[u], w_row0 + r[u], a[u], b[u], TWO ? row : epi.row(w_row0 + r[u]), pre[u]);
            }
        }
    }
    __syncwarp();                                 // (outputs that are not there, and the functions' branches, part a warp's lanes)
    if (slices > 1) tc_cluster_sync();            // (no CTA leaves while another reads its sums)
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    if (tid == 0 && *abort_flag) atomicExch(p.status, 1);
}

// ---- host ---------------------------------------------------------------------------------------------------------------
// Slices of K: CTAs enough for a step of a few hundred tokens, four blocks of K each at least.  By W's shape alone: see above.
static inline int split_slices(long long row_tiles, int K) {
    const int blocks = (K + TC_BK - 1) / TC_BK;
    int s = 1;
    while (s < 8 && row_tiles * s * 4 < 148 && blocks / (2 * s) >= 4) s *= 2;
    return s;
}

template <int BN, bool TWO, class Epi>
static int launch_split(const CUtensorMap& mw, const SplitParams& p, const Epi& epi, int slices, long long row_tiles, cudaStream_t stream) {
    using Sh = SplitShape<BN>;
    const long long tok_tiles = ((long long)p.n + BN - 1) / BN;
    if (tok_tiles > 65535 || row_tiles > 65535) return XR_ERR_ARG;
    static bool ready[XR_DEVICES];
    if (!xr_once_per_device(ready, [] { return xr_allow_smem(k_split_product<BN, TWO, Epi>, Sh::SMEM); })) return XR_ERR_LAUNCH;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(slices, (unsigned)tok_tiles, (unsigned)row_tiles); cfg.blockDim = dim3(Sh::THREADS); cfg.dynamicSmemBytes = Sh::SMEM; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = slices; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = xr_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, k_split_product<BN, TWO, Epi>, mw, p, epi);
    return xr_launch_status();
}
// What the copies and the 16-byte loads need; `W` [w_rows][K] bfloat16.
static inline bool split_takes(const float* x, int n, long long ldx, const void* W, int K) {
    return K % 8 == 0 && ldx % 4 == 0 && (long long)n * ldx < (1LL << 34) && !(((uintptr_t)x | (uintptr_t)W) & 15);
}
// What the grid holds: `rows` rows of W (TWO: features) a block.
template <bool TWO> static inline bool split_fits(int n, int rows, int blocks) {
    constexpr int per = TWO ? TC_BM / 2 : TC_BM;
    return (long long)((rows + per - 1) / per) * blocks <= 65535 && n <= 65535 * 64;
}
// `blocks` blocks of X's columns.  64 tokens a tile, or 32 while these still fit the SMs at once; 16 for a few.
template <bool TWO, class Epi>
static int run_split(const void* W, long long w_rows, SplitParams p, const Epi& epi, int blocks, cudaStream_t stream) {
    CUtensorMap mw;
    if (!make_map(&mw, W, w_rows, p.K, p.K, TC_BM / 2)) return -3;
    p.tiles = (p.rows + (TWO ? TC_BM / 2 : TC_BM) - 1) / (TWO ? TC_BM / 2 : TC_BM);
    const long long row_tiles = (long long)p.tiles * blocks;
    const int slices = split_slices(row_tiles, p.K);
    if (p.n <= 16) return launch_split<16, TWO>(mw, p, epi, slices, row_tiles, stream);
    if (p.n <= 32 || row_tiles * slices * ((p.n + 31) / 32) <= xr_sm_count()) return launch_split<32, TWO>(mw, p, epi, slices, row_tiles, stream);
    return launch_split<64, TWO>(mw, p, epi, slices, row_tiles, stream);
}
