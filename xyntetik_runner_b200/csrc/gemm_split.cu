// out[t][r] = sum_k X[t][k] W[r][k], X float32 and W bfloat16, in float32's precision on the tensor cores: see split_product.cuh.
#include "split_product.cuh"
#include "activation.cuh"

// (not inlined: see the end of k_split_product)
__device__ __noinline__ float split_act(int act, float v) { return xr_activation(act, v); }
__device__ __noinline__ float split_gate(int act, float limit, float g, float u) { return xr_gate(act, limit, g, u); }

struct SplitStore {
    float* out; long long ldo;
    const float* bias;           // [rows] or null
    int add, act;
    float alpha;
    struct Row {};
    using Pre = float2;          // bias, the output as it stands
    __device__ __forceinline__ Row row(int) const { return {}; }
    __device__ __forceinline__ Pre pre(int t, int r) const {
        return make_float2(bias ? bias[r] : 0.f, add ? xr_ld_now(out + (size_t)t * ldo + r) : 0.f);
    }
    __device__ __forceinline__ void put(int t, int r, float a, float, Row, Pre q) const {
        float v = alpha * a;
        if (bias) v += q.x;
        if (act) v = split_act(act, v);
        out[(size_t)t * ldo + r] = add ? q.y + v : v;
    }
};
struct SplitGate {
    float* out; long long ldo;
    int act;
    float limit;
    struct Row {};
    struct Pre {};
    __device__ __forceinline__ Row row(int) const { return {}; }
    __device__ __forceinline__ Pre pre(int, int) const { return {}; }
    __device__ __forceinline__ void put(int t, int f, float g, float u, Row, Pre) const { out[(size_t)t * ldo + f] = split_gate(act, limit, g, u); }
};

// X: [n][K] float32, rows ldx apart; W: [n_out][K] bfloat16, dense, finite (a piece of X that is zero times an infinite weight is no
// number); out float32, rows ldo apart.  accumulate: out += alpha sum + bias, else out = act(alpha sum + bias).
// gated: W [2 n_out][K], out = act(sum of row f) * (sum of row n_out + f); no bias, alpha or accumulation.
XR_EXPORT int xr_gemm_split(const void* X, const void* W, const float* bias, void* out, int accumulate, int gated, int act, float limit, float alpha,
                            int n, int n_out, int K, long long ldx, long long ldo, int* status, cudaStream_t stream) {
    if (n < 1 || n_out < 1 || K < 1 || ldx < K || ldo < n_out || act < 0 || act > 4 || (act == 3 && !gated) || (accumulate && (act || gated)) ||
        (gated && (bias || alpha != 1.f)) || n_out > (1 << 30) || !split_takes((const float*)X, n, ldx, W, K))
        return XR_ERR_ARG;
    SplitParams p{(const float*)X, ldx, n, K, n_out, n_out, 0, status};
    if (gated) return run_split<true>(W, 2LL * n_out, p, SplitGate{(float*)out, ldo, act, limit}, 1, stream);
    return run_split<false>(W, n_out, p, SplitStore{(float*)out, ldo, bias, accumulate, act, alpha}, 1, stream);
}
