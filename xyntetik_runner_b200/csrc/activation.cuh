// A feed-forward's activation in full precision (expf and tanhf): what the true 32-bit path computes.
// act 1: SiLU, g / (1 + exp(-g)), 0 for g < -80 (src/model.c:4451-4452; the reference's kernel is src/kernels.cu:2868-2874); act 2:
// tanh-GELU, 0.5 g (1 + tanh(0.7978845608 (g + 0.044715 g^3))) (src/model.c:4438-4441); act 4: the square of relu; act 0: none.
#pragma once

__device__ __forceinline__ float xr_activation(int act, float g) {
    if (act == 1) return g < -80.0f ? 0.0f : g / (1.0f + expf(-g));
    if (act == 2) return 0.5f * g * (1.0f + tanhf(0.7978845608f * (g + 0.044715f * g * g * g)));
    if (act == 4) { const float r = fmaxf(g, 0.f); return r * r; }
    return g;
}

// act 3 (gated only): with g' = min(g, limit) and u' = u clamped to [-limit, limit], h = g' sigmoid(1.702 g') (u' + 1).
__device__ __forceinline__ float xr_gate(int act, float limit, float g, float u) {
    if (act == 3) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
    }
    return xr_activation(act, g) * u;
}
