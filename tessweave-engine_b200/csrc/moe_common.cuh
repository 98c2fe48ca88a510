// What the kernels of routed experts share (moe.cu, moe_smallm.cu).
#pragma once

#include "common.cuh"

// what an expert makes of its gate and up products: 0 silu(g) u;  1 with g = min(g, limit), u = clamp(u, -limit, limit):
// g sigmoid(alpha g) (u + 1)
__device__ __forceinline__ float tw_glu(float g, float u, int act, float limit, float alpha) {
    if (act == 1) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
    }
    return g / (1.0f + expf(-g)) * u;
}
