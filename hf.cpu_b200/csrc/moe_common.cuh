// What the grouped products of a mixture of experts share: the activations of their epilogues.
#pragma once
#include "common.cuh"

namespace hfb {

__device__ __forceinline__ float moe_act(float v, int act)
{
    if (act == HFB_ACT_RELU2) { v = fmaxf(v, 0.f); v *= v; }
    else if (act == HFB_ACT_RELU) v = fmaxf(v, 0.f);
    else if (act == HFB_ACT_SILU) v = v / (1.0f + expf(-v));
    else if (act == HFB_ACT_GELU_TANH) v = 0.5f * v * (1.0f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
    return v;
}

// The two halves of a gated pair: act(g) * u, or, for HFB_ACT_CLAMPED_GLU, min(g, limit) sigmoid(alpha min(g, limit)) *
// (clamp(u, -limit, limit) + offset).
struct GluClamp { float limit, alpha, offset; };

__device__ __forceinline__ float moe_glu(float g, float u, int act, const GluClamp &c)
{
    if (act == HFB_ACT_CLAMPED_GLU) {
        g = fminf(g, c.limit);
        u = fminf(fmaxf(u, -c.limit), c.limit);
        return g / (1.0f + expf(-c.alpha * g)) * (u + c.offset);
    }
    return moe_act(g, act) * u;
}

}  // namespace hfb
