#pragma once

#include "common.cuh"

namespace {

// What the two products of a gated expert become.  kind 1: silu(g) * u.  kind 2: g <- min(g, limit), u <- clamp(u, -limit, limit) where limit > 0,
// then g * sigmoid(alpha g) * (u + up_offset).
struct ExpertGate {
    int kind;
    float alpha, limit, up_offset;
};
__device__ __forceinline__ float expert_gate(float g, float u, const ExpertGate& shape) {
    if (shape.kind == 2) {
        if (shape.limit > 0.0f) {
            g = fminf(g, shape.limit);
            u = fminf(fmaxf(u, -shape.limit), shape.limit);
        }
        return g / (1.0f + expf(-shape.alpha * g)) * (u + shape.up_offset);
    }
    return g / (1.0f + expf(-g)) * u;
}


}  // namespace
