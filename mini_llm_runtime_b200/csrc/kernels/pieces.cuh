// A contribution to the residual stream that has not been added up: what routed experts leave (`experts.cu`) for whoever adds it into
// the stream.  Row t is
//     sum_j weights[t, j] * y[row_of_pair[t, j]]      (j = 0 .. top-1 in order; a row of -1 is an identity expert: no row of y)
//   + identity[t] * x[t]                              (with identity experts: the weights of those chosen, times the sub-layer's input)
//   + gate[t] * shared[t]                             (with a shared expert; gate null: as it is)
// in float32.  y null: there is none.
#pragma once

#include "common.cuh"

struct Pieces {
    const float* y;
    long long ldy;
    const int* row_of_pair;
    const float* weights;
    int top;
    const float* shared;
    long long ld_shared;
    const float* gate;
    const void* x;
    long long ld_x;
    int x_bf16;
    const float* identity;
};
constexpr int kMaxPieces = 32;

struct StagedPieces {
    float weight[kMaxPieces];
    long long from[kMaxPieces];       // offset of the piece's row in y, or -1
};

// Leaves a row's weights and places in shared memory; the caller meets at a barrier before `piece_sum`.
__device__ __forceinline__ void stage_pieces(const Pieces& p, int row, StagedPieces& s) {
    if (threadIdx.x < p.top) {
        const int from = __ldcg(p.row_of_pair + static_cast<size_t>(row) * p.top + threadIdx.x);
        s.weight[threadIdx.x] = __ldcg(p.weights + static_cast<size_t>(row) * p.top + threadIdx.x);
        s.from[threadIdx.x] = from < 0 ? -1 : static_cast<long long>(from) * p.ldy;
    }
}

// Columns i .. i + 3 of a row (VEC), or column i alone in `.x`.
template <bool VEC>
__device__ __forceinline__ float4 piece_sum(const Pieces& p, const StagedPieces& s, int row, int i) {
    auto load = [](const float* q, int at) {
        if constexpr (VEC) return __ldcg(reinterpret_cast<const float4*>(q + at));
        else return make_float4(__ldcg(q + at), 0.0f, 0.0f, 0.0f);
    };
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto add = [&](float w, const float4& e) {
        v.x = fmaf(w, e.x, v.x);
        if constexpr (VEC) { v.y = fmaf(w, e.y, v.y); v.z = fmaf(w, e.z, v.z); v.w = fmaf(w, e.w, v.w); }
    };
#pragma unroll 4
    for (int j = 0; j < p.top; ++j)
        if (s.from[j] >= 0) add(s.weight[j], load(p.y + s.from[j], i));
    if (p.identity) {
        const float w = __ldcg(p.identity + row);
        float e[4] = {};
        const size_t at = static_cast<size_t>(row) * p.ld_x + i;
        if (p.x_bf16) {
            const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(p.x) + at;
            if constexpr (VEC) mlr_load4(x, e);
            else e[0] = mlr_load(x, 0);
        } else {
            const float* x = static_cast<const float*>(p.x) + at;
            if constexpr (VEC) mlr_load4(x, e);
            else e[0] = mlr_load(x, 0);
        }
        add(w, make_float4(e[0], e[1], e[2], e[3]));
    }
    if (p.shared) add(p.gate ? __ldcg(p.gate + row) : 1.0f, load(p.shared + static_cast<size_t>(row) * p.ld_shared, i));
    return v;
}

// The same for NQ groups of four columns of a row, i + k * step (k = 0 .. NQ - 1, those below `width`): a piece's loads are on
// their way together, the order of every sum is that of `piece_sum`.
template <int NQ>
__device__ __forceinline__ void piece_sums(const Pieces& p, const StagedPieces& s, int row, int i, int step, int width, float4 (&v)[NQ]) {
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto add = [&](float w, const float4 (&e)[NQ]) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            v[k].x = fmaf(w, e[k].x, v[k].x); v[k].y = fmaf(w, e[k].y, v[k].y);
            v[k].z = fmaf(w, e[k].z, v[k].z); v[k].w = fmaf(w, e[k].w, v[k].w);
        }
    };
#pragma unroll
    for (int k = 0; k < NQ; ++k) v[k] = zero;
    float4 shared[NQ], passed[NQ];            // asked for first, added last
    float w_shared = 0.0f, w_passed = 0.0f;
    if (p.shared) {
#pragma unroll
        for (int k = 0; k < NQ; ++k)
            shared[k] = i + k * step < width ? __ldcg(reinterpret_cast<const float4*>(p.shared + static_cast<size_t>(row) * p.ld_shared + i + k * step)) : zero;
        w_shared = p.gate ? __ldcg(p.gate + row) : 1.0f;
    }
    if (p.identity) {
        w_passed = __ldcg(p.identity + row);
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            passed[k] = zero;
            if (i + k * step >= width) continue;
            float e[4];
            const size_t at = static_cast<size_t>(row) * p.ld_x + i + k * step;
            if (p.x_bf16) mlr_load4(static_cast<const __nv_bfloat16*>(p.x) + at, e);
            else mlr_load4(static_cast<const float*>(p.x) + at, e);
            passed[k] = make_float4(e[0], e[1], e[2], e[3]);
        }
    }
#pragma unroll 4
    for (int j = 0; j < p.top; ++j) {
        const long long from = s.from[j];
        float4 e[NQ];
#pragma unroll
        for (int k = 0; k < NQ; ++k) e[k] = from >= 0 && i + k * step < width ? __ldcg(reinterpret_cast<const float4*>(p.y + from + i + k * step)) : zero;
        if (from >= 0) add(s.weight[j], e);
    }
    if (p.identity) add(w_passed, passed);
    if (p.shared) add(w_shared, shared);
}

static int check_pieces(const Pieces& p, int width, const char* who) {
    MLR_REQUIRE(p.top >= 1 && p.top <= kMaxPieces && p.row_of_pair && p.weights && p.ldy >= width && (!p.shared || p.ld_shared >= width) &&
                    (!p.identity || (p.x && p.ld_x >= width)),
                "%s: a contribution in pieces has 1 to %d pieces a row, with their places, weights and row strides", who, kMaxPieces);
    return 0;
}

// Whether four columns may be read at once.
static bool pieces_aligned(const Pieces& p) {
    const auto fits = [](const void* q, size_t bytes) { return reinterpret_cast<uintptr_t>(q) % bytes == 0; };
    return fits(p.y, 16) && p.ldy % 4 == 0 && (!p.shared || (fits(p.shared, 16) && p.ld_shared % 4 == 0)) &&
           (!p.identity || (fits(p.x, p.x_bf16 ? 8 : 16) && p.ld_x % 4 == 0));
}
