// Layer norm with weight and bias, fused with what a block does to the residual stream around it:
//
//   x   = h[row] + (d1[row] + d2[row] + bias)                 the sub-layers' results, if the block hands any over
//   history[n_prev][row] = x;  x = sum_{j <= n_prev} w[j] * history[j][row]       the depth-weighted average, if asked for
//   h[row] = x                                                                      unless only wanted rows are normed
//   out[r] = (x - mean) / sqrt(var + eps) * weight + bias_n   var = mean of the squared deviations; if a norm is named
//
// `history` holds the stream's earlier states of this step, [states][rows][width] float32, `slot_stride` values apart: state 0
// is what the embedding made, state j + 1 what layer j computed before its own averaging.  A launch with n_prev = 0 and w = {1}
// starts the history (it stores the stream as state 0).  Everything is float32; `out` is float32 or bfloat16.  One block per
// row, the row in registers or in shared memory, sums by a fixed tree (a row's result depends on that row only).
#include "common.cuh"

namespace {

constexpr int kThreads = 256;

// The row in shared memory: rows too wide for the kernel below, and results or norm weights that start off the borders it wants.
template <typename TO>
__global__ void __launch_bounds__(kThreads) depth_norm_kernel(float* h, const float* d1, long long ld1, const float* d2, long long ld2,
                                                              const float* bias, float* history, long long slot_stride, int n_prev,
                                                              const float* dwa, const float* norm_w, const float* norm_b, float eps,
                                                              TO* out, long long ld_out, const int* want_rows, int width, int store_h) {
    mlr_grid_wait();
    extern __shared__ __align__(16) float xs[];       // [width]
    __shared__ float scratch[32];
    const int r = blockIdx.x;
    const int row = want_rows ? want_rows[r] : r;
    float* hrow = h + static_cast<size_t>(row) * width;
    const bool vec = width % 4 == 0 && ld1 % 4 == 0 && ld2 % 4 == 0 && slot_stride % 4 == 0;
    float sum = 0.0f;
    auto value_at = [&](int c, float x) {
        // x: the stream's value; returns what the stream becomes
        float add = 0.0f;
        bool any = false;
        if (d1) { add = __ldcg(d1 + static_cast<size_t>(row) * ld1 + c); any = true; }
        if (d2) { add += __ldcg(d2 + static_cast<size_t>(row) * ld2 + c); any = true; }
        if (bias) { add += bias[c]; any = true; }
        if (any) x += add;
        if (history) {
            history[static_cast<size_t>(n_prev) * slot_stride + static_cast<size_t>(row) * width + c] = x;
            float mixed = 0.0f;
            for (int j = 0; j < n_prev; ++j)
                mixed = fmaf(dwa[j], __ldcg(history + static_cast<size_t>(j) * slot_stride + static_cast<size_t>(row) * width + c), mixed);
            x = fmaf(dwa[n_prev], x, mixed);
        }
        return x;
    };
    if (vec) {
        for (int c = threadIdx.x * 4; c < width; c += kThreads * 4) {
            float4 x = __ldcg(reinterpret_cast<const float4*>(hrow + c));
            float v[4] = {x.x, x.y, x.z, x.w};
            float add[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            bool any = false;
            if (d1) {
                const float4 a = __ldcg(reinterpret_cast<const float4*>(d1 + static_cast<size_t>(row) * ld1 + c));
                add[0] = a.x; add[1] = a.y; add[2] = a.z; add[3] = a.w;
                any = true;
            }
            if (d2) {
                const float4 a = __ldcg(reinterpret_cast<const float4*>(d2 + static_cast<size_t>(row) * ld2 + c));
                add[0] += a.x; add[1] += a.y; add[2] += a.z; add[3] += a.w;
                any = true;
            }
            if (bias) {
                const float4 a = *reinterpret_cast<const float4*>(bias + c);
                add[0] += a.x; add[1] += a.y; add[2] += a.z; add[3] += a.w;
                any = true;
            }
            if (any) {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] += add[e];
            }
            if (history) {
                float* slot = history + static_cast<size_t>(row) * width + c;
                *reinterpret_cast<float4*>(slot + static_cast<size_t>(n_prev) * slot_stride) = make_float4(v[0], v[1], v[2], v[3]);
                float mixed[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                int j = 0;
                for (; j + 4 <= n_prev; j += 4) {      // four states on their way at a time
                    float4 s[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) s[u] = __ldcg(reinterpret_cast<const float4*>(slot + static_cast<size_t>(j + u) * slot_stride));
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float w = dwa[j + u];
                        mixed[0] = fmaf(w, s[u].x, mixed[0]); mixed[1] = fmaf(w, s[u].y, mixed[1]);
                        mixed[2] = fmaf(w, s[u].z, mixed[2]); mixed[3] = fmaf(w, s[u].w, mixed[3]);
                    }
                }
                for (; j < n_prev; ++j) {
                    const float4 s = __ldcg(reinterpret_cast<const float4*>(slot + static_cast<size_t>(j) * slot_stride));
                    const float w = dwa[j];
                    mixed[0] = fmaf(w, s.x, mixed[0]); mixed[1] = fmaf(w, s.y, mixed[1]);
                    mixed[2] = fmaf(w, s.z, mixed[2]); mixed[3] = fmaf(w, s.w, mixed[3]);
                }
                const float w = dwa[n_prev];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = fmaf(w, v[e], mixed[e]);
            }
            if (store_h) *reinterpret_cast<float4*>(hrow + c) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(xs + c) = make_float4(v[0], v[1], v[2], v[3]);
            sum += (v[0] + v[1]) + (v[2] + v[3]);
        }
    } else {
        for (int c = threadIdx.x; c < width; c += kThreads) {
            const float v = value_at(c, __ldcg(hrow + c));
            if (store_h) hrow[c] = v;
            xs[c] = v;
            sum += v;
        }
    }
    mlr_grid_dependents_may_start();     // only now: waiting blocks of the next grid take room that this one's need
    if (!out) return;
    const float mean = mlr_block_sum(sum, scratch) / static_cast<float>(width);
    float squares = 0.0f;
    for (int c = threadIdx.x; c < width; c += kThreads) {       // the row is whole after the sum's barriers
        const float d = xs[c] - mean;
        squares = fmaf(d, d, squares);
    }
    const float inv = 1.0f / sqrtf(mlr_block_sum(squares, scratch) / static_cast<float>(width) + eps);
    TO* orow = out + static_cast<size_t>(r) * ld_out;
    for (int c = threadIdx.x; c < width; c += kThreads) {
        float v = (xs[c] - mean) * inv * norm_w[c];
        if (norm_b) v += norm_b[c];
        mlr_store(orow, c, v);
    }
}

// The same for rows of up to 16 values a thread that can be read four at a time (the number of threads depends on the width alone):
// a thread keeps its values in registers, and the loads of its four groups of columns, of the stream, of the results and of
// every earlier state, are on their way together.  The kernel above goes through shared memory and back to memory for every group,
// which one row of a decode step pays in full.  Measured with rows of 4096 in a step: one row 14.8 -> 4.8 us, 2048 rows 47 -> 40 us.
constexpr int kQuads = 4;

// NQ: a thread's groups of four columns.  THREADS: the most a block has (what it leaves each thread in registers).  Rows of up to 2048 columns have a
// thread for every group: empty groups cost their registers and instructions (2048 rows with four states: of
// 512 17.2 -> 6.7 us, of 1024 18.5 -> 11.0 us, of 2048 33.8 -> 27.9 us).
template <typename TO, int NQ, int THREADS>
__global__ void __launch_bounds__(THREADS) depth_norm_quads_kernel(float* h, const float* d1, long long ld1, const float* d2, long long ld2,
                                                                const float* bias, float* history, long long slot_stride, int n_prev,
                                                                const float* dwa, const float* norm_w, const float* norm_b, float eps,
                                                                TO* out, long long ld_out, const int* want_rows, int width, int store_h) {
    mlr_grid_dependents_may_start();
    mlr_grid_wait();
    __shared__ float scratch[32];
    const int r = blockIdx.x;
    const int row = want_rows ? want_rows[r] : r;
    float* hrow = h + static_cast<size_t>(row) * width;
    const int c0 = threadIdx.x * 4, step = blockDim.x * 4;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto load = [&](const float* p, float4 (&v)[NQ]) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) v[k] = c0 + k * step < width ? __ldcg(reinterpret_cast<const float4*>(p + c0 + k * step)) : zero;
    };
    auto store = [&](float* p, const float4 (&v)[NQ]) {
#pragma unroll
        for (int k = 0; k < NQ; ++k)
            if (c0 + k * step < width) *reinterpret_cast<float4*>(p + c0 + k * step) = v[k];
    };
    auto plus = [](float4 (&v)[NQ], const float4 (&a)[NQ]) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) { v[k].x += a[k].x; v[k].y += a[k].y; v[k].z += a[k].z; v[k].w += a[k].w; }
    };
    float4 x[NQ];
    load(hrow, x);
    if (d1 || d2 || bias) {
        float4 add[NQ], more[NQ];
        if (d1) load(d1 + static_cast<size_t>(row) * ld1, add);
        else {
#pragma unroll
            for (int k = 0; k < NQ; ++k) add[k] = zero;
        }
        if (d2) {
            load(d2 + static_cast<size_t>(row) * ld2, more);
            plus(add, more);
        }
        if (bias) {
            load(bias, more);
            plus(add, more);
        }
        plus(x, add);
    }
    if (history) {
        float* slot = history + static_cast<size_t>(row) * width;
        float4 mixed[NQ];
#pragma unroll
        for (int k = 0; k < NQ; ++k) mixed[k] = zero;
        auto mix = [&](float w, const float4 (&s)[NQ]) {
#pragma unroll
            for (int k = 0; k < NQ; ++k) {
                mixed[k].x = fmaf(w, s[k].x, mixed[k].x); mixed[k].y = fmaf(w, s[k].y, mixed[k].y);
                mixed[k].z = fmaf(w, s[k].z, mixed[k].z); mixed[k].w = fmaf(w, s[k].w, mixed[k].w);
            }
        };
        constexpr int kAhead = NQ == 1 ? 4 : 2;             // states on their way at a time
        int j = 0;
        for (; j + kAhead <= n_prev; j += kAhead) {
            float4 s[kAhead][NQ];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) load(slot + static_cast<size_t>(j + u) * slot_stride, s[u]);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) mix(dwa[j + u], s[u]);
        }
        for (; j < n_prev; ++j) {
            float4 s[NQ];
            load(slot + static_cast<size_t>(j) * slot_stride, s);
            mix(dwa[j], s);
        }
        store(slot + static_cast<size_t>(n_prev) * slot_stride, x);
        const float w = dwa[n_prev];
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            x[k].x = fmaf(w, x[k].x, mixed[k].x); x[k].y = fmaf(w, x[k].y, mixed[k].y);
            x[k].z = fmaf(w, x[k].z, mixed[k].z); x[k].w = fmaf(w, x[k].w, mixed[k].w);
        }
    }
    if (store_h) store(hrow, x);
    if (!out) return;
    float4 weight[NQ], shift[NQ];
    load(norm_w, weight);
    if (norm_b) load(norm_b, shift);
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < NQ; ++k) sum += (x[k].x + x[k].y) + (x[k].z + x[k].w);      // columns past the row are zeros
    const float mean = mlr_block_sum(sum, scratch) / static_cast<float>(width);
    float squares = 0.0f;
#pragma unroll
    for (int k = 0; k < NQ; ++k)
        if (c0 + k * step < width) {
            x[k].x -= mean; x[k].y -= mean; x[k].z -= mean; x[k].w -= mean;
            squares = fmaf(x[k].x, x[k].x, squares); squares = fmaf(x[k].y, x[k].y, squares);
            squares = fmaf(x[k].z, x[k].z, squares); squares = fmaf(x[k].w, x[k].w, squares);
        }
    const float inv = 1.0f / sqrtf(mlr_block_sum(squares, scratch) / static_cast<float>(width) + eps);
    TO* orow = out + static_cast<size_t>(r) * ld_out;
#pragma unroll
    for (int k = 0; k < NQ; ++k)
        if (c0 + k * step < width) {
            float4 v = make_float4(x[k].x * inv * weight[k].x, x[k].y * inv * weight[k].y, x[k].z * inv * weight[k].z, x[k].w * inv * weight[k].w);
            if (norm_b) { v.x += shift[k].x; v.y += shift[k].y; v.z += shift[k].z; v.w += shift[k].w; }
            mlr_store4(orow + c0 + k * step, v.x, v.y, v.z, v.w);
        }
}

}  // namespace

// h: float32 [*, width] (row stride width).  d1, d2: float32 results to add (row strides ld1, ld2) or null; bias: float32 [width] or null.
// history: float32 or null; with it, state n_prev is written and the stream becomes the average over states 0..n_prev with the
// weights dwa (float32 [n_prev + 1]).  norm_w, norm_b: float32 [width] (norm_b may be null); out: [rows, width] with row stride
// ld_out in float32 or bfloat16, or null for no norm.  want_rows: int32 [rows] or null (all rows 0..rows-1).
MLR_API int mlr_depth_norm(float* h, const float* d1, long long ld1, const float* d2, long long ld2, const float* bias, float* history,
                           long long slot_stride, int n_prev, const float* dwa, const float* norm_w, const float* norm_b, float eps, void* out,
                           long long ld_out, int out_bf16, const int* want_rows, int rows, int width, int store_h, cudaStream_t stream) {
    MLR_REQUIRE(h && width > 0 && n_prev >= 0, "depth_norm: bad arguments");
    MLR_REQUIRE(!history || (dwa && slot_stride >= 0), "depth_norm: a history needs its weights");
    MLR_REQUIRE(!out || norm_w, "depth_norm: a norm needs its weight");
    MLR_REQUIRE(!(want_rows && (store_h || history)), "depth_norm: a launch over wanted rows leaves the stream as it is");
    MLR_REQUIRE(reinterpret_cast<uintptr_t>(h) % 16 == 0 && reinterpret_cast<uintptr_t>(d1) % 16 == 0 && reinterpret_cast<uintptr_t>(d2) % 16 == 0 &&
                    reinterpret_cast<uintptr_t>(history) % 16 == 0 && reinterpret_cast<uintptr_t>(bias) % 16 == 0,
                "depth_norm: buffers must start on 16-byte borders");
    const size_t shared = sizeof(float) * static_cast<size_t>(width);
    MLR_REQUIRE(shared <= 200 * 1024, "depth_norm: a row of %d values does not fit shared memory", width);
    if (rows <= 0) return 0;
    const auto fits = [](const void* p, size_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; };
    const bool quads = width % 4 == 0 && (n_prev == 0 || slot_stride >= width) && width <= 1024 * 4 * kQuads && ld1 % 4 == 0 && ld2 % 4 == 0 && slot_stride % 4 == 0 && ld_out % 4 == 0 &&
                       fits(out, out_bf16 ? 8 : 16) && fits(norm_w, 16) && fits(norm_b, 16);
    int threads = 128;
    while (threads < 2 * kThreads && threads * 4 < width) threads <<= 1;
    if (width > 4 * threads) threads = kThreads;
    while (threads < 1024 && threads * 4 * kQuads < width) threads <<= 1;
#define MLR_GO(TO)                                                                                                                         \
    do {                                                                                                                                   \
        if (quads) {                                                                                                                       \
            mlr_launch((threads <= 2 * kThreads && width <= 4 * threads ? depth_norm_quads_kernel<TO, 1, 2 * kThreads>                     \
                        : threads == kThreads                           ? depth_norm_quads_kernel<TO, kQuads, kThreads>                    \
                                                                        : depth_norm_quads_kernel<TO, kQuads, 1024>),                      \
                       dim3(rows), dim3(threads), 0, stream, h, d1, ld1, d2, ld2, bias, history, slot_stride, n_prev, dwa, norm_w, norm_b, eps,        \
                       static_cast<TO*>(out), ld_out, want_rows, width, store_h);                                                          \
            break;                                                                                                                         \
        }                                                                                                                                  \
        if (shared > 48 * 1024) cudaFuncSetAttribute(depth_norm_kernel<TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared)); \
        mlr_launch((depth_norm_kernel<TO>), dim3(rows), dim3(kThreads), shared, stream, h, d1, ld1, d2, ld2, bias, history, slot_stride,   \
                   n_prev, dwa, norm_w, norm_b, eps, static_cast<TO*>(out), ld_out, want_rows, width, store_h);                            \
    } while (0)
    if (out_bf16) MLR_GO(__nv_bfloat16);
    else MLR_GO(float);
#undef MLR_GO
    return mlr_launched("depth_norm");
}
