// Walks of a matrix state (see recurrence.cu) sixteen tokens at a time, for portions of many rows in bfloat16.
//
// With D_t the diagonal of token t's decays, P_t = D_1 .. D_t within a chunk of sixteen tokens and S the state before it, all three rules are
//     u_t = v_t (decay, step)    or    U = M (V - K~ S),  M = (I + diag(beta) A)^-1 diag(beta),  K~_t = P_t k_t   (delta)
//     o_t = S^T (P_t q_t) + sum_{s <= t} B_ts u_s,   S <- P_16 S + sum_s (P_16 / P_s) k_s u_s^T
//     A_ts = k_t . (P_t / P_s) k_s (s < t),   B_ts = q_t . (P_t / P_s) k_s
// (the step rule's dt_s are part of B and of what is added to S).  A, B, M and the scaled vectors need no state:
// `chunk_prepare_kernel` makes them for all chunks side by side.  What is left for the walk are three products of 16 rows a chunk with the state
// of a block's columns.  Quotients of decays are made as products of the decays between the two tokens: nothing is divided by a decay, however
// small.
//
// The walk's products are on the tensor cores, each float32 operand split into three bfloat16 parts (24 bits; the six largest of the nine
// products), sums in float32; the state itself is decayed and added to in float32 on the CUDA cores.  A value that is not finite breaks such
// products (an infinity minus its first part, zeros of B times a later token's value): a block that finds one in its outputs or its end of the
// state throws them away and walks its columns again token by token, so such values reach what the rules say and nothing else.
//
// Measured, both kernels against the walk token by token (B200, states of 128 x 128, one request of 2048 tokens): delta rule, 16 heads 59 + 118
// instead of 358 us; with decays per channel 90 + 111 instead of 404 us; gated linear attention, 16 heads 50 + 87 instead of 312 us; retention,
// 8 heads 15 + 95 instead of 242 us (in pieces 173 us); the step rule, 1999 tokens of 128 heads of 128 x 64 in 8 groups, 40 + 241 instead of 475 us.  What a
// chunk takes, 0.7 to 0.9 us (1.9 us for the step rule's 256 blocks, two an SM), is the chain from one state to the next: splitting it, a product, the
// meeting of the warps, a product.  Distance of the outputs from 64 bits over 2048 tokens: 1.4e-7 with the delta rule (token by token 1.3e-7), 1.0e-7 (2.0e-7)
// retention, 1.7e-7 (1.7e-7) gated linear attention, 2.8e-8 (2.8e-8) step; held beside the walk token by token by tests/test_recurrence_chunks.py.
//
// Sixteen tokens a chunk are the rows of one instruction.  Two column tiles a block where the tiles outnumber the SMs: what a block reads of W, Q
// and K serves both.
#pragma once

constexpr int kChunk = 16;                 // tokens
constexpr int kChunkPrepareThreads = 256;
constexpr int kChunkEnds = 36;             // values of `ends` a chunk and head without decays per channel

// Buffers between the two kernels.  The operands W, Q and K of the walk's products are laid out as its lanes take them (`chunk_operand`):
// [chunk place][head][slice of 16 values][part][lane][4] words of two bfloat16.
struct ChunkBuffers {
    const float* qf;                       // [rows][qk_heads * dim] prepared q and k
    const float* kf;
    const float* df;                       // [rows][heads * dim] decays per channel
    const float* gates;                    // [rows][2 * heads]
    uint32_t* w;                           // M K~ (delta)
    uint32_t* q;                           // q (of the qk_heads); with decays per channel P_t q_t (of the heads)
    uint32_t* k;                           // k; with decays per channel (P_16 / P_s) k_s
    float* bm;                             // [rows][heads * 16] B
    float* ends;                           // [chunk place][heads * dim] P_16 (decays per channel), or [chunk place][heads * 36] P_t, P_16 / P_t and what P_16's rounding lost
    float* obuf;                           // [rows][heads * vdim] M V (delta), then the outputs
};
constexpr int kSliceWords = 3 * 32 * 4;    // of an operand's slice of 16 values

// A segment's chunk c has place (first + 16 c) / 16 + segment: segments lie in the order of their rows, so no two chunks share one.
__host__ __device__ inline int chunk_places(int rows, int segments) { return (rows + kChunk - 1) / kChunk + segments; }

__device__ __forceinline__ void dot4(float4 a, float4 b, float4& acc) {
    acc.x = fmaf(a.x, b.x, acc.x);
    acc.y = fmaf(a.y, b.y, acc.y);
    acc.z = fmaf(a.z, b.z, acc.z);
    acc.w = fmaf(a.w, b.w, acc.w);
}
__device__ __forceinline__ float whole4(float4 a) { return (a.x + a.y) + (a.z + a.w); }
__device__ __forceinline__ float4 times4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }

// Two float32 numbers as three pairs of bfloat16 numbers, largest first; the first number in the lower half.
struct Split {
    uint32_t part[3];
};
__device__ __forceinline__ Split split_pair(float x0, float x1) {
    Split s;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(s.part[i]) : "f"(x1), "f"(x0));
        if (i < 2) {
            x0 -= __uint_as_float(s.part[i] << 16);
            x1 -= __uint_as_float(s.part[i] & 0xffff0000u);
        }
    }
    return s;
}
__device__ __forceinline__ void mma_chunk(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Lane's words of an operand's slice: the four pairs in each of their parts.
__device__ __forceinline__ void store_operand(uint32_t* slice, int lane, const Split (&pairs)[4]) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
        *reinterpret_cast<uint4*>(slice + (i * 32 + lane) * 4) = make_uint4(pairs[0].part[i], pairs[1].part[i], pairs[2].part[i], pairs[3].part[i]);
}
__device__ __forceinline__ void load_operand(const uint32_t* slice, int lane, Split (&pairs)[4]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint4 x = *reinterpret_cast<const uint4*>(slice + (i * 32 + lane) * 4);
        pairs[0].part[i] = x.x; pairs[1].part[i] = x.y; pairs[2].part[i] = x.z; pairs[3].part[i] = x.w;
    }
}
// The six products of two split operands, smallest first: parts of A and of B.  The last, largest one has a sum of its own: the tensor cores cut
// sums off where float32 additions round.
constexpr int kSplitProducts = 6;
__host__ __device__ constexpr int split_a(int i) { return i == 1 ? 2 : i == 2 || i == 4 ? 1 : 0; }
__host__ __device__ constexpr int split_b(int i) { return i == 0 ? 2 : i == 2 || i == 3 ? 1 : 0; }
// d += product i of A [16][16] and B [16][8].
__device__ __forceinline__ void mma_product(float (&d)[4], const Split (&a)[4], const Split& b0, const Split& b1, int i) {
    mma_chunk(d, a[0].part[split_a(i)], a[1].part[split_a(i)], a[2].part[split_a(i)], a[3].part[split_a(i)], b0.part[split_b(i)], b1.part[split_b(i)]);
}

// Solves (I + diag(beta) A) x = beta_j e_j for column j (a thread each) and leaves column j of M.
__device__ __forceinline__ void chunk_solve(const float (*a)[kChunk + 4], const float* beta, float (*m)[kChunk + 4], int j) {
    float x[kChunk];
#pragma unroll
    for (int i = 0; i < kChunk; ++i) {
        float row[kChunk];
#pragma unroll
        for (int s = 0; s < i; s += 4) mlr_load4(&a[i][s], reinterpret_cast<float (&)[4]>(row[s]));
        float sum = 0.0f;
#pragma unroll
        for (int s = 0; s < i; ++s) sum = fmaf(row[s], x[s], sum);
        x[i] = i < j ? 0.0f : beta[i] * ((i == j ? 1.0f : 0.0f) - sum);
        m[i][j] = x[i];
    }
}

// out[t * stride] = sum_{s <= t} M_ts x_s for the first n tokens.
__device__ __forceinline__ void chunk_apply(const float (*m)[kChunk + 4], const float (&x)[kChunk], float* out, size_t stride, int n) {
#pragma unroll
    for (int t = 0; t < kChunk; ++t) {
        float sum = 0.0f;
#pragma unroll
        for (int s = 0; s <= t; s += 4) {
            float row[4];
            mlr_load4(&m[t][s], row);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (s + i <= t) sum = fmaf(row[i], x[s + i], sum);
        }
        if (t < n) out[t * stride] = sum;
    }
}

template <int DIM, bool CH>
constexpr size_t chunk_prepare_shared() { return sizeof(float) * (DIM + 4) * (CH ? 104 : 48); }

// One block a chunk and `heads_a_block` heads that share q and k (one with the delta rule and with decays per channel).  A thread has a pair of tokens for A and B; then the
// threads of the first half have a value of k each, those of the second a column of V, whose loads have been on their way since the start.
template <typename T, int DIM, int RULE, bool CH>
__global__ void __launch_bounds__(kChunkPrepareThreads, RULE == 1 ? 2 : CH ? 3 : 4) chunk_prepare_kernel(ChunkBuffers b, const T* proj, int ld, const int* segment_info,
                                                                                        int segments, RecurrenceSpec s, int heads_a_block) {
    mlr_grid_wait();
    constexpr int LD = DIM + 4, kHalf = kChunkPrepareThreads / 2;      // LD: eight rows of a vector access fall into different banks
    extern __shared__ __align__(16) float chunk_smem[];
    __shared__ int chunk_first, chunk_rows;
    __shared__ __align__(16) float a[kChunk][kChunk + 4], m[kChunk][kChunk + 4];
    __shared__ __align__(16) float gs[kChunk];
    __shared__ float beta[kChunk], ps[kChunk];
    float* qs = chunk_smem;                // [16][LD]
    float* ks = qs + kChunk * LD;
    float* ws = ks + kChunk * LD;          // RULE 1: W, at last (in the place of `ds` where there are decays per channel)
    float* ds = ks + kChunk * LD;          // with decays per channel: the decays, k and q times the decays since their group of four began,
    float* kl = ds + kChunk * LD;          // and k times the decays up to the beginning of each later group of four (4 + 8 + 12 rows)
    float* ql = kl + kChunk * LD;
    float* kr = ql + kChunk * LD;
    const int tid = threadIdx.x, place = blockIdx.x;
    bool found = false;
    for (int i = tid; i < segments; i += kChunkPrepareThreads) {
        const int from = segment_info[4 * i], count = segment_info[4 * i + 1], c = place - (from / kChunk + i);
        if (c >= 0 && c * kChunk < count) {
            chunk_first = from + c * kChunk;
            chunk_rows = min(kChunk, count - c * kChunk);
            found = true;
        }
    }
    if (!__syncthreads_or(found)) return;  // no chunk has this place
    const int first = chunk_first, n = chunk_rows;
    const int group = s.heads / s.qk_heads;
    const int head0 = blockIdx.y * heads_a_block, qk_head = head0 / group;
    const size_t qk_ld = static_cast<size_t>(s.qk_heads) * DIM, d_ld = static_cast<size_t>(s.heads) * DIM;

    T v[RULE == 1 ? kChunk : 1];           // a column of V of this thread's first head
    auto load_v = [&](int head, int c) {
        if constexpr (RULE == 1) {
            const T* at = proj + static_cast<size_t>(first) * ld + s.col_v + head * s.vdim + c;
#pragma unroll
            for (int r = 0; r < kChunk; ++r) v[r] = at[static_cast<size_t>(r < n ? r : 0) * ld];
        }
    };
    if (tid >= kHalf && tid - kHalf < s.vdim) load_v(head0, tid - kHalf);
    float gate[2] = {1.0f, 0.0f};          // of token `tid`, this block's first head
    auto load_gates = [&](int head) {
        if (tid < n) {
            const float* at = b.gates + static_cast<size_t>(first + tid) * 2 * s.heads + head;
            if constexpr (!CH) gate[0] = RULE == 0 ? s.decay[head] : __ldcg(at);
            if constexpr (RULE != 0) gate[1] = __ldcg(at + s.heads);
        }
    };
    load_gates(head0);

    const int t = tid / kChunk, x = tid % kChunk;              // this thread's pair: token t with token x
    float4 kk[2] = {}, qk[2] = {};         // eight sums each: chains of DIM / 8 terms
    float kt[kChunk];                      // RULE 1: P_t k_t of value `tid`
    if constexpr (!CH) {
        for (int i = tid; i < kChunk * DIM / 4; i += kChunkPrepareThreads) {
            const int row = i / (DIM / 4), c = i % (DIM / 4) * 4;
            const size_t at = static_cast<size_t>(first + row) * qk_ld + static_cast<size_t>(qk_head) * DIM + c;
            const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            *reinterpret_cast<float4*>(qs + row * LD + c) = row < n ? __ldcg(reinterpret_cast<const float4*>(b.qf + at)) : zero;
            *reinterpret_cast<float4*>(ks + row * LD + c) = row < n ? __ldcg(reinterpret_cast<const float4*>(b.kf + at)) : zero;
        }
        __syncthreads();
        if (x <= t) {
#pragma unroll 8
            for (int c = 0; c < DIM; c += 4) {
                const float4 right = *reinterpret_cast<const float4*>(ks + x * LD + c);
                dot4(*reinterpret_cast<const float4*>(qs + t * LD + c), right, qk[c / 4 % 2]);
                if constexpr (RULE == 1) dot4(*reinterpret_cast<const float4*>(ks + t * LD + c), right, kk[c / 4 % 2]);
            }
        }
    } else {
        if (tid < DIM) {                   // a value of the head a thread
            float q[kChunk], k[kChunk], d[kChunk];
            const size_t q_at = static_cast<size_t>(first) * qk_ld + static_cast<size_t>(qk_head) * DIM + tid;
            const size_t d_at = static_cast<size_t>(first) * d_ld + static_cast<size_t>(head0) * DIM + tid;
#pragma unroll
            for (int r = 0; r < kChunk; ++r) {
                q[r] = r < n ? __ldcg(b.qf + q_at + r * qk_ld) : 0.0f;
                k[r] = r < n ? __ldcg(b.kf + q_at + r * qk_ld) : 0.0f;
                d[r] = r < n ? __ldcg(b.df + d_at + r * d_ld) : 1.0f;
            }
            float from_group = 1.0f;
#pragma unroll
            for (int r = 0; r < kChunk; ++r) {
                from_group = r % 4 ? from_group * d[r] : d[r];
                qs[r * LD + tid] = q[r];
                ks[r * LD + tid] = k[r];
                ds[r * LD + tid] = d[r];
                ql[r * LD + tid] = from_group * q[r];
                kl[r * LD + tid] = from_group * k[r];
            }
#pragma unroll
            for (int later = 1; later < 4; ++later) {
                float run = 1.0f;
#pragma unroll
                for (int r = 4 * later - 1; r >= 0; --r) {
                    kr[(2 * later * (later - 1) + r) * LD + tid] = run * k[r];
                    run *= d[r];
                }
            }
        }
        __syncthreads();
        if (x <= t && x / 4 < t / 4) {
            const float* right_row = kr + (2 * (t / 4) * (t / 4 - 1) + x) * LD;
#pragma unroll 8
            for (int c = 0; c < DIM; c += 4) {
                const float4 right = *reinterpret_cast<const float4*>(right_row + c);
                dot4(*reinterpret_cast<const float4*>(ql + t * LD + c), right, qk[c / 4 % 2]);
                if constexpr (RULE == 1) dot4(*reinterpret_cast<const float4*>(kl + t * LD + c), right, kk[c / 4 % 2]);
            }
        }
        // Pairs of one group of four: the decays between them one by one.
        const bool near = x <= t && x / 4 == t / 4;
        if (near) {
            const float4 one = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
#pragma unroll 4
            for (int c = 0; c < DIM; c += 4) {
                float4 right = *reinterpret_cast<const float4*>(ks + x * LD + c);
#pragma unroll
                for (int back = 0; back < 3; ++back)
                    right = times4(right, t - back > x ? *reinterpret_cast<const float4*>(ds + (t - back) * LD + c) : one);
                dot4(*reinterpret_cast<const float4*>(qs + t * LD + c), right, qk[c / 4 % 2]);
                if constexpr (RULE == 1) dot4(*reinterpret_cast<const float4*>(ks + t * LD + c), right, kk[c / 4 % 2]);
            }
        }
    }

    for (int head = head0; head < head0 + heads_a_block; ++head) {
        if (head > head0) load_gates(head);
        if (tid < kChunk) {
            gs[tid] = gate[0];
            beta[tid] = gate[1];
        }
        __syncthreads();
        float between = 1.0f;              // the decays behind token x up to token t
        if constexpr (!CH) {
#pragma unroll
            for (int r = 1; r < kChunk; r += 1) between *= r > x && r <= t ? gs[r] : 1.0f;
        }
        float value = between * (whole4(qk[0]) + whole4(qk[1]));
        if constexpr (RULE == 1) a[t][x] = x < t ? between * (whole4(kk[0]) + whole4(kk[1])) : 0.0f;
        if constexpr (RULE == 2) value *= beta[x];
        if (t < n) b.bm[(static_cast<size_t>(first + t) * s.heads + head) * kChunk + x] = x <= t ? value : 0.0f;
        if constexpr (!CH) {
            // A fixed decay in 64 bits: its powers would have the same rounding error in every chunk.
            using Wide = std::conditional_t<RULE == 0, double, float>;
            if (tid < 2 * kChunk) {
                const int r0 = tid % kChunk;
                const bool after = tid >= kChunk;              // the decays behind token r0, or those up to it
                Wide p = 1;
#pragma unroll
                for (int r = 0; r < kChunk; ++r) p *= (r > r0) == after ? gs[r] : 1.0f;
                float* at = b.ends + (static_cast<size_t>(place) * s.heads + head) * kChunkEnds;
                const float rounded = static_cast<float>(p);
                at[tid] = RULE == 2 && after ? rounded * beta[r0] : rounded;
                if (!after) ps[r0] = rounded;
                if (tid == kChunk - 1) *reinterpret_cast<float4*>(at + 2 * kChunk) = make_float4(static_cast<float>(p - rounded), 0.0f, 0.0f, 0.0f);
            }
        }
        if constexpr (RULE == 1 || CH) __syncthreads();
        if constexpr (RULE == 1) {
            if (tid >= kHalf && tid < kHalf + kChunk) chunk_solve(a, beta, m, tid - kHalf);
        }
        if constexpr (CH) {
            if (tid < DIM) {               // q and k of the walk; the pairs have been multiplied
                float from_start = 1.0f, to_end = 1.0f, d[kChunk];
#pragma unroll
                for (int r = 0; r < kChunk; ++r) {
                    d[r] = ds[r * LD + tid];
                    from_start *= d[r];
                    ql[r * LD + tid] = from_start * qs[r * LD + tid];
                    if constexpr (RULE == 1) kt[r] = from_start * ks[r * LD + tid];
                }
                b.ends[static_cast<size_t>(place) * d_ld + static_cast<size_t>(head) * DIM + tid] = from_start;
#pragma unroll
                for (int r = kChunk - 1; r >= 0; --r) {
                    kl[r * LD + tid] = to_end * ks[r * LD + tid];
                    to_end *= d[r];
                }
            }
        }
        if constexpr (RULE == 1) {
            __syncthreads();
            if (tid < DIM) {
                if constexpr (!CH) {
#pragma unroll
                    for (int r = 0; r < kChunk; ++r) kt[r] = ps[r] * ks[r * LD + tid];
                }
                chunk_apply(m, kt, ws + tid, LD, kChunk);
            }
            if (tid >= kHalf) {
                const size_t o_ld = static_cast<size_t>(s.heads) * s.vdim;
                for (int c = tid - kHalf; c < s.vdim; c += kHalf) {
                    if (head > head0 || c >= kHalf) load_v(head, c);
                    float values[kChunk];
#pragma unroll
                    for (int r = 0; r < kChunk; ++r) values[r] = r < n ? act_in(mlr_load(&v[r], 0), s.in_act) : 0.0f;
                    chunk_apply(m, values, b.obuf + static_cast<size_t>(first) * o_ld + static_cast<size_t>(head) * s.vdim + c, o_ld, n);
                }
            }
        }
        if constexpr (RULE == 1 || CH) __syncthreads();
        // The walk's operands: a warp a slice of 16 values.
        const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
        if (warp < DIM / 16) {
            auto rows_of = [&](const float* from, uint32_t* to) {
                Split pairs[4];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    const float4 row = *reinterpret_cast<const float4*>(from + (nt * 8 + g) * LD + warp * 16 + t4 * 4);
                    pairs[nt * 2] = split_pair(row.x, row.z);
                    pairs[nt * 2 + 1] = split_pair(row.y, row.w);
                }
                store_operand(to, lane, pairs);
            };
            const size_t at = ((static_cast<size_t>(place) * s.heads + head) * (DIM / 16) + warp) * kSliceWords;
            if constexpr (RULE == 1) rows_of(ws, b.w + at);
            if (CH || head % group == 0) {
                const size_t qk_at = CH ? at : ((static_cast<size_t>(place) * s.qk_heads + qk_head) * (DIM / 16) + warp) * kSliceWords;
                rows_of(CH ? ql : qs, b.q + qk_at);
                const float* from = (CH ? kl : ks) + warp * 16 + 2 * g;
                Split pairs[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 k0 = *reinterpret_cast<const float2*>(from + (h * 8 + 2 * t4) * LD), k1 = *reinterpret_cast<const float2*>(from + (h * 8 + 2 * t4 + 1) * LD);
                    pairs[h] = split_pair(k0.x, k1.x);
                    pairs[2 + h] = split_pair(k0.y, k1.y);
                }
                store_operand(b.k + qk_at, lane, pairs);
            }
        }
        if (head + 1 < head0 + heads_a_block) __syncthreads();               // the next head's decays, A and M
    }
    mlr_grid_dependents_may_start();
}

// Shared memory in floats (words).  Every warp copies what it needs of a chunk itself, into stages of its own.
template <int DIM, int RULE, bool CH, int NC>
struct ChunkStage {
    static constexpr int kSlices = DIM / 16, kWarps = kSlices + 4, kCols = 16 * NC;
    // Two leave room for two blocks an SM.  With 128 decays per channel a block has its SM alone, by three stages' room: two long portions' blocks on one SM
    // slow each other (gated linear attention, 16 heads, portions of 18, 1664 and four of 1: 198 us alone, 270 us side by side; the delta rule, whose registers leave one, has three as well).
    static constexpr int kStages = RULE != 1 && NC == 2 && !(CH && DIM == 128) ? 2 : 3;
    // a warp with a slice of the state: W, Q, K and the ends
    static constexpr int w = 0, q = w + (RULE == 1 ? kSliceWords : 0), k = q + kSliceWords, ends = k + kSliceWords, slice = ends + (CH ? 16 : 8);
    // a warp that makes U^T of eight tokens: M V in float32 or V in bfloat16, and the weights P_16 / P_t
    static constexpr int kVStride = RULE == 1 ? kCols + 4 : kCols + 8;             // floats, or bfloat16
    static constexpr int weights = 8 * kVStride / (RULE == 1 ? 1 : 2), makes_u = weights + 8;
    // a warp that finishes the outputs of eight tokens: their rows of B, P_t, and (step) V
    static constexpr int kBStride = kChunk + 4, powers = 8 * kBStride, skipped = powers + 8, finishes = skipped + (RULE == 2 ? 8 * kVStride / 2 : 0);
    static constexpr int stage = kSlices * slice + 2 * makes_u + 2 * finishes;
    static constexpr int sums = 2 * NC * kSlices * 32 * 4;                         // [column tile][token tile][slice][lane][4]
    static constexpr int kUSets = CH ? 1 : 2;                                      // U^T, and U^T times the weights
    static constexpr int u = kUSets * NC * kSliceWords;
    static constexpr int floats = kStages * stage + (RULE == 1 ? 3 : 2) * sums + 2 * u;
    static constexpr size_t bytes() { return sizeof(float) * floats; }
};

// Meetings of some of a block's warps (barrier 0 is the whole block's).
template <int ID, int THREADS>
__device__ __forceinline__ void chunk_arrive() { asm volatile("bar.arrive %0, %1;\n" ::"n"(ID), "n"(THREADS) : "memory"); }
template <int ID, int THREADS>
__device__ __forceinline__ void chunk_meet() { asm volatile("bar.sync %0, %1;\n" ::"n"(ID), "n"(THREADS) : "memory"); }

// A block's columns of a segment token by token on the CUDA cores, eight lanes a column, for the values that products of parts cannot take.  `room`: shared
// memory, whose other uses are over.  It is rare, and the walk in chunks must not pay for it: the state is in shared memory and the block's place is asked
// for anew, since with the state in registers the step rule's walk took 92 registers instead of 80, one block an SM instead of two (1999 tokens of 128
// heads 325 -> 367 us; so 330 us, the other rules' walks within 3 % of those without it).  2048 tokens of 16 heads, all columns: 2.0 ms.
template <int DIM, int COLS>
__host__ __device__ constexpr int by_token_floats() { return kChunk * (3 * DIM + COLS + 2) + COLS * (DIM + 8); }
template <typename T, int DIM, int RULE, bool CH, int COLS>
__device__ __forceinline__ void chunk_walk_by_token(const ChunkBuffers& b, const T* proj, int ld, float* state, long long state_stride, const int* segment_info,
                                                    const RecurrenceSpec& s, float* room) {
    constexpr int kLanes = 8, kThreads = (DIM / 16 + 4) * 32, LD = DIM + 8;                // LD: a warp's four columns fall into different banks
    static_assert(COLS * kLanes <= kThreads);
    float *ks = room, *qs = ks + kChunk * DIM, *ds = qs + kChunk * DIM, *vs = ds + kChunk * DIM, *gs = vs + kChunk * COLS, *S = gs + 2 * kChunk;
    const int tid = threadIdx.x, sub = tid % kLanes, col = tid / kLanes;
    // Asked for anew: nothing is kept for this through the walk in chunks.
    const volatile int* info = segment_info + 4 * blockIdx.x;
    const int first = info[0], count = info[1], slot = info[3], head = blockIdx.y, block_col = blockIdx.z * COLS;
    float* columns = state + static_cast<size_t>(slot) * state_stride + (static_cast<size_t>(head) * s.vdim + block_col) * DIM;
    const size_t qk_ld = static_cast<size_t>(s.qk_heads) * DIM, d_ld = static_cast<size_t>(s.heads) * DIM, o_ld = static_cast<size_t>(s.heads) * s.vdim;
    const size_t qk_at = static_cast<size_t>(head / (s.heads / s.qk_heads)) * DIM, d_at = static_cast<size_t>(head) * DIM, v_at = head * s.vdim + block_col;
#pragma unroll 1
    for (int i = tid; i < COLS * DIM; i += kThreads) S[i / DIM * LD + i % DIM] = columns[i];
#pragma unroll 1
    for (int base = 0; base < count; base += kChunk) {
        const int n = min(kChunk, count - base);
        const size_t row0 = static_cast<size_t>(first) + base;
#pragma unroll 1
        for (int i = tid; i < n * DIM; i += kThreads) {
            const size_t row = row0 + i / DIM;
            ks[i] = __ldcg(b.kf + row * qk_ld + qk_at + i % DIM);
            qs[i] = __ldcg(b.qf + row * qk_ld + qk_at + i % DIM);
            if constexpr (CH) ds[i] = __ldcg(b.df + row * d_ld + d_at + i % DIM);
        }
#pragma unroll 1
        for (int i = tid; i < n * COLS; i += kThreads) vs[i] = act_in(mlr_load(proj + (row0 + i / COLS) * ld + s.col_v + v_at, i % COLS), s.in_act);
        if (tid < n) {
            const float* gate = b.gates + (row0 + tid) * 2 * s.heads + head;
            if constexpr (!CH) gs[tid] = RULE == 0 ? s.decay[head] : __ldcg(gate);
            if constexpr (RULE != 0) gs[kChunk + tid] = __ldcg(gate + s.heads);
        }
        __syncthreads();
        if (col < COLS) {                  // whole warps
            float* mine = S + col * LD + sub;                  // every eighth value of the column
#pragma unroll 1
            for (int t = 0; t < n; ++t) {
                const float *k = ks + t * DIM + sub, *q = qs + t * DIM + sub, *d = ds + t * DIM + sub;
                const float v = vs[t * COLS + col];
                float held = 0.0f, o = 0.0f;
                if constexpr (RULE == 1) {
#pragma unroll 4
                    for (int j = 0; j < DIM; j += kLanes) held = fmaf((CH ? d[j] : gs[t]) * mine[j], k[j], held);
#pragma unroll
                    for (int step = 1; step < kLanes; step *= 2) held += __shfl_xor_sync(0xffffffffu, held, step);
                }
                const float write = RULE == 0 ? v : gs[kChunk + t] * (v - held);
#pragma unroll 4
                for (int j = 0; j < DIM; j += kLanes) {
                    const float decay = CH ? d[j] : gs[t];
                    const float value = RULE == 1 ? fmaf(k[j], write, decay * mine[j]) : fmaf(decay, mine[j], k[j] * write);
                    mine[j] = value;
                    o = fmaf(value, q[j], o);
                }
#pragma unroll
                for (int step = 1; step < kLanes; step *= 2) o += __shfl_xor_sync(0xffffffffu, o, step);
                if (RULE == 2) o = fmaf(s.skip[head], v, o);
                if (sub == 0) b.obuf[(row0 + t) * o_ld + v_at + col] = o;
            }
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int i = tid; i < COLS * DIM; i += kThreads) columns[i] = S[i / DIM * LD + i % DIM];
}

// A block walks a segment for 16 * NC columns of a head's state.  Warp w of the first ones keeps the values 16 w .. 16 w + 15 of every column, as
// the accumulators of a product with the state's columns as its rows: they are the first operand of the products S^T W^T and S^T Q^T as they are.
// The slices' sums meet in shared memory: two more warps add up the first and make U^T of it, the first operand of what is added to the state,
// while the slices' warps are at the second; two others finish the outputs while the slices' warps are at the next chunk.  Within a slice, lane (g, t) has the values 4 t .. 4 t + 3 of columns g
// and g + 8.
template <typename T, int DIM, int RULE, bool CH, int NC>
__global__ void __launch_bounds__((DIM / 16 + 4) * 32) chunk_walk_kernel(ChunkBuffers b, const T* proj, int ld, float* state, long long state_stride,
                                                                        const int* segment_info, RecurrenceSpec s) {
    mlr_grid_wait();
    using Stage = ChunkStage<DIM, RULE, CH, NC>;
    constexpr int kSlices = Stage::kSlices;
    constexpr int kSummed = 1, kMade = 2, kRead = 3;           // barriers: W's sums are there; U^T is; it and Q's sums are, for the outputs
    constexpr int kToTwo = (kSlices + 2) * 32, kToAll = Stage::kWarps * 32;
    extern __shared__ __align__(16) float chunk_smem[];
    uint32_t* uset = reinterpret_cast<uint32_t*>(chunk_smem + Stage::kStages * Stage::stage);        // [2][set][column tile] operands
    float4* ysum = reinterpret_cast<float4*>(uset + 2 * Stage::u);                                 // [2]
    float4* xsum = ysum + 2 * Stage::sums / 4;
    const int segment = blockIdx.x, head = blockIdx.y, block_col = blockIdx.z * Stage::kCols;
    const int first = segment_info[4 * segment], count = segment_info[4 * segment + 1], slot = segment_info[4 * segment + 3];
    if (count <= 0) return;
    const size_t place0 = first / kChunk + segment;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    int broken;                            // some result of the block is not finite
    const size_t d_ld = static_cast<size_t>(s.heads) * DIM, o_ld = static_cast<size_t>(s.heads) * s.vdim;
    const size_t ends_ld = CH ? d_ld : static_cast<size_t>(s.heads) * kChunkEnds;
    const float* ends0 = b.ends + place0 * ends_ld + static_cast<size_t>(head) * (CH ? DIM : kChunkEnds);
    auto wait_stage = [] {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(Stage::kStages - 2) : "memory");
        __syncwarp();
    };
    // Calls `fetch(stage)` for the first chunks, then `chunk(stage, c)` for every chunk, whose copies have landed, behind the call that starts a later one's.
    auto walk = [&](auto fetch, auto chunk) {
        int left = count, fill = 0;        // rows not yet on their way; the stage that is filled next
        auto next = [&] {
            if (left > 0) fetch(fill, left);
            mlr_async_commit();
            left -= kChunk;
            fill = fill + 1 == Stage::kStages ? 0 : fill + 1;
        };
#pragma unroll
        for (int i = 0; i < Stage::kStages - 1; ++i) next();
        for (int rows = count, stage = 0, odd = 0; rows > 0; rows -= kChunk, stage = stage + 1 == Stage::kStages ? 0 : stage + 1, odd ^= 1) {
            wait_stage();                  // (and the warp is done with the stage that is filled now)
            next();
            chunk(stage, rows, odd);
        }
    };

    if (warp < kSlices) {
        float* mine = chunk_smem + warp * Stage::slice;
        const int qk_heads = CH ? s.heads : s.qk_heads, qk_head = CH ? head : head / (s.heads / s.qk_heads);
        const uint32_t* wnext = b.w + ((place0 * s.heads + head) * kSlices + warp) * kSliceWords + lane * 4;
        const size_t qk_at = ((place0 * qk_heads + qk_head) * kSlices + warp) * kSliceWords + lane * 4;
        const uint32_t *qnext = b.q + qk_at, *knext = b.k + qk_at;
        const float* enext = ends0 + (CH ? warp * 16 + lane * 4 : lane == 0 ? kChunk - 4 : 2 * kChunk);
        const size_t w_step = static_cast<size_t>(s.heads) * kSlices * kSliceWords, qk_step = static_cast<size_t>(qk_heads) * kSlices * kSliceWords;
        auto fetch = [&](int stage, int) {
            float* to = mine + stage * Stage::stage + lane * 4;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                if constexpr (RULE == 1) mlr_async_copy16(to + Stage::w + i * 128, wnext + i * 128);
                mlr_async_copy16(to + Stage::q + i * 128, qnext + i * 128);
                mlr_async_copy16(to + Stage::k + i * 128, knext + i * 128);
            }
            if (lane < (CH ? 4 : 2)) mlr_async_copy16(to + Stage::ends, enext);
            wnext += w_step;
            qnext += qk_step;
            knext += qk_step;
            enext += ends_ld;
        };
        float S[NC][2][4];                 // [column tile][j][(g, 4t + j), (g, 4t + 2 + j), (g + 8, ..), (g + 8, ..)]
        float* my_state = state + static_cast<size_t>(slot) * state_stride + (static_cast<size_t>(head) * s.vdim + block_col + g) * DIM + warp * 16 + 4 * t;
#pragma unroll
        for (int m = 0; m < NC; ++m)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) S[m][j][i] = my_state[(m * 16 + (i >> 1) * 8) * DIM + (i & 1) * 2 + j];
        walk(fetch, [&](int stage, int, int odd) {
            const float* now = mine + stage * Stage::stage;
            const auto operand = [&](int at) { return reinterpret_cast<const uint32_t*>(now + at); };
            {
                Split parts[NC][4], rows16[4];
#pragma unroll
                for (int m = 0; m < NC; ++m)
#pragma unroll
                    for (int i = 0; i < 4; ++i) parts[m][i] = split_pair(S[m][i >> 1][(i & 1) * 2], S[m][i >> 1][(i & 1) * 2 + 1]);
                // S^T times sixteen rows: columns g (+ 8) of the state, tokens 8 nt + 2t (+ 1).
                auto rows_times_state = [&](float4* to) {
                    float sum[2][NC][2][4] = {};           // [the largest product, the others]
#pragma unroll
                    for (int i = 0; i < kSplitProducts; ++i)               // independent sums side by side
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                            for (int m = 0; m < NC; ++m) mma_product(sum[i + 1 < kSplitProducts][m][nt], parts[m], rows16[2 * nt], rows16[2 * nt + 1], i);
#pragma unroll
                    for (int m = 0; m < NC; ++m)
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt)
                            to[((m * 2 + nt) * kSlices + warp) * 32 + lane] = make_float4(sum[0][m][nt][0] + sum[1][m][nt][0], sum[0][m][nt][1] + sum[1][m][nt][1],
                                                                                            sum[0][m][nt][2] + sum[1][m][nt][2], sum[0][m][nt][3] + sum[1][m][nt][3]);
                };
                if constexpr (RULE == 1) {
                    load_operand(operand(Stage::w), lane, rows16);
                    rows_times_state(xsum);
                }
                chunk_arrive<kSummed, kToTwo>();
                load_operand(operand(Stage::q), lane, rows16);
                rows_times_state(ysum + odd * (Stage::sums / 4));
            }
            Split k[4];
            load_operand(operand(Stage::k), lane, k);
            float decay[4], rest = 0.0f;   // of the values 4t ..
            if constexpr (CH) {
                mlr_load4(now + Stage::ends + 4 * t, decay);
            } else {
                decay[0] = decay[1] = decay[2] = decay[3] = now[Stage::ends + 3];
                rest = now[Stage::ends + 4];
            }
            chunk_meet<kMade, kToAll>();
            chunk_arrive<kRead, kToTwo>();
            const uint32_t* made = uset + odd * Stage::u + (Stage::kUSets - 1) * NC * kSliceWords;
            float sum[2][NC][2][4] = {};
            Split u[NC][4];
#pragma unroll
            for (int m = 0; m < NC; ++m) load_operand(made + m * kSliceWords, lane, u[m]);
#pragma unroll
            for (int i = 0; i < kSplitProducts; ++i)
#pragma unroll
                for (int m = 0; m < NC; ++m)
#pragma unroll
                    for (int j = 0; j < 2; ++j) mma_product(sum[i + 1 < kSplitProducts][m][j], u[m], k[2 * j], k[2 * j + 1], i);
#pragma unroll
            for (int m = 0; m < NC; ++m)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float added = sum[0][m][j][i] + sum[1][m][j][i];
                        if constexpr (!CH) added = fmaf(rest, S[m][j][i], added);
                        S[m][j][i] = fmaf(decay[(i & 1) * 2 + j], S[m][j][i], added);
                    }
        });
        float finite = 0.0f;               // stays zero while the state is finite
#pragma unroll
        for (int i = 0; i < NC * 8; ++i) finite = fmaf((&S[0][0][0])[i], 0.0f, finite);
        broken = __syncthreads_or(finite != 0.0f);
        if (!broken) {
#pragma unroll
            for (int m = 0; m < NC; ++m)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) my_state[(m * 16 + (i >> 1) * 8) * DIM + (i & 1) * 2 + j] = S[m][j][i];
        }
    } else {
        const int nt = warp & 1;           // tokens 8 nt .. 8 nt + 7 (kSlices is even)
        float finite = 0.0f;               // stays zero while the outputs are finite
        // The slices' sums of a tile, added up.
        auto summed = [&](const float4* sums, int m) {
            const float4* from = sums + (m * 2 + nt) * kSlices * 32 + lane;
            float4 x[kSlices];
#pragma unroll
            for (int w = 0; w < kSlices; ++w) x[w] = from[w * 32];
#pragma unroll
            for (int step = kSlices / 2; step > 0; step /= 2)
#pragma unroll
                for (int w = 0; w < step; ++w) {
                    x[w].x += x[w + step].x; x[w].y += x[w + step].y; x[w].z += x[w + step].z; x[w].w += x[w + step].w;
                }
            return x[0];
        };
        if (warp < kSlices + 2) {
            float* mine = chunk_smem + kSlices * Stage::slice + nt * Stage::makes_u;
            constexpr int kUnits = (RULE == 1 ? 4 : 2) * NC;   // 16-byte units of a row of M V or V
            const float* unext = b.obuf + static_cast<size_t>(first + nt * 8) * o_ld + static_cast<size_t>(head) * s.vdim + block_col;
            const T* vnext = proj + static_cast<size_t>(first + nt * 8) * ld + s.col_v + head * s.vdim + block_col;
            const float* wnext = ends0 + kChunk + nt * 8 + lane * 4;
            auto fetch = [&](int stage, int left) {            // rows past the segment become zeros
                float* to = mine + stage * Stage::stage;
#pragma unroll
                for (int i = lane; i < 8 * kUnits; i += 32) {
                    const int r = i / kUnits, u = i % kUnits;
                    const bool real = nt * 8 + r < left;
                    if constexpr (RULE == 1) mlr_async_copy16(to + r * Stage::kVStride + u * 4, real ? unext + r * o_ld + u * 4 : b.obuf, real);
                    else mlr_async_copy16(reinterpret_cast<T*>(to) + r * Stage::kVStride + u * 8, real ? vnext + static_cast<size_t>(r) * ld + u * 8 : proj, real);
                }
                if (!CH && lane < 2) mlr_async_copy16(to + Stage::weights + lane * 4, wnext);
                unext += kChunk * o_ld;
                vnext += static_cast<size_t>(kChunk) * ld;
                wnext += ends_ld;
            };
            walk(fetch, [&](int stage, int, int odd) {
                const float* now = mine + stage * Stage::stage;
                uint32_t* made = uset + odd * Stage::u;
                float2 weight = make_float2(1.0f, 1.0f);
                if constexpr (!CH) weight = *reinterpret_cast<const float2*>(now + Stage::weights + 2 * t);
                float u[NC][4];
#pragma unroll
                for (int m = 0; m < NC; ++m) {
                    if constexpr (RULE == 1) {
                        const float* at = now + 2 * t * Stage::kVStride + m * 16 + g;
                        u[m][0] = at[0]; u[m][1] = at[Stage::kVStride]; u[m][2] = at[8]; u[m][3] = at[Stage::kVStride + 8];
                    } else {
                        const T* at = reinterpret_cast<const T*>(now) + 2 * t * Stage::kVStride + m * 16 + g;
                        u[m][0] = act_in(mlr_load(at, 0), s.in_act);
                        u[m][1] = act_in(mlr_load(at, Stage::kVStride), s.in_act);
                        u[m][2] = act_in(mlr_load(at, 8), s.in_act);
                        u[m][3] = act_in(mlr_load(at, Stage::kVStride + 8), s.in_act);
                    }
                }
                chunk_meet<kSummed, kToTwo>();
#pragma unroll
                for (int m = 0; m < NC; ++m) {
                    if constexpr (RULE == 1) {
                        const float4 held = summed(xsum, m);
                        u[m][0] -= held.x; u[m][1] -= held.y; u[m][2] -= held.z; u[m][3] -= held.w;
                    }
#pragma unroll
                    for (int set = 0; set < Stage::kUSets; ++set) {
                        if (set == 1) { u[m][0] *= weight.x; u[m][1] *= weight.y; u[m][2] *= weight.x; u[m][3] *= weight.y; }
                        const Split upper = split_pair(u[m][0], u[m][1]), lower = split_pair(u[m][2], u[m][3]);
#pragma unroll
                        for (int i = 0; i < 3; ++i)
                            *reinterpret_cast<uint2*>(made + (set * NC + m) * kSliceWords + (i * 32 + lane) * 4 + nt * 2) = make_uint2(upper.part[i], lower.part[i]);
                    }
                }
                chunk_arrive<kMade, kToAll>();
            });
        } else {
            float* mine = chunk_smem + kSlices * Stage::slice + 2 * Stage::makes_u + nt * Stage::finishes;
            const float* bnext = b.bm + (static_cast<size_t>(first + nt * 8 + lane / 4) * s.heads + head) * kChunk + lane % 4 * 4;
            const float* pnext = ends0 + nt * 8 + lane * 4;
            const T* vnext = proj + static_cast<size_t>(first + nt * 8) * ld + s.col_v + head * s.vdim + block_col;
            const float skip = RULE == 2 ? s.skip[head] : 0.0f;
            float* outputs = b.obuf + static_cast<size_t>(first + nt * 8 + 2 * t) * o_ld + static_cast<size_t>(head) * s.vdim + block_col + g;
            auto fetch = [&](int stage, int left) {
                float* to = mine + stage * Stage::stage;
                const bool real = nt * 8 + lane / 4 < left;
                mlr_async_copy16(to + lane / 4 * Stage::kBStride + lane % 4 * 4, real ? bnext : b.bm, real);
                if (!CH && lane < 2) mlr_async_copy16(to + Stage::powers + lane * 4, pnext);
                if constexpr (RULE == 2) {
#pragma unroll
                    for (int i = lane; i < 8 * 2 * NC; i += 32) {
                        const int r = i / (2 * NC), u = i % (2 * NC);
                        const bool in = nt * 8 + r < left;
                        mlr_async_copy16(reinterpret_cast<T*>(to + Stage::skipped) + r * Stage::kVStride + u * 8, in ? vnext + static_cast<size_t>(r) * ld + u * 8 : proj, in);
                    }
                    vnext += static_cast<size_t>(kChunk) * ld;
                }
                bnext += static_cast<size_t>(kChunk) * s.heads * kChunk;
                pnext += ends_ld;
            };
            walk(fetch, [&](int stage, int rows, int odd) {
                chunk_arrive<kMade, kToAll>();             // done with the chunk before: its places may be written again after this one's
                const float* now = mine + stage * Stage::stage;
                const float2 lo = *reinterpret_cast<const float2*>(now + g * Stage::kBStride + 2 * t), hi = *reinterpret_cast<const float2*>(now + g * Stage::kBStride + 8 + 2 * t);
                const Split b0 = split_pair(lo.x, lo.y), b1 = split_pair(hi.x, hi.y);
                float2 power = make_float2(1.0f, 1.0f);
                if constexpr (!CH) power = *reinterpret_cast<const float2*>(now + Stage::powers + 2 * t);
                chunk_meet<kRead, kToTwo>();
#pragma unroll
                for (int m = 0; m < NC; ++m) {
                    const float4 y = summed(ysum + odd * (Stage::sums / 4), m);
                    Split u[4];
                    load_operand(uset + odd * Stage::u + m * kSliceWords, lane, u);
                    float sum[2][4] = {};
#pragma unroll
                    for (int i = 0; i < kSplitProducts; ++i) mma_product(sum[i + 1 < kSplitProducts], u, b0, b1, i);
                    float o[4] = {fmaf(power.x, y.x, sum[0][0] + sum[1][0]), fmaf(power.y, y.y, sum[0][1] + sum[1][1]),
                                  fmaf(power.x, y.z, sum[0][2] + sum[1][2]), fmaf(power.y, y.w, sum[0][3] + sum[1][3])};
                    if constexpr (RULE == 2) {
                        const T* v = reinterpret_cast<const T*>(now + Stage::skipped) + 2 * t * Stage::kVStride + m * 16 + g;
#pragma unroll
                        for (int i = 0; i < 4; ++i) o[i] = fmaf(skip, act_in(mlr_load(v, (i & 1) * Stage::kVStride + (i >> 1) * 8), s.in_act), o[i]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) finite = fmaf(o[i], 0.0f, finite);         // one instruction a value
                    float* to = outputs + m * 16;
                    if (nt * 8 + 2 * t < rows) {
                        to[0] = o[0];
                        to[8] = o[2];
                    }
                    if (nt * 8 + 2 * t + 1 < rows) {
                        to[o_ld] = o[1];
                        to[o_ld + 8] = o[3];
                    }
                }
                outputs += kChunk * o_ld;
            });
        }
        broken = __syncthreads_or(finite != 0.0f);
    }
    if (broken) {
        static_assert(by_token_floats<DIM, Stage::kCols>() <= Stage::floats);
        chunk_walk_by_token<T, DIM, RULE, CH, Stage::kCols>(b, proj, ld, state, state_stride, segment_info, s, chunk_smem);
    }
    mlr_grid_dependents_may_start();
}
