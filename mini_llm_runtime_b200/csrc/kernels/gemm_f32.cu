// True 32-bit matrix product on the CUDA cores: C[M,N] = A[M,K] * W[N,K]^T, all
// row-major float32, `y = x W^T` as the reference defines its products
// (include/minillm/cuda/matrix.h:35; it calls cublasGemmEx in pedantic FP32 mode,
// src/minillm/cuda/matrix.cpp:30-36).  No tensor cores, no TF32, no split-K.
//
// Every output element is one accumulator that adds its K products in the order
// k = 0, 1, ..., K-1 with fused multiply-adds.  The value of C[m,n] therefore depends
// only on row m of A and row n of W, not on M, on the tile the element falls in, or on
// what else is in the batch: the same token gives the same bits however the work is cut,
// and both kernels below give the same bits.
//
// Measured (one product, W from memory; before: one kernel of 64 x 64 tiles that waited for every 16 values of K):
//   2 x 1024 x 3072 (M, N, K): 243 -> 22 us, bound by one thread's chain of multiply-adds; 2 x 151936 x 1024: 574 -> 100 us, 6.2 TB/s;
//   129 x 1024 x 3072: 225 -> 55 us and 129 x 4096 x 1024: 164 -> 46 us, a few warps an SM, bound by their reads of shared memory;
//   2048 x 4096 x 4096: 1970 -> 1620 us, 42 TFLOP/s, bound by shared memory.
// Both stage rows of A and W as they lie in memory (asynchronous copies, several stages of K in
// flight) with their stride padded by 16 bytes, so that 8 neighbouring rows read 4 values of K
// each from different banks.
#include "common.cuh"

#include <algorithm>
#include <climits>

namespace {

// 16 bytes at column k of a row of K values, zeros past its end.
template <bool kVector>
__device__ __forceinline__ void stage4(float* dst, const float* row, int k, int K, bool real) {
    const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    if (kVector) {
        const int bytes = real ? max(0, min(16, (K - k) * 4)) : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(bytes ? row + k : row), "r"(bytes) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int bytes = real && k + i < K ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(to + 4 * i), "l"(bytes ? row + k + i : row), "r"(bytes) : "memory");
        }
    }
}
template <int N>
__device__ __forceinline__ void stages_left() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---- a tile of BM x BN outputs a block, TM x TN of them a thread (rows and columns dealt round the block) ----
// Shared memory hands a warp 32 registers a cycle, however few addresses they come from, and the SM's schedulers issue four
// multiply-adds a warp in that cycle: a thread's TM + TN values of a k for TM * TN multiply-adds bind all tiles but the largest.
// START, RATE, ROUND: what the tile measured, see tile_cost.
template <int BM, int BN, int TM, int TN, int STAGES, int KK, int START, int RATE, int ROUND>
struct Tile {
    static constexpr int kRows = BM, kColumns = BN, kThreadRows = TM, kThreadColumns = TN;
    static constexpr int kThreads = (BM / TM) * (BN / TN);
    static constexpr int kStages = STAGES, kK = KK, kLd = kK + 4;
    static constexpr int kStart = START, kRate = RATE, kRound = ROUND;
    static constexpr size_t kShared = sizeof(float) * kStages * (BM + BN) * kLd;
};

template <bool kVector, typename T>
__global__ void __launch_bounds__(T::kThreads) gemm_f32_tile_kernel(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                                                                    int ldc) {
    constexpr int BM = T::kRows, BN = T::kColumns, TM = T::kThreadRows, TN = T::kThreadColumns;
    extern __shared__ __align__(16) float staged[];           // per stage: A [BM][kLd], W [BN][kLd]
    constexpr int kAcross = BN / TN, kDown = BM / TM, kStage = (BM + BN) * T::kLd, kChunks = T::kK / 4;
    const int tid = threadIdx.x, tx = tid % kAcross, ty = tid / kAcross;
    // Neighbouring blocks share W's rows, so that they come from memory once.  All tiles in one dimension of the grid: the others take 65535.
    const int row_tiles = (M + BM - 1) / BM, m0 = blockIdx.x % row_tiles * BM, n0 = blockIdx.x / row_tiles * BN;
    const int steps = (K + T::kK - 1) / T::kK;
    auto fetch_a = [&](int step) {
        float* to = staged + (step % T::kStages) * kStage;
#pragma unroll
        for (int i = tid; i < BM * kChunks; i += T::kThreads) {
            const int r = i / kChunks, c = (i % kChunks) * 4;
            stage4<kVector>(to + r * T::kLd + c, m0 + r < M ? A + static_cast<size_t>(m0 + r) * lda : A, step * T::kK + c, K, m0 + r < M);
        }
    };
    auto fetch_w = [&](int step) {
        float* to = staged + (step % T::kStages) * kStage + BM * T::kLd;
#pragma unroll
        for (int i = tid; i < BN * kChunks; i += T::kThreads) {
            const int r = i / kChunks, c = (i % kChunks) * 4;
            stage4<kVector>(to + r * T::kLd + c, n0 + r < N ? W + static_cast<size_t>(n0 + r) * ldw : W, step * T::kK + c, K, n0 + r < N);
        }
    };
    mlr_grid_wait();
    for (int step = 0; step < T::kStages - 1; ++step) {
        if (step < steps) { fetch_w(step); fetch_a(step); }
        mlr_async_commit();
    }
    float acc[TM][TN] = {};
    for (int step = 0; step < steps; ++step) {
        stages_left<T::kStages - 2>();
        __syncthreads();           // this step's stage has landed for everyone, and everyone is done with the one refilled next
        if (step + T::kStages - 1 < steps) { fetch_w(step + T::kStages - 1); fetch_a(step + T::kStages - 1); }
        mlr_async_commit();
        const float* as = staged + (step % T::kStages) * kStage + ty * T::kLd;
        const float* ws = staged + (step % T::kStages) * kStage + (BM + tx) * T::kLd;
#pragma unroll
        for (int kk = 0; kk < T::kK; kk += 4) {
            float a[TM][4], w[TN][4];
#pragma unroll
            for (int i = 0; i < TM; ++i) mlr_load4(as + i * kDown * T::kLd + kk, a[i]);
#pragma unroll
            for (int j = 0; j < TN; ++j) mlr_load4(ws + j * kAcross * T::kLd + kk, w[j]);
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i][q], w[j][q], acc[i][j]);
        }
    }
    mlr_grid_dependents_may_start();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + i * kDown;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * kAcross;
            if (n < N) C[static_cast<size_t>(m) * ldc + n] = acc[i][j];
        }
    }
}

// ---- up to four rows (a decode step): a pass over W.  A block takes BN rows of W; thread (n, g) has row n of them and the rows g, g + G,
// .. of A, G = 128 / BN.  With `static_w` (no kernel in flight writes W: it holds weights) W's first stages are on their way before the
// kernel before this one has ended.
constexpr int kFewRows = 4, kFewThreads = 128, kFewK = 64, kFewLd = kFewK + 4;
constexpr size_t few_shared(int bn, int stages, int rows) { return sizeof(float) * stages * (bn + rows) * kFewLd; }

template <bool kVector, int BN, int STAGES, int MT>
__global__ void __launch_bounds__(kFewThreads) gemm_f32_few_kernel(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                                                                   int ldc, int static_w) {
    extern __shared__ __align__(16) float staged[];           // per stage: W [BN][kFewLd], A [M][kFewLd]
    constexpr int kGroups = kFewThreads / BN, kChunks = kFewK / 4;
    const int tid = threadIdx.x, n = tid % BN, g = tid / BN;
    const int n0 = blockIdx.x * BN, stage_floats = (BN + M) * kFewLd;
    const int steps = (K + kFewK - 1) / kFewK;
    auto fetch_w = [&](int step) {
        float* to = staged + (step % STAGES) * stage_floats;
#pragma unroll
        for (int i = tid; i < BN * kChunks; i += kFewThreads) {
            const int r = i / kChunks, c = (i % kChunks) * 4;
            stage4<kVector>(to + r * kFewLd + c, n0 + r < N ? W + static_cast<size_t>(n0 + r) * ldw : W, step * kFewK + c, K, n0 + r < N);
        }
    };
    auto fetch_a = [&](int step) {
        float* to = staged + (step % STAGES) * stage_floats + BN * kFewLd;
        for (int i = tid; i < M * kChunks; i += kFewThreads) {
            const int r = i / kChunks, c = (i % kChunks) * 4;
            stage4<kVector>(to + r * kFewLd + c, A + static_cast<size_t>(r) * lda, step * kFewK + c, K, true);
        }
    };
    if (!static_w) mlr_grid_wait();
    for (int step = 0; step < STAGES - 1 && step < steps; ++step) fetch_w(step);
    if (static_w) mlr_grid_wait();
    // The first group to complete holds all of W's first stages and A's first; the later ones A's alone.
    for (int step = 0; step < STAGES - 1; ++step) {
        if (step < steps) fetch_a(step);
        mlr_async_commit();
    }
    float acc[MT] = {};
    for (int step = 0; step < steps; ++step) {
        stages_left<STAGES - 2>();
        __syncthreads();
        if (step + STAGES - 1 < steps) { fetch_w(step + STAGES - 1); fetch_a(step + STAGES - 1); }
        mlr_async_commit();
        if ((tid & ~31) / BN >= M) continue;          // none of this warp's threads has a row of A (it still fetches for the others)
        const float* ws = staged + (step % STAGES) * stage_floats + n * kFewLd;
        const float* as = staged + (step % STAGES) * stage_floats + BN * kFewLd;
#pragma unroll 8
        for (int kk = 0; kk < kFewK; kk += 4) {
            float w[4];
            mlr_load4(ws + kk, w);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                float a[4];
                mlr_load4(as + min(g + i * kGroups, M - 1) * kFewLd + kk, a);
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i] = fmaf(a[q], w[q], acc[i]);
            }
        }
    }
    mlr_grid_dependents_may_start();
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        const int m = g + i * kGroups;
        if (m < M && n0 + n < N) C[static_cast<size_t>(m) * ldc + n0 + n] = acc[i];
    }
}

template <typename Kernel>
int allow_shared(Kernel kernel, size_t bytes) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    return e == cudaSuccess ? 0 : mlr_fail("gemm_f32: cannot use %zu bytes of shared memory: %s", bytes, cudaGetErrorString(e));
}

struct Product {
    const float *A, *W;
    float* C;
    int M, N, K, lda, ldw, ldc, static_w;
    cudaStream_t stream;
};

// Blocks on the busiest SM when a grid is dealt out evenly.
long long busiest_blocks(long long blocks) { return (blocks + mlr_sm_count() - 1) / mlr_sm_count(); }

// Shared memory of a block of which `each` fit an SM and no more.  Blocks are placed while blocks of the kernel before still hold part of the SMs:
// a grid that could have an SM each ends up with two or three on some of them (a product of 129 rows of 6144 x 1024 behind its norm: 129 us, 59 us
// so) unless more do not fit.
size_t shared_for(long long each) {
    constexpr long long kSm = 228 * 1024, kMostOfBlock = 227 * 1024, kReserved = 1024;       // what sm_100 has, gives a block, and keeps of each block's
    return static_cast<size_t>(std::max(0ll, std::min(kMostOfBlock, kSm / each / 128 * 128 - kReserved)));
}

template <bool kVector, typename T>
int launch_tile(const Product& p) {
    const long long blocks = ((p.M + T::kRows - 1LL) / T::kRows) * ((p.N + T::kColumns - 1LL) / T::kColumns);
    MLR_REQUIRE(blocks <= INT_MAX, "gemm_f32: M=%d N=%d need more than %d tiles", p.M, p.N, INT_MAX);
    const size_t bytes = std::max(T::kShared, shared_for(busiest_blocks(blocks)));
    if (allow_shared(gemm_f32_tile_kernel<kVector, T>, shared_for(1))) return 1;         // the same limit at every call: threads may launch side by side
    mlr_launch((gemm_f32_tile_kernel<kVector, T>), dim3(static_cast<unsigned>(blocks)), dim3(T::kThreads), bytes, p.stream, p.A, p.W, p.C, p.M, p.N,
               p.K, p.lda, p.ldw, p.ldc);
    return 0;
}

template <bool kVector, int BN, int STAGES, int MT>
int launch_few(const Product& p) {
    if (allow_shared(gemm_f32_few_kernel<kVector, BN, STAGES, MT>, few_shared(BN, STAGES, kFewRows))) return 1;
    mlr_launch((gemm_f32_few_kernel<kVector, BN, STAGES, MT>), dim3((p.N + BN - 1) / BN), dim3(kFewThreads), few_shared(BN, STAGES, p.M), p.stream, p.A, p.W,
               p.C, p.M, p.N, p.K, p.lda, p.ldw, p.ldc, p.static_w);
    return 0;
}

// What a tile costs a value of K, in cycles, with n blocks on the busiest SM: START + RATE * n, n rounded up to ROUND (2 where blocks run in pairs and a
// block alone takes a pair's time).  The numbers are fits to every tile at 5 to 2048 rows of ten shapes (1024 x 1024 to 151936 x 1024); by them
// the choice is within 1 % of the best tile on average, 9 % at worst.  (Computing them from the registers that are read from shared memory missed the
// largest tile's single round by half: 256 x 4096 x 1024 114 us, with 64 x 64 tiles 66 us.)
template <typename T>
int tile_cost(int M, int N) {
    const long long busiest = busiest_blocks(((M + T::kRows - 1LL) / T::kRows) * ((N + T::kColumns - 1LL) / T::kColumns));
    return static_cast<int>(std::min<long long>(T::kStart + T::kRate * ((busiest + T::kRound - 1) / T::kRound * T::kRound), INT_MAX));
}

template <bool kVector, typename... Tiles>
int launch_cheapest(const Product& p) {
    const int costs[] = {tile_cost<Tiles>(p.M, p.N)...};
    int (*const launches[])(const Product&) = {launch_tile<kVector, Tiles>...};
    int best = 0;
    for (int i = 1; i < static_cast<int>(sizeof...(Tiles)); ++i)
        if (costs[i] < costs[best]) best = i;
    return launches[best](p);
}

template <bool kVector>
int choose(const Product& p) {
    if (p.M <= kFewRows) {
        // Wide blocks where they still give every SM two; with narrow ones a thread's chain of K multiply-adds is the bound, and
        // sixteen stages hold most of its K in flight.
        if (p.N >= 64 * 2 * mlr_sm_count()) return p.M <= 2 ? launch_few<kVector, 64, 4, 1>(p) : launch_few<kVector, 64, 4, 2>(p);
        if (p.N >= 16 * 2 * mlr_sm_count()) return launch_few<kVector, 16, 16, 1>(p);
        return launch_few<kVector, 8, 16, 1>(p);
    }
    return launch_cheapest<kVector, Tile<64, 128, 8, 8, 3, 32, 10, 100, 2>, Tile<48, 128, 6, 8, 3, 32, 30, 74, 1>, Tile<64, 64, 8, 4, 3, 32, 20, 55, 1>,
                           Tile<32, 128, 4, 8, 3, 32, 22, 56, 1>, Tile<32, 64, 4, 4, 4, 32, 20, 30, 1>, Tile<48, 32, 3, 4, 4, 64, 15, 26, 1>,
                           Tile<16, 64, 2, 4, 4, 64, 12, 24, 1>, Tile<16, 128, 8, 4, 4, 32, 2, 41, 2>, Tile<8, 128, 4, 4, 4, 32, 0, 30, 2>,
                           Tile<16, 32, 2, 2, 5, 64, 10, 13, 1>, Tile<8, 32, 1, 2, 5, 64, 7, 11, 1>>(p);
}

int product(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int static_w, cudaStream_t stream) {
    MLR_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    MLR_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: a leading dimension is smaller than its row");
    if (M == 0) return 0;
    const bool vector = lda % 4 == 0 && ldw % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
                        reinterpret_cast<uintptr_t>(W) % 16 == 0;
    const Product p = {A, W, C, M, N, K, lda, ldw, ldc, static_w, stream};
    if (vector ? choose<true>(p) : choose<false>(p)) return 1;
    return mlr_launched("gemm_f32");
}

}  // namespace

MLR_API int mlr_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                         int ldc, cudaStream_t stream) {
    return product(A, W, C, M, N, K, lda, ldw, ldc, 0, stream);
}

// The same for a W that no kernel in flight writes (it holds weights): a few-row product fetches it before the kernels before it are done.
MLR_API int mlr_gemm_f32_weights(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                                 int ldc, cudaStream_t stream) {
    return product(A, W, C, M, N, K, lda, ldw, ldc, 1, stream);
}
