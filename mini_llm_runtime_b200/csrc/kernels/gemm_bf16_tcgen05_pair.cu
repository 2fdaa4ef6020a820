// bfloat16 matrix product for many rows (prompt portions) on pairs of SMs:
//     out[p, q] (+)= sum_k X[p, k] * W[q, k]          (both operands row-major, K contiguous)
// Two thread blocks of a cluster share one 256 x 256 output tile.  Each loads its own 128 rows
// of X and its own 128 rows of W per 64-wide block of K (TMA, 128-byte swizzle); block 0 issues
// one tcgen05.mma.cta_group::2 (M = 256, N = 256, K = 16) per 16 of K, which both SMs' tensor
// cores execute, each reading the other's half of W from its shared memory; each block ends
// up with its 128 rows of the accumulator in its own tensor memory.  Against one block per
// 128 x 256 tile this cuts what every SM fetches from L2 per flop by a third.
//
// Per block six warps, as in the one-block kernel:
//   warp 0      one lane issues the block's TMA loads; their bytes are counted on the "full"
//               barrier of the stage in block 0, which expects both blocks' bytes;
//   warp 1      allocates tensor memory (both blocks' warps together); in block 0 one lane
//               issues the instructions, frees a stage in both blocks with a multicast
//               tcgen05.commit and hands a finished accumulator to both blocks' store warps;
//   warps 2-5   read the block's accumulator rows (tcgen05.ld), apply the epilogue, store, and
//               give the accumulator back to block 0 (a remote arrival for block 1).
// Epilogues: bfloat16 or float32 store; float32 add into `out` (a product that ends a
// sub-layer adds into the residual stream); SiLU gate, for a stacked weight matrix whose rows
// alternate 128 of the gate with the 128 of "up" that belong to the same outputs, so that
// columns c and c + 128 of a tile meet in one thread: out[p, q/2 + c] = silu(g) * u.
// GROUPED: the rows of X are cut into groups (experts), each with a matrix of its own out of a stack [groups * Q, K]; a list on the
// device names the row tiles {group, first row, rows}, and a tile's rows past its group are worked out and not stored.  Plain: float32
// store.  With a gate (routed experts) block 0 loads 128 rows of the first stack and block 1 the same rows of the second, so that again
// columns c and c + 128 of a tile meet in one thread.  Against tiles of 64 rows on mma.sync, gate/up and down together with the gather:
// 15,452 rows of 16 experts of 1024 x 2048: 678 -> 246 us; 6,400 rows of 16 experts of 2048 x 4096: 1044 -> 338 us.
// Every barrier wait gives up after about two seconds, sets MLR_STATUS_TIMEOUT and lets both
// blocks leave through the common exit, which frees the tensor memory.
//
// The reference calls cublasGemmEx for every product (src/minillm/cuda/matrix.cpp:30-36).
#include "expert_gate.cuh"
#include "tcgen05.cuh"

namespace {

using namespace mlr_tc;

constexpr int kThreads = 192;
constexpr int kRows = 128;          // rows of X, and of W, per block and stage
constexpr int kTileK = 64;          // 64 bf16 = 128 bytes = one swizzle row
constexpr int kTileN = 256;         // columns of the pair's tile
constexpr int kOperandBytes = kRows * kTileK * 2;
constexpr int kStageBytes = 2 * kOperandBytes;          // per block
constexpr int kStages = 7;
constexpr int kTmemColumns = 2 * kTileN;                // two accumulators
enum Epilogue : int { kStoreBf16 = 0, kStoreF32 = 1, kAddF32 = 2, kSiluGateBf16 = 3, kSquaredReluBf16 = 4 };

// dst[0..3] += (a, b, c, d), done by the memory system: the thread does not wait for the old
// values.  Every element is added to by exactly one thread, once, so the result does not
// depend on any order (the adder flushes subnormal sums to zero).
__device__ __forceinline__ void add_to_float4(float4* dst, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

struct Groups {
    const int* tiles;           // {group, first row, rows} per tile
    const int* n_tiles;
    ExpertGate gate;            // kind 0: none
};

template <bool GROUPED>
__global__ void __launch_bounds__(kThreads) gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                     const __grid_constant__ CUtensorMap map_w,
                                                                     const __grid_constant__ CUtensorMap map_w2,
                                                                     void* __restrict__ out, long long ldo, int P, int Q, int K,
                                                                     int epilogue, int* status, Groups groups) {
    mlr_grid_dependents_may_start();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long barriers[2 * kStages + 4];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int fault;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_base = smem_u32(barriers);
    auto full_bar = [&](int s) { return bar_base + s * 8; };
    auto empty_bar = [&](int s) { return bar_base + (kStages + s) * 8; };
    auto acc_full_bar = [&](int a) { return bar_base + (2 * kStages + a) * 8; };
    auto acc_empty_bar = [&](int a) { return bar_base + (2 * kStages + 2 + a) * 8; };
    auto tile_x = [&](int s) { return smem_base + s * kStageBytes; };
    auto tile_w = [&](int s) { return smem_base + s * kStageBytes + kOperandBytes; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();          // 0 leads
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    if (threadIdx.x == 0) {
        fault = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);             // used in block 0: its loader's arrival with both blocks' bytes
            mbar_init(empty_bar(s), 1);            // in both blocks: the multicast commit
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full_bar(a), 1);         // in both blocks: the multicast commit
            mbar_init(acc_empty_bar(a), 8);        // used in block 0: four store warps of each block
        }
        mbar_init_done();
    }
    if (warp == 1) tmem_alloc_pair(&tmem_base_slot, kTmemColumns);
    tmem_fence_before();
    cluster_sync();                                // barriers and tensor memory of both blocks exist
    tmem_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    // GROUPED: the list of tiles was written by an earlier kernel; every role reads it after its wait.
    const bool gated = GROUPED && groups.gate.kind != 0;
    const int tile_q = gated ? kTileN / 2 : kTileN;         // columns of the result (and rows of a matrix) a tile stands for
    int tiles_p = (P + 2 * kRows - 1) / (2 * kRows), tiles = 0;
    const int tiles_q = (Q + tile_q - 1) / tile_q;
    auto count_tiles = [&]() {
        if (GROUPED) tiles_p = __ldcg(groups.n_tiles);
        tiles = tiles_p * tiles_q;
    };
    const int k_blocks = (K + kTileK - 1) / kTileK;

    if (warp == 0) {
        // ---------------- loads (each block its halves)
        if (lane == 0) {
            mlr_grid_wait();
            count_tiles();
            bool ok = true;
            int it = 0;
            for (int tile = pair; tile < tiles && ok; tile += pairs) {
                int p0 = (tile % tiles_p) * 2 * kRows + rank * kRows;
                int q0 = (tile / tiles_p) * tile_q + (gated ? 0 : rank * kRows);
                if (GROUPED) {
                    p0 = __ldcg(groups.tiles + 3 * (tile % tiles_p) + 1) + rank * kRows;
                    q0 += __ldcg(groups.tiles + 3 * (tile % tiles_p)) * Q;
                }
                const CUtensorMap* w_map = gated && rank ? &map_w2 : &map_w;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int stage = it % kStages;
                    if (it >= kStages) ok = mbar_wait(empty_bar(stage), ((it / kStages) - 1) & 1);
                    if (!ok) break;
                    if (rank == 0) mbar_expect_tx(full_bar(stage), 2 * kStageBytes);
                    const uint32_t leader_full = in_block_of_rank(full_bar(stage), 0);
                    tma_load_2d_pair(tile_x(stage), &map_x, kb * kTileK, p0, leader_full);
                    tma_load_2d_pair(tile_w(stage), w_map, kb * kTileK, q0, leader_full);
                }
            }
            if (!ok) fault = 2;
        }
    } else if (warp == 1) {
        // ---------------- tensor-core instructions (block 0 only)
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = instruction_descriptor_m256(kTileN);
            if (GROUPED) mlr_grid_wait();
            count_tiles();
            bool ok = true;
            int it = 0, local = 0;
            for (int tile = pair; tile < tiles && ok; tile += pairs, ++local) {
                const int acc = local & 1;
                if (local >= 2) ok = mbar_wait(acc_empty_bar(acc), ((local >> 1) - 1) & 1);
                if (!ok) break;
                tmem_fence_after();
                const uint32_t tmem_d = tmem_base + acc * kTileN;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int stage = it % kStages;
                    ok = mbar_wait(full_bar(stage), (it / kStages) & 1);
                    if (!ok) break;
                    tmem_fence_after();
                    const uint64_t desc_x = smem_descriptor(tile_x(stage)), desc_w = smem_descriptor(tile_w(stage));
#pragma unroll
                    for (int k = 0; k < kTileK / 16; ++k)
                        umma_bf16_pair(tmem_d, desc_x + 2 * k, desc_w + 2 * k, idesc, kb > 0 || k > 0);
                    umma_commit_pair(empty_bar(stage), 3);      // both blocks' loaders may refill the stage
                }
                if (!ok) break;
                umma_commit_pair(acc_full_bar(acc), 3);         // both blocks' store warps may read
            }
            if (!ok) fault = 2;
        }
    } else {
        // ---------------- stores: warp w reads lanes 32 (w % 4) .. of this block's accumulator rows
        const int quarter = warp & 3;
        mlr_grid_wait();
        count_tiles();
        const uint32_t leader_acc_empty[2] = {in_block_of_rank(acc_empty_bar(0), 0), in_block_of_rank(acc_empty_bar(1), 0)};
        bool ok = true;
        int local = 0;
        for (int tile = pair; tile < tiles; tile += pairs, ++local) {
            const int acc = local & 1;
            int p = (tile % tiles_p) * 2 * kRows + rank * kRows + quarter * 32 + lane, p_end = P;
            const int q0 = (tile / tiles_p) * tile_q;
            if (GROUPED) {
                const int* at = groups.tiles + 3 * (tile % tiles_p);
                p = __ldcg(at + 1) + rank * kRows + quarter * 32 + lane;
                p_end = __ldcg(at + 1) + __ldcg(at + 2);
            }
            ok = __all_sync(0xffffffffu, mbar_wait(acc_full_bar(acc), (local >> 1) & 1));     // the whole warp goes on, or none of it
            if (!ok) break;
            tmem_fence_after();
            const uint32_t row_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * kTileN;
            if (gated) {
                // Columns c (first matrix) and c + 128 (second) of the tile give output column q0 + c.
                __nv_bfloat16* dst_row = static_cast<__nv_bfloat16*>(out) + static_cast<size_t>(p) * ldo + q0;
                const int width = Q - q0;
#pragma unroll 2
                for (int c = 0; c < kTileN / 2; c += 16) {
                    uint32_t g[16], u[16];
                    __syncwarp();           // the load takes the whole warp, rows past the tile's last one included
                    tmem_load16(row_base + c, g);
                    tmem_load16(row_base + kTileN / 2 + c, u);
                    if (p >= p_end) continue;
                    uint32_t w[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const __nv_bfloat162 h = __floats2bfloat162_rn(expert_gate(__uint_as_float(g[2 * j]), __uint_as_float(u[2 * j]), groups.gate),
                                                                       expert_gate(__uint_as_float(g[2 * j + 1]), __uint_as_float(u[2 * j + 1]), groups.gate));
                        w[j] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    if (c + 16 <= width && (ldo & 7) == 0) {
                        uint4* dst = reinterpret_cast<uint4*>(dst_row + c);
                        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c + j < width) dst_row[c + j] = reinterpret_cast<const __nv_bfloat16*>(w)[j];
                    }
                }
            } else if (epilogue == kSiluGateBf16) {
                // Columns c (gate) and c + 128 (up) of the tile give output column q0 / 2 + c.
                __nv_bfloat16* dst_row = static_cast<__nv_bfloat16*>(out) + static_cast<size_t>(p) * ldo + q0 / 2;
                const int width = Q / 2 - q0 / 2;       // output columns left from this tile's first
#pragma unroll 2
                for (int c = 0; c < kTileN / 2; c += 16) {
                    uint32_t g[16], u[16];
                    __syncwarp();           // as above
                    tmem_load16(row_base + c, g);
                    tmem_load16(row_base + kTileN / 2 + c, u);
                    if (p < P) {
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            // The gate is rounded to bfloat16 first, as the unfused path stores it.
                            const float gate = __bfloat162float(__float2bfloat16_rn(__uint_as_float(g[j])));
                            const float up = __bfloat162float(__float2bfloat16_rn(__uint_as_float(u[j])));
                            v[j] = __fdividef(gate, 1.0f + __expf(-gate)) * up;
                        }
                        if (c + 16 <= width && (ldo & 7) == 0) {
                            uint32_t w[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                                w[j] = *reinterpret_cast<const uint32_t*>(&h);
                            }
                            uint4* dst = reinterpret_cast<uint4*>(dst_row + c);
                            dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                            dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (c + j < width) dst_row[c + j] = __float2bfloat16_rn(v[j]);
                        }
                    }
                }
            } else {
#pragma unroll 4
                for (int c = 0; c < kTileN; c += 16) {
                    uint32_t r[16];
                    __syncwarp();           // as above
                    tmem_load16(row_base + c, r);
                    if (p >= p_end) continue;
                    const bool whole = q0 + c + 16 <= Q && (ldo & 7) == 0;
                    if (epilogue == kSquaredReluBf16) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const float v = fmaxf(__uint_as_float(r[j]), 0.0f);
                            r[j] = __float_as_uint(v * v);
                        }
                    }
                    if (epilogue == kStoreBf16 || epilogue == kSquaredReluBf16) {
                        __nv_bfloat16* dst_row = static_cast<__nv_bfloat16*>(out) + static_cast<size_t>(p) * ldo + q0 + c;
                        if (whole) {
                            uint32_t w[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
                                w[j] = *reinterpret_cast<const uint32_t*>(&h);
                            }
                            uint4* dst = reinterpret_cast<uint4*>(dst_row);
                            dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                            dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (q0 + c + j < Q) dst_row[j] = __float2bfloat16_rn(__uint_as_float(r[j]));
                        }
                    } else {
                        float* dst_row = static_cast<float*>(out) + static_cast<size_t>(p) * ldo + q0 + c;
                        const bool add = epilogue == kAddF32;
                        if (whole) {
                            float4* dst = reinterpret_cast<float4*>(dst_row);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                if (add)
                                    add_to_float4(dst + j, __uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                  __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                                else
                                    dst[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                         __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (q0 + c + j < Q) dst_row[j] = __uint_as_float(r[j]) + (add ? dst_row[j] : 0.0f);
                        }
                    }
                }
            }
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_acc_empty[acc]);
        }
        if (!ok) fault = 2;
    }
    tmem_fence_before();
    __syncthreads();
    if (fault && warp == 1) {
        // Give work that may still be in flight time to finish before the memory goes back.
        for (int i = 0; i < 100; ++i) __nanosleep(1000);
    }
    cluster_sync();                                // neither block's memory goes away under the other
    if (warp == 1) tmem_free_pair(tmem_base, kTmemColumns);
    if (fault && threadIdx.x == 0 && status) atomicOr(status, MLR_STATUS_TIMEOUT);
}

int make_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld) {
    EncodeTiled encode = encode_tiled();
    MLR_REQUIRE(encode != nullptr, "gemm_bf16_tcgen05_pair: the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    const cuuint32_t box[2] = {kTileK, kRows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    MLR_REQUIRE(r == CUDA_SUCCESS, "gemm_bf16_tcgen05_pair: cuTensorMapEncodeTiled failed with code %d", static_cast<int>(r));
    return 0;
}

int sm_count() {
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms;
}

template <bool GROUPED>
int launch(const CUtensorMap& map_x, const CUtensorMap& map_w, const CUtensorMap& map_w2, int pairs, void* out, long long ldo, int P, int Q, int K,
           int epilogue, int* status, const Groups& groups, cudaStream_t stream) {
    const size_t bytes = static_cast<size_t>(kStages) * kStageBytes + 1024;
    static thread_local bool allowed = false;
    if (!allowed) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_pair_kernel<GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(bytes));
        if (e != cudaSuccess) return mlr_fail("gemm_bf16_tcgen05_pair: cannot use %zu bytes of shared memory: %s", bytes, cudaGetErrorString(e));
        allowed = true;
    }
    mlr_launch_cluster(gemm_tcgen05_pair_kernel<GROUPED>, dim3(2 * pairs), dim3(kThreads), 2, bytes, stream, map_x, map_w, map_w2, out, ldo, P, Q, K,
                       epilogue, status, groups);
    return mlr_launched("gemm_bf16_tcgen05_pair");
}

}  // namespace

// out[p, q] = sum_k X[p, k] W[q, k] for X [P, K] (row stride ldx) and W [Q, K] (row stride ldw),
// bfloat16.  epilogue: 0 stores bfloat16, 1 stores float32, 2 adds into float32 `out`, 3 takes
// W as 128 gate rows alternating with their 128 "up" rows (Q a multiple of 256) and stores
// bfloat16 silu(gate) * up at out[p, Q / 2 columns], 4 stores bfloat16 relu(x)^2.  Row stride of out: ldo elements.
MLR_API int mlr_gemm_bf16_tcgen05_pair(const void* X, long long ldx, int P, const void* W, long long ldw, int Q, int K, void* out,
                                       long long ldo, int epilogue, int* status, cudaStream_t stream) {
    MLR_REQUIRE(epilogue >= 0 && epilogue <= 4, "gemm_bf16_tcgen05_pair: epilogue must be 0..4, got %d", epilogue);
    MLR_REQUIRE(P >= 1 && Q >= 1 && K >= 8, "gemm_bf16_tcgen05_pair: bad sizes P=%d Q=%d K=%d", P, Q, K);
    MLR_REQUIRE(K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 && ldx >= K && ldw >= K,
                "gemm_bf16_tcgen05_pair: K and the operand row strides must be multiples of 8 elements (16 bytes), got K=%d", K);
    MLR_REQUIRE(reinterpret_cast<uintptr_t>(X) % 16 == 0 && reinterpret_cast<uintptr_t>(W) % 16 == 0,
                "gemm_bf16_tcgen05_pair: the operands must be 16-byte aligned");
    MLR_REQUIRE(epilogue != kSiluGateBf16 || Q % 256 == 0, "gemm_bf16_tcgen05_pair: the gated epilogue wants Q %% 256 == 0, got %d", Q);
    MLR_REQUIRE(ldo >= (epilogue == kSiluGateBf16 ? Q / 2 : Q), "gemm_bf16_tcgen05_pair: the output row stride is smaller than the row");
    MLR_REQUIRE(reinterpret_cast<uintptr_t>(out) % 16 == 0, "gemm_bf16_tcgen05_pair: the output must be 16-byte aligned");
    CUtensorMap map_x, map_w;
    if (int e = make_map(&map_x, X, P, K, ldx)) return e;
    if (int e = make_map(&map_w, W, Q, K, ldw)) return e;
    const int tiles = ((P + 2 * kRows - 1) / (2 * kRows)) * ((Q + kTileN - 1) / kTileN), most = sm_count() / 2;
    return launch<false>(map_x, map_w, map_w, tiles < most ? tiles : most, out, ldo, P, Q, K, epilogue, status, Groups{}, stream);
}

// Products of groups of rows with a matrix each.  X: bfloat16 [P, K], P = rows * top, a group's rows side by side; W (and W2 with a gate): bfloat16
// [groups, Q, K]; tiles, n_tiles (device memory): {group, first row, rows} of every row tile, a tile being at most 256 rows of one group.
// out: without a gate (gate_kind 0) float32 [P, Q] = x W^T; with one bfloat16 [P, Q] = gate(x W^T, x W2^T), 1: silu(g) * u,
// 2: the clamped shape of alpha, limit and up_offset.
MLR_API int mlr_grouped_product_bf16(const void* X, long long ldx, int rows, int top, const void* W, const void* W2, int groups, int gate_kind, int Q, int K, void* out,
                                     long long ldo, const int* tiles, const int* n_tiles, float alpha, float limit, float up_offset, int* status,
                                     cudaStream_t stream) {
    MLR_REQUIRE(X && W && out && tiles && n_tiles && (gate_kind == 0 || W2) && gate_kind >= 0 && gate_kind <= 2, "grouped_product_bf16: bad arguments");
    if (rows <= 0) return 0;
    const int P = rows * top;
    MLR_REQUIRE(P >= 1 && Q >= 1 && groups >= 1 && K >= 8 && K % 8 == 0 && ldx % 8 == 0 && ldx >= K && ldo >= Q,
                "grouped_product_bf16: bad sizes P=%d Q=%d K=%d (K and the row stride of X are multiples of 8)", P, Q, K);
    const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    MLR_REQUIRE(aligned(X) && aligned(W) && aligned(W2) && aligned(out), "grouped_product_bf16: the operands must be 16-byte aligned");
    CUtensorMap map_x, map_w, map_w2;
    if (int e = make_map(&map_x, X, P, K, ldx)) return e;
    if (int e = make_map(&map_w, W, static_cast<long long>(groups) * Q, K, K)) return e;
    if (int e = make_map(&map_w2, gate_kind ? W2 : W, static_cast<long long>(groups) * Q, K, K)) return e;
    const Groups list = {tiles, n_tiles, {gate_kind, alpha, limit, up_offset}};
    return launch<true>(map_x, map_w, map_w2, sm_count() / 2, out, ldo, P, Q, K, kStoreF32, status, list, stream);
}
