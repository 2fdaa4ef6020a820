// The prompt portions of `attention_masked.cu` on the fifth-generation tensor cores: what that file's head says of masks, scores, sinks,
// rotation, gates and the cache holds here, for bfloat16, one attention map a head, key rows of up to 128 values and tiles of 128 query rows.
//
// One block per (128 query rows of one request, query head); two blocks share an SM.  Six warps, as in `attention_tcgen05.cu`:
//   warps 0-3   thread t owns query row t.  First the rows themselves: rotated in float32, rounded to bfloat16 and stored to shared
//               memory with the 128-byte swizzle.  Then per tile of 64 keys: its 64 scores from tensor memory, scaled (or capped),
//               biased, masked; the running maximum in log2 units (the accumulator is rescaled only when it grows by more than
//               2^8) and the sum in float32; the weights back to tensor memory as TWO bfloat16 terms (p = hi + lo, 16 bits of
//               mantissa) over the scores' 64 columns; at the end the division by the sum, the gate and the store.
//   warp 4      TMA copies of the keys and values of a tile through tensor maps over the paged cache (128-byte swizzle, one box
//               per page and 64 values; a row's values past its end read as zero).
//   warp 5      one lane issues tcgen05.mma: S = Q K^T (M 128, N 64) into one of two score buffers; O += hi V and O += lo V
//               (M 128, N value size) with the weights read from tensor memory.  S of the next tile is issued first.
// Values that are the start of their keys (shared_kv) are read from the keys' tile, which then has four stages instead of two.
// Rows of a tile that no query of the block may see are not copied; their values are zeroed before P V (0 * garbage must stay 0).
// Every wait gives up after about two seconds and sets MLR_STATUS_TIMEOUT; the block then leaves through the common exit.
//
// Tiles of 64 rows on `mma.sync` (a block of four warps, an eighth of the tensor cores' rate, scores and weights through registers) were
// bound by the issue of those instructions and their fragment loads.  2048 rows, window 1024: 32 heads of 128 with a cap 439 -> 117 us, 32
// heads over latents of 128 (values 96) 264 -> 84 us, 16 rotated and gated heads of 128 209 -> 67 us.
#include "attention_spec.cuh"
#include "tcgen05.cuh"

#include <type_traits>

namespace {

using namespace mlr_tc;

constexpr int kThreads = 192;
constexpr int kRows = 128;          // query rows per block
constexpr int kKeys = 64;           // keys per tile
constexpr int kRowBytes = 128;      // of a row's 64 values in shared memory
constexpr int kQHalfBytes = kRows * kRowBytes, kTileHalfBytes = kKeys * kRowBytes;
constexpr int kTmemColumns = 256;   // O: 128, two score buffers of 64
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleStep = 8.0f;    // log2 units by which the maximum may lag

enum Barrier { kQFull = 0, kKFull = 1, kKEmpty = 5, kVFull = 9, kVEmpty = 11, kSFull = 13, kPFull = 15, kODone = 17, kBarriers = 18 };

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float exp2_raw(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, int w, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ int first_visible(int position, const MaskedAttentionSpec& s) {
    int lo = 0;
    if (s.window > 0) lo = max(lo, position - s.window + 1);
    if (s.chunk > 0) lo = max(lo, (position / s.chunk) * s.chunk);
    return lo;
}
__device__ __forceinline__ float gate_value(float g, int kind) {
    const float sig = 1.0f / (1.0f + expf(-g));
    return kind == 2 ? g * sig : sig;
}

// KH, VH: pieces of 64 values of a key and of a value.
template <int KH, int VH, bool SHARED>
__global__ void __launch_bounds__(kThreads, 2) attention_masked_wide_kernel(const __grid_constant__ CUtensorMap map_k,
                                                                            const __grid_constant__ CUtensorMap map_v, const __nv_bfloat16* q,
                                                                            int ldq, const __nv_bfloat16* gate, int ld_gate, int gate_octets,
                                                                            __nv_bfloat16* out, int ldo, int num_pages, const int* tiles,
                                                                            const int* segment_info, const int* block_table, int table_stride,
                                                                            int page_size, MaskedAttentionSpec s, int* status) {
    mlr_grid_wait();
    constexpr int kStages = SHARED ? 4 : 2;
    constexpr int kQBytes = KH * kQHalfBytes, kKBytes = KH * kTileHalfBytes, kVBytes = VH * kTileHalfBytes;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long barriers[kBarriers];
    __shared__ uint32_t tmem_slot;
    __shared__ int bad_page, gave_up;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char* smem_ptr = smem_raw + (smem_base - smem_u32(smem_raw));
    auto k_offset = [&](int stage) { return kQBytes + stage * kKBytes; };
    auto v_offset = [&](int stage) { return SHARED ? k_offset(stage) : kQBytes + kStages * kKBytes + stage * kVBytes; };
    const uint32_t bar_base = smem_u32(barriers);
    auto bar = [&](int which, int i = 0) { return bar_base + (which + i) * 8; };

    const int head = blockIdx.x, kv_head = head / (s.heads / s.kv_heads);
    const int segment = tiles[blockIdx.y * 2], tile_token = tiles[blockIdx.y * 2 + 1];
    const int first = segment_info[segment * 4], count = segment_info[segment * 4 + 1], start = segment_info[segment * 4 + 2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile_rows = min(kRows, count - tile_token);
    const int first_pos = start + tile_token, last_pos = first_pos + tile_rows - 1;
    const int lo_min = first_visible(first_pos, s), keep_first = s.window > 0 ? s.keep_first : 0;
    // Tiles of keys in the order they are walked: those of the kept first tokens that lie before the window's first tile, then the others.
    const int kt_first = lo_min / kKeys * kKeys;
    const int early_tiles = (min(keep_first, kt_first) + kKeys - 1) / kKeys;
    const int n_tiles = early_tiles + (last_pos - kt_first) / kKeys + 1;
    auto tile_start = [&](int j) { return j < early_tiles ? j * kKeys : kt_first + (j - early_tiles) * kKeys; };

    if (threadIdx.x == 0) {
        bad_page = 0;
        gave_up = 0;
        for (int i = 0; i < kBarriers; ++i) mbar_init(bar(i), i == kQFull || i == kPFull || i == kPFull + 1 ? 4 : 1);
        mbar_init_done();
    }
    if (warp == 5) tmem_alloc(&tmem_slot, kTmemColumns);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem_o = tmem_slot;
    auto tmem_s = [&](int b) { return tmem_o + 128 + b * kKeys; };     // scores; then hi over the first 32 columns and lo over the others
    auto wait = [&](uint32_t b, uint32_t parity) {
        if (mbar_wait(b, parity, &gave_up)) return true;
        gave_up = 1;
        return false;
    };

    if (warp == 4) {
        // ---------------- loads.  Lane 2 i + h copies piece h of the rows [i * rows_per_copy, ..) of a tile.
        const int page_shift = 31 - __clz(page_size), rows_per_copy = min(page_size, kKeys);
        const int sub = lane >> 1, half = lane & 1;
        const int* table = block_table + static_cast<size_t>(segment) * table_stride;
        constexpr int kNotMine = -2;
        auto lookup = [&](int j) {          // the page, two tiles ahead of its use
            const int row0 = (j < n_tiles ? tile_start(j) : 0) + sub * rows_per_copy;
            if (j >= n_tiles || sub * rows_per_copy >= kKeys || row0 > last_pos || (row0 + rows_per_copy <= lo_min && row0 >= keep_first)) return kNotMine;
            return __ldg(table + (row0 >> page_shift));
        };
        auto issue = [&](int j, bool value, int page) {
            const int stage = j % kStages;
            const bool mine = page != kNotMine && half < (value ? VH : KH);
            const unsigned mask = __ballot_sync(0xffffffffu, mine);
            const uint32_t full = bar(value ? kVFull : kKFull, stage);
            if (lane == 0) mbar_expect_tx(full, __popc(mask) * rows_per_copy * kRowBytes);
            __syncwarp();
            if (mine) {
                if (page < 0 || page >= num_pages) {
                    bad_page = 1;
                    page = 0;               // still copy something so that the tile's byte count is met
                }
                const int in_page = (tile_start(j) + sub * rows_per_copy) & (page_size - 1);
                const uint32_t dst = smem_base + (value ? v_offset(stage) : k_offset(stage)) + half * kTileHalfBytes + sub * rows_per_copy * kRowBytes;
                if (value) tma_load_4d(dst, &map_v, half * 64, in_page, kv_head, page, full);
                else tma_load_4d(dst, &map_k, half * 64, in_page, kv_head, page, full);
            }
        };
        int page_now = lookup(0), page_next = lookup(1);
        bool ok = true;
        if constexpr (SHARED) {
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int page_after = lookup(j + 2);
                if (j >= kStages) ok = wait(bar(kKEmpty, j % kStages), ((j / kStages) - 1) & 1);
                if (!ok) break;
                issue(j, false, page_now);
                page_now = page_next;
                page_next = page_after;
            }
        } else {
            issue(0, false, page_now);
            for (int j = 0; j < n_tiles && ok; ++j) {
                if (j + 1 < n_tiles) {
                    if (j + 1 >= 2) ok = wait(bar(kKEmpty, (j + 1) & 1), (((j + 1) >> 1) - 1) & 1);
                    if (!ok) break;
                    issue(j + 1, false, page_next);
                }
                const int page_after = lookup(j + 2);
                if (j >= 2) ok = wait(bar(kVEmpty, j & 1), ((j >> 1) - 1) & 1);
                if (!ok) break;
                issue(j, true, page_now);
                page_now = page_next;
                page_next = page_after;
            }
        }
    } else if (warp == 5) {
        // ---------------- tensor-core instructions
        if (lane == 0) {
            constexpr uint32_t idesc_s = instruction_descriptor(kKeys);
            const uint32_t idesc_o = instruction_descriptor((s.vdim + 15) / 16 * 16, true);
            bool ok = wait(bar(kQFull), 0);
            // Descriptors of the tiles, made once: an instruction adds a constant to them.
            const uint64_t desc_q = smem_descriptor(smem_base);
            uint64_t desc_k[kStages], desc_v[kStages];
#pragma unroll
            for (int i = 0; i < kStages; ++i) {
                desc_k[i] = smem_descriptor(smem_base + k_offset(i));
                desc_v[i] = smem_descriptor(smem_base + v_offset(i), kTileHalfBytes, 1024);
            }
            auto of_stage = [](const uint64_t (&d)[kStages], int stage) {
                uint64_t v = d[0];
#pragma unroll
                for (int i = 1; i < kStages; ++i)
                    if (stage == i) v = d[i];
                return v;
            };
            // A key's values past its end are zeros in both operands: whole pieces of 64.
            auto issue_s = [&](int j) {
                const int stage = j % kStages;
                if (!wait(bar(kKFull, stage), (j / kStages) & 1)) return false;
                tmem_fence_after();
                const uint32_t tmem_d = tmem_s(j & 1);
                const uint64_t dk = of_stage(desc_k, stage);
#pragma unroll
                for (int h = 0; h < KH; ++h)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint64_t da = desc_q + (h * (kQHalfBytes >> 4) + 2 * k), db = dk + (h * (kTileHalfBytes >> 4) + 2 * k);
                        if (h == 0 && k == 0) umma_bf16(tmem_d, da, db, idesc_s, 0u);
                        else umma_bf16(tmem_d, da, db, idesc_s, 1u);
                    }
                if (!SHARED) umma_commit(bar(kKEmpty, stage));
                umma_commit(bar(kSFull, j & 1));
                return true;
            };
            if (ok) ok = issue_s(0);
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int stage = j % kStages;
                if (j + 1 < n_tiles) ok = issue_s(j + 1);
                if (!ok) break;
                ok = wait(bar(kPFull, j & 1), (j >> 1) & 1);
                if (!SHARED && ok) ok = wait(bar(kVFull, stage), (j / kStages) & 1);
                if (!ok) break;
                tmem_fence_after();
                // hi: 32 columns of two weights each, then lo; four steps of 16 keys each.
                const uint32_t tmem_p = tmem_s(j & 1);
                const uint64_t dv = of_stage(desc_v, stage);
                umma_bf16_tmem_a(tmem_o, tmem_p, dv, idesc_o, j > 0);
#pragma unroll
                for (int k = 1; k < 8; ++k) umma_bf16_tmem_a(tmem_o, tmem_p + 8 * k, dv + (k & 3) * ((16 * kRowBytes) >> 4), idesc_o, 1u);
                umma_commit(bar(SHARED ? kKEmpty : kVEmpty, stage));
                umma_commit(bar(kODone));
            }
        }
    } else {
        // ---------------- a thread per query row
        const int row = threadIdx.x, pos = first_pos + row;
        const bool valid = row < tile_rows;
        const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
        {
            // The row, rotated, to shared memory: 16-byte piece c of 64 values sits at c ^ (row & 7).
            const __nv_bfloat16* from = q + static_cast<size_t>(first + tile_token + (valid ? row : 0)) * ldq + static_cast<size_t>(head) * s.dim;
            const int rotated = s.rot_dims / 16;            // pieces of the first half of the rotated values
            auto load8 = [&](int c, float (&v)[8]) {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = 0.0f;
                if (valid && c * 8 < s.dim) mlr_load8(from + c * 8, v);
            };
            auto store8 = [&](int c, const float (&v)[8]) {
                *reinterpret_cast<uint4*>(smem_ptr + (c >> 3) * kQHalfBytes + row * kRowBytes + (((c & 7) ^ (row & 7)) << 4)) =
                    make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
            };
            for (int c = 0; c < rotated; ++c) {
                float a[8], b[8], x[8], y[8];
                load8(c, a);
                load8(c + rotated, b);
#pragma unroll 1
                for (int e = 0; e < 8; ++e) {               // the angle's functions are long: they stand once
                    float sn, cs;
                    sincosf(static_cast<float>(pos) * s.freq[c * 8 + e], &sn, &cs);
                    float u = 0.0f, v = 0.0f;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (i == e) u = a[i], v = b[i];
                    }
                    const float first_value = u * cs - v * sn, second_value = v * cs + u * sn;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (i == e) x[i] = first_value, y[i] = second_value;
                    }
                }
                store8(c, x);
                store8(c + rotated, y);
            }
            for (int c = 2 * rotated; c < KH * 8; ++c) {
                float a[8];
                load8(c, a);
                store8(c, a);
            }
            fence_async_proxy();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kQFull));
        }
        const int lo = first_visible(pos, s);
        const bool capped = s.softcap > 0.0f;
        const float slope = s.slopes ? s.slopes[head] * kLog2e : 0.0f;
        // Without a cap a score in log2 units is raw * to_score; with one it is cap - 2 cap / (2^(raw * to_score) + 1), times log2(e).
        const float to_score = capped ? 2.0f * kLog2e * s.scale / s.softcap : s.scale * kLog2e;
        const float cap = s.softcap * kLog2e;
        float m_ref = s.sink ? (s.sinks ? s.sinks[head] : 0.0f) * kLog2e : -INFINITY, l = s.sink ? 1.0f : 0.0f;
        bool ok = true;
        for (int j = 0; j < n_tiles; ++j) {
            const int b = j & 1, key0 = tile_start(j);
            ok = __all_sync(0xffffffffu, wait(bar(kSFull, b), (j >> 1) & 1));
            if (!ok) break;
            tmem_fence_after();
            uint32_t raw[64];
            tmem_load32_nowait(tmem_s(b) + lane_base, raw);
            tmem_load32_nowait(tmem_s(b) + lane_base + 32, raw + 32);
            tmem_load_wait();
            // A tile that every row of the warp sees whole needs no mask.
            const bool open = key0 + kKeys - 1 <= first_pos + warp * 32 && key0 >= first_visible(first_pos + warp * 32 + 31, s);
            float part_max[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            auto shape = [&](auto capped_tag, auto masked_tag) {
                constexpr bool kCapped = decltype(capped_tag)::value, kMasked = decltype(masked_tag)::value;
                const float back = slope * static_cast<float>(key0 - pos);
#pragma unroll
                for (int c = 0; c < 64; ++c) {
                    float x = __uint_as_float(raw[c]) * to_score;
                    if (kCapped) {
                        float r;
                        asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(exp2_raw(x) + 1.0f));
                        x = fmaf(-2.0f * cap, r, cap);
                    }
                    if (s.slopes) x += fmaf(slope, static_cast<float>(c), back);
                    if (kMasked) {
                        const int key = key0 + c;
                        if (key > pos || (key < lo && key >= keep_first)) x = -INFINITY;
                    }
                    raw[c] = __float_as_uint(x);
                    part_max[c & 3] = fmaxf(part_max[c & 3], x);
                }
            };
            if (capped) {
                if (open) shape(std::true_type{}, std::false_type{});
                else shape(std::true_type{}, std::true_type{});
            } else {
                if (open) shape(std::false_type{}, std::false_type{});
                else shape(std::false_type{}, std::true_type{});
            }
            const float m_tile = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3]));
            const bool grow = m_tile > m_ref + kRescaleStep || (m_ref == -INFINITY && m_tile > -INFINITY);
            // P V of the tile before is waited for once per tile, in order (a wait by parity can tell a phase only from the one before it).
            bool o_seen = j == 0;
            if (__any_sync(0xffffffffu, grow)) {
                const float m_new = grow ? m_tile : m_ref;
                const float alpha = grow ? exp2_raw(m_ref - m_new) : 1.0f;
                m_ref = m_new;
                l *= alpha;
                if (j > 0) {
                    ok = __all_sync(0xffffffffu, wait(bar(kODone), (j - 1) & 1));
                    if (!ok) break;
                    o_seen = true;
                    tmem_fence_after();
#pragma unroll
                    for (int c = 0; c < VH * 64; c += 32) {
                        if (c >= s.vdim) continue;
                        uint32_t o[32];
                        tmem_load32_nowait(tmem_o + lane_base + c, o);
                        tmem_load_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_store32(tmem_o + lane_base + c, o);
                    }
                }
            }
            const float m_use = m_ref == -INFINITY ? 0.0f : m_ref;
            float sum[4] = {};
#pragma unroll
            for (int piece = 0; piece < 2; ++piece) {
                uint32_t hi[16], lo_term[16];
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    const float p0 = exp2_raw(__uint_as_float(raw[piece * 32 + c]) - m_use), p1 = exp2_raw(__uint_as_float(raw[piece * 32 + c + 1]) - m_use);
                    sum[(c >> 1) & 3] += p0 + p1;
                    const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
                    const float2 back = __bfloat1622float2(h);
                    hi[c >> 1] = *reinterpret_cast<const uint32_t*>(&h);
                    lo_term[c >> 1] = pack_bf16(p0 - back.x, p1 - back.y);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) raw[piece * 32 + i] = hi[i], raw[piece * 32 + 16 + i] = lo_term[i];
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            {
                uint32_t terms[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) terms[i] = raw[(i >> 4) * 32 + (i & 15)];
                tmem_store32(tmem_s(b) + lane_base, terms);
#pragma unroll
                for (int i = 0; i < 32; ++i) terms[i] = raw[(i >> 4) * 32 + 16 + (i & 15)];
                tmem_store32(tmem_s(b) + lane_base + 32, terms);
            }
            // Rows of values that no query of the block may see become zero.
            if (key0 + kKeys - 1 > last_pos || (key0 < lo_min && key0 + kKeys > keep_first)) {
                const int stage = j % kStages;
                ok = __all_sync(0xffffffffu, wait(bar(SHARED ? kKFull : kVFull, stage), (j / kStages) & 1));
                if (!ok) break;
                constexpr int kPieces = (SHARED ? KH : VH) * 8;
                for (int i = threadIdx.x; i < kKeys * kPieces; i += 128) {
                    const int key_row = i / kPieces, piece = i % kPieces, key = key0 + key_row;
                    if (key > last_pos || (key < lo_min && key >= keep_first))
                        *reinterpret_cast<uint4*>(smem_ptr + v_offset(stage) + (piece >> 3) * kTileHalfBytes + key_row * kRowBytes + (piece & 7) * 16) =
                            make_uint4(0u, 0u, 0u, 0u);
                }
                fence_async_proxy();
            }
            if (!o_seen) {
                ok = __all_sync(0xffffffffu, wait(bar(kODone), (j - 1) & 1));
                if (!ok) break;
            }
            tmem_store_wait();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kPFull, b));
        }
        if (ok) ok = __all_sync(0xffffffffu, wait(bar(kODone), (n_tiles - 1) & 1));
        if (ok) {
            tmem_fence_after();
            const size_t out_row = static_cast<size_t>(first + tile_token + (valid ? row : 0));
            float scale = l > 0.0f ? s.out_scale / l : 0.0f;
            if (gate && s.gate_kind == 3) scale *= gate_value(__bfloat162float(gate[out_row * ld_gate + head]), 3);
            const __nv_bfloat16* gate_row = gate ? gate + out_row * ld_gate + static_cast<size_t>(head) * s.vdim : nullptr;
            __nv_bfloat16* dst = out + out_row * ldo + static_cast<size_t>(head) * s.vdim;
#pragma unroll
            for (int c = 0; c < VH * 64; c += 32) {
                if (c >= s.vdim) continue;
                uint32_t o[32];
                tmem_load32_nowait(tmem_o + lane_base + c, o);
                tmem_load_wait();
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    if (!valid || c + i >= s.vdim) continue;
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(o[i + e]) * scale;
                    if (gate && s.gate_kind != 3) {
                        float g[8];
                        if (gate_octets) {
                            mlr_load8(gate_row + c + i, g);
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; ++e) g[e] = __bfloat162float(gate_row[c + i + e]);
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] *= gate_value(g[e], s.gate_kind);
                    }
                    mlr_store8(dst + c + i, v);
                }
                __syncwarp();           // the next load takes the whole warp
            }
        }
    }
    tmem_fence_before();
    mlr_grid_dependents_may_start();
    __syncthreads();
    if (warp == 5) {
        if (gave_up) {
            // Give work that may still be in flight time to finish before the memory goes back.
            for (int i = 0; i < 100; ++i) __nanosleep(1000);
        }
        tmem_free(tmem_o, kTmemColumns);
    }
    if (threadIdx.x == 0 && status && (gave_up || bad_page))
        atomicOr(status, (gave_up ? MLR_STATUS_TIMEOUT : 0) | (bad_page ? MLR_STATUS_BAD_PAGE : 0));
}

// Rows of `width` values of one kind in every page, as [value][token in page][kv head][page]: boxes of 64 values of up to 64 tokens.
int cache_map(CUtensorMap* map, const __nv_bfloat16* base, int width, int page_size, int kv_heads, int num_pages, size_t page_elems) {
    EncodeTiled encode = encode_tiled();
    MLR_REQUIRE(encode != nullptr, "attention_masked_wide: the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(width), static_cast<cuuint64_t>(page_size), static_cast<cuuint64_t>(kv_heads),
                                static_cast<cuuint64_t>(num_pages)};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(width) * 2, static_cast<cuuint64_t>(page_size) * width * 2, page_elems * 2};
    const cuuint32_t box[4] = {64, static_cast<cuuint32_t>(page_size < kKeys ? page_size : kKeys), 1, 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(base), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    MLR_REQUIRE(r == CUDA_SUCCESS, "attention_masked_wide: cuTensorMapEncodeTiled failed with code %d", static_cast<int>(r));
    return 0;
}

template <int KH, int VH, bool SHARED>
int launch(const CUtensorMap& map_k, const CUtensorMap& map_v, const void* q, int ldq, const void* gate, int ld_gate, void* out, int ldo, int num_pages,
           const int* tiles, int n_tiles, const int* segment_info, const int* block_table, int table_stride, int page_size,
           const MaskedAttentionSpec& s, int* status, cudaStream_t stream) {
    const size_t bytes = KH * kQHalfBytes + (SHARED ? 4 : 2) * KH * kTileHalfBytes + (SHARED ? 0 : 2 * VH * kTileHalfBytes) + 1024;
    const cudaError_t e = cudaFuncSetAttribute(attention_masked_wide_kernel<KH, VH, SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return mlr_fail("attention_masked_wide: cannot use %zu bytes of shared memory: %s", bytes, cudaGetErrorString(e));
    const int gate_octets = gate && s.gate_kind != 3 && ld_gate % 8 == 0 && reinterpret_cast<uintptr_t>(gate) % 16 == 0;
    mlr_launch((attention_masked_wide_kernel<KH, VH, SHARED>), dim3(s.heads, n_tiles), dim3(kThreads), bytes, stream, map_k, map_v,
               static_cast<const __nv_bfloat16*>(q), ldq, static_cast<const __nv_bfloat16*>(gate), ld_gate, gate_octets, static_cast<__nv_bfloat16*>(out),
               ldo, num_pages, tiles, segment_info, block_table, table_stride, page_size, s, status);
    return mlr_launched("attention_masked_wide");
}

}  // namespace

// Whether `mlr_attention_masked_wide` takes this description (host memory) and page size: 1 yes, 0 no.
MLR_API int mlr_attention_masked_wide_fit(const MaskedAttentionSpec* s, int page_size) {
    return s->maps <= 1 && !s->dense_cache && s->dim % 16 == 0 && s->dim >= 16 && s->dim <= 128 && s->vdim % 8 == 0 && s->vdim >= 8 && s->vdim <= 128 &&
           s->rot_dims % 16 == 0 && page_size >= 8 && page_size <= 256 && (page_size & (page_size - 1)) == 0;
}

// tiles: n_tiles pairs {segment, first token of a tile of up to 128 rows of that segment}; the rest as `mlr_attention_masked_tiles`.
MLR_API int mlr_attention_masked_wide(const MaskedAttentionSpec* spec, const void* q, int ldq, const void* gate, int ld_gate, void* out, int ldo,
                                      const void* cache, int num_pages, const int* tiles, int n_tiles, const int* segment_info, const int* block_table,
                                      int table_stride, int page_size, int* status, cudaStream_t stream) {
    MLR_REQUIRE(spec && mlr_attention_masked_wide_fit(spec, page_size) && spec->heads > 0 && spec->kv_heads > 0 && spec->heads % spec->kv_heads == 0 &&
                    (!spec->shared_kv || spec->vdim <= spec->dim) && (spec->rot_dims == 0 || spec->freq) && spec->rot_dims <= spec->dim,
                "attention_masked_wide: these sizes are not taken");
    MLR_REQUIRE(n_tiles >= 0 && n_tiles <= 65535 && num_pages > 0, "attention_masked_wide: bad tile count or pages");
    MLR_REQUIRE(ldq >= spec->heads * spec->dim && ldo >= spec->heads * spec->vdim && ldq % 8 == 0 && ldo % 8 == 0, "attention_masked_wide: bad row strides");
    MLR_REQUIRE((spec->gate_kind == 0) == (gate == nullptr), "attention_masked_wide: the description and the call disagree about a gate");
    const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    MLR_REQUIRE(aligned(q) && aligned(out) && aligned(cache), "attention_masked_wide: q, out and the cache start on 16-byte borders");
    if (n_tiles == 0) return 0;
    const MaskedAttentionSpec& s = *spec;
    const size_t keys = static_cast<size_t>(s.kv_heads) * page_size * s.dim;
    const size_t page_elems = s.shared_kv ? keys : keys + static_cast<size_t>(s.kv_heads) * page_size * s.vdim;
    const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(cache);
    CUtensorMap map_k, map_v;
    if (int e = cache_map(&map_k, base, s.dim, page_size, s.kv_heads, num_pages, page_elems)) return e;
    if (s.shared_kv) map_v = map_k;
    else if (int e = cache_map(&map_v, base + keys, s.vdim, page_size, s.kv_heads, num_pages, page_elems)) return e;
#define MLR_GO(KH, VH, SHARED)                                                                                                              \
    return launch<KH, VH, SHARED>(map_k, map_v, q, ldq, gate, ld_gate, out, ldo, num_pages, tiles, n_tiles, segment_info, block_table,       \
                                  table_stride, page_size, s, status, stream)
    const bool long_key = s.dim > 64, long_value = s.vdim > 64;
    if (s.shared_kv) {
        if (long_value) MLR_GO(2, 2, true);
        if (long_key) MLR_GO(2, 1, true);
        MLR_GO(1, 1, true);
    }
    if (long_key && long_value) MLR_GO(2, 2, false);
    if (long_key) MLR_GO(2, 1, false);
    if (long_value) MLR_GO(1, 2, false);
    MLR_GO(1, 1, false);
#undef MLR_GO
}
