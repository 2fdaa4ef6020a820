// What the kernels that stream weights through a ring of shared-memory slots have in common: bulk copies counted by mbarriers,
// waits that end, and the tensor-core instruction whose second operand is up to eight rows of activations.
#pragma once

#include "common.cuh"

namespace {

constexpr long long kWaitLimitCycles = 4000000000LL;      // about two seconds

__device__ __forceinline__ void mma_16x8x16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 load_shared16(uint32_t address) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(address));
    return v;
}

// ---- mbarriers and bulk copies (the ring of weights)
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
// Waits for a phase of a barrier, but not for ever.  A wait that runs out (about two seconds) sets the block's
// `failed` flag and MLR_STATUS_TIMEOUT; from then on no wait of the block waits, so that every thread still walks
// through the same barriers to the kernel's end (its results are then worthless, and the status says so).
__device__ __forceinline__ void wait_phase(uint32_t bar, uint32_t parity, volatile int* failed, int* status) {
    if (mbar_try_wait(bar, parity)) return;
    const long long start = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (*failed) return;
        if (clock64() - start > kWaitLimitCycles) {
            *failed = 1;
            if (status) atomicOr(status, MLR_STATUS_TIMEOUT);
            return;
        }
    }
}
// Bytes between rows of the activations in shared memory, and between a slot's rows of weights: the values and a
// pad that makes it 64 modulo 128, so that the 16-byte reads of the eight rows a quarter-warp touches fall into
// different banks.
__host__ __device__ inline int pitch_bytes(int values) { return values * 2 + ((64 - (values * 2) % 128) + 128) % 128; }

}  // namespace
