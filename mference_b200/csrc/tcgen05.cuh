// mbarrier, tensor-memory and descriptor helpers of the tcgen05 kernels.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace mfb {

constexpr long long TC_WAIT_CYCLES = 400000000ll;      // limit of every mbarrier wait, ~0.2 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait; false when the limit runs out.  Without a time hint: with one the compiler adds a sleep to each attempt.
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit = TC_WAIT_CYCLES) {
    const uint32_t addr = smem_u32(bar);
    if (mbar_try(addr, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t polls = 1;; ++polls) {
        // the clock is looked at every sixteenth poll: other warps want the issue slots
        if (mbar_try(addr, parity)) return true;
        if ((polls & 15u) == 0 && clock64() - t0 > limit) return false;
    }
}
// The same for a converged warp: one answer for all its lanes, also where the phase completes just as the limit runs out, since
// warp-wide instructions (tcgen05.ld / st, elect.sync) and named barriers follow.  The lanes vote only once their common first
// attempt has failed (a vote on every wait cost a prefill call 2 %).  If only some lanes' attempt failed, the phase is
// complete and cannot be followed by another before this warp has arrived, so they wait by themselves and succeed at once.
//
// A waiting warp shares its scheduler with the warps it waits for, so a poll is an attempt, a count and two branches: with a vote and a look
// at the clock in every poll, the polls were 40 % of the instructions of a prefill call with 48 rows per expert.
// IDLE: for warps that wait long and whose wake-up is not on the path of the MMAs; they sleep between two polls.
template <bool IDLE = false>
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, long long limit = TC_WAIT_CYCLES) {
    const uint32_t addr = smem_u32(bar);
    if (mbar_try(addr, parity)) return true;
    if (__activemask() != 0xFFFFFFFFu) return mbar_wait(bar, parity, limit);
    const long long t0 = clock64();
    for (;;) {
        uint32_t done = 0;
        if (IDLE) {
            for (uint32_t i = 0; i < 16 && !done; ++i) {
                __nanosleep(100);
                done = mbar_try(addr, parity);
            }
        } else {
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\t"
                "mov.u32 n, 64;\n"
                "POLL:\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "@p bra DONE;\n\t"
                "sub.u32 n, n, 1;\n\t"
                "setp.ne.u32 q, n, 0;\n\t"
                "@q bra POLL;\n"
                "DONE:\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        }
        if (__all_sync(0xFFFFFFFFu, done != 0)) return true;
        if (__any_sync(0xFFFFFFFFu, clock64() - t0 > limit)) return false;
    }
}
// Whether the phase has completed, without waiting (lanes may differ).
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// One thread of a converged warp.  The tensor and copy instructions take their operands from uniform registers: inside a
// branch on elect.sync of a warp-uniform path they issue back to back, inside `lane == 0` each of them cost ~55 cycles
// (and a commit ~125), more than the MMA itself up to N = 96.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory operand descriptor: K-major tile of 128-byte rows in the 128-byte swizzle, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t smem_desc(const void* tile) {
    const uint64_t addr = (smem_u32(tile) & 0x3FFFFu) >> 4;
    return addr | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Its two halves: what varies lies in the low one.
constexpr uint32_t SMEM_DESC_HI = (1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t smem_desc_lo(const void* tile) { return ((smem_u32(tile) & 0x3FFFFu) >> 4) | (1u << 16); }

}  // namespace mfb
