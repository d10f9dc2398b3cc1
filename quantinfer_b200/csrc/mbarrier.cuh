// mbarriers in shared memory, and waits on them that end.
//
// A wait gives up when kWaitNs of the global timer have passed, when another role of the block gave up (its abort flag in shared
// memory) or when any block recorded a wait that ran out in the device's status word. A time, not a count of polls: a poll may be
// suspended by the hardware for as long as it likes. mbar_wait() is for one thread; a whole warp uses mbar_wait_warp(), whose outcome is
// the same for all lanes, since what follows (tcgen05.ld, shuffles, barriers) needs all of them.
#pragma once

#include "common.cuh"

namespace qi_mbar {

constexpr unsigned long long kWaitNs = 1000000000ull;      // 1 s: a thousand times the longest launch of a step
constexpr unsigned long long kGraceNs = 200000ull;         // copies and MMAs that were issued have landed after a few microseconds

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

// Of a wait whose phase is not there after another 256 polls (`i` so far): whether it gives up. Looked at more often, a wait would notice its phase
// late.
__device__ __forceinline__ bool gives_up(uint32_t i, unsigned long long& until, const volatile int* abort_flag, const volatile int* status) {
    if (abort_flag && *abort_flag) return true;
    const unsigned long long now = now_ns();
    if (until == 0) until = now + kWaitNs;
    else if (now >= until) return true;
    return (i & 4095u) == 0u && status && (*status & qi::kStatusWaitTimeout);
}

// Waits for the phase with the given parity to complete; false when the wait gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* abort_flag = nullptr,
                                          const volatile int* status = nullptr) {
    unsigned long long until = 0;
    for (uint32_t i = 1;; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 0u && gives_up(i, until, abort_flag, status)) return false;
    }
}

// The same by all lanes of a warp, which poll together and vote on every poll: the loop's branches are the same for all lanes. (36 layers of the
// 8B sizes with one token: 3,200 us with lanes that poll by themselves, 3,170 with those and a vote at the end, 3,145 so; 64 tokens: 4,841
// and 4,746 us.)
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, const volatile int* abort_flag = nullptr,
                                               const volatile int* status = nullptr) {
    unsigned long long until = 0;
    for (uint32_t i = 1;; ++i) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if ((i & 255u) == 0u && __any_sync(0xffffffffu, gives_up(i, until, abort_flag, status))) return false;
    }
}

// A role whose wait gave up: the block's other roles and, through the status word, the other blocks leave too.
__device__ __forceinline__ void give_up(volatile int* abort_flag, int* status) {
    if (!*abort_flag) {
        *abort_flag = 1;
        if (status) atomicOr(status, qi::kStatusWaitTimeout);
    }
}

// Asked by one thread of a block beside the first products: after a wait that ran out in an earlier launch of the step there is
// nothing to compute from, and the block leaves.
__device__ __forceinline__ bool failed_before(const volatile int* status) { return status && (*status & qi::kStatusWaitTimeout); }

// Before a block that gave up leaves (one warp is enough: the block's memory stays its own until the last is gone), and after the barrier behind
// which no role issues anything any more: what is in flight still writes into its shared and tensor memory.
__device__ __forceinline__ void settle_in_flight() {
    const unsigned long long until = now_ns() + kGraceNs;
    while (now_ns() < until) __nanosleep(1000);
}

}  // namespace qi_mbar
