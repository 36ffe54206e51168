// Bounded waits on a shared-memory mbarrier: the tensor-core sweeps' and the
// self-test's (libconv_gb300_selftest_wait).
#pragma once
#include <stdint.h>

namespace lcg {

constexpr uint32_t kWaitSleep = 64;                          // ns between polls
constexpr uint32_t kWaitClocks = 200000;                     // SM clocks of polls between two looks at the timer
constexpr unsigned long long kWaitLimit = 2000000000ull;     // ns of the GPU's global timer

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Polls for the phase of the given parity, until it has come or kWaitClocks (about
// 100 us) and a poll (3.8 us when it fails) are over.  A waiting warp's polls come out
// of the working warps' issue slots, so the loop is a few instructions and ends by the
// clock: one that counts a known number of polls is unrolled (MagicFilter and kinetic
// on 32 x 128^3: 2.50 ms this way, 2.57 to 2.66 counting 16 to 256).
__device__ __forceinline__ bool bar_polls(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 t, n;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE_%=;\n\tmov.u32 t, %%clock;\n"
        "WAIT_%=:\n\tnanosleep.u32 %3;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE_%=;\n\tmov.u32 n, %%clock;\n\tsub.u32 n, n, t;\n\tsetp.lt.u32 q, n, %4;\n\t@q bra WAIT_%=;\n"
        "DONE_%=:\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "n"(kWaitSleep), "n"(kWaitClocks)
        : "memory");
    return ok != 0;
}

// The rest of a wait that one run of polls did not end: out of line, the working
// warps' loops stay short.
static __device__ __noinline__ bool bar_wait_long(uint32_t bar, uint32_t parity, unsigned long long limit_ns) {
    const unsigned long long t0 = global_ns();
    while (!bar_polls(bar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}

// Wait for the phase of the given parity; false when it has not come limit_ns
// (and at most two runs of polls) after the wait began.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns = kWaitLimit) {
    return bar_polls(bar, parity) || bar_wait_long(bar, parity, limit_ns);
}

}  // namespace lcg
