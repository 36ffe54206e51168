// Bounded waits on a shared-memory mbarrier: the tensor-core sweeps' and the
// self-test's (libconv_gb300_selftest_wait).
#pragma once
#include <stdint.h>

namespace lcg {

constexpr uint32_t kWaitSleep = 64;                          // ns between polls
constexpr uint32_t kWaitSuspend = 1000;                      // ns, hint: how long a poll may suspend its thread
constexpr uint32_t kWaitPolls = 16;                          // polls between two looks at the clock
constexpr unsigned long long kWaitLimit = 2000000000ull;     // ns of the GPU's global timer

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// kWaitPolls polls for the phase of the given parity.  A poll that fails takes 3.8 us
// (measured; the hint is not kept to), so a run of them 60 us.
// The loop is a few instructions, because a waiting warp's polls come out of the
// working warps' issue slots.
__device__ __forceinline__ bool bar_polls(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\tmov.u32 n, %3;\n"
        "WAIT_%=:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %5;\n\t@p bra DONE_%=;\n\t"
        "nanosleep.u32 %4;\n\tsub.u32 n, n, 1;\n\tsetp.ne.u32 q, n, 0;\n\t@q bra WAIT_%=;\n"
        "DONE_%=:\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "n"(kWaitPolls), "n"(kWaitSleep), "r"(kWaitSuspend)
        : "memory");
    return ok != 0;
}

// The rest of a wait that kWaitPolls polls did not end: out of line, the working
// warps' loops stay short.
static __device__ __noinline__ bool bar_wait_long(uint32_t bar, uint32_t parity, unsigned long long limit_ns) {
    const unsigned long long t0 = global_ns();
    while (!bar_polls(bar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}

// Wait for the phase of the given parity; false when it has not come limit_ns
// (and at most two runs of kWaitPolls polls) after the wait began.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns = kWaitLimit) {
    return bar_polls(bar, parity) || bar_wait_long(bar, parity, limit_ns);
}

}  // namespace lcg
