// Bounded wait on a shared-memory mbarrier: the tensor-core sweeps' and the
// self-test's (libconv_gb300_selftest_wait).
#pragma once
#include <stdint.h>

namespace lcg {

constexpr uint32_t kWaitSleep = 64;                          // ns between polls
constexpr uint32_t kWaitClocks = 200000;                     // SM clocks of polls between two looks at the timer
constexpr unsigned long long kWaitLimit = 2000000000ull;     // ns of the GPU's global timer

// Wait for the phase of the given parity; false when it has not come limit_ns (and
// at most two runs of polls, some 100 us each, a failing poll taking 3.8 us) after
// the wait began.  A waiting warp's polls come out of the working warps' issue
// slots, so a poll is a few instructions, the timer is read between runs only, and
// all is one statement: a run of a known number of polls gets unrolled and an
// out-of-line rest costs registers around every wait (MagicFilter and kinetic on
// 32 x 128^3: 2.44 ms this way, as without a limit in time; 2.57 to 2.66 with runs
// of 16 to 256 polls, 2.49 with the timer in a function of its own).
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns = kWaitLimit) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 c, n;\n\t.reg .u64 s, t;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE_%=;\n\t"
        "mov.u64 s, 0;\n"                                    // the timer after the first run
        "RUN_%=:\n\tmov.u32 c, %%clock;\n"
        "WAIT_%=:\n\tnanosleep.u32 %3;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE_%=;\n\t"
        "mov.u32 n, %%clock;\n\tsub.u32 n, n, c;\n\tsetp.lt.u32 q, n, %4;\n\t@q bra WAIT_%=;\n\t"
        "mov.u64 t, %%globaltimer;\n\tsetp.eq.u64 q, s, 0;\n\tselp.u64 s, t, s, q;\n\t"
        "sub.u64 t, t, s;\n\tsetp.le.u64 q, t, %5;\n\t@q bra RUN_%=;\n"
        "DONE_%=:\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "n"(kWaitSleep), "n"(kWaitClocks), "l"(limit_ns)
        : "memory");
    return ok != 0;
}

}  // namespace lcg
