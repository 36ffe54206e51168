// tcgen05 tensor-core sweep, shared by the exact-digit and split-precision
// forms (instantiated in sweep_tc_exact.cu, sweep_tc_bf16x3.cu, sweep_tc_tf32x3.cu
// and sweep_tc_fd.cu).
//
// One sweep = one banded Toeplitz product per 16-output block:
//   D[line, n] = sum_kk A[line, kk] * B[kk, n]
// A holds a window of input elements (128 lines x K elements), B the filter:
// B[kk, n] = f_{c,c'}(kk/NCH - n/NCH) with c = n mod NCH, c' = kk mod NCH, where
// NCH = 1 for a convolution and 2 for the wavelet polyphase pairs (elements are
// (pair, channel), interleaved), so K = 32 or 48 for every filter here.
//
// Scheme SCH_EXACT (FP64-accurate, exact integer arithmetic on FP16 operands)
//   * each line is scaled by the power of two above its largest magnitude
//     (line_exp_kernel, or the sweep before: Sweep::le_next), each window of 64
//     outputs of a long periodic one by its own (window_exp_kernel, Sweep::le_win),
//     to signed 62-bit integers X = x 2^(62-E) (|X| <=
//     2^62, truncated toward zero); X is cut into 8 balanced byte digits
//     d_0 (top) .. d_7 in [-128, 127], X = sum_s d_s 256^(7-s): the bytes
//     of X + 0x8080808080808080 minus 128.  The operand keeps the bytes d_s +
//     128 themselves, as FP16 subnormals (units of 2^-24), and the 128 leaves
//     with a constant per order, 128 sum_t<=k sum_taps e_t;
//   * the filter, with the operator scalar a folded in exactly (128-bit
//     product of the two mantissas), is cut the same way into e_0..e_7;
//   * every partial sum of byte products stays within 2^22 units (checked on
//     the filter's digits, tc_filter_digits); every TMEM accumulator starts at
//     1.5 * 2^23 units (one MMA of a constant tile per output block), so all
//     its values are integers in [2^23, 2^24] units, where FP32 is exact, and
//     its bits are kAccBias plus the sum (the filter's digits are stored times
//     2^8, so the unit is 2^-16);
//   * the 36 pairs of order k = s + t <= 7 are accumulated, one TMEM
//     accumulator per order; the epilogue recombines
//     Y = sum_k Acc_k 2^(46-8k) in int64 (the orders 6-7 rounded to an
//     integer first), converts once and rescales the exponent.
//   Dropped orders (k >= 8) weigh below 2^-70 of the product of the line and
//   filter scales; the data truncation (2^-62 of the line scale) and the
//   final roundings stay below the rounding of an FP64 FMA chain.
//   Lines never share a scale; a line or window holding an Inf or NaN gives NaN.
//
// Split-precision schemes (FP32-class accuracy, reported per operator)
//   * every element is rounded to FP32 (magnitudes outside the normal float
//     range flush to zero / infinity), every filter tap times a likewise;
//   * SCH_BF16X3: three bfloat16 terms x = x0 + x1 + x2 (exact split of the
//     24-bit value), the 6 products of order <= 2, kind::f16 with BF16 inputs;
//   * SCH_TF32X3: two tf32 terms x = hi + lo (about 23 bits, both rounded to
//     nearest), the 3 products hi.hi + hi.lo + lo.hi, kind::tf32 (4-byte
//     elements, K = 8 per MMA);
//   * one FP32 accumulator per output: relative error near 1e-7.
//
// Persistent, warp-specialised CTA (one per SM), 512 threads at 128 registers.
// The unit of work is a strip: 128 lines and a run of consecutive 16-element
// output blocks along them (the whole line, or one of the segments it is cut
// into when a launch has few lines, tc_prepare).  Along a strip the input is cut
// into 16-element slabs; output block j reads slabs j .. j + W - 1 (W = 2, or 3
// for 29 and 2 x 16 taps), so neighbouring blocks share them: each element is
// converted once per strip, and the operand buffer is a ring of 6 slabs that
// conversion, MMAs and epilogue walk at their own pace, across strip ends too:
//   warps 0-7  producers: thread = (row, half of the slab's 16 elements); exact
//              scheme: byte digits; split schemes: bfloat16 / tf32 terms;
//              coalesced or vector loads, the next slab's in flight;
//   warps 8-15 epilogue: thread = TMEM lane = row; warps 8-11 take the even
//              blocks, warps 12-15 the odd ones; TMEM -> FP64 -> global.  Before
//              it drains a block, one of the group's warps in turn (lane 0,
//              unrolled) issues the MMAs of the group's next one into the other
//              of its two TMEM slots.
// Hand-offs (mbarriers): full[slab] producers -> issuer, empty[slab] MMAs ->
// producers (every block that reads a slab commits to it; the issuer of the
// first reader adds the arrivals of the readers a strip's ends do not have),
// tfull[slot] MMAs and issuer -> epilogue, drained[slot] epilogue -> issuer.
// No phase can run two ahead of its waiter; every wait gives up after kWaitLimit
// (lcg_wait.cuh: status word set, TMEM freed, kernel returns).  In single-sweep launches
// every role skips the strips of an array whose S0.active flag is 0 (flags fixed
// for the launch), so the roles still meet on the same strips.
//
// What bounds it (32 grids of 128^3, a launch of 67 M outputs): the instructions
// of the two roles and their latency with 16 warps per SM.  Before, tiles of 64
// outputs held the whole operand buffer, so conversion, MMAs and drain of a tile
// ran one after the other, and every tile converted its halo again; the kernel
// was 190 KB of code with one epilogue for every case.  MagicFilter sweep 520 ->
// 286 us (340 handing on exponents), kinetic sweep along x 600 -> 328 us, with
// partial sums 640 -> 470 us (issue slots 45 %, FP64 pipe 33-48 %, HBM 30-36 %).
// What mattered: the ring; one kernel per form of sweep with a short straight
// epilogue loop (no spills, 50 KB: 436 -> 325 us for the MagicFilter sweep alone);
// digits as FP16 subnormals; polls and shared-memory stores in few instructions;
// the slab after the next prefetched to L2.  Measured and slower: three epilogue
// groups and an issuer warp on 24 warps (80 registers: 1.58 ms against 1.52 for
// MagicFilter3D), TMEM loads one step ahead, global loads two slabs ahead in
// registers (kinetic 1.60 -> 1.65 ms), larger unrolled loops.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <type_traits>

#include "lcg_sweep.cuh"
#include "lcg_tc.cuh"
#include "lcg_wait.cuh"

namespace lcg {
namespace tck {

constexpr int kM = 128;          // lines per strip (MMA M)
constexpr int kSlots = 6;        // slabs in the operand ring
constexpr int kTmemSlots = 4;    // output blocks in TMEM
// Strips whose row exponents are kept.  Producers write strip s's once slab W s - 1
// of strips of one block (the shortest: W slabs) is in the ring, so once slab
// W s - 1 - kSlots has left it and block s - ceil((kSlots + 1) / W) was issued; that took
// every warp of its group past the block kTmemSlots before, and of the same group.  An
// epilogue warp still to read its exponents is then less than ceil((kSlots + 1) / W)
// + kTmemSlots strips behind: 8 for W = 2, the ring's length (tests/test_tc_ring.py).
constexpr int kExpRing = 8;
constexpr int kThreads = 512;    // 8 producer warps + 8 epilogue warps
constexpr int kProdWarps = 8, kEpiWarps = 8;
static_assert(kEpiWarps == kTcDotSlots, "dot partials per CTA");

// Forms of a sweep, one kernel each, so that the epilogue of the common ones is
// a short loop (code and registers): plain stores; plus a partial sum x2; plus
// the next sweep's line exponents, a warp's rows in one of its lines (HAND) or
// in one or two (HAND2); anything (dot products, a_x, a_y).
enum Form { FORM_PLAIN = 0, FORM_X2 = 1, FORM_HAND = 2, FORM_ANY = 3, FORM_HAND2 = 4 };
// How a block's outputs lie in memory: 32-byte runs, anyhow, anyhow and the
// line ends within the block.
enum Run { RUN_VEC = 0, RUN_ANY = 1, RUN_PART = 2 };

template <int KIND, int NT, int SCH> struct Geom {
    static constexpr int NCH = KIND == KCONV ? 1 : 2;            // elements per position
    static constexpr int PROD = NCH * NT;                        // products per output
    static constexpr int KB = ((NCH * (16 / NCH + NT - 1)) + 15) / 16 * 16;   // K per block
    static constexpr int W = KB / 16;                            // slabs a block reads
    static constexpr int PB = 16 / NCH;                          // positions per block or slab
    static constexpr int ESZ = SCH == SCH_TF32X3 ? 4 : 2;         // operand element bytes
    static constexpr int CE = 16 / ESZ;                          // elements per core-matrix row
    static constexpr int ND = SCH == SCH_EXACT ? 8 : SCH == SCH_BF16X3 ? 3 : 2;
    static constexpr int ORD = ND;                               // order accumulators per block
    // operand planes interleaved along K: the exact scheme keeps its digit
    // planes in pairs (K index = 2 * element + plane within the pair), so one
    // byte permute builds both FP16 digits of an element; split schemes one
    // plane per slice
    static constexpr int PL = SCH == SCH_EXACT ? 2 : 1;
    static constexpr int NS = ND / PL;                           // A slices (MMAs per K step)
    static constexpr int BN = 16 * ORD;                          // rows of the stacked filter
    static constexpr int LBO_B = BN * 16;                        // its K-direction chunk stride
    // a slab: NS slices of CH core-matrix columns (kM rows x 16 bytes each)
    static constexpr int CH = 16 * PL / CE;
    static constexpr int SLICE = CH * kM * 16;
    static constexpr int SLAB = NS * SLICE;
    static constexpr int KS = CH / 2;                            // MMA K steps per slab and slice
    static constexpr int A_BYTES = kSlots * SLAB;
    static constexpr int KBP = KB * PL;                          // K of a block window
    static constexpr int B_BYTES = BN * KBP * ESZ;
    // exact scheme: a 128 x 16 FP16 tile holding 8 at K = 0, 1, 2 of every row;
    // as both operands of an N = 128 MMA it sets an output block's eight order
    // accumulators to 3 * 8^2 = 192 = 1.5 * 2^23 units of 2^-16
    static constexpr int Z_BYTES = SCH == SCH_EXACT ? kM * 16 * 2 : 0;
    // barriers and TMEM address; row exponents of the last kExpRing strips
    static constexpr int AUX = 256 + kExpRing * kM * 2;
    static constexpr int SMEM = A_BYTES + B_BYTES + Z_BYTES + AUX + 1024;
    static constexpr int SLOT_COLS = ORD * 16;                   // one TMEM slot (a block)
    static constexpr uint32_t TMEM_COLS = kTmemSlots * SLOT_COLS <= 128 ? 128 : kTmemSlots * SLOT_COLS <= 256 ? 256 : 512;
    static_assert(kTmemSlots * SLOT_COLS <= 512, "TMEM columns");
    static_assert(W >= 2 && W < kSlots, "slab ring");
    static_assert(kExpRing >= (kSlots + W) / W + kTmemSlots, "row exponents in use");
    static_assert(ND % PL == 0 && CH % 2 == 0, "plane slices");
    static_assert(SMEM <= 232448, "shared memory");
    // Instruction descriptor (kind::f16 / kind::tf32): D F32; A and B F16
    // (exact), BF16 or TF32 (formats 0, 1, 2); both K-major; M = 128; N is
    // added per MMA (idesc()).
    static constexpr uint32_t FMT = SCH == SCH_EXACT ? 0u : SCH == SCH_BF16X3 ? 1u : 2u;
    static constexpr uint32_t IDESC0 = (1u << 4) | (FMT << 7) | (FMT << 10) |
                                       ((uint32_t)(kM >> 4) << 24);
    static constexpr uint32_t idesc(int n) { return IDESC0 | ((uint32_t)(n >> 3) << 17); }
};

// ---- PTX wrappers ----------------------------------------------------------------
__device__ __forceinline__ uint32_t saddr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    // K-major, no swizzle: start, leading (K-direction) and stride (8-row)
    // byte offsets in 16-byte units; bits 46-47 = 1 (descriptor version).
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

template <bool TF32>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t IDESC,
                                    uint32_t accum) {
    if (TF32)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
            "l"(a), "l"(b), "r"(IDESC), "r"(accum)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
            "l"(a), "l"(b), "r"(IDESC), "r"(accum)
            : "memory");
}

__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
        : "memory");
}

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}\n" ::"r"(bar)
        : "memory");
}

__device__ __forceinline__ void bar_arrive_n(uint32_t bar, uint32_t n) {
    asm volatile(
        "{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0], %1;\n\t}\n" ::"r"(bar), "r"(n)
        : "memory");
}

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}

// The line of a mapped address on its way to L2.
__device__ __forceinline__ void prefetch_l2(const void *p) {
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// 32 bytes from global memory (a 32-byte aligned address) in one load.  It keeps its
// place among the waits and stores around it: the kernels before may still be
// writing what it reads until griddepcontrol.wait, and y is read and rewritten.
__device__ __forceinline__ void ld256(const long long *p, long long &a, long long &b, long long &c,
                                      long long &d) {
    asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(a), "=l"(b), "=l"(c), "=l"(d)
                 : "l"(p)
                 : "memory");
}

// 32 bytes to global memory (a 32-byte aligned address) in one store.
__device__ __forceinline__ void st256(double *p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(__double_as_longlong(a)),
                 "l"(__double_as_longlong(b)), "l"(__double_as_longlong(c)), "l"(__double_as_longlong(d))
                 : "memory");
}

__device__ __forceinline__ int imod(int a, int n) {
    int r = a % n;
    return r < 0 ? r + n : r;
}

// Y * 2^se as an FP64, Y rounded to 53 bits to nearest-even, when every non-zero
// result is a normal number (-1022 <= se <= 961): one conversion instruction,
// and se added to its exponent field.  On this GPU the FP64 pipe takes 2 lanes a
// clock per SM and the integer pipes 64 each, so one FP64 instruction per output
// (1.0 K of a block's 3.1 K cycles) costs less than the ~27 integer instructions
// of the same normalisation, and a second one (a multiply by 2^se) already sets
// the pace: MagicFilter3D on 32 x 128^3 1.87 ms all integer, 1.80 with conversion
// and multiply, 1.56 with the conversion alone (64-output tiles).
__device__ __forceinline__ double ll_scaled_fast(long long Y, int se) {
    const double t = __ll2double_rn(Y);
    int hi = __double2hiint(t);
    if (hi) hi += se << 20;
    return __hiloint2double(hi, __double2loint(t));
}

// Y = sum_k Acc_k 2^(46 - 8k) over the 8 order accumulators of one output
// (channel c of the filter), orders 6-7 as the nearest integer of Acc_6 / 4 +
// Acc_7 / 1024, from the accumulators' bits b_k = kAccBias + Acc_k + C_k (C_k:
// the digits' offset of 128, tc_filter_digits).  Two neighbouring orders fit
// one 32-bit word: w = 256 b_k + b_{k+1} modulo 2^32 stays within [0x43000000,
// 0xC3800000], so it can be taken as unsigned, and biases and offsets of all
// orders leave by two constants (F.k64, F.k67).  One multiply-add per pair and
// three 32x32+64 ones to join them, with multipliers the compiler cannot turn
// into shifts (F.c...): they run on the multiply-add pipe, beside the
// producers' ALU work.  The wrap-around is exact because the true sum fits in
// 62 bits.
template <int ORD>
__device__ __forceinline__ long long horner_bal(const uint32_t (&b)[ORD], const TcFilter &F, int c) {
    static_assert(ORD == 8, "eight order accumulators");
    const uint32_t w01 = b[0] * F.c256 + b[1], w23 = b[2] * F.c256 + b[3], w45 = b[4] * F.c256 + b[5];
    const int lo = (int)(b[6] * F.c256 + b[7] + F.k67[c]) >> 10;
    long long v;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(v) : "r"(w45), "r"(F.c64), "l"(F.k64[c]));
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(v) : "r"(w23), "r"(F.c22));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(v) : "r"(lo), "r"(F.c1));
    return v + (long long)((unsigned long long)(w01 * F.c64) << 32);
}

// FP32 bits -> FP64 value, integer only (normal, zero, subnormal flushed, inf/nan).
__device__ __forceinline__ double f32_to_f64(uint32_t f) {
    const uint32_t sgn = f >> 31, ex = (f >> 23) & 0xFF, man = f & 0x7FFFFF;
    unsigned long long b = (unsigned long long)sgn << 63;
    if (ex == 0xFF) b |= 0x7FF0000000000000ull | ((unsigned long long)man << 29);
    else if (ex != 0) b |= ((unsigned long long)(ex - 127 + 1023) << 52) | ((unsigned long long)man << 29);
    return __longlong_as_double((long long)b);
}

// Balanced fixed point of one FP64 bit pattern against its line's largest
// exponent field mx (>= 1): U = X + 0x8080808080808080 with X = x 2^(62-E),
// E = mx - 1022, truncated toward zero; integer only, no branch: the 53-bit
// mantissa shifted up by 10 (below 2^63), then right by 10 - sh in [0, 63]
// where X = mant 2^sh (sh <= 9 since the element's exponent is at most mx;
// a shift of 63 leaves 0), sign applied in two's complement, bias added.
__device__ __forceinline__ void fixed_bal(long long bits, int mx, uint32_t &ul, uint32_t &uh) {
    const uint32_t lo = (uint32_t)bits, hi = (uint32_t)((unsigned long long)bits >> 32);
    const int ex = (int)((hi >> 20) & 0x7FF);
    const uint32_t mh = (hi & 0xFFFFFu) | (ex ? 0x100000u : 0u);
    const int c = min(max(mx - max(ex, 1) + 1, 0), 63);         // 10 - sh
    const unsigned long long m10 = (((unsigned long long)mh << 32) | lo) << 10;
    const unsigned long long M = m10 >> c;
    const unsigned long long sg = (unsigned long long)(bits >> 63);   // 0 or all ones
    const unsigned long long U = (M ^ sg) + (sg & 1ull) + 0x8080808080808080ull;
    ul = (uint32_t)U;
    uh = (uint32_t)(U >> 32);
}

// The same for a row whose largest exponent field mx is at least 64, with mxs =
// (mx + 1) << 20: a zero or subnormal element then lies below one unit, and its
// shift of mx + 1 > 64 gives 0 whatever the mantissa's leading bit, so neither
// it nor the shift needs a special case.  c10 = 1024 (a multiplier the compiler
// cannot turn into shifts: the multiply-add pipe has room, the ALU pipe has not).
__device__ __forceinline__ void fixed_fast(long long bits, uint32_t mxs, uint32_t c10, uint32_t &ul, uint32_t &uh) {
    const uint32_t lo = (uint32_t)bits, hi = (uint32_t)((unsigned long long)bits >> 32);
    const uint32_t c = (mxs - (hi & 0x7FF00000u)) >> 20;        // mx + 1 - ex
    const uint32_t mh = (hi & 0xFFFFFu) | 0x100000u;
    unsigned long long m = (unsigned long long)lo * c10;
    m += (unsigned long long)(mh * c10) << 32;
    asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(c));              // 0 for c > 63
    const uint32_t sg = (uint32_t)((int)hi >> 31);              // 0 or all ones
    // (m ^ sg) - sg + 0x8080808080808080
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, %5;"
        : "=r"(ul), "=r"(uh)
        : "r"((uint32_t)m ^ sg), "r"(0x80808080u | (sg & 1u)), "r"((uint32_t)(m >> 32) ^ sg), "r"(0x80808080u));
}

// FP16 pair of digits 2p, 2p+1 (bytes 7-2p and 6-2p) of one biased fixed point
// (ul/uh): PRMT takes the two bytes with a zero byte above each.  As FP16 bits
// a byte u is the subnormal u 2^-24, exact; the operand is the balanced digit
// plus 128, and the 128 leaves with the accumulators' bias (horner_bal).  The
// lower half is plane 2p (the more significant digit).
__device__ __forceinline__ uint32_t digit_pair_elem(int p, uint32_t ul, uint32_t uh) {
    const uint32_t w = p < 2 ? uh : ul;
    // bytes (3, 2) of the word for even p, (1, 0) for odd p; selector 4 = 0
    const uint32_t sel = (p & 1) ? 0x4041u : 0x4243u;
    uint32_t t;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(t) : "r"(w), "r"(0u), "r"(sel));
    return t;
}

// FP64 bit pattern -> FP32 bit pattern, rounded to nearest (ties away) on the
// magnitude, integer only; magnitudes outside the normal float range flush to
// a signed zero or overflow to infinity.
__device__ __forceinline__ uint32_t f64_to_f32_bits(long long bits) {
    const uint32_t lo = (uint32_t)bits, hi = (uint32_t)((unsigned long long)bits >> 32);
    const uint32_t sg = hi & 0x80000000u;
    const int e = (int)((hi >> 20) & 0x7FF) - 1023 + 127;
    if (e <= 0) return sg;
    if (e >= 255) return sg | 0x7F800000u;
    // the rounding carry may step into the exponent (and up to infinity): exact
    return sg | ((((uint32_t)e << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29)) + ((lo >> 28) & 1u));
}

// Split of an FP32 value into SPLITS terms (bfloat16: 3 x 8 significant bits,
// an exact split; tf32: 2 x 11 bits), as FP32 bit patterns whose low bits are
// zero.  Each term is the remainder rounded to nearest (half an ulp added to
// the magnitude bits, ties away from zero; a carry steps into the exponent),
// and each remainder is formed exactly in FP32.
template <int SPLITS, uint32_t MASK>
__device__ __forceinline__ void split_f32(uint32_t f, uint32_t (&h)[SPLITS]) {
    constexpr uint32_t HALF = (~MASK + 1u) >> 1;
    uint32_t r = f;
#pragma unroll
    for (int i = 0; i < SPLITS; ++i) {
        h[i] = (r + HALF) & MASK;
        if (i + 1 < SPLITS) r = __float_as_uint(__uint_as_float(r) - __uint_as_float(h[i]));
    }
}

// Issue the MMAs of one output block.  The filter planes t = 0..ORD-1 are
// stacked along N in one matrix (rows 16t + n), and the ORD accumulators of the
// block (order k = s + t at columns 16k of its TMEM slot) are contiguous, so
// ONE MMA per data plane s covers all its pairs at once: D = columns 16s.. of
// the slot, N = 16 (ORD - s) (a prefix of the stacked filter), giving pair
// (s, t) at order s + t.  The s = 0 MMA of the first K step initialises every
// order (split schemes); in the exact scheme one MMA of the constant tile
// (z_desc, N = 128) first sets all eight orders to 1.5 * 2^23 and every data
// MMA accumulates.  One MMA covers 32 bytes of K (two core matrices); a[w] is
// the descriptor of the window's slab w.  Descriptors are advanced by adding
// the (16-byte unit) offset to the start-address field (addresses < 256 KB
// never carry out of it).
template <int KIND, int NT, int SCH>
__device__ __forceinline__ void issue_block(uint32_t d0, const uint64_t (&a)[Geom<KIND, NT, SCH>::W],
                                            uint64_t b_desc0, uint64_t z_desc) {
    using G = Geom<KIND, NT, SCH>;
    constexpr bool TF = SCH == SCH_TF32X3;
    constexpr bool EX = SCH == SCH_EXACT;
    if (EX) mma<false>(d0, z_desc, z_desc, G::idesc(16 * G::ORD), 0u);
#pragma unroll
    for (int sl = 0; sl < G::NS; ++sl) {
        const int sd = sl * G::PL;                               // first plane (order) of the slice
        const uint32_t id = G::idesc(16 * (G::ORD - sd));
#pragma unroll
        for (int w = 0; w < G::W; ++w) {
#pragma unroll
            for (int ks = 0; ks < G::KS; ++ks) {
                const uint64_t ad = a[w] + (uint64_t)((sl * G::SLICE + 2 * ks * 2048) >> 4);
                const uint64_t bd = b_desc0 + (uint64_t)((2 * (w * G::KS + ks) * G::LBO_B) >> 4);
                mma<TF>(d0 + (uint32_t)(sd * 16), ad, bd, id, (EX || sl > 0 || w > 0 || ks > 0) ? 1u : 0u);
            }
        }
    }
}

// Filter of output channel c, input channel c2 within the flat digit table
// (convolution: 0; wavelets: LE | LO | HE | HO, each NT taps).
template <int KIND>
__device__ __forceinline__ int filter_index(int c, int c2) {
    if (KIND == KCONV) return 0;
    if (KIND == KDEC) return c == 0 ? (c2 == 0 ? 0 : 1) : (c2 == 0 ? 2 : 3);
    return c == 0 ? (c2 == 0 ? 1 : 3) : (c2 == 0 ? 0 : 2);          // KREC
}

// floor(n / d) for n < 2^31 with d's multiplicative inverse (tc_prepare).
__device__ __forceinline__ uint32_t fdiv(uint32_t n, uint32_t m, uint32_t s) {
    return (uint32_t)(((unsigned long long)n * m) >> s);
}

// Where strip `strip` of a launch lives: its sweep, its segment `seg` along the
// lines, its block of kM lines `lb` and its array.  Strips are numbered
// segment fastest, then line block, then array.  A batched launch (BATCH)
// covers a list of sweeps of the same kind and filter, one per grid of a
// batch of uneven grids, whose strips are numbered consecutively (prefix[i] =
// first strip of sweep i).
struct StripLoc {
    const Sweep *S;
    int seg;
    uint32_t lb;
    int arr;
};

template <bool BATCH>
__device__ __forceinline__ StripLoc locate(const Sweep &S0, const Sweep *descs,
                                           const long long *prefix, int nsweeps, long long strip) {
    const Sweep *S = &S0;
    uint32_t t = (uint32_t)strip;
    if (BATCH) {
        int lo = 0, hi = nsweeps - 1;                    // last i with prefix[i] <= strip
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (prefix[mid] <= strip) lo = mid;
            else hi = mid - 1;
        }
        S = descs + lo;
        t = (uint32_t)(strip - prefix[lo]);
    }
    const uint32_t q = fdiv(t, S->tdiv_m[0], S->tdiv_s[0]);          // t / segments
    const uint32_t arr = fdiv(q, S->tdiv_m[1], S->tdiv_s[1]);        // / line blocks
    return {S, (int)(t - q * S->tdiv_d[0]), q - arr * S->tdiv_d[1], (int)arr};
}

// Output blocks of segment `seg` of a sweep (PB positions each).
template <int PB>
__device__ __forceinline__ int strip_blocks(const Sweep &S, int seg) {
    return min(S.seg_blocks, (S.qhi - S.qlo + PB) / PB - seg * S.seg_blocks);
}

// Line g of a sweep as (l, r): g = l + nL r.
__device__ __forceinline__ void line_lr(const Sweep &S, uint32_t g, uint32_t &l, uint32_t &r) {
    r = fdiv(g, S.tdiv_m[2], S.tdiv_s[2]);
    l = g - r * S.tdiv_d[2];
}

template <int KIND, int NT, int SCH, bool BATCH, int FORM>
__global__ void __launch_bounds__(kThreads, 1)
sweep_tc_kernel(const __grid_constant__ Sweep S0, const __grid_constant__ TcFilter F, int *status,
                const Sweep *__restrict__ descs, const long long *__restrict__ prefix, int nsweeps,
                const int *lineE) {      // no __restrict__: a kernel still running may write it
    using G = Geom<KIND, NT, SCH>;
    constexpr int NCH = G::NCH, W = G::W, PB = G::PB;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *A = smem;
    uint8_t *B = smem + G::A_BYTES;
    uint8_t *Z = B + G::B_BYTES;                      // exact scheme: accumulator bias tile
    uint8_t *aux = Z + G::Z_BYTES;
    uint32_t *tslot = (uint32_t *)(aux + 192);
    short *rowE = (short *)(aux + 256);               // row exponents, by strip mod kExpRing
    const uint32_t bar0 = saddr(aux);
    auto full = [&](uint32_t s) { return bar0 + 8 * s; };
    auto empty = [&](uint32_t s) { return bar0 + 8 * (kSlots + s); };
    auto tfull = [&](uint32_t s) { return bar0 + 8 * (2 * kSlots + s); };
    auto drained = [&](uint32_t s) { return bar0 + 8 * (2 * kSlots + kTmemSlots + s); };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // window offset of the convolution sweeps (0 in batched launches)
    const int woff = (!BATCH && KIND == KCONV) ? S0.woff : 0;
    // the next kernel of the stream may start its own prologue (it waits below)
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         saddr(tslot)),
                     "r"(G::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kSlots; ++s) {
            bar_init(full(s), kProdWarps);
            bar_init(empty(s), W);                    // one arrival per block of a window
        }
        for (int s = 0; s < kTmemSlots; ++s) {
            bar_init(tfull(s), 2);                    // the issuer's commit and its own arrival
            bar_init(drained(s), kEpiWarps / 2);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // Toeplitz filter tiles B_t[n][kk], K-major core matrices, a 16-byte row of one
    // per thread and step.  The filter's digits come through shared memory (the
    // operand ring, not in use yet): read where they are, in the parameters, a
    // warp's 32 addresses take turns.  A launch of a few blocks is mostly this
    // prologue: MagicFilter3D of one 32^3 grid 39 us, element by element from the
    // parameters 50
    static_assert(TcFilter::kSlices * TcFilter::kMaxTaps == 4 * 128, "digit table");
    uint32_t *const dig = (uint32_t *)A;
    if (tid < 128) ((uint4 *)dig)[tid] = ((const uint4 *)F.dig)[tid];
    __syncthreads();
    for (int idx = tid; idx < G::ORD * 16 * (G::KBP / G::CE); idx += kThreads) {
        const int row = idx % (G::ORD * 16), kc = idx / (G::ORD * 16);
        const int t = row / 16, n = row % 16;            // stacked filter planes
        uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int e = 0; e < G::CE; ++e) {
            // K index k2 = element kk, data plane pj within the slice: the pair
            // (slice plane pj, filter digit t - pj) lands on order column t
            const int k2 = kc * G::CE + e, kk = k2 / G::PL, pj = k2 % G::PL;
            const int ti = kk / NCH - n / NCH - woff;
            const uint32_t v = (ti >= 0 && ti < NT && t >= pj)
                                   ? dig[(t - pj) * TcFilter::kMaxTaps + filter_index<KIND>(n % NCH, kk % NCH) * NT + ti]
                                   : 0u;
            if (G::ESZ == 4) w[e % 4] = v;
            else w[e / 2] |= (v & 0xFFFFu) << (16 * (e & 1));
        }
        sts128(saddr(B) + kc * G::LBO_B + (row >> 3) * 128 + (row & 7) * 16, w[0], w[1], w[2], w[3]);
    }
    // bias tile, K-major core matrices like A: (row, k) at (k / 8) * 2048 +
    // (row / 8) * 128 + (row % 8) * 16 + (k % 8) * 2; FP16 8 = 0x4800 at k < 3
    for (int idx = tid; idx < G::Z_BYTES / 16; idx += kThreads)
        sts128(saddr(Z) + 16 * idx, idx < kM ? 0x48004800u : 0u, idx < kM ? 0x4800u : 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tslot;
    bool alive = true;
    // everything above touches parameters and this CTA's own memory only; from here on
    // the work of the kernels before is complete
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const long long nstrips =
        BATCH ? prefix[nsweeps]
              : ((long long)S0.nL * S0.nR + kM - 1) / kM * (long long)S0.tdiv_d[0] * S0.narr;
    // the strip after `strip` for this CTA, skipping inactive arrays
    auto skip_inactive = [&](long long strip) -> long long {
        if (!BATCH && S0.active)
            while (strip < nstrips && !S0.active[locate<BATCH>(S0, descs, prefix, nsweeps, strip).arr])
                strip += gridDim.x;
        return strip;
    };
    if (!BATCH && (FORM == FORM_HAND || FORM == FORM_HAND2) && S0.le_zero)
        for (long long i = (long long)blockIdx.x * kThreads + tid; i < S0.le_zero_n; i += (long long)gridDim.x * kThreads)
            S0.le_zero[i] = 0;

    if (warp < kProdWarps) {
        // ============ producers: thread = (row, half of every slab); lanes 0-15
        // take 16 consecutive rows' elements 0-7, lanes 16-31 elements 8-15
        constexpr int PG = 8 / NCH;                      // positions of a thread's group
        const int half = lane >> 4;
        const int row = warp * 16 + (lane & 15);
        const uint32_t a_addr = saddr(A);
        // the strip being loaded: the row's line, and the thread's next group of 8
        // elements: its position in the line and the used positions left
        const Sweep *S = &S0;
        const long long *base = nullptr;
        long long stride = 0;
        int ps = 0, left = 0, nsl = 0;
        int wrap = 0, last = 0;                          // ps wraps at; runs end by `last`
        int mx = 0;                                      // largest exponent field of the row
        // the group's elements; those past the used positions, and outside a free
        // boundary's line, are zero
        auto load8 = [&](long long (&bits)[8]) {
            if (left >= PG && ps >= 0 && ps + PG <= last) {      // one run of positions
                // the slab after this one on its way to L2: its loads, a slab's work
                // from now, then take an L2 latency instead of a memory one (one
                // slab ahead in registers is all there is room for).  One line per
                // thread: strided, 16 neighbouring rows share the lines of 8
                // positions; contiguous, a row's own run.  32 x 128^3: MagicFilter3D
                // 1155 -> 1098 us; two slabs ahead 1113, three 1125
                if (left >= PG + PB && ps + PG + PB <= last) {
                    const int k = lane & 7;
                    prefetch_l2(base + (KIND == KREC ? (long long)ps + PB + ((k & 4) ? S->in_ext : 0) + (k & 3)
                                                     : (long long)(NCH * (ps + PB)) + (stride == 1 ? 0 : k)) * stride);
                }
                if (KIND == KREC) {
                    // channel c of position ps at ps + in_ext c: two runs of 4,
                    // interleaved into the group
                    const long long *qL = base + (long long)ps * stride;
                    const long long *qH = qL + (long long)S->in_ext * stride;
                    if (stride == 1 && ((((uintptr_t)qL) | ((uintptr_t)qH)) & 31) == 0) {
                        ld256(qL, bits[0], bits[2], bits[4], bits[6]);
                        ld256(qH, bits[1], bits[3], bits[5], bits[7]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            bits[2 * j] = qL[j * stride];
                            bits[2 * j + 1] = qH[j * stride];
                        }
                    }
                } else {
                    const long long *q = base + (long long)(NCH * ps) * stride;
                    if (stride == 1 && (((uintptr_t)q) & 31) == 0) {
                        ld256(q, bits[0], bits[1], bits[2], bits[3]);
                        ld256(q + 4, bits[4], bits[5], bits[6], bits[7]);
                    } else if (stride == 1 && (((uintptr_t)q) & 15) == 0) {
                        const double2 *v = reinterpret_cast<const double2 *>(q);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const double2 t = v[e];
                            bits[2 * e] = __double_as_longlong(t.x);
                            bits[2 * e + 1] = __double_as_longlong(t.y);
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            bits[e] = *q;
                            q += stride;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) bits[e] = 0ll;
                const int n = S->n, bc = S->bc;
                int p = ps;
                if (bc == BC_PERIODIC && n < 32) p = imod(p, n);
#pragma unroll
                for (int j = 0; j < PG; ++j) {
                    if (bc == BC_PERIODIC && p >= n) p -= n;
                    if (j < left && (bc == BC_PERIODIC || bc == BC_SHRINK || (p >= 0 && p < n))) {
                        const long long *q = base + (long long)(KIND == KDEC ? 2 * p : p) * stride;
                        if (KIND == KCONV) {
                            bits[j] = *q;
                        } else {
                            bits[2 * j] = *q;
                            bits[2 * j + 1] = q[(KIND == KDEC ? 1 : S->in_ext) * stride];
                        }
                    }
                    ++p;
                }
            }
            ps += PB;                                    // on to the next slab
            if (ps >= wrap) ps -= wrap;
            left -= PB;
        };
        auto open = [&](long long strip) {               // make `strip` the strip being loaded
            const StripLoc loc = locate<BATCH>(S0, descs, prefix, nsweeps, strip);
            if (BATCH) S = loc.S;
            const uint32_t nlines = (uint32_t)S->nL * (uint32_t)S->nR;
            const uint32_t g = loc.lb * kM + row;
            const bool valid = g < nlines;
            uint32_t l = 0, r = 0;
            if (valid) line_lr(*S, g, l, r);
            stride = S->nL;
            base = reinterpret_cast<const long long *>(S->x) + (long long)loc.arr * S->x_arr + l +
                   stride * ((long long)S->in_ext * NCH) * r;
            const int nb = strip_blocks<PB>(*S, loc.seg);
            nsl = nb + W - 1;
            const int p0 = S->qlo + loc.seg * S->seg_blocks * PB + S->lowfil - woff;   // window start
            // positions the strip's outputs use, none past the sweep's last input
            left = min(nb * PB + NT - 1 + woff, S->qhi + S->lowfil + NT - p0) - half * PG;
            ps = p0 + half * PG;
            wrap = 0x40000000;
            last = S->n;
            if (S->bc == BC_SHRINK) {
                ps -= S->in_lo;
                last = 0x40000000;
            } else if (S->bc == BC_PERIODIC) {
                // filters reach less than 32 positions: shorter lines may wrap more
                // than once and go element by element
                if (last < 32) {
                    last = -1;
                } else {
                    wrap = last;
                    ps = ps < 0 ? ps + last : ps >= last ? ps - last : ps;
                }
            }
            // largest exponent field of the line, or of the strip's window of it; a row
            // past the last line is all zeros under any scale
            mx = 0x7FE;
            if (!valid) left = 0;
            else if (SCH == SCH_EXACT) {
                long long le = S->le_off + (long long)loc.arr * nlines + g;
                if (!BATCH && KIND == KCONV && S->le_win)            // the window (4 blocks) of the strip
                    le += (long long)((loc.seg * S->seg_blocks) >> 2) * nlines * S->narr;
                mx = lineE[le];
            }
        };
        long long strip = skip_inactive(blockIdx.x);
        uint32_t slot = 0, par = 1;                      // ring position; empty phase to wait for
        uint32_t si = 0;                                 // strips begun
        long long bits[8];
        int sl = 0, n_cur = 0, mxe = 1;                  // slab in `bits`, slabs of its strip
        uint32_t mxs = 0;
        bool fast = true;
#pragma unroll 1
        for (bool first = true;; first = false) {
            // the slab's elements as operands-to-be in registers; then the next
            // slab's loads (of the next strip after the last one) into the registers
            // these leave, in flight while the operands wait for their slot and are
            // stored
            uint32_t ul[8], uh[8];                       // exact: biased fixed point
            if (!first) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    if (SCH == SCH_EXACT) fixed_fast(bits[e], mxs, F.c10, ul[e], uh[e]);
                    else ul[e] = f64_to_f32_bits(bits[e]);
                }
                if (SCH == SCH_EXACT && !fast) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) fixed_bal(bits[e], mxe, ul[e], uh[e]);
                }
            }
            const bool ends = sl + 1 >= n_cur;           // the strip's last slab
            if (ends) {
                if (!first) strip = skip_inactive(strip + gridDim.x);
                left = 0;
                if (strip < nstrips) open(strip);
            }
            load8(bits);
            if (!first) {
                if (!bar_wait(empty(slot), par)) {       // the ring's first pass finds it free
                    alive = false;
                    break;
                }
                const uint32_t dst = a_addr + slot * G::SLAB + half * (8 * G::PL / G::CE) * 2048 +
                                     (row >> 3) * 128 + (row & 7) * 16;
                if (SCH == SCH_EXACT) {
                    // slice p holds digit planes 2p, 2p+1 = bytes 7-2p, 6-2p: one
                    // 16-byte core-matrix row per 4 elements
#pragma unroll
                    for (int s = 0; s < G::NS; ++s) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t wds[4];
#pragma unroll
                            for (int w = 0; w < 4; ++w)
                                wds[w] = digit_pair_elem(s, ul[4 * h + w], uh[4 * h + w]);
                            sts128(dst + s * G::SLICE + h * 2048, wds[0], wds[1], wds[2], wds[3]);
                        }
                    }
                } else if (SCH == SCH_BF16X3) {
                    uint32_t h[8][3];
#pragma unroll
                    for (int e = 0; e < 8; ++e) split_f32<3, 0xFFFF0000u>(ul[e], h[e]);
#pragma unroll
                    for (int sd = 0; sd < 3; ++sd) {
                        uint32_t wds[4];
#pragma unroll
                        for (int w = 0; w < 4; ++w) wds[w] = (h[2 * w][sd] >> 16) | (h[2 * w + 1][sd] & 0xFFFF0000u);
                        sts128(dst + sd * G::SLICE, wds[0], wds[1], wds[2], wds[3]);
                    }
                } else {
                    uint32_t h[8][2];
#pragma unroll
                    for (int e = 0; e < 8; ++e) split_f32<2, 0xFFFFE000u>(ul[e], h[e]);
#pragma unroll
                    for (int sd = 0; sd < 2; ++sd) {
                        sts128(dst + sd * G::SLICE, h[0][sd], h[1][sd], h[2][sd], h[3][sd]);
                        sts128(dst + sd * G::SLICE + 2048, h[4][sd], h[5][sd], h[6][sd], h[7][sd]);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) bar_arrive(full(slot));
                if (++slot == kSlots) {
                    slot = 0;
                    par ^= 1;
                }
            }
            ++sl;
            if (ends) {
                if (strip >= nstrips) break;
                sl = 0;
                n_cur = nsl;
                mxe = max(mx, 1);
                mxs = (uint32_t)(mx + 1) << 20;
                fast = !__any_sync(0xffffffffu, mx < 64);
                if (SCH == SCH_EXACT && half == 0)
                    rowE[si % kExpRing * kM + row] = (short)(mx == 0x7FF ? 0x7FFF : mxe - 1022);
                ++si;
            }
        }
    } else {
        // ============ epilogue: thread = TMEM lane = row; group hf takes the blocks
        // whose number is hf modulo 2
        const int ew = warp - kProdWarps;
        const int lq = ew & 3, hf = ew >> 2;
        const int row = lq * 32 + lane;
        const uint64_t a_desc0 = umma_desc(saddr(A), 2048, 128);
        const uint64_t b_desc0 = umma_desc(saddr(B), G::LBO_B, 128);
        const uint64_t z_desc = umma_desc(saddr(Z), 2048, 128);
        // the block to be issued next by some warp: strip, block j of nb, its
        // number blk, and the number of its first slab since the launch began
        long long istrip = skip_inactive(blockIdx.x);
        int ij = 0, inb = 0;
        uint32_t islab = 0, iblk = 0;
        auto istrip_blocks = [&]() {
            if (istrip < nstrips) {
                const StripLoc loc = locate<BATCH>(S0, descs, prefix, nsweeps, istrip);
                inb = strip_blocks<PB>(*loc.S, loc.seg);
            }
        };
        istrip_blocks();
        // step to the next block
        auto istep = [&]() {
            ++iblk;
            ++islab;
            if (++ij == inb) {
                islab += W - 1;
                ij = 0;
                istrip = skip_inactive(istrip + gridDim.x);
                istrip_blocks();
            }
        };
        // block iblk (one of this group's): issued by one of the group's warps in
        // turn once its TMEM slot is drained and its slabs are full; every warp
        // steps to the group's next block
        auto issue_next = [&]() -> bool {
            if (istrip >= nstrips) return true;
            if (lq == (int)((iblk >> 1) & 3)) {
                const uint32_t ts = iblk % kTmemSlots, last = islab + W - 1;
                if (iblk >= kTmemSlots && !bar_wait(drained(ts), (iblk / kTmemSlots - 1) & 1)) return false;
                if (!bar_wait(full(last % kSlots), (last / kSlots) & 1)) return false;
                if (lane == 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    uint32_t sl[W];
                    uint64_t a[W];
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        sl[w] = (islab + w) % kSlots;
                        a[w] = a_desc0 + (uint64_t)((sl[w] * (uint32_t)G::SLAB) >> 4);
                    }
                    issue_block<KIND, NT, SCH>(tmem + ts * G::SLOT_COLS, a, b_desc0, z_desc);
                    commit(tfull(ts));
                    bar_arrive(tfull(ts));
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        commit(empty(sl[w]));
                        // slab ij + w is read by `readers` blocks; the first of
                        // them stands in for the W - readers others
                        const int k = ij + w, first = max(0, k - W + 1);
                        const int readers = min(k, inb - 1) - first + 1;
                        if (first == ij && readers < W) bar_arrive_n(empty(sl[w]), W - readers);
                    }
                }
                __syncwarp();
            }
            istep();
            if (istrip < nstrips) istep();
            return true;
        };
        if (hf == 1 && istrip < nstrips) istep();        // the group's first block
        if (!issue_next()) alive = false;

        // dot products per array: each epilogue warp owns the slot
        // dot_part[(arr * gridDim.x + blockIdx.x) * kTcDotSlots + ew] of every array it
        // visits (strips are array-major, so a CTA meets the arrays in order)
        double dot = 0.0;
        int dot_arr = -1;
        auto flush_dot = [&]() {
            for (int o = 16; o > 0; o >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, o);
            if (lane == 0) S0.dot_part[((long long)dot_arr * gridDim.x + blockIdx.x) * kTcDotSlots + ew] = dot;
            dot = 0.0;
        };
        uint32_t blk0 = 0, si = 0;                       // strip's first block, strips begun
        int nb = 0;
        for (long long strip = skip_inactive(blockIdx.x); alive && strip < nstrips;
             strip = skip_inactive(strip + gridDim.x), ++si, blk0 += (uint32_t)nb) {
            const StripLoc loc = locate<BATCH>(S0, descs, prefix, nsweeps, strip);
            const Sweep &S = *loc.S;
            const int arr = loc.arr;
            if (!BATCH && FORM == FORM_ANY && S0.has_dot && arr != dot_arr) {
                if (dot_arr >= 0) flush_dot();
                dot_arr = arr;
            }
            nb = strip_blocks<PB>(S, loc.seg);
            const int qs = S.qlo + loc.seg * S.seg_blocks * PB;
            const long long out_pext = (long long)S.out_ext * NCH;
            const uint32_t nlines = (uint32_t)S.nL * (uint32_t)S.nR;
            const uint32_t g = loc.lb * kM + row;
            const bool valid = g < nlines;
            uint32_t l32 = 0, r32 = 0;
            if (valid) line_lr(S, g, l32, r32);
            const long long l = l32, rr = r32;
            double *__restrict__ y = S.y + (long long)arr * S.y_arr;
            const double *__restrict__ xa = S.x + (long long)arr * S.x_arr;
            constexpr bool kMayX2 = KIND == KCONV && (FORM == FORM_X2 || FORM == FORM_ANY);
            const double *__restrict__ x2 = kMayX2 && S.x2 ? S.x2 + (long long)arr * S.x_arr : nullptr;
            // this row's output element (position p, channel c) sits at
            // yrow + yps p + ycs c; its x2 partial at x2row + x2s q; its input
            // at xrow + nL ps (row bases formed once per strip)
            const long long ys = S.transpose ? S.nR : S.nL;
            double *const yrow = S.transpose ? y + rr : y + l + (long long)S.nL * out_pext * rr;
            const long long yps = KIND == KREC ? 2 * ys : ys;
            const long long ycs = KIND == KREC ? ys : ys * S.out_ext;
            const bool grow = S.bc == BC_GROW;
            const double *const x2row = !x2 ? nullptr
                : grow ? (S.transpose ? x2 + rr : x2 + l + (long long)S.nL * S.out_ext * rr)
                       : x2 + l + (long long)S.nL * S.in_ext * rr;
            const long long x2s = grow ? ys : S.nL;
            const int x2lo = grow ? S.out_lo : S.in_lo;
            const double *const xrow = xa + l + (long long)S.nL * S.in_ext * rr;
            // no dot, a_x or a_y term: every output is its value (plus x2), stored
            const bool lean = FORM != FORM_ANY || (!S.has_dot && !S.has_ax && S.ay_mode == 0);
            constexpr bool hands = FORM == FORM_HAND || FORM == FORM_HAND2;
            int se = 0;
            bool farrow = false;
            double scale = 1.0, scale2 = 1.0;                // 2^se = scale (scale scale2 in a far row)
            const int j0 = (int)((blk0 ^ (uint32_t)hf) & 1u);   // the group's first block of the strip
            if (SCH == SCH_EXACT && j0 < nb) {
                // known with the strip's first slab; a row holding an Inf or NaN
                // gives NaN; farrow: 2^se is outside the range of the fast
                // conversion (two multiplications, the first one exact)
                if (!bar_wait(tfull((blk0 + j0) % kTmemSlots), ((blk0 + j0) / kTmemSlots) & 1)) { alive = false; break; }
                const int Er = rowE[si % kExpRing * kM + row];
                const bool nanrow = Er == 0x7FFF;
                se = nanrow ? 0 : max(Er + F.ef - 58, -2000);
                farrow = valid && (nanrow || se < -1022 || se > 961);
                const int e1 = farrow ? se / 2 : se;
                scale = __longlong_as_double(nanrow ? 0x7FF8000000000000LL : (long long)(e1 + 1023) << 52);
                scale2 = __longlong_as_double((long long)(se - e1 + 1023) << 52);
            }
            // next sweep's line exponents: the warp's 32 rows lie in one of its lines in
            // every output column, or in two neighbouring ones (run_plan: lines of at
            // least 32), so one or two maxima per column and an atomic from the
            // lanes that keep them
            const uint32_t g0 = loc.lb * kM + 32 * lq, ln = hands ? g0 / (uint32_t)max(S0.le_n1, 1) : 0;
            const uint32_t cut = (ln + 1) * (uint32_t)S0.le_n1;      // first row of the second line
            const bool two = FORM == FORM_HAND2 && g0 + 32 > cut && cut < nlines;
            int *const le_col = !hands ? nullptr : S0.le_next + (long long)arr * S0.le_next_lines + ln;
            const uint32_t sel = !valid ? 0u : g < cut || !two ? 0x7FFFFFFFu : 0u;     // rows of the first line
            auto hand_on = [&](auto &v, int q0, auto N) {    // N outputs from position q0 on
                constexpr int n = decltype(N)::value;
                const int p = q0 + lane / NCH, c = lane % NCH;
                const int e = KIND == KREC ? 2 * (p - S.out_lo) + c : p - S.out_lo + S.out_ext * c;
                int *const le = le_col + (long long)S0.le_n2 * e;
                const bool keeps = lane < n && p <= S.qhi && g0 < nlines;
                uint32_t mask = sel;
#pragma unroll 1
                for (int line = 0;; ++line) {
                    uint32_t m[n];
#pragma unroll
                    for (int i = 0; i < n; ++i) m[i] = __reduce_max_sync(0xffffffffu, (uint32_t)__double2hiint(v[i]) & mask);
                    // m[lane % n], by the lane's bits (log2 n predicates instead of n:
                    // MagicFilter3D on 32 x 128^3 1.055 -> 1.044 ms)
#pragma unroll
                    for (int w = 1; w < n; w *= 2)
#pragma unroll
                        for (int i = 0; i < n; i += 2 * w) m[i] = lane & w ? m[i + w] : m[i];
                    if (keeps) atomicMax(le + line, (int)(m[0] >> 20));
                    if (!two || line == 1) break;
                    mask = valid ? 0x7FFFFFFFu - sel : 0u;
                }
            };
            // blocks of far rows, and of sweeps that hot does not take; four outputs at a time
            auto cold_block = [&](int j) {
                const uint32_t blk = blk0 + j;
#pragma unroll 1
                for (int st = 0; st < 4; ++st) {
                    const int q0 = qs + j * PB + st * (4 / NCH);    // first output position of the step
                    const int nv = (S.qhi - q0 + 1) * NCH;          // valid elements of the step
                    const bool plain = lean && nv >= 4;
                    uint32_t acc[G::ORD][4];
#pragma unroll
                    for (int k = 0; k < G::ORD; ++k)
                        tmem_ld4(tmem + ((uint32_t)(lq * 32) << 16) +
                                     (uint32_t)((blk % kTmemSlots) * G::SLOT_COLS + k * 16 + 4 * st),
                                 acc[k]);
                    double add[4];
                    if (kMayX2 && x2 && valid) {
                        const double *xp = x2row + x2s * (q0 - x2lo);
#pragma unroll
                        for (int n = 0; n < 4; ++n) {
                            add[n] = n < nv ? *xp : 0.0;
                            xp += x2s;
                        }
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    if (st == 3) {                        // the slot may be reissued
                        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) bar_arrive(drained(blk % kTmemSlots));
                    }
                    if ((!hands && !valid) || nv <= 0) continue;
                    double *const ystep = yrow + yps * (q0 - S.out_lo);
                    // the outputs' values first (independent chains), then their memory side
                    double outv[4];
                    if constexpr (SCH == SCH_EXACT) {
                        long long Y[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            uint32_t bb[G::ORD];
#pragma unroll
                            for (int k = 0; k < G::ORD; ++k) bb[k] = acc[k][i];
                            Y[i] = horner_bal<G::ORD>(bb, F, i % NCH);
                        }
                        if (farrow) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                outv[i] = __ll2double_rn(Y[i]) * scale * scale2;
                                if (kMayX2 && x2 && plain) outv[i] += add[i];
                            }
                        } else if (kMayX2 && x2 && plain) {
                            // scale and partial sum in one FP64 instruction (the
                            // product is exact)
#pragma unroll
                            for (int i = 0; i < 4; ++i) outv[i] = fma(__ll2double_rn(Y[i]), scale, add[i]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) outv[i] = ll_scaled_fast(Y[i], se);
                        }
                    } else {                          // sum of the order accumulators
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float f = __uint_as_float(acc[0][i]);
#pragma unroll
                            for (int k = 1; k < G::ORD; ++k) f += __uint_as_float(acc[k][i]);
                            outv[i] = f32_to_f64(__float_as_uint(f));
                        }
                    }
                    if (hands) {
                        hand_on(outv, q0, std::integral_constant<int, 4>());
                        if (!valid) continue;
                    }
                    double *yq = ystep;
                    if (plain) {
                        if (SCH != SCH_EXACT && kMayX2 && x2) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) outv[i] += add[i];
                        }
                        // a contiguous output line takes the step's 4 outputs as one run
                        // of 32 bytes (convolution; synthesis, whose channels interleave)
                        if (KIND != KDEC && ys == 1 && (((uintptr_t)ystep) & 31) == 0) {
                            st256(ystep, outv[0], outv[1], outv[2], outv[3]);
                        } else if (KIND == KDEC && ys == 1 && ((((uintptr_t)ystep) | ((uintptr_t)(ystep + ycs))) & 15) == 0) {
                            *reinterpret_cast<double2 *>(ystep) = make_double2(outv[0], outv[2]);
                            *reinterpret_cast<double2 *>(ystep + ycs) = make_double2(outv[1], outv[3]);
                        } else {
#pragma unroll
                            for (int n = 0; n < 4; ++n) {
                                const int c = n % NCH;
                                *(c ? yq + ycs * c : yq) = outv[n];
                                if (c == NCH - 1) yq += yps;
                            }
                        }
                        continue;
                    }
                    if constexpr (FORM != FORM_ANY) {        // a partial step
#pragma unroll
                        for (int n = 0; n < 4; ++n) {
                            const int c = n % NCH;
                            if (n < nv) *(c ? yq + ycs : yq) = kMayX2 && x2 ? outv[n] + add[n] : outv[n];
                            if (c == NCH - 1) yq += yps;
                        }
                        continue;
                    }
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        const int q = q0 + n / NCH, c = n % NCH;
                        if (n >= nv) break;
                        double out = outv[n];
                        double *const yp = c ? yq + ycs * c : yq;
                        if (KIND == KCONV) {
                            const bool want_dot = !BATCH && S.has_dot;   // batched sweeps have no dot
                            if ((want_dot || S.has_ax) && (!grow || (q >= 0 && q < S.n))) {
                                                            const double xq = xrow[(long long)S.nL * (q - S.in_lo)];
                                if (want_dot) dot = fma(xq, out, dot);
                                if (S.has_ax) out = fma(xq, S.a_x, out);
                            }
                            if (kMayX2 && x2) out += add[n];
                        }
                        if (S.ay_mode == 2) out += *yp;
                        else if (S.ay_mode == 1) out = fma(S.a_y, *yp, out);
                        *yp = out;
                        if (c == NCH - 1) yq += yps;
                    }
                }
            };
            // the common case, a whole block of a plain sweep: one tight loop of straight
            // runs of eight outputs, so that recombination, conversion (the narrow
            // FP64 pipe) and stores of neighbouring outputs overlap
            constexpr std::integral_constant<int, RUN_VEC> vec_run{};
            constexpr std::integral_constant<int, RUN_ANY> any_run{};
            constexpr std::integral_constant<int, RUN_PART> last_run{};
            auto full_block = [&](int j) { return j < nb && qs + (j + 1) * PB - 1 <= S.qhi; };
            auto hot_block = [&](auto MODE, int j) {
                constexpr bool kHands = hands, kVec = MODE.value == RUN_VEC;
                const uint32_t blk = blk0 + j;
                double *yb = yrow + yps * (qs + j * PB - S.out_lo);
                const uint32_t ta = tmem + ((uint32_t)(lq * 32) << 16) + (blk % kTmemSlots) * G::SLOT_COLS;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    uint32_t acc[G::ORD][8];
#pragma unroll
                    for (int k = 0; k < G::ORD; ++k) tmem_ld8(ta + k * 16 + 8 * h, acc[k]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    if (h == 1) {             // the slot may be reissued
                        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) bar_arrive(drained(blk % kTmemSlots));
                    }
                    double v[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if constexpr (SCH == SCH_EXACT) {
                            uint32_t bb[G::ORD];
#pragma unroll
                            for (int k = 0; k < G::ORD; ++k) bb[k] = acc[k][i];
                            const long long Y = horner_bal<G::ORD>(bb, F, i % NCH);
                            v[i] = ll_scaled_fast(Y, se);
                        } else {                         // sum of the order accumulators
                            float f = __uint_as_float(acc[0][i]);
#pragma unroll
                            for (int k = 1; k < G::ORD; ++k) f += __uint_as_float(acc[k][i]);
                            v[i] = f32_to_f64(__float_as_uint(f));
                        }
                        if (!kVec) {
                            const int c = i % NCH;
                            if (valid) *(c ? yb + ycs : yb) = v[i];
                            if (c == NCH - 1) yb += yps;
                        }
                    }
                    if (kVec) {
                        // a contiguous output line takes its 8 outputs as two 32-byte
                        // runs: elements 0-7 (convolution; synthesis, whose channels
                        // interleave), or channel 0 and channel 1 (analysis)
                        if (valid) {
                            if (KIND == KDEC) {
                                st256(yb, v[0], v[2], v[4], v[6]);
                                st256(yb + ycs, v[1], v[3], v[5], v[7]);
                            } else {
                                st256(yb, v[0], v[1], v[2], v[3]);
                                st256(yb + 4, v[4], v[5], v[6], v[7]);
                            }
                        }
                        yb += 8 / NCH * yps;
                    }
                    if (kHands) hand_on(v, qs + j * PB + h * (8 / NCH), std::integral_constant<int, 8>());
                }
            };
            // a whole block with partial sums, dot product, a_x and a_y terms: four
            // outputs at a time, the next four's operands in flight meanwhile and the
            // group's next block's on their way to L2.  Bound by the chain of operand
            // latency, conversion and FP64 arithmetic in two warps per scheduler;
            // four outputs a step keep everything in registers (eight a step, and
            // operands two or four steps ahead, spill or outgrow the loop: kinetic
            // sweep with partial sums, 32 x 128^3, 580 us at eight, 480 at four, 515
            // with operands two steps ahead).  Kinetic sweeps with energies (and a_y),
            // 110^3 x 8, went through cold_block before: 213-349 us, now 164-199
            // a partial block in the same loop pays where the general block would have
            // the more to do (110^3 x 8 with energies: 3 % of the Hamiltonian), not
            // for partial sums alone (its code costs 32 x 128^3 2 %)
            constexpr bool kPartial = FORM == FORM_ANY;
            const bool want_dot = !BATCH && FORM == FORM_ANY && S.has_dot;
            const bool want_x = FORM == FORM_ANY && (want_dot || S.has_ax), want_y = FORM == FORM_ANY && S.ay_mode != 0;
            double ta[4], tx[4], ty[4];                  // the next four outputs' x2, x and y
            auto load_terms = [&](auto MODE, int q) {
                if (!valid) return;
                auto run = [&](double (&d)[4], const double *p, long long st) {
                    if constexpr (MODE.value == RUN_VEC) {
                        long long b0, b1, b2, b3;
                        ld256(reinterpret_cast<const long long *>(p), b0, b1, b2, b3);
                        d[0] = __longlong_as_double(b0), d[1] = __longlong_as_double(b1);
                        d[2] = __longlong_as_double(b2), d[3] = __longlong_as_double(b3);
                    } else {
#pragma unroll
                        for (int n = 0; n < 4; ++n) {
                            if (MODE.value != RUN_PART || q + n <= S.qhi) d[n] = *p;
                            p += st;
                        }
                    }
                };
                if (x2) run(ta, x2row + x2s * (q - x2lo), x2s);
                if (want_x) run(tx, xrow + (long long)S.nL * (q - S.in_lo), S.nL);
                if (want_y) run(ty, yrow + yps * (q - S.out_lo), yps);
            };
            auto term_block = [&](auto MODE, int j) {
                constexpr bool kVec = MODE.value == RUN_VEC, kPart = MODE.value == RUN_PART;
                const uint32_t blk = blk0 + j;
                const int q0 = qs + j * PB;
                const uint32_t tb = tmem + ((uint32_t)(lq * 32) << 16) + (blk % kTmemSlots) * G::SLOT_COLS;
                const bool more = full_block(j + 2), part = !more && j + 2 < nb;
                int nv = kPart ? S.qhi - q0 + 1 : 16;            // outputs left
                if (more && valid) {                     // the group's next block on its way to L2
                    const int q = q0 + 2 * PB + (lane & 15);
                    if (x2) prefetch_l2(x2row + x2s * (q - x2lo));
                    if (want_x) prefetch_l2(xrow + (long long)S.nL * (q - S.in_lo));
                    if (want_y) prefetch_l2(yrow + yps * (q - S.out_lo));
                }
                double *yb = yrow + yps * (q0 - S.out_lo);
#pragma unroll 1
                for (int st = 0; st < 4; ++st) {
                    uint32_t acc[G::ORD][4];
#pragma unroll
                    for (int k = 0; k < G::ORD; ++k) tmem_ld4(tb + k * 16 + 4 * st, acc[k]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    if (st == 3) {                       // the slot may be reissued
                        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) bar_arrive(drained(blk % kTmemSlots));
                    }
                    double v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if constexpr (SCH == SCH_EXACT) {
                            uint32_t bb[G::ORD];
#pragma unroll
                            for (int k = 0; k < G::ORD; ++k) bb[k] = acc[k][i];
                            const long long Y = horner_bal<G::ORD>(bb, F, 0);
                            // x2 alone: scale and partial sum in one FP64
                            // instruction (the product is exact)
                            if (x2 && !want_x) v[i] = fma(__ll2double_rn(Y), scale, ta[i]);
                            else v[i] = ll_scaled_fast(Y, se);
                        } else {
                            float f = __uint_as_float(acc[0][i]);
#pragma unroll
                            for (int k = 1; k < G::ORD; ++k) f += __uint_as_float(acc[k][i]);
                            v[i] = f32_to_f64(__float_as_uint(f));
                            if (x2 && !want_x) v[i] += ta[i];
                        }
                    }
                    if (want_x) {
                        if (want_dot && valid) {
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (!kPart || i < nv) dot = fma(tx[i], v[i], dot);
                        }
                        if (S.has_ax) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) v[i] = fma(tx[i], S.a_x, v[i]);
                        }
                        if (x2) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) v[i] += ta[i];
                        }
                    }
                    if (want_y) {
                        const double ay = S.ay_mode == 1 ? S.a_y : 1.0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) v[i] = fma(ay, ty[i], v[i]);
                    }
                    if (st < 3) load_terms(MODE, q0 + 4 * st + 4);
                    else if (more) load_terms(MODE, q0 + 2 * PB);
                    else if (kPartial && part) load_terms(last_run, q0 + 2 * PB);
                    if (valid) {
                        if (kVec) {
                            st256(yb, v[0], v[1], v[2], v[3]);
                        } else {
                            double *yp = yb;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (!kPart || i < nv) *yp = v[i];
                                yp += yps;
                            }
                        }
                    }
                    if (kPart) {
                        nv -= 4;
                        if (nv <= 0 && st < 3) {         // the rest of the block is not there
                            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                            __syncwarp();
                            if (lane == 0) bar_arrive(drained(blk % kTmemSlots));
                            break;
                        }
                    }
                    yb += 4 * yps;
                }
            };
            const bool vec = ys == 1 && (KIND == KDEC ? ((((uintptr_t)yrow | (uintptr_t)(yrow + ycs)) & 31) == 0)
                                                      : (((uintptr_t)yrow) & 31) == 0) &&
                             (yps * (qs - S.out_lo)) % 4 == 0;
            // cold_block: far rows, and a dot product or a_x term of a growing sweep,
            // whose input has no element for its outer outputs
            constexpr bool kTerms = KIND == KCONV && (FORM == FORM_ANY || FORM == FORM_X2);
            const bool hot = (kTerms || FORM != FORM_ANY) && !__any_sync(0xffffffffu, farrow) && !(want_x && grow);
            auto unit = [&](const double *p, long long st) { return st == 1 && (((uintptr_t)p) & 31) == 0; };
            const bool tvec = vec && (!x2 || unit(x2row + x2s * (qs - x2lo), x2s)) &&
                              (!want_x || unit(xrow + (long long)S.nL * (qs - S.in_lo), S.nL));
            const bool vecs = __all_sync(0xffffffffu, (kTerms ? tvec : vec) || !valid);
            if constexpr (kTerms)
                if (hot && j0 < nb) {
                    if (!full_block(j0)) { if (kPartial) load_terms(last_run, qs + j0 * PB); }
                    else if (vecs) load_terms(vec_run, qs + j0 * PB);
                    else load_terms(any_run, qs + j0 * PB);
                }
#pragma unroll 1
            for (int j = j0; j < nb; j += 2) {
                const uint32_t blk = blk0 + j;
                // issuing after the wait keeps the phases apart: the slabs that
                // block blk + 2's replaced in the ring were read by block blk or
                // an earlier one, so their phase is known to be over
                if (!bar_wait(tfull(blk % kTmemSlots), (blk / kTmemSlots) & 1) || !issue_next()) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                if (!hot || (!kPartial && !full_block(j))) {
                    cold_block(j);
                } else if constexpr (kTerms) {
                    if (kPartial && !full_block(j)) term_block(last_run, j);
                    else if (vecs) term_block(vec_run, j);
                    else term_block(any_run, j);
                } else if (vecs) {
                    hot_block(vec_run, j);
                } else {
                    hot_block(any_run, j);
                }
            }
        }
        if (!BATCH && FORM == FORM_ANY && S0.has_dot && dot_arr >= 0) flush_dot();
    }

    if (!alive) atomicExch(status, 1);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                     "r"(G::TMEM_COLS)
                     : "memory");
}

template <int KIND, int NT, int SCH, bool BATCH, int FORM>
cudaError_t set_smem_attr() {
    using G = Geom<KIND, NT, SCH>;
    static bool attr[64] = {};   // the attribute is set once per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr[dev]) {
        cudaError_t e = cudaFuncSetAttribute(sweep_tc_kernel<KIND, NT, SCH, BATCH, FORM>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr[dev] = true;
    }
    return cudaSuccess;
}

// The sweep may start while the kernels before it in the stream finish: its
// prologue (filter tiles, barriers, TMEM) needs nothing of theirs, and it waits
// for their completion before its first access to the caller's or the scratch
// memory (griddepcontrol.wait).  MagicFilter3D of one 32^3 grid 36 -> 28 us,
// Hamiltonian 48^3 x 8 1655 -> 1589 us
template <class Kernel, class... Args>
void launch_early(Kernel *kernel, unsigned grid, int smem, cudaStream_t st, const Args &...args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int KIND, int NT, int SCH, int FORM>
cudaError_t launch_form(const Sweep &S, const TcFilter &F, int *status, const int *lineE, cudaStream_t st) {
    using G = Geom<KIND, NT, SCH>;
    cudaError_t e = set_smem_attr<KIND, NT, SCH, false, FORM>();
    if (e != cudaSuccess) return e;
    launch_early(sweep_tc_kernel<KIND, NT, SCH, false, FORM>, (unsigned)sweep_tc_blocks(S), G::SMEM, st, S, F, status,
                 (const Sweep *)nullptr, (const long long *)nullptr, 0, lineE);
    return cudaGetLastError();
}

template <int KIND, int NT, int SCH>
cudaError_t launch(const Sweep &S_in, const TcFilter &F, int *status, const int *lineE,
                   cudaStream_t st) {
    using G = Geom<KIND, NT, SCH>;
    Sweep S = S_in;
    if (!tc_prepare(S)) return cudaErrorInvalidValue;
    if (S.has_dot || S.has_ax || S.ay_mode || (S.x2 && NT != 29))
        return launch_form<KIND, NT, SCH, FORM_ANY>(S, F, status, lineE, st);
    if constexpr (KIND == KCONV && NT == 29)
        if (S.x2) return launch_form<KIND, NT, SCH, FORM_X2>(S, F, status, lineE, st);
    if constexpr (SCH == SCH_EXACT && (KIND != KCONV || NT == 16))
        if (S.le_next) {
            // MagicFilter3D on 32 x 128^3: 1.083 ms this way, 1.114 with HAND2 for all
            if (S.le_n1 % 32 == 0 && (long long)S.nL * S.nR % 32 == 0)
                return launch_form<KIND, NT, SCH, FORM_HAND>(S, F, status, lineE, st);
            return launch_form<KIND, NT, SCH, FORM_HAND2>(S, F, status, lineE, st);
        }
    return launch_form<KIND, NT, SCH, FORM_PLAIN>(S, F, status, lineE, st);
}

// Batched launch over nsweeps descriptors (device arrays) of the form of `like`;
// S0 only carries has_dot = 0.  One CTA per SM.  lineE (exact scheme, or null):
// line exponent maxima of every sweep's lines, sweep i's at descs[i].le_off.
template <int KIND, int NT, int SCH, int FORM>
cudaError_t launch_batch_form(const Sweep *descs, const long long *prefix, int nsweeps,
                              const TcFilter &F, int *status, const int *lineE, cudaStream_t st) {
    using G = Geom<KIND, NT, SCH>;
    cudaError_t e = set_smem_attr<KIND, NT, SCH, true, FORM>();
    if (e != cudaSuccess) return e;
    Sweep S0{};
    launch_early(sweep_tc_kernel<KIND, NT, SCH, true, FORM>, (unsigned)sm_count(), G::SMEM, st, S0, F, status, descs,
                 prefix, nsweeps, lineE);
    return cudaGetLastError();
}

template <int KIND, int NT, int SCH>
cudaError_t launch_batch(const Sweep &like, const Sweep *descs, const long long *prefix, int nsweeps,
                         const TcFilter &F, int *status, const int *lineE, cudaStream_t st) {
    if constexpr (NT == 29) {
        if (like.has_ax || like.ay_mode)
            return launch_batch_form<KIND, NT, SCH, FORM_ANY>(descs, prefix, nsweeps, F, status, lineE, st);
        if (like.x2)
            return launch_batch_form<KIND, NT, SCH, FORM_X2>(descs, prefix, nsweeps, F, status, lineE, st);
    } else if (like.has_ax || like.ay_mode || like.x2) {
        return cudaErrorInvalidValue;
    }
    return launch_batch_form<KIND, NT, SCH, FORM_PLAIN>(descs, prefix, nsweeps, F, status, lineE, st);
}

}  // namespace tck
}  // namespace lcg
