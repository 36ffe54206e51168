// Tensor-core (tcgen05) sweeps: operand schemes, filter digits and launchers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "lcg_sweep.cuh"

namespace lcg {

// Operand schemes of the tensor-core sweep.
enum Scheme { SCH_EXACT = 0, SCH_BF16X3 = 1, SCH_TF32X3 = 2 };

// Filter operand planes, one entry per tap of the flat filter (convolution:
// the taps; wavelets: LE | LO | HE | HO), operator scalar folded in.
//   SCH_EXACT: balanced byte digits (in [-128, 127]) of the signed 62-bit
//     fixed point, times 2^8, as FP16 bit patterns, a*tap = 2^(ef-62) * sum_s
//     digit[s] 256^(7-s);
//   SCH_BF16X3: three bfloat16 terms (low 16 bits of dig[0..2]);
//   SCH_TF32X3: two tf32 terms (FP32 bit patterns in dig[0..1]).
struct TcFilter {
    static constexpr int kSlices = 8;
    static constexpr int kMaxTaps = 64;
    uint32_t dig[kSlices][kMaxTaps];
    int ef;
    // exact scheme, per output channel: what the recombination adds to the orders
    // 0-5 and to 256 times order 6 plus order 7 (the accumulators' biases and the
    // data digits' offsets leave, 512 rounds the latter)
    long long k64[2];
    uint32_t k67[2];
    // powers of two the kernel multiplies by, as values the compiler does not know
    uint32_t c1 = 1, c64 = 64, c256 = 256, c10 = 1024, c22 = 1u << 22;
};
// Bits of an FP32 accumulator at 1.5 * 2^23 units of 2^-16 (192).
constexpr uint32_t kAccBias = 0x43400000u;

// Host: operand planes of a * taps[0..ntaps) for scheme sch.
// (exact: kind and flat filter of the sweep, which fix the taps of each output channel).
void tc_filter_digits(int kind, const double *taps, int ntaps, double a, TcFilter &F);
void tc_filter_split(const double *taps, int ntaps, double a, int sch, TcFilter &F);
bool sweep_tc_supported(const Sweep &S);
// Fill S's strip length and strip-index divisors (Sweep::seg_blocks, tdiv_*) for
// a launch of `blocks` 128-line blocks (0: S's own); false when the sweep has
// 2^31 or more strips or lines (the kernel's 32-bit strip arithmetic).
bool tc_prepare(Sweep &S, long long blocks = 0);
long long sweep_tc_line_blocks(const Sweep &S);
// CTAs of the (non-batched) tensor-core sweep of S.  Its dot partials: one per
// epilogue warp, kTcDotSlots per CTA per array, array-major; the
// slots of an array a CTA has no strip of are not written.
constexpr int kTcDotSlots = 8;
long long sweep_tc_blocks(const Sweep &S);
// Windows of a line whose exponents an exact sweep takes one by one in its own
// pass (one per run of 64 outputs, over the elements that run reads), for periodic
// convolutions along lines at least as long as one window (16 taps 80 elements,
// 29 taps 96); 0 for other sweeps, which have one exponent per line.
int tc_windows(const Sweep &S);
// Exponents of S: one per line, or per line and window when S.le_win is set
// (entry window * sweep_tc_lines(S) + line).
long long sweep_tc_exps(const Sweep &S);
// status (device int) is set non-zero if a tensor-core wait timed out.
// lineE (exact scheme, or null): device scratch of sweep_tc_exps(S) ints; the
// largest exponent of each line or window is computed into it first (one read of
// the input), so the tensor-core sweep reads its input once.
// lineE_ready: lineE already holds the exponents (launch_line_exp3, or the lines'
// handed on); no pre-pass.
cudaError_t launch_sweep_tc(const Sweep &S, const TcFilter &F, int sch, int *status, int *lineE,
                            cudaStream_t st, bool lineE_ready = false);
// Line exponents of narr n0 x n1 x n2 grids along all three axes in one read
// of x (e0: n1 n2 narr, e1: n0 n2 narr, e2: n0 n1 narr ints), in the line
// order of the non-rotating sweeps along axes 0, 1, 2; wins (or null): the axes'
// exponent windows (tc_windows; 0: one exponent per line), each axis's ints times
// as many, for sweeps that line_exp3_windows takes.  active (or null):
// grids with active[a] == 0 are skipped (their entries stay 0).
bool line_exp3_windows(const Sweep &S);
cudaError_t launch_line_exp3(const double *x, int n0, int n1, int n2, int narr, const int *wins, int *e0, int *e1,
                             int *e2, cudaStream_t st, const int *active = nullptr);
long long sweep_tc_lines(const Sweep &S);
// Strips of one sweep (the unit a batched launch numbers consecutively).
long long sweep_tc_strips(const Sweep &S);
bool sweep_tc_batch_supported(int kind, int ntaps);
// One persistent launch over nsweeps sweeps (device descriptor array, strip
// prefix sums with prefix[nsweeps] = total) of one kind and filter.  Exact
// scheme with lineE: first one launch computes the largest exponent of every
// line of every sweep into lineE (sweep i's lines from descs[i].le_off on,
// exp_blocks blocks per sweep), so the sweeps read their input once.
cudaError_t launch_sweep_tc_batch(int kind, int ntaps, const Sweep &like, const Sweep *descs, const long long *prefix,
                                  int nsweeps, const TcFilter &F, int sch, int *status,
                                  int *lineE, int exp_blocks, cudaStream_t st, bool lineE_ready = false);
// Line exponents along all three axes of the grids of a batch in one read of x:
// descriptors (device) of the non-rotating sweeps along axes 0, 1, 2, exponent
// arrays of lines0, lines1 and lines2 ints; at most tiles tiles of 32 x 8 columns per
// grid, each in nseg segments of the third axis (line_exp3_batch_segments).
cudaError_t launch_line_exp3_batch(const Sweep *d0, const Sweep *d1, const Sweep *d2, int nsweeps, int *e0,
                                   long long lines0, int *e1, long long lines1, int *e2, long long lines2, int tiles,
                                   int nseg, cudaStream_t st);
int line_exp3_batch_segments(int tiles, int n2, int ngrids);
// Blocks per sweep of the batched line-exponent pass for ngrids sweeps whose largest
// line count (lines x narr) is max_lines, contiguous lines (nL == 1) or not.
int line_exp_batch_blocks(long long max_lines, bool contiguous, int ngrids);

namespace tck {
// 17-tap convolution (the Poisson finite differences), every scheme; its own
// translation unit.
cudaError_t launch_fd(const Sweep &S, const TcFilter &F, int sch, int *status, const int *lineE,
                      cudaStream_t st);
int sm_count();
// Per-scheme launchers (one translation unit each).
cudaError_t launch_exact(const Sweep &S, const TcFilter &F, int *status, const int *lineE,
                          cudaStream_t st);
cudaError_t launch_bf16x3(const Sweep &S, const TcFilter &F, int *status, const int *lineE,
                          cudaStream_t st);
cudaError_t launch_tf32x3(const Sweep &S, const TcFilter &F, int *status, const int *lineE,
                          cudaStream_t st);
cudaError_t launch_exact_batch(int kind, int ntaps, const Sweep &like, const Sweep *descs, const long long *prefix,
                               int nsweeps, const TcFilter &F, int *status, const int *lineE,
                               cudaStream_t st);
cudaError_t launch_bf16x3_batch(int kind, int ntaps, const Sweep &like, const Sweep *descs, const long long *prefix,
                                int nsweeps, const TcFilter &F, int *status, cudaStream_t st);
cudaError_t launch_tf32x3_batch(int kind, int ntaps, const Sweep &like, const Sweep *descs, const long long *prefix,
                                int nsweeps, const TcFilter &F, int *status, cudaStream_t st);
}  // namespace tck

}  // namespace lcg
