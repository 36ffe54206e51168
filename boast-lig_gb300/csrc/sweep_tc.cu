// Host side of the tensor-core sweeps: filter operand planes, support test,
// grid size and scheme dispatch.  The kernel itself is tc_kernel.cuh.
#include <cuda_fp16.h>
#include <math.h>
#include <string.h>

#include <algorithm>

#include "lcg_tc.cuh"

namespace lcg {
namespace tck {

namespace {
int g_sms[64] = {0};
}

constexpr int kWindow = 64;                  // outputs of an exponent window (tc_windows)

int sm_count() {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!g_sms[dev]) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        g_sms[dev] = n > 0 ? n : 148;
    }
    return g_sms[dev];
}

// Largest exponent field over the elements each line of S uses (positions
// 0..plen-1 of every channel; ld padding is not read), one int per line of
// every array.  Contiguous lines (nL == 1): a warp per line, lanes along the
// line, L of them at a time with I loads each in flight (1 and 4: 110^3 x 8 16 us,
// 25 one by one; a batch's short lines 4 and 2); strided lines: a thread per line,
// consecutive lines in a warp.
template <int L, int I>
__device__ __forceinline__ void line_exp_lines(const Sweep &S, int plen, int *out, long long first,
                                               long long step) {
    const int nchan = S.kind == KCONV ? 1 : 2;
    const long long nlines = (long long)S.nL * S.nR, total = nlines * S.narr;
    const long long pext = (long long)S.in_ext * nchan;
    auto offset = [&](int e) -> long long {          // element e of the used run
        if (S.kind == KCONV || S.kind == KDEC) return e;   // interleaved pairs: contiguous
        return e < plen ? e : (long long)(e - plen) + S.in_ext;   // blocked channels
    };
    const long long *xb = reinterpret_cast<const long long *>(S.x);
    const int count = plen * nchan;
    if (S.nL == 1) {
        const int lane = threadIdx.x & 31;
        const long long warps = step >> 5;
        const bool packed = S.x_arr == pext * nlines;    // line w of all arrays at pext w
        for (long long w = first >> 5; w < total; w += L * warps) {
            const long long *base[L];
            uint32_t mx[L];
#pragma unroll
            for (int k = 0; k < L; ++k) {
                const long long v = min(w + k * warps, total - 1);
                base[k] = xb + (packed ? pext * v : v / nlines * S.x_arr + pext * (v % nlines));
                mx[k] = 0;
            }
            for (int e0 = lane; e0 < count; e0 += 32 * I) {
                long long h[L][I];
#pragma unroll
                for (int i = 0; i < I; ++i) {
                    const int e = e0 + 32 * i;
#pragma unroll
                    for (int k = 0; k < L; ++k) h[k][i] = e < count ? base[k][offset(e)] : 0ll;
                }
#pragma unroll
                for (int k = 0; k < L; ++k)
#pragma unroll
                    for (int i = 0; i < I; ++i)
                        mx[k] = max(mx[k], (uint32_t)((unsigned long long)h[k][i] >> 32) & 0x7FF00000u);
            }
#pragma unroll
            for (int k = 0; k < L; ++k) {
                const uint32_t m = __reduce_max_sync(0xffffffffu, mx[k]);
                if (lane == 0 && w + k * warps < total) out[w + k * warps] = (int)(m >> 20);
            }
        }
    } else {
        for (long long t = first; t < total; t += step) {
            const long long arr = t / nlines, g = t % nlines;
            const long long l = g % S.nL, r = g / S.nL;
            const long long *base = xb + arr * S.x_arr + l + (long long)S.nL * pext * r;
            uint32_t mx = 0;
#pragma unroll 8
            for (int e = 0; e < count; ++e)
                mx = max(mx, (uint32_t)((unsigned long long)base[offset(e) * S.nL] >> 32) & 0x7FF00000u);
            out[t] = (int)(mx >> 20);
        }
    }
}

template <int I>
__global__ void line_exp_kernel(const Sweep S, int plen, int *out) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");   // the sweep's prologue may begin
    if (S.le_next)                       // the exponents that the sweep will hand on
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < S.le_next_lines * S.narr;
             i += (long long)gridDim.x * blockDim.x)
            S.le_next[i] = 0;
    line_exp_lines<1, I>(S, plen, out, (long long)blockIdx.x * blockDim.x + threadIdx.x,
                         (long long)gridDim.x * blockDim.x);
}

// Input positions 0..plen-1 a sweep's outputs read along its line: the whole
// line, or the used part of a shrink input.
__host__ __device__ __forceinline__ int line_exp_plen(const Sweep &S) {
    const int up = S.lowfil + S.ntaps - 1;
    return S.bc == BC_SHRINK ? S.qhi + up - S.in_lo + 1 : S.n;
}

// Exponents per line and window (Sweep::le_win): window w of a line is what its
// outputs 64 w .. 64 w + 63 read, positions qlo + 64 w + lowfil - woff on, at most
// 63 + ntaps + woff of them.  Contiguous lines: a warp per window (along x of 32 x
// 128^3, 16 taps: 117 us element by element, 102 with four elements a lane where
// windows start on 32 bytes; HBM 79); strided lines: a thread per line, a warp's
// windows one after another.  Windows of one line are neighbours, so what two of them
// read comes from L1 or L2 the second time.  by: divisors wins, nL nR and nL.
struct FastDiv {
    uint32_t d, m, s;
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const {
        return (uint32_t)(((unsigned long long)n * m) >> s);
    }
};
struct WindowDivs { FastDiv wins, lines, left; };

__global__ void __launch_bounds__(256, 8) window_exp_kernel(const Sweep S, const WindowDivs by, int *out) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");   // the sweep's prologue may begin
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    if (S.le_next)                       // the exponents that the sweep will hand on
        for (long long i = first; i < S.le_next_lines * S.narr; i += step) S.le_next[i] = 0;
    const long long *xb = reinterpret_cast<const long long *>(S.x);
    const uint32_t nlines = by.lines.d, total = nlines * (uint32_t)S.narr;
    const int n = S.n, lane = threadIdx.x & 31;
    const uint32_t wins = by.wins.d, warps = step >> 5;
    constexpr uint32_t kExp = 0x7FF00000u;
    auto start = [&](int w) { return S.qlo + kWindow * w + S.lowfil - S.woff; };
    auto count = [&](int w) {
        return min(kWindow + S.ntaps - 1 + S.woff, S.qhi + S.lowfil + S.ntaps - start(w));
    };
    auto field = [&](long long h) { return (uint32_t)((unsigned long long)h >> 32) & kExp; };
    // contiguous lines whose windows start on 32-byte boundaries: four elements a lane
    const bool quads = S.nL == 1 && n % 4 == 0 && S.in_ext % 4 == 0 && S.x_arr % 4 == 0 && start(0) % 4 == 0 &&
                       (((uintptr_t)S.x) & 31) == 0;
    if (quads) {
        const uint32_t units = total * wins;
        for (uint32_t u = first >> 5; u < units; u += warps) {
            const uint32_t line = by.wins(u), w = u - line * wins, arr = by.lines(line);
            const long long *base = xb + arr * S.x_arr + (long long)S.in_ext * (line - arr * nlines);
            const int p = start(w) + 4 * lane, q = p < 0 ? p + n : p >= n ? p - n : p;
            const int left = count(w) - 4 * lane;        // elements from the lane's first on
            uint32_t m = 0;
            if (left > 0) {
                const longlong4_32a h = *reinterpret_cast<const longlong4_32a *>(base + q);
                m = field(h.x);
                if (left > 1) m = max(m, field(h.y));
                if (left > 2) m = max(m, field(h.z));
                if (left > 3) m = max(m, field(h.w));
            }
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) out[w * total + line] = (int)(m >> 20);
        }
    } else if (S.nL == 1) {
        constexpr int L = 2, I = 3;                      // windows, and loads that cover one
        const uint32_t units = total * wins;
        for (uint32_t u = first >> 5; u < units; u += L * warps) {
            long long h[L][I];
            uint32_t at[L];
#pragma unroll
            for (int k = 0; k < L; ++k) {
                const uint32_t v = min(u + k * warps, units - 1), line = by.wins(v), w = v - line * wins;
                const uint32_t arr = by.lines(line);
                const long long *base = xb + arr * S.x_arr + (long long)S.in_ext * (line - arr * nlines);
                const int c = count(w);
                at[k] = w * total + line;
                int p = start(w) + lane;
#pragma unroll
                for (int i = 0; i < I; ++i) {
                    const int q = p < 0 ? p + n : p >= n ? p - n : p;
                    h[k][i] = lane + 32 * i < c ? base[q] : 0ll;
                    p += 32;
                }
            }
#pragma unroll
            for (int k = 0; k < L; ++k) {
                uint32_t m = 0;
#pragma unroll
                for (int i = 0; i < I; ++i) m = max(m, field(h[k][i]));
                m = __reduce_max_sync(0xffffffffu, m);
                if (lane == 0 && u + k * warps < units) out[at[k]] = (int)(m >> 20);
            }
        }
    } else {
        const uint32_t units = (total + 31) / 32 * wins;
        for (uint32_t u = first >> 5; u < units; u += warps) {
            const uint32_t block = by.wins(u), w = u - block * wins, line = block * 32 + lane;
            if (line >= total) continue;
            const uint32_t arr = by.lines(line), g = line - arr * nlines, r = by.left(g);
            const long long *base = xb + arr * S.x_arr + (g - r * S.nL) + (long long)S.nL * S.in_ext * r;
            const int c = count(w);
            int p = start(w);
            if (p < 0) p += n;
            uint32_t m = 0;
            for (int e = 0; e < c;) {                    // up to the line's end, then from its start
                const int run = min(c - e, n - p);
                const long long *q = base + (long long)S.nL * p;
#pragma unroll 8
                for (int i = 0; i < run; ++i) {
                    m = max(m, field(*q));
                    q += S.nL;
                }
                e += run;
                p = 0;
            }
            out[w * total + line] = (int)(m >> 20);
        }
    }
}

// The same maxima for a batch of sweeps: blockIdx.y = sweep, its lines'
// maxima written from out + le_off on.
__global__ void line_exp_batch_kernel(const Sweep *__restrict__ descs, int *out) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const Sweep &S = descs[blockIdx.y];
    line_exp_lines<4, 2>(S, line_exp_plen(S), out + S.le_off,
                   (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

// Per-line exponent maxima of one n0 x n1 x n2 grid (narr of them, back to
// back) along all three axes in one read: e0[i1 + n1 (i2 + n2 a)] over i0,
// e1[i0 + n0 (i2 + n2 a)] over i1, e2[i0 + n0 (i1 + n1 a)] over i2 -- the
// line orders of the three non-rotating sweeps of the grid.  Block: 32 i0 x
// 8 i1 threads over one segment of i2 (blockIdx.z = a nseg + segment), in
// chunks of 8 planes (the next chunk's 8 loads in flight while one chunk is
// reduced).  e2 is a thread's own maximum; each chunk is staged in shared
// memory (rows padded to 33 words, so the row and the column reads below are
// free of bank conflicts), where 4 threads per (plane, i1) row reduce the 32
// i0 values for e0 and one thread per (plane, i0) column the 8 i1 values for
// e1.  Partial maxima are
// combined across blocks with atomicMax (e0, e1 and, with several segments,
// e2 zeroed first).
constexpr int kExpChunk = 8;
// Exponent windows of the three axes (0: the axis has one exponent per line), each
// axis's lines in all grids, and its pieces of 8.
struct Exp3Windows {
    int wins[3] = {0, 0, 0};
    long long lines[3] = {0, 0, 0};
};

// Raise to m the exponent of the line at e, or those of its windows that read piece c
// (elements 8 c .. 8 c + 7 of n): a 17-tap window, elements 64 w - 8 .. 64 w + 71, is
// ten such pieces, the first and the last of them its neighbours' too.
__device__ __forceinline__ void exp3_edges(int *e, int c, int n, int wins, long long lines, int m) {
    const int w = c >> 3;
    if ((c & 7) == 0) atomicMax(e + (w ? w - 1 : wins - 1) * lines, m);
    if ((c & 7) == 7 || 8 * (c + 1) >= n) atomicMax(e + (w + 1 < wins ? w + 1 : 0) * lines, m);
}
template <bool WIN>
__device__ __forceinline__ void exp3_raise(int *e, int c, int n, int wins, long long lines, int m) {
    if (!WIN || !wins) {
        atomicMax(e, m);
        return;
    }
    atomicMax(e + (c >> 3) * lines, m);
    exp3_edges(e, c, n, wins, lines, m);
}

// The block's 32 i0 x 8 i1 columns from (b0, b1) on, planes [zb, ze) of one grid.
// WIN: some axis has windows (its extent and zb are multiples of 8).
template <bool WIN>
__device__ __forceinline__ void line_exp3_block(const double *__restrict__ x, int n0, int n1, int n2, int b0, int b1,
                                                int zb, int ze, int *__restrict__ e0, int *__restrict__ e1,
                                                int *__restrict__ e2, const Exp3Windows &W = Exp3Windows()) {
    __shared__ int ys[kExpChunk][8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i0 = b0 + tx, i1 = b1 + ty;
    const bool valid = i0 < n0 && i1 < n1;
    const long long plane = (long long)n0 * n1;
    const unsigned long long *xa = reinterpret_cast<const unsigned long long *>(x) + i0 + (long long)n0 * i1;
    // e1 reader: column (c1, tx) of the chunk; e0 reader: quarter q0 of row (c0r, r0)
    const int c1 = ty, row = threadIdx.x >> 2, q0 = threadIdx.x & 3;
    const int c0r = row >> 3, r0 = row & 7;
    const int i1r = b1 + r0;
    int *const column = e2 + i0 + (long long)n0 * i1;
    int zmax = 0;
    // the next chunk's loads are in flight while this chunk is reduced
    unsigned long long raw[kExpChunk];
#pragma unroll
    for (int c = 0; c < kExpChunk; ++c) raw[c] = (valid && zb + c < ze) ? xa[plane * (zb + c)] : 0ull;
    for (int c0 = zb; c0 < ze; c0 += kExpChunk) {
        int e[kExpChunk];
#pragma unroll
        for (int c = 0; c < kExpChunk; ++c) e[c] = (int)((raw[c] >> 52) & 0x7FF);
        const int c1n = c0 + kExpChunk;
#pragma unroll
        for (int c = 0; c < kExpChunk; ++c) raw[c] = (valid && c1n + c < ze) ? xa[plane * (c1n + c)] : 0ull;
        if (WIN && W.wins[2]) zmax = 0;
#pragma unroll
        for (int c = 0; c < kExpChunk; ++c) {
            zmax = max(zmax, e[c]);
            ys[c][ty][tx] = e[c];
        }
        if (WIN && W.wins[2] && valid) exp3_raise<true>(column, c0 / 8, n2, W.wins[2], W.lines[2], zmax);
        __syncthreads();
        if (c0 + c1 < ze && i0 < n0) {
            int m = ys[c1][0][tx];
#pragma unroll
            for (int r = 1; r < 8; ++r) m = max(m, ys[c1][r][tx]);
            exp3_raise<WIN>(e1 + i0 + (long long)n0 * (c0 + c1), b1 / 8, n1, W.wins[1], W.lines[1], m);
        }
        {
            int m = ys[c0r][r0][8 * q0];
#pragma unroll
            for (int k = 1; k < 8; ++k) m = max(m, ys[c0r][r0][8 * q0 + k]);
            const bool keeps = c0 + c0r < ze && i1r < n1;
            int *const line = e0 + i1r + (long long)n1 * (c0 + c0r);
            // the four quarters lie in one run of 64; its ends are the outer ones'
            if (WIN && W.wins[0] && keeps && b0 + 8 * q0 < n0) exp3_edges(line, b0 / 8 + q0, n0, W.wins[0], W.lines[0], m);
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
            if (q0 == 0 && keeps) atomicMax(line + (WIN && W.wins[0] ? (b0 >> 6) * W.lines[0] : 0), m);
        }
        __syncthreads();
    }
    if (valid && !(WIN && W.wins[2])) {
        if (zb == 0 && ze == n2) *column = zmax;
        else atomicMax(column, zmax);
    }
}

template <bool WIN>
__global__ void __launch_bounds__(256)
line_exp3_kernel(const double *__restrict__ x, int n0, int n1, int n2, int nseg, int seglen,
                 int *__restrict__ e0, int *__restrict__ e1, int *__restrict__ e2,
                 const int *__restrict__ active, const __grid_constant__ Exp3Windows W) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const long long a = blockIdx.z / nseg;
    if (active && !active[a]) return;                   // grid skipped (uniform over the block)
    const int zb = blockIdx.z % nseg * seglen;
    if (zb >= n2) return;                               // more segments than seglen fills
    line_exp3_block<WIN>(x + a * n0 * n1 * n2, n0, n1, n2, blockIdx.x * 32, blockIdx.y * 8, zb, min(n2, zb + seglen),
                         e0 + a * n1 * n2, e1 + a * n0 * n2, e2 + a * n0 * n1, W);
}

// The same for the grids of a batch: d0, d1, d2 describe the non-rotating sweeps
// along axes 0, 1, 2 of each grid (all read the same x), whose exponents start at
// their le_off.  blockIdx.y = grid, whose 32 x 8 columns and nseg segments of the third
// axis its blocks share.
__global__ void __launch_bounds__(256)
line_exp3_batch_kernel(const Sweep *__restrict__ d0, const Sweep *__restrict__ d1, const Sweep *__restrict__ d2,
                       int *__restrict__ e0, int *__restrict__ e1, int *__restrict__ e2, int nseg) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const Sweep &S = d1[blockIdx.y];
    const int n0 = S.nL, n1 = S.n, n2 = S.nR, gx = (n0 + 31) / 32, tiles = gx * ((n1 + 7) / 8);
    const int seglen = (n2 + nseg - 1) / nseg;
    for (int t = blockIdx.x; t < tiles * nseg; t += gridDim.x) {
        const int tile = t % tiles, zb = t / tiles * seglen;
        if (zb < n2)
            line_exp3_block<false>(S.x, n0, n1, n2, tile % gx * 32, tile / gx * 8, zb, min(n2, zb + seglen),
                            e0 + d0[blockIdx.y].le_off, e1 + S.le_off, e2 + d2[blockIdx.y].le_off);
    }
}

}  // namespace tck

constexpr int kExpChunkHost = tck::kExpChunk;

long long sweep_tc_lines(const Sweep &S) { return (long long)S.nL * S.nR * S.narr; }

// A window's scale is its own, so small values far from a line's large ones keep 62
// bits below their neighbours' magnitude, and an Inf or NaN spoils 64 outputs, not the
// line.  Only where a line's exponents come from the sweep's own pass: handed-on and
// shared ones are the line's, as are those of lines of less than a window, of other
// boundaries and of wavelets.
int tc_windows(const Sweep &S) {
    if (S.kind != KCONV || S.bc != BC_PERIODIC || S.n < tck::kWindow - 16 + (S.ntaps + 30) / 16 * 16) return 0;
    return (S.qhi - S.qlo + tck::kWindow) / tck::kWindow;
}

long long sweep_tc_exps(const Sweep &S) { return sweep_tc_lines(S) * (S.le_win > 0 ? S.le_win : 1); }

// Extents whose exponent windows the shared pass can take: the windows of a 17-tap
// filter (8 elements on each side) over whole pieces of 8.
bool line_exp3_windows(const Sweep &S) { return S.ntaps == 17 && S.lowfil == -8 && S.qlo == 0 && S.n % 8 == 0; }

cudaError_t launch_line_exp3(const double *x, int n0, int n1, int n2, int narr, const int *wins, int *e0, int *e1,
                             int *e2, cudaStream_t st, const int *active) {
    if (n0 < 1 || n1 < 1 || n2 < 1 || narr < 1 || narr > 65535) return cudaErrorInvalidValue;
    const long long gx = (n0 + 31) / 32, gy = (n1 + 7) / 8;
    // segments of i2 so that a few grids still give the GPU about 8 blocks per SM
    const long long want = 8LL * tck::sm_count();
    long long nseg = (want + gx * gy * narr - 1) / (gx * gy * narr);
    const long long most = (n2 + kExpChunkHost - 1) / kExpChunkHost;
    if (nseg > most) nseg = most;
    if (nseg > 65535 / narr) nseg = 65535 / narr;
    if (nseg < 1) nseg = 1;
    int seglen = (int)((n2 + nseg - 1) / nseg);
    tck::Exp3Windows W;
    size_t c[3] = {(size_t)n1 * n2 * narr, (size_t)n0 * n2 * narr, (size_t)n0 * n1 * narr};
    bool win = false;
    for (int k = 0; k < 3; ++k) {
        W.lines[k] = (long long)c[k];
        W.wins[k] = wins ? wins[k] : 0;
        if (W.wins[k] > 0) win = true, c[k] *= (size_t)W.wins[k];
    }
    if (W.wins[2] > 0) seglen = (seglen + 7) / 8 * 8;
    // one clear when the three lie back to back
    const bool clear2 = nseg > 1 || W.wins[2] > 0;
    cudaError_t e;
    if (e1 == e0 + c[0] && e2 == e1 + c[1]) {
        e = cudaMemsetAsync(e0, 0, (c[0] + c[1] + (clear2 ? c[2] : 0)) * sizeof(int), st);
    } else {
        e = cudaMemsetAsync(e0, 0, c[0] * sizeof(int), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(e1, 0, c[1] * sizeof(int), st);
        if (e == cudaSuccess && clear2) e = cudaMemsetAsync(e2, 0, c[2] * sizeof(int), st);
    }
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)(narr * nseg));
    if (win) tck::line_exp3_kernel<true><<<grid, 256, 0, st>>>(x, n0, n1, n2, (int)nseg, seglen, e0, e1, e2, active, W);
    else tck::line_exp3_kernel<false><<<grid, 256, 0, st>>>(x, n0, n1, n2, (int)nseg, seglen, e0, e1, e2, active, W);
    return cudaGetLastError();
}

// Divisor d with its inverse for n < 2^31: s = 31 + ceil(log2 d),
// m = ceil(2^s / d) < 2^32, floor(n / d) = (n m) >> s (the error term
// n (m - 2^s / d) / 2^s stays below 1 / d).
static void fast_div(unsigned int d, unsigned int &dd, unsigned int &m, unsigned int &s) {
    unsigned int l = 0;
    while ((1ull << l) < d) ++l;
    dd = d;
    s = 31 + l;
    m = (unsigned int)(((1ull << s) + d - 1) / d);
}

// 128-line blocks of one sweep (all narr arrays), 16-element output blocks
// along a line, and slabs a block reads (Geom::W).
static long long line_blocks(const Sweep &S) {
    return ((long long)S.nL * S.nR + 127) / 128 * S.narr;
}
static int out_blocks(const Sweep &S) {
    const int pb = S.kind == KCONV ? 16 : 8;
    return (S.qhi - S.qlo + pb) / pb;
}
static int window_slabs(const Sweep &S) {
    const int nch = S.kind == KCONV ? 1 : 2;
    return (nch * (16 / nch + S.ntaps - 1) + 15) / 16;
}

// Output blocks per strip, for `blocks` line blocks in the launch: the split
// of the lines that gives the busiest CTA the least slabs to convert (its
// strips times nb + W - 1); whole lines unless a launch has few of them.  With an
// exponent per window (4 blocks) a strip is a window, or a half or a quarter of one.
static int strip_blocks(const Sweep &S, long long blocks) {
    const int n = out_blocks(S), halo = window_slabs(S) - 1, sms = tck::sm_count();
    int best = n;
    long long cost = -1;
    auto consider = [&](int nb) {
        const long long strips = blocks * ((n + nb - 1) / nb);
        const long long c = (strips + sms - 1) / sms * (nb + halo);
        if (cost < 0 || c < cost) {
            cost = c;
            best = nb;
        }
    };
    if (S.le_win > 0) {
        for (int nb = tck::kWindow / 16; nb >= 1; nb /= 2) consider(nb);
    } else {
        // as many segments as give every CTA a strip: 64 at most left 88 of 152 SMs idle
        // for a few long lines (one of 10^6 points, kinetic filter, BF16x3: 2540 us, now
        // 1084; 1217 as tiles of 64 outputs)
        const long long most = std::max<long long>(64, (sms + blocks - 1) / blocks);
        for (int seg = 1; seg <= n && seg <= most; ++seg) consider((n + seg - 1) / seg);
    }
    return best;
}

bool tc_prepare(Sweep &S, long long blocks) {
    const long long nlines = (long long)S.nL * S.nR, nlb = (nlines + 127) / 128;
    S.seg_blocks = strip_blocks(S, blocks > 0 ? blocks : line_blocks(S));
    const long long seg = (out_blocks(S) + S.seg_blocks - 1) / S.seg_blocks;
    if (nlines < 1 || nlines >= (1LL << 31) || seg * nlb * S.narr >= (1LL << 31)) return false;
    fast_div((unsigned int)seg, S.tdiv_d[0], S.tdiv_m[0], S.tdiv_s[0]);
    fast_div((unsigned int)nlb, S.tdiv_d[1], S.tdiv_m[1], S.tdiv_s[1]);
    fast_div((unsigned int)S.nL, S.tdiv_d[2], S.tdiv_m[2], S.tdiv_s[2]);
    return true;
}

bool sweep_tc_supported(const Sweep &S) {
    if (S.kind == KCONV) return S.ntaps == 16 || S.ntaps == 17 || S.ntaps == 29;
    return (S.kind == KDEC || S.kind == KREC) && (S.ntaps == 8 || S.ntaps == 16);
}

long long sweep_tc_strips(const Sweep &S) {
    const int nb = S.seg_blocks > 0 ? S.seg_blocks : strip_blocks(S, line_blocks(S));
    return line_blocks(S) * ((out_blocks(S) + nb - 1) / nb);
}

long long sweep_tc_line_blocks(const Sweep &S) { return line_blocks(S); }

long long sweep_tc_blocks(const Sweep &S) {
    const long long strips = sweep_tc_strips(S);
    const int sms = tck::sm_count();
    return strips < sms ? strips : sms;
}

// Filter digits with the operator scalar folded in exactly: a*f is formed as
// the 106-bit product of the two mantissas, then rounded once to the signed
// fixed point F = a f 2^(62 - ef), |F| <= 2^62 (ef: power of two above the
// largest |a f| of the whole flat filter, so every channel pair shares one
// scale; raised further while the sum of |a f| reaches 8 * 2^ef, which keeps
// the kernel's recombined 64-bit result below 2^61).  F is cut into 8
// balanced byte digits e_0 (top) .. e_7 in [-128, 127]:
// F = sum_t e_t 256^(7-t), the bytes of F + 0x8080808080808080 minus 128.
// The operand holds the data's balanced digits plus 128 (0..255), so order k's
// accumulator lies between minus and plus 255 times the sums of the negative
// and of the positive digits e_0 .. e_k of an output's taps; both must stay
// within the 2^22 units that the biased FP32 accumulator holds exactly.  The
// library's filters reach half of that; where a scalar's digits do not fit, ef
// is raised by one and the digits cut again.
void tc_filter_digits(int kind, const double *taps, int ntaps, double a, TcFilter &F) {
    F = TcFilter{};
    memset(F.dig, 0, sizeof(F.dig));
    int ea = 0;
    const double fa = frexp(fabs(a), &ea);                          // |a| = fa 2^ea
    const unsigned long long ma = (unsigned long long)ldexp(fa, 53);  // 53-bit integer
    unsigned __int128 prod[TcFilter::kMaxTaps];
    int ep[TcFilter::kMaxTaps];
    int ef = -100000;
    double sum = 0.0;
    for (int i = 0; i < ntaps; ++i) {
        int e = 0;
        const double ff = frexp(fabs(taps[i]), &e);
        const unsigned long long mf = (unsigned long long)ldexp(ff, 53);
        prod[i] = (unsigned __int128)ma * mf;
        ep[i] = (ea - 53) + (e - 53);                               // |a f| = prod 2^ep
        sum += fabs(a * taps[i]);
        if (prod[i]) {
            int bl = 0;
            for (unsigned __int128 t = prod[i]; t; t >>= 1) ++bl;
            if (bl + ep[i] > ef) ef = bl + ep[i];                   // |a f| < 2^(bl + ep)
        }
    }
    if (ef == -100000) ef = 0;
    while (sum >= ldexp(8.0, ef)) ++ef;
    // output channel of a tap of the flat filter: wavelet decompose LE, LO give
    // the first and HE, HO the second; recompose LO, HO the first, LE, HE the second
    const int nt = kind == KCONV ? ntaps : ntaps / 4;
    auto channel = [&](int i) {
        return kind == KCONV ? 0 : kind == KDEC ? (i / nt >= 2) : (i / nt) % 2 == 0;
    };
    constexpr long long kMost = 1ll << 22;
    for (bool fits = false; !fits; ++ef) {
        F.ef = ef;
        long long esum[TcFilter::kSlices][2] = {}, pos[2] = {}, neg[2] = {};
        fits = true;
        for (int t = 0; t < TcFilter::kSlices; ++t)
            for (int i = 0; i < ntaps; ++i) {
                const int sh = ep[i] + 62 - ef;                     // |F| = prod 2^sh <= 2^62
                const unsigned __int128 v = prod[i];
                unsigned long long M;
                if (sh >= 0) M = (unsigned long long)(v << sh);
                else if (-sh >= 127) M = 0;
                else M = (unsigned long long)((v + ((unsigned __int128)1 << (-sh - 1))) >> (-sh));
                const bool negative = (a < 0) != (taps[i] < 0);
                const unsigned long long X = negative ? 0ull - M : M;   // two's complement
                const unsigned long long U = X + 0x8080808080808080ull;
                const int digit = (int)((U >> (8 * (7 - t))) & 0xFF) - 128, c = channel(i);
                F.dig[t][i] = __half_as_ushort(__int2half_rn(digit * 256));
                esum[t][c] += digit;
                (digit > 0 ? pos[c] : neg[c]) += digit > 0 ? digit : -digit;
                fits = fits && 255 * pos[c] <= kMost && 255 * neg[c] <= kMost;
            }
        // biases of the eight accumulators (modulo 2^32 for a pair of orders) and the
        // offsets C_k = 128 sum_t<=k esum[t] of the data digits, subtracted
        constexpr uint32_t kPair = 257u * kAccBias;
        for (int c = 0; c < 2; ++c) {
            unsigned long long k64 = (unsigned long long)kPair * ((1ull << 38) + (1ull << 22) + (1ull << 6));
            long long ck = 0;
            for (int k = 0; k < 6; ++k) {
                ck += 128 * esum[k][c];
                k64 += (unsigned long long)ck << (46 - 8 * k);
            }
            const long long c6 = ck + 128 * esum[6][c], c7 = c6 + 128 * esum[7][c];
            F.k64[c] = (long long)(0ull - k64);
            F.k67[c] = 512u - kPair - (uint32_t)(256 * c6 + c7);
        }
    }
}

// bfloat16 x 3 or tf32 x 2 terms of the FP32 value of a*f (rounded to
// nearest); each term is its remainder rounded to nearest (ties away from
// zero), each remainder exact in FP32 -- the split the kernel applies to x.
void tc_filter_split(const double *taps, int ntaps, double a, int sch, TcFilter &F) {
    memset(&F, 0, sizeof(F));
    const int nsplit = sch == SCH_BF16X3 ? 3 : 2;
    const uint32_t mask = sch == SCH_BF16X3 ? 0xFFFF0000u : 0xFFFFE000u;
    const uint32_t half = (~mask + 1u) >> 1;
    for (int i = 0; i < ntaps; ++i) {
        float r = (float)(a * taps[i]);
        for (int s = 0; s < nsplit; ++s) {
            uint32_t b;
            memcpy(&b, &r, 4);
            const uint32_t h = (b + half) & mask;
            float hf;
            memcpy(&hf, &h, 4);
            F.dig[s][i] = sch == SCH_BF16X3 ? (h >> 16) : h;
            r = r - hf;
        }
    }
}

bool sweep_tc_batch_supported(int kind, int ntaps) {
    return kind == KCONV && (ntaps == 16 || ntaps == 29);
}

int line_exp_batch_blocks(long long max_lines, bool contiguous, int ngrids) {
    // four lines a warp; each block first waits for its descriptor, so not too many
    // of them (128 grids, axes 24-72, a MagicFilter and kinetic run: 1349, 1306, 1319 and
    // 1384 us with at most 16, 32, 64 and 256 per grid), but two for every SM in all:
    // with these and the segments of the shared pass, runs over one grid of 72^3
    // 126 -> 87 us, two 158 -> 123, three of 120^3 579 -> 419, four of 40-72 125 -> 113
    const long long threads = contiguous ? max_lines * (32 / 4) : max_lines;
    const long long want = (threads + 255) / 256;
    const long long most = std::max<long long>(32, (2LL * tck::sm_count() + ngrids - 1) / ngrids);
    return (int)(want < 1 ? 1 : want > most ? most : want);
}

cudaError_t launch_line_exp3_batch(const Sweep *d0, const Sweep *d1, const Sweep *d2, int nsweeps, int *e0,
                                   long long lines0, int *e1, long long lines1, int *e2, long long lines2, int tiles,
                                   int nseg, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(e0, 0, (size_t)lines0 * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(e1, 0, (size_t)lines1 * sizeof(int), st);
    if (e == cudaSuccess && nseg > 1) e = cudaMemsetAsync(e2, 0, (size_t)lines2 * sizeof(int), st);
    if (e != cudaSuccess) return e;
    const int blocks = std::min(256, tiles * nseg);
    tck::line_exp3_batch_kernel<<<dim3(blocks < 1 ? 1 : blocks, nsweeps), 256, 0, st>>>(d0, d1, d2, e0, e1, e2, nseg);
    return cudaGetLastError();
}

// Segments of the third axis (n2 long) that give ngrids grids of `tiles` 32 x 8 column
// tiles two blocks for every SM; chunks of 8 planes are the shortest.
int line_exp3_batch_segments(int tiles, int n2, int ngrids) {
    const long long blocks = std::max(1LL, (long long)tiles * ngrids), want = 2LL * tck::sm_count();
    const long long most = (n2 + kExpChunkHost - 1) / kExpChunkHost;
    return (int)std::max(1LL, std::min(most, (want + blocks - 1) / blocks));
}

cudaError_t launch_sweep_tc_batch(int kind, int ntaps, const Sweep &like, const Sweep *descs, const long long *prefix,
                                  int nsweeps, const TcFilter &F, int sch, int *status,
                                  int *lineE, int exp_blocks, cudaStream_t st, bool lineE_ready) {
    if (sch == SCH_EXACT) {
        if (lineE && !lineE_ready) {
            if (exp_blocks < 1 || nsweeps > 65535) return cudaErrorInvalidValue;
            tck::line_exp_batch_kernel<<<dim3(exp_blocks, nsweeps), 256, 0, st>>>(descs, lineE);
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
        return tck::launch_exact_batch(kind, ntaps, like, descs, prefix, nsweeps, F, status, lineE, st);
    }
    if (sch == SCH_BF16X3) return tck::launch_bf16x3_batch(kind, ntaps, like, descs, prefix, nsweeps, F, status, st);
    if (sch == SCH_TF32X3) return tck::launch_tf32x3_batch(kind, ntaps, like, descs, prefix, nsweeps, F, status, st);
    return cudaErrorInvalidValue;
}

cudaError_t launch_sweep_tc(const Sweep &S_in, const TcFilter &F, int sch, int *status, int *lineE,
                            cudaStream_t st, bool lineE_ready) {
    Sweep S = S_in;
    // contiguous periodic lines of a filter whose K blocks leave room: start
    // the window on a 4-element boundary (32-byte aligned groups)
    if (S.kind == KCONV && 16 * window_slabs(S) - 15 - S.ntaps >= 3 && S.nL == 1 && S.bc == BC_PERIODIC &&
        S.n % 4 == 0 && S.in_ext % 4 == 0 && S.x_arr % 4 == 0 && (((uintptr_t)S.x) & 31) == 0)
        S.woff = ((S.qlo + S.lowfil) % 4 + 4) % 4;
    if (sch == SCH_EXACT) {
        if (S.le_win > 0 && !lineE) return cudaErrorInvalidValue;
        if (lineE && !lineE_ready) {
            const long long total = sweep_tc_lines(S);
            // threads with something to do: a warp per contiguous line or window, a
            // thread per strided line (and window)
            const long long units = S.nL == 1 ? total : (total + 31) / 32;
            const long long want = (units * (S.le_win > 0 ? S.le_win : 1) + 7) / 8;
            const int grid = (int)(want < 8LL * tck::sm_count() ? want : 8LL * tck::sm_count());
            if (S.le_win > 0) {
                if (sweep_tc_exps(S) >= (1LL << 31)) return cudaErrorInvalidValue;   // 32-bit window numbers
                tck::WindowDivs by;
                fast_div((unsigned int)S.le_win, by.wins.d, by.wins.m, by.wins.s);
                fast_div((unsigned int)(total / S.narr), by.lines.d, by.lines.m, by.lines.s);
                fast_div((unsigned int)S.nL, by.left.d, by.left.m, by.left.s);
                tck::window_exp_kernel<<<grid > 0 ? grid : 1, 256, 0, st>>>(S, by, lineE);
            } else {
                // a warp or two an SM: more loads in flight for each (one line of 10^6 points,
                // kinetic filter: the call 2773 us with four, 2121 with eight)
                const int plen = tck::line_exp_plen(S);
                if (units < 2LL * tck::sm_count()) tck::line_exp_kernel<8><<<grid > 0 ? grid : 1, 256, 0, st>>>(S, plen, lineE);
                else tck::line_exp_kernel<4><<<grid, 256, 0, st>>>(S, plen, lineE);
            }
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
        return tck::launch_exact(S, F, status, lineE, st);
    }
    if (sch == SCH_BF16X3) return tck::launch_bf16x3(S, F, status, nullptr, st);
    if (sch == SCH_TF32X3) return tck::launch_tf32x3(S, F, status, nullptr, st);
    return cudaErrorInvalidValue;
}

}  // namespace lcg
