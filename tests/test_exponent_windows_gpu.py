"""Exact sweeps of long periodic lines scale each run of 64 outputs by the largest magnitude
that run reads, not by the line's: small values far from a line's large ones keep the accuracy
of an FP64 chain, and an Inf or NaN stays within the runs that read it.

A run's bound: its outputs' error against the oracle is at most 1e-13 times the largest input the
run reads times the filter's absolute sum (the data truncation is 2^-62 of that input, the rest are
roundings of the results)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-13
OPS = {'d_s0s0_1d_sym8_md': (-8, 16), 'd_s0s0_1d_sym8_imd': (-7, 16), 'd_s0s0_1d_sym8_d1': (-14, 29),
       'd_s0s0_1d_sym8_d2_dotin': (-14, 29)}


@pytest.fixture(autouse=True)
def exact(pkg):
    with pkg.mode(pkg.MODE_TC_EXACT):
        yield


def steep(seed, lines, n, step=45, width=100):
    """Lines whose magnitude falls by 2^-step every `width` positions (wrapping to 1), each from
    another position on."""
    r = np.random.default_rng(seed)
    x = r.uniform(-1.0, 1.0, (lines, n))
    k = (np.arange(n)[None, :] + 37 * np.arange(lines)[:, None]) // width % 3
    return x * 2.0 ** (-step * k)


def run_scales(x, low, taps):
    """Largest input that each 64-output run of a periodic line reads (up to 3 elements more, which a
    contiguous 29-tap line's aligned loads take in), per output."""
    n = x.shape[-1]
    out = np.zeros_like(x)
    for q in range(0, n, 64):
        at = np.arange(q + low - 3, min(q + 64, n) + low + taps - 1) % n
        out[..., q:q + 64] = np.abs(x[..., at]).max(axis=-1, keepdims=True)
    return out


def apply_1d(pkg, O, op, x, idim, both=True):
    """The operator along the last axis of x (lines, n), laid out with the lines' axis first or last."""
    lines, n = x.shape
    shape = [n, lines] if idim == 0 else [lines, n]
    lay = (lambda v: v) if idim == 0 else np.transpose
    xi = np.ascontiguousarray(lay(x)).ravel()
    y, yo = np.zeros_like(xi), np.zeros_like(xi)
    args = [2, idim, shape, 0, shape, shape, 1, xi]
    tail = (1.0, 0.0, 0.0)
    if op.endswith('dotin'):
        st = pkg.Kernel(op).run(*args, y, *tail, None)
        d = ctypes.c_double(0.0)
        if both:
            assert O.call('oracle_' + op, *args, yo, *tail, ctypes.pointer(d)) == 0
            assert abs(st['reference_return']['dot_in'] - d.value) <= TOL * (np.abs(xi) * np.abs(yo)).sum() * 4
    else:
        pkg.Kernel(op).run(*args, y, *tail)
        if both:
            assert O.call('oracle_' + op, *args, yo, *tail) == 0
    back = lambda v: lay(v.reshape(lay(x).shape))   # noqa: E731
    return back(y), back(yo)


def tap_sum(O, op):
    """Sum of the filter's magnitudes, from its response to a unit impulse."""
    n = 128
    x, y = np.zeros(n), np.zeros(n)
    x[64] = 1.0
    dot = [ctypes.pointer(ctypes.c_double(0.0))] if op.endswith('dotin') else []
    assert O.call('oracle_' + op, 1, 0, [n], 0, [n], [n], 1, x, y, 1.0, 0.0, 0.0, *dot) == 0
    return np.abs(y).sum()


# from one run's window (80 elements of 16 taps, 96 of 29) to several, whole and partial runs;
# few lines (strips of less than a run), a block of lines and more
@pytest.mark.parametrize('lines', [1, 3, 129, 5000])
@pytest.mark.parametrize('n', [96, 97, 128, 131, 192, 300, 1024])
@pytest.mark.parametrize('idim', [0, 1])
@pytest.mark.parametrize('op', sorted(OPS))
def test_small_values_of_a_line(pkg, O, op, idim, n, lines):
    if lines == 5000 and n > 200:
        lines = 600
    low, taps = OPS[op]
    x = steep(n + lines, lines, n)
    y, yo = apply_1d(pkg, O, op, x, idim)
    bound = TOL * tap_sum(O, op) * run_scales(x, low, taps)
    assert np.all(np.abs(y - yo) <= bound)


@pytest.mark.parametrize('bad', [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize('idim', [0, 1])
@pytest.mark.parametrize('op', sorted(set(OPS) - {'d_s0s0_1d_sym8_d2_dotin'}))
def test_a_nan_stays_in_the_runs_that_read_it(pkg, O, op, idim, bad):
    """The other runs give the bits they give without it."""
    low, taps = OPS[op]
    lines, n, at = 3, 320, 150
    x = steep(5, lines, n)
    clean = apply_1d(pkg, O, op, x, idim, both=False)[0]
    x[1, at] = bad
    y = apply_1d(pkg, O, op, x, idim, both=False)[0]
    reads = np.isinf(run_scales(np.where(np.arange(n) == at, np.inf, 0.0)[None], low, taps)[0])
    assert np.array_equal(y[[0, 2]], clean[[0, 2]])
    assert np.array_equal(y[1, ~reads], clean[1, ~reads])
    assert np.isnan(y[1, at - low - taps + 1:at - low + 1]).all()


@pytest.mark.parametrize('n', [[96, 40, 112], [110, 131, 96], [256, 33, 20]])
def test_magicfilter3d_of_long_lines(pkg, n):
    """Every sweep over periodic lines of 80 points or more takes its runs' exponents: the 3D operator
    gives the bits of three 1D calls.  (Lines of exactly 128 points whose exponents the sweep before
    hands on have the line's.)"""
    r = np.random.default_rng(sum(n))
    N, narr = int(np.prod(n)), 2
    x = r.uniform(-1, 1, (narr, n[2], n[1], n[0]))
    x = (x * 2.0 ** (-30.0 * (np.arange(n[0]) // 90)) * 2.0 ** (-25.0 * (np.arange(n[2])[:, None, None] // 85))).ravel()
    y, w1, w2 = np.zeros(N * narr), np.zeros(N * narr), np.zeros(N * narr)
    pkg.Kernel('d_sfrf_ld_narr').run(3, n, [0, 0, 0], n, n, narr, x, y, w1, w2)
    cur = x
    for i in range(3):
        step = np.zeros(N * narr)
        pkg.Kernel('d_s0s0_1d_sym8_md').run(3, i, n, 0, n, n, narr, cur, step, 1.0, 0.0, 0.0)
        cur = step
    assert np.array_equal(y, cur)


@pytest.mark.parametrize('nord', [2, 16])
def test_poisson_derivatives_of_long_lines(pkg, O, nord):
    """nabla along three periodic axes: each axis's runs keep their own scale."""
    n, h = [112, 96, 81], np.array([0.1, 0.12, 0.09])
    N = int(np.prod(n))
    r = np.random.default_rng(nord)
    k = [np.arange(v) // 60 for v in n]
    u = r.uniform(-1, 1, n[::-1]) * 2.0 ** (-40.0 * (k[0][None, None, :] + k[1][None, :, None] + k[2][:, None, None]))
    du, do = pkg.Poisson().nabla_u(2, n, u.ravel(), nord, h), np.zeros(3 * N)
    assert O.call('oracle_nabla_u', 2, *n, u.ravel(), do, nord, h) == 0
    for axis in range(3):
        line = np.moveaxis(u, 2 - axis, -1)
        taps = 40.0 / h[axis]                        # bounds the stencils' absolute sums
        bound = np.moveaxis(TOL * taps * run_scales(line, -8, 17), -1, 2 - axis)
        err = np.abs(np.asarray(du).ravel()[axis * N:(axis + 1) * N] - do[axis * N:(axis + 1) * N])
        assert np.all(err.reshape(u.shape) <= bound), axis


# windows shared by the three axes' sweeps (whole pieces of 8; runs of 64 whole and partial, the
# last one a single piece), mixed with axes below a window, and extents that keep passes of their own
@pytest.mark.parametrize('geocode', [1, 2, 3])
@pytest.mark.parametrize('n', [[96, 88, 80], [128, 64, 72], [136, 200, 64], [40, 96, 264], [90, 96, 104], [80, 80, 81]])
def test_shared_windows_are_those_of_single_sweeps(pkg, n, geocode):
    """nabla, whose three sweeps share one exponent pass, gives the bits of three single derivatives."""
    h = np.array([0.1, 0.12, 0.09])
    N = int(np.prod(n))
    r = np.random.default_rng(N + geocode)
    u = r.uniform(-1, 1, n[::-1])
    for ax in range(3):
        k = np.arange(n[ax]) * 3 // n[ax] - 1
        u = u * (2.0 ** (-35.0 * k * k)).reshape([-1 if 2 - d == ax else 1 for d in range(3)])
    u[3, 5] = 0.0
    u = u.ravel()
    P = pkg.Poisson()
    bc = {1: [-2, -2, -2], 2: [0, 0, 0], 3: [0, -2, 0]}[geocode]
    du = np.asarray(P.nabla_u(geocode, n, u, 16, h)).ravel()
    for ax in range(3):
        one = np.asarray(P.broker(16, ax, n, bc[ax], u, 1.0 / h[ax])).ravel()
        assert np.array_equal(du[ax * N:(ax + 1) * N], one), ax
