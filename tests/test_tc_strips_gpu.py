"""Exact tensor-core sweeps at the edges of their work split: blocks of 16
outputs, strips of 128 lines that may be cut into segments, the kernel's forms
(plain, partial sums, line exponents handed on, any), against the oracle.
Tolerance: 1e-13 of each line's largest output, as for every FP64-level
operator; a handed-on exponent must give the very bits of separate sweeps,
which take it from a pre-pass."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-13
TAPS = {'d_s0s0_1d_sym8_md': 16, 'd_s0s0_1d_sym8_d1': 29, 'd_s0s0_1d_sym8_d2_dotin': 29,
        'd_s0s1_1d_sym8': 8, 'd_s1s0_1d_sym8': 8}


@pytest.fixture(autouse=True)
def exact(pkg):
    with pkg.mode(pkg.MODE_TC_EXACT):
        yield


def data(seed, shape, axis=-1):
    """Uniform values, each line along `axis` with its own magnitude."""
    r = np.random.default_rng(seed)
    x = r.uniform(-1.0, 1.0, shape)
    lines = np.ones_like(np.take(x, [0], axis=axis))
    return x * lines * 2.0 ** r.integers(-30, 30, lines.shape)


# positions per line: below, at and above one block and one slab, windows that wrap
# more than once, and lines long enough to be cut into segments
@pytest.mark.parametrize('n', [3, 7, 15, 16, 17, 31, 32, 33, 48, 113, 2051])
@pytest.mark.parametrize('op', sorted(TAPS))
def test_lines_of_every_length(pkg, O, op, n):
    wav = op in ('d_s0s1_1d_sym8', 'd_s1s0_1d_sym8')
    m = 2 if wav else 1
    for bc, lines, idim in ((0, 1, 0), (0, 130, 1), (2, 33, 0), (1, 3, 1), (-1, 129, 0)):
        if n == 2051:
            lines = min(lines, 5)
        shape = [n, n]
        shape[1 - idim] = lines
        nx, ny = list(shape), list(shape)
        nx[idim] += TAPS[op] - 1 if bc == -1 else 0
        ny[idim] += TAPS[op] - 1 if bc == 1 else 0
        x = data(abs(n + 10 * bc), (m * nx[1], m * nx[0]), axis=1 - idim)
        y = np.zeros((m * ny[1], m * ny[0]))
        yo = np.zeros_like(y)
        args = [2, idim, shape, bc, nx, ny, 1, np.ascontiguousarray(x).ravel()]
        tail = (1.0, 0.0) if wav else (0.7, 0.0, 0.0)
        if op.endswith('dotin'):
            st = pkg.Kernel(op).run(*args, y.ravel(), *tail, None)
            d = ctypes.c_double(0.0)
            assert O.call('oracle_' + op, *args, yo.ravel(), *tail, ctypes.pointer(d)) == 0
            # the sum of the products' magnitudes bounds what rounding can move
            assert abs(st['reference_return']['dot_in'] - d.value) <= TOL * np.abs(x).max() * np.abs(yo).sum()
        else:
            pkg.Kernel(op).run(*args, y.ravel(), *tail)
            assert O.call('oracle_' + op, *args, yo.ravel(), *tail) == 0
        err = np.abs(y - yo).max(axis=1 - idim)
        ref = np.abs(yo).max(axis=1 - idim)
        assert np.all(err <= TOL * ref), (op, n, bc, lines, idim)


# line counts and lengths that are multiples of 32 (a warp's rows lie in one line of the
# next sweep), that are not (in one or two), and lengths below 32 (pre-pass instead)
@pytest.mark.parametrize('bcs', [[0, 0, 0], [2, 2, 2], [1, 0, 2], [0, 2, 1], [-1, -1, -1]])
@pytest.mark.parametrize('n', [[32, 32, 32], [64, 32, 96], [96, 160, 32], [48, 32, 64], [34, 46, 66], [32, 24, 130], [62, 64, 34]])
@pytest.mark.parametrize('op', ['magicfilter', 'd_dwt_sym8', 'd_idwt_sym8'])
def test_handed_on_exponents(pkg, op, n, bcs):
    """The 3D operator, whose sweeps hand on line exponents, gives the bits of three 1D calls."""
    mf = op == 'magicfilter'
    m, taps = (1, 16) if mf else (2, 8)
    ni = n if mf else [v // 2 for v in n]             # input positions, filtered, output positions
    nf = [v - (taps - 1) * (b == -1) for v, b in zip(ni, bcs)]
    no = [v + (taps - 1) * (b == 1) for v, b in zip(nf, bcs)]
    narr = 2
    x = data(n[0] + n[1], (narr, m * ni[2], m * ni[1], m * ni[0]))
    x[0, 3, 5] = 0.0                                  # a line of zeros
    big = narr * int(np.prod([m * max(v, w) for v, w in zip(ni, no)]))
    y = np.zeros(narr * int(np.prod([m * v for v in no])))
    w1, w2 = np.zeros(big), np.zeros(big)
    if mf:
        pkg.Kernel('d_sfrf_ld_narr').run(3, nf, bcs, ni, no, narr, x.ravel(), y, w1, w2)
    else:
        pkg.Kernel(op + '_narr').run(3, nf, bcs, narr, x.ravel(), y, w1, w2)
    name = {'magicfilter': 'd_s0s0_1d_sym8_md', 'd_dwt_sym8': 'd_s0s1_1d_sym8', 'd_idwt_sym8': 'd_s1s0_1d_sym8'}[op]
    cur, ext = x.ravel(), list(ni)
    for i in range(3):
        mid, out = list(ext), list(ext)
        mid[i], out[i] = nf[i], no[i]
        step = np.zeros(narr * int(np.prod([m * v for v in out])))
        pkg.Kernel(name).run(3, i, mid, bcs[i], ext, out, narr, cur, step, 1.0, *((0.0, 0.0) if mf else (0.0,)))
        cur, ext = step, out
    assert np.array_equal(y, cur)


@pytest.mark.parametrize('a_x,a_y', [(0.0, 0.0), (0.5, 0.0), (0.0, -1.0)])
@pytest.mark.parametrize('n', [[16, 32, 48], [33, 48, 65], [130, 17, 31]])
def test_partial_sums_and_terms(pkg, O, n, a_x, a_y):
    """Kinetic sweeps of whole and partial blocks: partial sums, a_x and a_y terms."""
    N = int(np.prod(n))
    r = np.random.default_rng(N)
    a = [-0.5 / 0.5 ** 2, -0.5 / 0.6 ** 2, -0.5 / 0.7 ** 2]
    for bcs in ([0, 0, 0], [2, 0, 2]):
        x, y0 = r.uniform(-1, 1, N), r.uniform(-1, 1, N)
        yg, yo, w = y0.copy(), y0.copy(), np.zeros(N)
        pkg.Kernel('d_kin').run(3, n, bcs, x, yg, w, w, a, a_x, a_y)
        assert O.call('oracle_d_kin', 3, n, bcs, x, yo, np.zeros(N), np.zeros(N), np.array(a), a_x, a_y) == 0
        assert np.abs(yg - yo).max() <= TOL * np.abs(yo).max(), bcs


# 128 lines or fewer: lines are cut into as many segments as there are SMs, the last one shorter
@pytest.mark.parametrize('mode,tol', [('MODE_TC_EXACT', 1e-13), ('MODE_TC_BF16X3', 1e-5)])
@pytest.mark.parametrize('lines,idim', [(1, 0), (3, 0), (2, 1), (130, 1)])
@pytest.mark.parametrize('op', ['d_s0s0_1d_sym8_md', 'd_s0s0_1d_sym8_d1', 'd_s0s1_1d_sym8', 'd_s1s0_1d_sym8'])
def test_few_long_lines(pkg, O, op, lines, idim, mode, tol):
    wav = op in ('d_s0s1_1d_sym8', 'd_s1s0_1d_sym8')
    m, n = (2, 6007) if wav else (1, 12007)
    shape = [n, n]
    shape[1 - idim] = lines
    r = np.random.default_rng(n + lines)
    x = r.uniform(-1, 1, m * m * n * lines)
    for bc in (0, 1, 2):
        ny = list(shape)
        ny[idim] += TAPS[op] - 1 if bc == 1 else 0
        y = np.zeros(m * m * int(np.prod(ny)))
        yo = np.zeros_like(y)
        args = [2, idim, shape, bc, shape, ny, 1, x]
        tail = (1.0, 0.0) if wav else (0.7, 0.0, 0.0)
        with pkg.mode(getattr(pkg, mode)):
            pkg.Kernel(op).run(*args, y, *tail)
        assert O.call('oracle_' + op, *args, yo, *tail) == 0
        assert np.abs(y - yo).max() <= tol * np.abs(yo).max(), bc
