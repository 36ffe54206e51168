"""The filter operands of the exact sweeps as the library forms them (tc_filter_digits, on the host),
filters whose digits do not fit the accumulators included: their scale is raised and they are cut
again."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from test_tc_recombination import constants

MOST = 2 ** 22


def cut(taps, a, ef):
    """Digits [8][taps] of round(a f 2^(62 - ef)), halves away from zero."""
    out = []
    for t in taps:
        v = Fraction(float(a)) * Fraction(float(t)) * Fraction(2) ** (62 - ef)
        F = int(abs(v) + Fraction(1, 2)) * (1 if v >= 0 else -1)
        U = (F + 0x8080808080808080) % 2 ** 64
        out.append([((U >> (8 * (7 - s))) & 0xFF) - 128 for s in range(8)])
        assert sum(d * 256 ** (7 - s) for s, d in enumerate(out[-1])) == F
    return np.array(out, dtype=object).T


def first_scale(taps, a):
    af = [abs(Fraction(float(a)) * Fraction(float(t))) for t in taps]
    ef = -1080
    while any(v >= Fraction(2) ** ef for v in af) or sum(af) >= 8 * Fraction(2) ** ef:
        ef += 1
    return ef


def channels(kind, ntaps):
    """Taps of each output channel."""
    if kind == 0:
        return [list(range(ntaps)), []]
    q = [list(range(k * ntaps // 4, (k + 1) * ntaps // 4)) for k in range(4)]     # LE, LO, HE, HO
    return [q[0] + q[1], q[2] + q[3]] if kind == 1 else [q[1] + q[3], q[0] + q[2]]


def fits(e, ch):
    return all(255 * sum(int(abs(v)) for v in e[:, ch].ravel() if (v > 0) == up) <= MOST for up in (True, False))


def library(pkg, kind, taps, a):
    n = len(taps)
    dig, ef = (ctypes.c_int * (8 * n))(), ctypes.c_int()
    k64, k67 = (ctypes.c_longlong * 2)(), (ctypes.c_uint * 2)()
    f = pkg.lib().libconv_gb300_selftest_digits
    f.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_double), ctypes.c_int, ctypes.c_double] + [ctypes.c_void_p] * 4
    assert f(kind, (ctypes.c_double * n)(*taps), n, a, dig, ctypes.byref(ef), k64, k67) == 0
    return np.array(dig[:], dtype=object).reshape(8, n), ef.value, list(k64), list(k67)


def heavy(n, sign, ef):
    """n equal taps whose sum stays just below 8 * 2^ef, the first scale, and whose digits below the
    top one are 127 there: their absolute sums exceed the accumulators' bound."""
    F = 0x117F7F7F7F7F7F00 if n == 29 else 0x077F7F7F7F7F7F00      # 53 bits at most
    return [sign * float(F) * 2.0 ** (ef - 62)] * n


CASES = {
    'md-like': (0, lambda r: r.uniform(-0.5, 0.5, 16), 1.0),
    'scaled': (0, lambda r: r.uniform(-1, 1, 29), -2.469135802469136),
    'heavy up': (0, lambda r: np.array(heavy(29, 1.0, 0)), 1.0),
    'heavy down': (0, lambda r: np.array(heavy(29, -1.0, 3)), 1.0),
    'heavy negated': (0, lambda r: np.array(heavy(29, 1.0, -2)), -1.0),
    'heavy scaled': (0, lambda r: np.array(heavy(29, 1.0, 1)) * r.uniform(0.9, 1.0, 29), 1.0 + 2.0 ** -30),
    'heavy analysis': (1, lambda r: np.array(heavy(64, 1.0, 0)), 1.0),
    'heavy synthesis': (2, lambda r: np.array(heavy(64, 1.0, 0)) * np.repeat([1.0, -1.0, 1.0, -1.0], 16), 1.0),
    'zero scalar': (0, lambda r: r.uniform(-1, 1, 17), 0.0),
    'tiny': (0, lambda r: r.uniform(-1, 1, 16) * 2.0 ** -900, 1.0),
}
RAISED = {'heavy up', 'heavy down', 'heavy negated', 'heavy analysis', 'heavy synthesis'}


@pytest.mark.parametrize('name', sorted(CASES))
def test_filter_digits(pkg, name):
    """Digits, scale and constants are those of the first scale whose digits fit; the named filters
    do not fit at their first one."""
    kind, make, a = CASES[name]
    taps = make(np.random.default_rng(7))
    e, ef, k64, k67 = library(pkg, kind, taps, a)
    want = first_scale(taps, a) if a else 0
    ch = channels(kind, len(taps))
    raised = 0
    while not all(fits(cut(taps, a, want), c) for c in ch if c):
        want, raised = want + 1, raised + 1
    assert (ef, bool(raised)) == (want, name in RAISED)
    assert np.array_equal(e, cut(taps, a, ef))
    for c in range(2):
        k = constants([int(e[t][ch[c]].sum()) if ch[c] else 0 for t in range(8)])
        assert (k64[c] % 2 ** 64, k67[c]) == k
