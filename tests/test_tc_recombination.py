"""The exact sweep's recombination of the eight order accumulators, replayed on
the CPU with the word sizes the kernel uses, and its conversion's scaling on
the GPU."""
import numpy as np
import pytest

M32, M64 = 2 ** 32 - 1, 2 ** 64 - 1
BIAS = 0x4B400000


def recombine(acc):
    """horner_bal: neighbouring orders in one 32-bit word, two 32x32+64 multiply-adds."""
    b = [(BIAS + int(v)) & M32 for v in acc]
    pair = (257 * BIAS) & M32
    minus = (-(pair * (2 ** 38 + 2 ** 22 + 2 ** 6))) & M64
    w01, w23, w45 = ((256 * b[k] + b[k + 1]) & M32 for k in (0, 2, 4))
    lo = (256 * b[6] + b[7] + 512 - pair) & M32
    lo = (lo - 2 ** 32 if lo >> 31 else lo) >> 10
    low = (minus & M32) + lo
    assert 0 <= low <= M32                       # no carry out of the low word
    v = ((minus >> 32) << 32) | low
    v = (v + w45 * 64) & M64
    v = (v + w23 * 2 ** 22) & M64
    v = (v + (((w01 * 64) & M32) << 32)) & M64
    return v - 2 ** 64 if v >> 63 else v


@pytest.mark.parametrize('kind', ['random', 'extreme'])
def test_recombination_equals_the_sum_of_orders(kind):
    r = np.random.default_rng(5)
    top = 2 ** 22
    for i in range(400):
        if kind == 'random':
            acc = r.integers(-top, top + 1, 8) >> int(r.integers(0, 22))
        else:
            acc = r.choice([-top, -top + 1, -1, 0, 1, top - 1, top], 8)
        acc = [int(v) for v in acc]
        Y = sum(acc[k] * 2 ** (46 - 8 * k) for k in range(6)) + ((acc[6] * 256 + acc[7] + 512) >> 10)
        if abs(Y) >= 2 ** 63:                    # the filter scale keeps |Y| below 2^62
            continue
        assert recombine(acc) == Y


@pytest.mark.gpu
@pytest.mark.parametrize('k', [-1010, -960, -900, 0, 900, 955, 1000])
@pytest.mark.parametrize('op', ['d_s0s0_1d_sym8_md', 'd_kin'])
def test_power_of_two_scaling_is_exact(pkg, op, k):
    """Exact sweeps scale with their lines: x 2^k gives y 2^k bit for bit, on both sides of the
    scales where the kernel changes its conversion (2^se with se in [-1022, 961]); a line of
    zeros stays zero.  The inputs are multiples of 2^-20 in [-1, 1) and every result is normal."""
    from boast_lig_gb300 import inputs
    n = [33, 20, 24]
    x = np.floor(inputs.uniform(9, int(np.prod(n))) * 2 ** 20) * 2.0 ** -20
    x.reshape(n[::-1])[3, 5] = 0.0

    def run(v):
        y, w1, w2 = np.zeros_like(v), np.zeros_like(v), np.zeros_like(v)
        with pkg.mode(pkg.MODE_TC_EXACT):
            if op == 'd_kin':
                pkg.Kernel(op).run(3, n, [0, 0, 0], v, y, w1, w2, [0.5, 0.25, 1.0], 0.0, 0.0)
            else:
                pkg.Kernel(op).run(3, 0, n, 0, n, n, 1, v, y, 1.0, 0.0, 0.0)
        return y

    y0, yk = run(x), run(np.ldexp(x, k))
    big = np.abs(np.ldexp(y0, k)) >= 2.0 ** -1021
    assert big.mean() > 0.9
    assert np.array_equal(yk[big], np.ldexp(y0, k)[big])
    if op != 'd_kin':
        assert not yk.reshape(n[::-1])[3, 5].any()
